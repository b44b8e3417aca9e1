"""The work that programs have this library do, as cases for timing it.

    plane     one small plane through Resize: a thumbnail or a preview, where the call itself counts
    batch     many planes of one or several sizes through Batch: transcoding and machine-learning input
    depth     planes of a frame through Depth: float masters to 8-bit delivery
    frame     a whole YUV or RGB frame through Graph, as video filters call it: 8-bit scaling, 10-bit to
              8-bit with error diffusion, HDR to SDR
    unresize  the planes of a frame through Unresize: undoing an upscale

A case is a dict of plain values; `draw` gives others of the same ranges.
"""
import math

import numpy as np
import torch

import zimg_gb300 as zg

WORD, FLOAT = "word", "float"


# ------------------------------------------------------------------ the cases --

def listed():
    return [
        # a preview of a 10-bit plane: the call's latency, a width that is no multiple of 8
        dict(name="plane_preview", family="plane", type=WORD, depth=10, sw=320, sh=180, dw=426, dh=240,
             filter="bicubic", a=0.0, b=0.5),
        # the headline: full HD to UHD, 10 bits, Lanczos-3, frames by the batch
        dict(name="batch_fhd_uhd", family="batch", type=WORD, depth=10, sizes="1920x1080", dw=3840, dh=2160,
             planes=32, chroma=False, fields=False, filter="lanczos", a=3.0, b=0.0),
        # digital cinema masters of 16 bits to 2K flat: lines that are no multiple of 16 bytes
        dict(name="batch_deep_dci", family="batch", type=WORD, depth=16, sizes="3996x2160", dw=1998, dh=1080,
             planes=16, chroma=False, fields=False, filter="spline36", a=0.0, b=0.0),
        # a transcoder's ladder: 4:2:0 frames of mixed sizes to full HD, MPEG-2 siting
        dict(name="batch_yuv420", family="batch", type=WORD, depth=10,
             sizes="1280x720,3840x2160,720x480,1920x1080", dw=1920, dh=1080, planes=32, chroma=True, fields=False,
             filter="spline36", a=0.0, b=0.0),
        # linear-light float frames 4:4:4 to 720p
        dict(name="batch_bicubic", family="batch", type=FLOAT, depth=32, sizes="1920x1080", dw=1280, dh=720,
             planes=96, chroma=False, fields=False, filter="bicubic", a=0.0, b=0.5),
        # 8K float planes to thumbnails, 128 taps an output
        dict(name="batch_wide", family="batch", type=FLOAT, depth=32, sizes="7680x4320", dw=480, dh=270, planes=8,
             chroma=False, fields=False, filter="lanczos", a=4.0, b=0.0),
        # the ends of the ratios' range: icons to posters
        dict(name="batch_extreme_up", family="batch", type=FLOAT, depth=32, sizes="64x64", dw=6400, dh=6400,
             planes=6, chroma=False, fields=False, filter="lanczos", a=3.0, b=0.0),
        # a float master frame to 8-bit delivery, ordered dither
        dict(name="depth_uhd", family="depth", width=3840, height=2160, planes=3, in_type=FLOAT, in_depth=32,
             out_type="byte", out_depth=8, dither="ordered"),
        # everyday video: an 8-bit 4:2:0 frame scaled to 480p (a chroma width of 427)
        dict(name="frame_8bit", family="frame", sw=1920, sh=1080, dw=854, dh=480, in_type="byte", in_depth=8,
             out_type="byte", out_depth=8, sub=1, hdr="", dither="none", filter="bicubic"),
        # a 10-bit frame delivered at 8 bits with error diffusion, the size kept
        dict(name="frame_diffusion", family="frame", sw=1920, sh=1080, dw=1920, dh=1080, in_type=WORD, in_depth=10,
             out_type="byte", out_depth=8, sub=1, hdr="", dither="error_diffusion", filter="bicubic"),
        # an HDR10 UHD frame to an SDR full HD one
        dict(name="frame_hdr", family="frame", sw=3840, sh=2160, dw=1920, dh=1080, in_type=WORD, in_depth=10,
             out_type="byte", out_depth=8, sub=1, hdr="pq", dither="ordered", filter="spline36"),
        # a frame that was upscaled from 720p, taken back
        dict(name="unresize_720p", family="unresize", width=1920, height=1080, ow=1280, oh=720, planes=3),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi):
    """A width and, at one of the usual aspect ratios, its height."""
    w = _log(rng, lo, hi)
    return w, max(16, int(w / rng.choice([16 / 9, 16 / 9, 4 / 3, 2.39, 1.85, 1.0])))


def _filter(rng):
    k = rng.choice(["bilinear", "bicubic", "spline16", "spline36", "spline64", "lanczos", "lanczos"])
    a = {"bicubic": rng.choice([0.0, 1.0 / 3.0]), "lanczos": float(rng.choice([2, 3, 4]))}.get(k, 0.0)
    b = 0.5 if k == "bicubic" and a == 0.0 else 1.0 / 3.0 if k == "bicubic" else 0.0
    return dict(filter=k, a=a, b=b)


def draw(rng):
    family = rng.choice(["plane", "batch", "batch", "batch", "batch", "depth", "frame", "frame", "unresize"])
    if family == "plane":
        t = rng.choice([WORD, FLOAT])
        (sw, sh), dw = _size(rng, 96, 1280), _log(rng, 96, 1280)
        return dict(family=family, type=t, depth=rng.choice([8, 10, 12, 16]) if t == WORD else 32,
                    sw=sw, sh=sh, dw=dw, dh=max(16, round(sh * dw / sw)), **_filter(rng))
    if family == "batch":
        t = rng.choice([WORD, WORD, FLOAT])
        depth = rng.choice([8, 9, 10, 10, 12, 14, 16]) if t == WORD else 32
        sw, sh = _size(rng, 480, 4096)
        ratio = math.exp(rng.uniform(math.log(0.1 if t == FLOAT else 0.3), math.log(min(3.0, 4096 / sw))))
        dw, dh = max(32, int(sw * ratio)), max(18, int(sh * ratio))
        if rng.random() < 0.5:  # most programs' widths are multiples of 8
            sw, dw = sw // 8 * 8, max(32, dw // 8 * 8)
        chroma = t == WORD and rng.random() < 0.3
        if chroma:
            sw, sh, dw, dh = (v // 2 * 2 for v in (sw, sh, dw, dh))
        each = (sw * sh + dw * dh) * (2 if t == WORD else 4) * (1.5 if chroma else 1.0)
        planes = max(1, min(_log(rng, 4, 64), int(500e6 / each)))
        return dict(family=family, type=t, depth=depth, sizes="%dx%d" % (sw, sh), dw=dw, dh=dh, planes=planes,
                    chroma=chroma, fields=not chroma and rng.random() < 0.15, **_filter(rng))
    if family == "depth":
        i, o = rng.choice([(FLOAT, "byte"), (FLOAT, WORD), (WORD, "byte"), (WORD, FLOAT), ("byte", FLOAT)])
        bits = {FLOAT: 32, "byte": 8}
        w, h = _size(rng, 320, 3840)
        return dict(family=family, width=w, height=h, planes=3, in_type=i,
                    in_depth=bits.get(i) or rng.choice([10, 12, 16]), out_type=o,
                    out_depth=bits.get(o) or rng.choice([10, 12, 16]),
                    dither="none" if o == FLOAT else rng.choice(["none", "ordered", "random"]))
    if family == "unresize":
        (ow, oh), up = _size(rng, 320, 1280), rng.uniform(1.2, 1.5)
        return dict(family=family, width=int(ow * up), height=int(oh * up), ow=ow, oh=oh, planes=3)
    kind = rng.choice(["8bit", "8bit", "10bit", "diffusion", "hdr"])
    sw, sh = (v // 2 * 2 for v in _size(rng, 480, 1920 if kind == "diffusion" else 3840))
    dw = sw if kind == "diffusion" and rng.random() < 0.5 else _log(rng, 480, 1920) // 2 * 2
    i, o = ("byte" if kind == "8bit" else WORD), (WORD if kind == "10bit" else "byte")
    return dict(family=family, sw=sw, sh=sh, dw=dw, dh=round(sh * dw / sw) // 2 * 2, in_type=i,
                in_depth=8 if kind == "8bit" else 10 if kind == "10bit" else rng.choice([10, 12]), out_type=o,
                out_depth=10 if kind == "10bit" else 8, sub=rng.choice([0, 1, 1]),
                hdr=rng.choice(["pq", "hlg"]) if kind == "hdr" else "",
                dither="error_diffusion" if kind == "diffusion" else rng.choice(["none", "ordered", "random"]),
                filter=rng.choice(["bilinear", "bicubic", "spline36", "lanczos"]))


# ---------------------------------------------------------------------- inputs --

DTYPE = {"byte": torch.uint8, WORD: torch.int16, FLOAT: torch.float32}
SIZE = {"byte": 1, WORD: 2, FLOAT: 4}


def _content(gen, n, h, w, kind, depth):
    """n planes: 16x16 blocks, half of them noise and half of them smooth
    waves, over the type's range (float: [0, 1] with values a little outside)."""
    dev = "cuda"
    p = torch.rand(n, 3, generator=gen, device=dev)
    lx, ly, ph = 64 + 448 * p[:, 0], 64 + 448 * p[:, 1], 2 * math.pi * p[:, 2]
    x = torch.arange(w, device=dev, dtype=torch.float32)
    y = torch.arange(h, device=dev, dtype=torch.float32)
    out = torch.empty(n, h, w, dtype=DTYPE[kind], device=dev)
    for k in range(n):
        wave = 0.5 + 0.5 * torch.sin(2 * math.pi * (x[None, :] / lx[k] + y[:, None] / ly[k]) + ph[k])
        noise = torch.rand(h, w, generator=gen, device=dev)
        pick = torch.rand((h + 15) // 16, (w + 15) // 16, generator=gen, device=dev) < 0.5
        pick = pick.repeat_interleave(16, 0)[:h].repeat_interleave(16, 1)[:, :w]
        v = torch.where(pick, noise, wave)
        if kind == FLOAT:
            out[k] = v * 1.04 - 0.02
        elif kind == "byte":
            out[k] = torch.round(v * 255).to(torch.uint8)
        else:
            out[k] = torch.round(v * ((1 << depth) - 1)).to(torch.int32).to(torch.int16)
    return out


def _jobs(case):
    """(source size, output size, shift_w, shift_h) of a batch's planes."""
    sizes = [tuple(int(v) for v in s.split("x")) for s in case["sizes"].split(",")]
    dw, dh, jobs = case["dw"], case["dh"], []
    for k in range(case["planes"]):
        sw, sh = sizes[k % len(sizes)]
        field = (-0.125 if k % 2 == 0 else 0.125) if case["fields"] else 0.0
        jobs.append((sw, sh, dw, dh, 0.0, field))
        if case["chroma"]:
            shift = 0.25 - 0.25 / ((dw // 2) / (sw // 2))
            jobs += [(sw // 2, sh // 2, dw // 2, dh // 2, shift, 0.0)] * 2
    return jobs


def _conversion(case, job):
    sw, sh, dw, dh, shift_w, shift_h = job
    return zg.ResizeConversion(sw, sh, case["type"]).set_depth(case["depth"]) \
        .set_filter(case["filter"], case["a"], case["b"]).set_dst_width(dw).set_dst_height(dh) \
        .set_shift_w(shift_w).set_shift_h(shift_h)


def _batch_inputs(case, gen):
    """The planes of each size, side by side in one tensor, in the jobs' order."""
    jobs, at = _jobs(case), {}
    for j in jobs:
        at.setdefault((j[0], j[1]), []).append(j)
    stacks = {s: iter(_content(gen, len(v), s[1], s[0], case["type"], case["depth"])) for s, v in at.items()}
    return jobs, [next(stacks[(j[0], j[1])]) for j in jobs]


def _frame_formats(case):
    yuv = dict(color_family=2, matrix_coefficients=1, transfer_characteristics=1, color_primaries=1)
    src, dst = dict(yuv), dict(yuv)
    if case["hdr"]:
        src.update(matrix_coefficients=9, color_primaries=9, transfer_characteristics={"pq": 16, "hlg": 18}[case["hdr"]])
    for f, t, d in ((src, "in_type", "in_depth"), (dst, "out_type", "out_depth")):
        f.update(pixel_type=case[t], depth=case[d], subsample_w=case["sub"], subsample_h=case["sub"])
    p = zg.graph_params(resample_filter=case["filter"], resample_filter_uv=case["filter"],
                        dither_type=["none", "ordered", "random", "error_diffusion"].index(case["dither"]))
    return zg.image_format(case["sw"], case["sh"], **src), zg.image_format(case["dw"], case["dh"], **dst), p


def _frame_planes(w, h, sub):
    return [(w, h), (w >> sub, h >> sub), (w >> sub, h >> sub)]


def _bytes(n):
    return torch.empty(max(n, 1), dtype=torch.uint8, device="cuda")


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    family = case["family"]
    if family == "plane":
        r = _conversion(case, (case["sw"], case["sh"], case["dw"], case["dh"], 0.0, 0.0)).create()
        src = _content(gen, 1, case["sh"], case["sw"], case["type"], case["depth"])[0]
        dst = torch.empty(case["dh"], case["dw"], dtype=DTYPE[case["type"]], device="cuda")
        return dict(family=family, plan=r, src=src, dst=dst, tmp=_bytes(r.tmp_size))
    if family == "batch":
        jobs, srcs = _batch_inputs(case, gen)
        count, at = {}, {}
        for j in jobs:
            count[(j[2], j[3])] = count.get((j[2], j[3]), 0) + 1
        outs = {s: torch.empty(n, s[1], s[0], dtype=DTYPE[case["type"]], device="cuda") for s, n in count.items()}
        dsts = []
        for j in jobs:
            s = (j[2], j[3])
            at[s] = at.get(s, -1) + 1
            dsts.append(outs[s][at[s]])
        b = zg.Batch([_conversion(case, j) for j in jobs])
        b.set_io(srcs, dsts)
        return dict(family=family, plan=b, src=srcs, dst=list(outs.values()), views=dsts, tmp=_bytes(b.tmp_size))
    if family == "depth":
        w, h, n = case["width"], case["height"], case["planes"]
        plans = [zg.DepthConversion(w, h).set_pixel_in(case["in_type"], case["in_depth"])
                 .set_pixel_out(case["out_type"], case["out_depth"]).set_dither_type(case["dither"]).set_plane(p)
                 .create() for p in range(n)]
        return dict(family=family, plan=plans, src=list(_content(gen, n, h, w, case["in_type"], case["in_depth"])),
                    dst=torch.empty(n, h, w, dtype=DTYPE[case["out_type"]], device="cuda"))
    if family == "unresize":
        u = zg.UnresizeConversion(case["width"], case["height"]).set_orig_width(case["ow"]) \
            .set_orig_height(case["oh"]).create()
        src = _content(gen, case["planes"], case["height"], case["width"], FLOAT, 32)
        dst = torch.empty(case["planes"], case["oh"], case["ow"], dtype=torch.float32, device="cuda")
        return dict(family=family, plan=u, src=list(src), dst=dst, tmp=_bytes(u.tmp_size))
    g = zg.Graph(*_frame_formats(case))
    src = [_content(gen, 1, h, w, case["in_type"], case["in_depth"])[0]
           for w, h in _frame_planes(case["sw"], case["sh"], case["sub"])]
    dst = [torch.empty(h, w, dtype=DTYPE[case["out_type"]], device="cuda")
           for w, h in _frame_planes(case["dw"], case["dh"], case["sub"])]
    return dict(family=family, plan=g, src=src, dst=dst, tmp=_bytes(g.tmp_size))


def run(state):
    plan, family = state["plan"], state["family"]
    if family == "plane":
        plan.process(state["src"], state["dst"], state["tmp"])
    elif family == "batch":
        plan.process(state["tmp"])
    elif family == "depth":
        for p, s, d in zip(plan, state["src"], state["dst"]):
            p.process(s, d)
    elif family == "unresize":
        for s, d in zip(state["src"], state["dst"]):
            plan.process(s, d, state["tmp"])
    else:
        plan.process(state["src"], state["dst"], state["tmp"])
    return state["dst"]


# ----------------------------------------------------------- what a pass needs --

SUPPORT = {"bilinear": 1, "bicubic": 2, "spline16": 2, "spline36": 3, "spline64": 4}


def _resize_flops(sw, sh, dw, dh, kind, a):
    """Multiply-adds of the two passes, in the cheaper order."""
    s = SUPPORT.get(kind) or int(a or 3)
    th, tv = (2 * s * max(1.0, n / m) if n != m else 0 for n, m in ((sw, dw), (sh, dh)))
    return 2 * min(dw * sh * th + dw * dh * tv, sw * dh * tv + dw * dh * th)


def work(case):
    family = case["family"]
    if family in ("plane", "batch"):
        jobs = _jobs(case) if family == "batch" else [(case["sw"], case["sh"], case["dw"], case["dh"])]
        return dict(bytes=sum((j[0] * j[1] + j[2] * j[3]) * SIZE[case["type"]] for j in jobs),
                    flops=sum(_resize_flops(*j[:4], case["filter"], case["a"]) for j in jobs))
    if family == "depth":
        n = case["width"] * case["height"] * case["planes"]
        return dict(bytes=n * (SIZE[case["in_type"]] + SIZE[case["out_type"]]), flops=4 * n)
    if family == "unresize":
        w, h, ow, oh, n = case["width"], case["height"], case["ow"], case["oh"], case["planes"]
        return dict(bytes=4 * n * (w * h + ow * oh), flops=n * (ow * h * (4 * w / ow + 5) + ow * oh * (4 * h / oh + 5)))
    src, dst = (_frame_planes(w, h, case["sub"]) for w, h in ((case["sw"], case["sh"]), (case["dw"], case["dh"])))
    n_out = sum(w * h for w, h in dst)
    flops = sum(_resize_flops(*s, *d, case["filter"], 3) for s, d in zip(src, dst)) + 4 * n_out
    if case["dither"] == "error_diffusion":
        flops += 10 * n_out
    if case["hdr"]:  # three matrices and two transfer functions a pixel, at the smaller size
        flops += min(case["sw"], case["dw"]) * min(case["sh"], case["dh"]) * (3 * 15 + 6 * 30)
    return dict(bytes=sum(w * h for w, h in src) * SIZE[case["in_type"]] + n_out * SIZE[case["out_type"]], flops=flops)


# ---------------------------------------------------------- outputs in 64 bits --

def _kernel(kind, a, b, x):
    x = np.abs(x)
    if kind == "bilinear":
        return np.maximum(1 - x, 0)
    if kind == "lanczos":
        n = int(a)
        return np.where(x < n, np.sinc(x) * np.sinc(x / n), 0)
    if kind == "bicubic":
        p = [((6 - 2 * a) / 6, 0, (-18 + 12 * a + 6 * b) / 6, (12 - 9 * a - 6 * b) / 6),
             ((8 * a + 24 * b) / 6, (-12 * a - 48 * b) / 6, (6 * a + 30 * b) / 6, (-a - 6 * b) / 6)]
        off = (0, 0)
    else:
        p = {"spline16": [(1, -1 / 5, -9 / 5, 1), (0, -7 / 15, 4 / 5, -1 / 3)],
             "spline36": [(1, -3 / 209, -453 / 209, 13 / 11), (0, -156 / 209, 270 / 209, -6 / 11),
                          (0, 26 / 209, -45 / 209, 1 / 11)],
             "spline64": [(1, -3 / 2911, -6387 / 2911, 49 / 41), (0, -2328 / 2911, 4032 / 2911, -24 / 41),
                          (0, 582 / 2911, -1008 / 2911, 6 / 41), (0, -97 / 2911, 168 / 2911, -1 / 41)]}[kind]
        off = (0, 1, 2, 3)
    y = np.zeros_like(x)
    for i, c in enumerate(p):
        t = x - off[i]
        y = np.where((x >= i) & (x < i + 1), c[0] + t * (c[1] + t * (c[2] + t * c[3])), y)
    return y


def _matrix(kind, a, b, src, dst, shift):
    """The resampling of a line as a matrix [dst, src]: edges mirrored."""
    if src == dst and shift == 0:
        return None
    scale = dst / src
    step = min(scale, 1.0)
    support = (SUPPORT.get(kind) or int(a)) / step
    n = max(int(math.ceil(support)) * 2, 1)
    pos = (np.arange(dst) + 0.5) / scale + shift
    at = np.floor(pos - n / 2 + 0.5)[:, None] + 0.5 + np.arange(n)[None, :]
    wt = _kernel(kind, a, b, (at - pos[:, None]) * step)
    wt /= wt.sum(1, keepdims=True)
    at = np.where(at < 0, -at, np.where(at >= src, 2.0 * src - at, at))
    at = np.floor(np.clip(at, 0, np.nextafter(float(src), 0))).astype(np.int64)
    m = np.zeros((dst, src))
    np.add.at(m, (np.arange(dst)[:, None], at), wt)
    return torch.from_numpy(m).cuda()


def _apply(v, h, x):
    x = x.double()
    x = x if v is None else v @ x
    return x if h is None else x @ h.T


def _unresize_matrix(orig, up):
    """The least-squares inverse of a bilinear upsampling orig -> up."""
    pos = (np.arange(up) + 0.5) * orig / up - 0.5
    left = np.clip(np.floor(pos), 0, orig - 1).astype(np.int64)
    dist = np.clip(pos, 0, orig - 1) - left
    m = np.zeros((up, orig))
    np.add.at(m, (np.arange(up), left), 1 - dist)
    np.add.at(m, (np.arange(up), np.minimum(left + 1, orig - 1)), dist)
    return torch.from_numpy(np.linalg.solve(m.T @ m, m.T)).cuda()


def exact(case, seed):
    family = case["family"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if family in ("plane", "batch") and case["type"] == FLOAT:
        if family == "plane":
            srcs = [_content(gen, 1, case["sh"], case["sw"], FLOAT, 32)[0]]
            jobs = [(case["sw"], case["sh"], case["dw"], case["dh"], 0.0, 0.0)]
        else:
            jobs, srcs = _batch_inputs(case, gen)
        made, outs = {}, {}
        for j, s in zip(jobs, srcs):
            for key in ((j[0], j[2], j[4]), (j[1], j[3], j[5])):
                if key not in made:
                    made[key] = _matrix(case["filter"], case["a"], case["b"], *key)
            outs.setdefault((j[2], j[3]), []).append(_apply(made[(j[1], j[3], j[5])], made[(j[0], j[2], j[4])], s))
        return outs.popitem()[1][0] if family == "plane" else [torch.stack(v) for v in outs.values()]
    if family == "unresize":
        h, v = _unresize_matrix(case["ow"], case["width"]), _unresize_matrix(case["oh"], case["height"])
        return torch.stack([_apply(v, h, s) for s in _content(gen, case["planes"], case["height"], case["width"],
                                                              FLOAT, 32)])
    if family == "depth" and case["out_type"] == FLOAT:
        # limited range: 16 to 235 of 8 bits are 0 to 1
        x = _content(gen, case["planes"], case["height"], case["width"], case["in_type"], case["in_depth"])
        x = x.to(torch.int32) & 0xFFFF
        return (x.double() - (16 << (case["in_depth"] - 8))) / (219 << (case["in_depth"] - 8))
    return None
