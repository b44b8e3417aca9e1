"""GPU parity of the chained u16 kernel's two forms, and its bounded waits.

The TMA form (producer warp, mbarrier pipeline) is the default wherever the
source planes admit a tensor map; ZG_CHAIN_TMA=0 selects the cp.async form,
which also runs planes that are not 16-byte aligned. The switch is read once
per process, so the conversions run in a child process with the variable
set; the parent checks the child's planes against the oracle (u16:
bit-exact against zimg's C path) and that no bounded pipeline wait ran out.

test_bounded_wait_runs_out makes one consumer wait of the TMA form run out
on purpose: a test hook stops the producer of CTA 0 from arming one group's
stage (no copy is issued for it) and shortens every wait to 1 ms. The
kernel must return on its own, the pipeline status must name the wait, and
the next conversion on the same context must be bit-exact again.
"""
import json
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# (src_w, src_h, dst_w, dst_h, filter, depth): H-first upscales, a V-first
# downscale with a 3-window vertical filter, odd sizes
SINGLE = [
    (1920, 1080, 3840, 2160, "lanczos", 10),
    (720, 480, 1920, 1080, "spline36", 10),
    (3840, 2160, 1920, 1080, "spline36", 10),
    (333, 97, 1001, 500, "lanczos", 8),
    (640, 480, 427, 320, "bicubic", 10),
]
BATCH = [(720, 480, 1920, 1080), (360, 240, 960, 540), (1280, 720, 1920, 1080), (640, 360, 960, 540),
         (1920, 1080, 1920, 1080)]

CHILD = r"""
import json, os, sys
import numpy as np
import torch
sys.path.insert(0, os.environ["ZG_ROOT"])
import zimg_gb300 as zg

out = sys.argv[1]
cfg = json.load(open(os.path.join(out, "cfg.json")))
lib = zg.load()
lib.zg_pipeline_status(1)
res = {"single_engines": [], "status": []}

def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a).view(np.int16)).cuda()

for i, (sw, sh, dw, dh, kind, depth) in enumerate(cfg["single"]):
    src = np.load(os.path.join(out, f"src{i}.npy"))
    conv = zg.ResizeConversion(sw, sh, "word").set_depth(depth).set_filter(kind).set_dst_width(dw).set_dst_height(dh)
    r = conv.create()
    d = torch.zeros((dh, dw), dtype=torch.int16, device="cuda")
    r.process(dev(src), d)
    torch.cuda.synchronize()
    np.save(os.path.join(out, f"got{i}.npy"), d.cpu().numpy().view(np.uint16))
    res["single_engines"].append(r.info["engine"])
res["status"].append(int(lib.zg_pipeline_status(1)))

convs, srcs, dsts = [], [], []
for i, (sw, sh, dw, dh) in enumerate(cfg["batch"]):
    src = np.load(os.path.join(out, f"bsrc{i}.npy"))
    convs.append(zg.ResizeConversion(sw, sh, "word").set_depth(10).set_filter("spline36")
                 .set_dst_width(dw).set_dst_height(dh))
    srcs.append(dev(src))
    dsts.append(torch.zeros((dh, dw), dtype=torch.int16, device="cuda"))
b = zg.Batch(convs)
b.set_io(srcs, dsts)
for mode in ("plain", "graph"):
    for d in dsts:
        d.zero_()
    (b.process if mode == "plain" else b.process_graph)()
    torch.cuda.synchronize()
    for i, d in enumerate(dsts):
        np.save(os.path.join(out, f"bgot_{mode}{i}.npy"), d.cpu().numpy().view(np.uint16))
res["status"].append(int(lib.zg_pipeline_status(1)))
json.dump(res, open(os.path.join(out, "res.json"), "w"))
"""


def test_cp_async_form_bitexact(cuda, oracle, tmp_path):
    rng = np.random.default_rng(0x7A)
    for i, (sw, sh, dw, dh, kind, depth) in enumerate(SINGLE):
        np.save(tmp_path / f"src{i}.npy", rng.integers(0, 1 << depth, size=(sh, sw), dtype=np.uint16))
    for i, (sw, sh, dw, dh) in enumerate(BATCH):
        np.save(tmp_path / f"bsrc{i}.npy", rng.integers(0, 1024, size=(sh, sw), dtype=np.uint16))
    json.dump({"single": SINGLE, "batch": BATCH}, open(tmp_path / "cfg.json", "w"))
    env = dict(os.environ, ZG_CHAIN_TMA="0", ZG_ROOT=ROOT)
    child = subprocess.run([sys.executable, "-c", CHILD, str(tmp_path)], env=env, capture_output=True, text=True,
                           timeout=600)
    assert child.returncode == 0, child.stderr[-3000:]
    res = json.load(open(tmp_path / "res.json"))
    assert res["status"] == [0, 0], "a pipelined kernel's bounded wait ran out"
    assert "tensor" in res["single_engines"]
    for i, (sw, sh, dw, dh, kind, depth) in enumerate(SINGLE):
        src = np.load(tmp_path / f"src{i}.npy")
        want = oracle.resize_plane(src, dw, dh, kind, depth=depth, mode="c", nthreads=16)
        np.testing.assert_array_equal(np.load(tmp_path / f"got{i}.npy"), want, err_msg=str(SINGLE[i]))
    for i, (sw, sh, dw, dh) in enumerate(BATCH):
        src = np.load(tmp_path / f"bsrc{i}.npy")
        want = oracle.resize_plane(src, dw, dh, "spline36", depth=10, mode="c", nthreads=16)
        for mode in ("plain", "graph"):
            np.testing.assert_array_equal(np.load(tmp_path / f"bgot_{mode}{i}.npy"), want,
                                          err_msg=f"{mode} {BATCH[i]}")


@pytest.mark.parametrize("sw,sh,dw,dh,kind", [
    (240, 96, 480, 192, "lanczos"),     # 2x up: kept products, four tiles a warp
    (1919, 70, 1279, 47, "spline36"),   # 1.5x down, odd lines
    (641, 131, 961, 197, "spline36"),   # 1.5x up
    (900, 65, 400, 29, "bicubic"),      # 2.25x down: strips narrower than seven warps' tiles
    (33, 17, 66, 34, "lanczos"),        # one strip, fewer lines than a window
    (320, 40, 426, 53, "bicubic"),      # a source for tensor copies, narrower strips, 4-byte stores
    (320, 40, 424, 53, "bicubic"),      # ... 16-byte stores
    (640, 64, 427, 43, "spline36"),     # ... single samples
    (17, 300, 23, 200, "bicubic")])
@pytest.mark.parametrize("pad,offset,flip", [(0, 0, False), (1, 1, False), (2, 4, False), (3, 7, False), (4, 2, True),
                                             (8, 8, False)])
def test_chained_kernel_any_alignment(cuda, oracle, sw, sh, dw, dh, kind, pad, offset, flip):
    """Planes at every offset of their lines in a 16-byte chunk, sources and
    destinations, bottom-up ones too, with all bits set between the lines
    (nothing there may reach a result) and kept between the output lines;
    single planes and a batch, bit for bit."""
    import torch
    import zimg_gb300 as zg
    rng = np.random.default_rng(sw * 17 + pad)
    src = rng.integers(0, 1024, size=(sh, sw), dtype=np.uint16)
    want = oracle.resize_plane(src, dw, dh, kind, depth=10, mode="c", nthreads=16)

    def plane(h, w):
        buf = torch.full((h * (w + pad) + offset,), -1, dtype=torch.int16, device="cuda")
        return buf, buf[offset:].view(h, w + pad)[:, :w]
    conv = zg.ResizeConversion(sw, sh, "word").set_depth(10).set_filter(kind).set_dst_width(dw).set_dst_height(dh)
    r = conv.create()
    assert r.info["engine"] == "tensor"
    sbuf, s = plane(sh, sw)
    host = src[::-1].copy() if flip else src
    s.copy_(torch.from_numpy(host.view(np.int16)))
    lib, stream = zg.load(), torch.cuda.current_stream().cuda_stream
    stride = (sw + pad) * 2
    sp, ss = (s.data_ptr() + (sh - 1) * stride, -stride) if flip else (s.data_ptr(), stride)
    dbuf, d = plane(dh, dw)
    assert lib.zg_resize_process(r.handle, sp, ss, d.data_ptr(), (dw + pad) * 2, None, stream) == 0
    torch.cuda.synchronize()
    np.testing.assert_array_equal(d.cpu().numpy().view(np.uint16), want)
    if pad:
        assert (dbuf[offset:].view(dh, dw + pad)[:, dw:] == -1).all()
    if not flip:
        planes = [plane(dh, dw)[1] for _ in range(3)]
        b = zg.Batch([conv] * 3)
        b.set_io([s] * 3, planes)
        b.process()
        torch.cuda.synchronize()
        for q in planes:
            np.testing.assert_array_equal(q.cpu().numpy().view(np.uint16), want)


@pytest.mark.parametrize("sw,sh,dw,dh,kind", [
    (640, 16, 272, 7, "bicubic"),    # a window of one block, the plane
    (640, 17, 272, 8, "bilinear"),   # the second of two in part
    (640, 79, 272, 33, "bicubic"),   # three blocks below the last group's row
    (640, 80, 272, 34, "bilinear"),  # ... and the plane ends with a block
    (640, 96, 320, 48, "bicubic"),   # whole groups
    (160, 16, 320, 33, "bicubic"),   # H first
    (160, 17, 320, 33, "lanczos")])
@pytest.mark.parametrize("pad,offset", [(0, 0), (1, 0), (8, 8)])
def test_windows_below_the_plane(cuda, oracle, sw, sh, dw, dh, kind, pad, offset):
    """Windows of whole 16-line blocks that end below the plane."""
    test_chained_kernel_any_alignment(cuda, oracle, sw, sh, dw, dh, kind, pad, offset, False)


@pytest.mark.parametrize("sw,sh,dw,dh,kind", [
    (640, 48, 800, 60, "bilinear"),    # H first, strips of 224 columns: four, the last one partial
    (256, 33, 448, 58, "bicubic"),     # two strips, whole
    (257, 33, 449, 58, "bicubic"),     # one column past them
    (300, 95, 330, 104, "bilinear"),   # nearly 1x
    (900, 40, 1283, 57, "spline16")])  # six strips
@pytest.mark.parametrize("pad,offset,flip", [(0, 0, False), (1, 1, False), (2, 4, True), (8, 8, False)])
def test_chained_kernel_narrow_strips(cuda, oracle, sw, sh, dw, dh, kind, pad, offset, flip):
    """Windows of 16 lines and columns in strips of two tiles a warp."""
    test_chained_kernel_any_alignment(cuda, oracle, sw, sh, dw, dh, kind, pad, offset, flip)


def test_narrow_strips_in_a_mixed_batch(cuda, oracle):
    """Jobs of two and of four tiles a warp, downscales and copies in one launch."""
    import torch
    import zimg_gb300 as zg
    rng = np.random.default_rng(0x7C)
    jobs = [(640, 48, 800, 60), (320, 64, 640, 128), (640, 96, 400, 64), (208, 160, 384, 176), (320, 64, 320, 64)] * 3
    convs, srcs, dsts, want = [], [], [], []
    for sw, sh, dw, dh in jobs:
        src = rng.integers(0, 1024, size=(sh, sw), dtype=np.uint16)
        want.append(oracle.resize_plane(src, dw, dh, "bilinear", depth=10, mode="c", nthreads=16))
        convs.append(zg.ResizeConversion(sw, sh, "word").set_depth(10).set_filter("bilinear").set_dst_width(dw)
                     .set_dst_height(dh))
        srcs.append(torch.from_numpy(src.view(np.int16)).cuda())
        dsts.append(torch.empty(dh, dw, dtype=torch.int16, device="cuda"))
    b = zg.Batch(convs)
    b.set_io(srcs, dsts)
    assert b.launch_count == 1
    for run in (b.process, b.process_graph):
        for d in dsts:
            d.zero_()
        run()
        torch.cuda.synchronize()
        for k, (d, w) in enumerate(zip(dsts, want)):
            np.testing.assert_array_equal(d.cpu().numpy().view(np.uint16), w, err_msg=str(jobs[k]))


@pytest.mark.parametrize("pad,offset", [(0, 0), (8, 8), (1, 3), (2, 0)])
def test_strips_of_two_and_four_tiles_in_one_launch(cuda, oracle, pad, offset):
    """Upscales of small windows, some in strips of four tiles a warp and some
    of two: one launch, whatever the planes' alignment."""
    import torch
    import zimg_gb300 as zg
    from test_gpu_resize import empty
    rng = np.random.default_rng(0x7E + pad)
    jobs = [(640, 48, 800, 60), (320, 64, 640, 128), (512, 33, 901, 58), (240, 40, 481, 80)] * 3
    convs, srcs, dsts, want = [], [], [], []
    for sw, sh, dw, dh in jobs:
        src = rng.integers(0, 1024, size=(sh, sw), dtype=np.uint16)
        want.append(oracle.resize_plane(src, dw, dh, "bilinear", depth=10, mode="c", nthreads=16))
        convs.append(zg.ResizeConversion(sw, sh, "word").set_depth(10).set_filter("bilinear").set_dst_width(dw)
                     .set_dst_height(dh))
        srcs.append(empty(sh, sw, np.uint16, pad=pad, offset=offset))
        srcs[-1].copy_(torch.from_numpy(src.view(np.int16)))
        dsts.append(empty(dh, dw, np.uint16, pad=pad, offset=offset))
    b = zg.Batch(convs)
    b.set_io(srcs, dsts)
    assert b.launch_count == 1
    for run in (b.process, b.process_graph):
        for d in dsts:
            d.zero_()
        run()
        torch.cuda.synchronize()
        for k, (d, w) in enumerate(zip(dsts, want)):
            np.testing.assert_array_equal(d.cpu().numpy().view(np.uint16), w, err_msg=str(jobs[k]))


FAULT_CHILD = r"""
import json, os, sys, time
import numpy as np
import torch
sys.path.insert(0, os.environ["ZG_ROOT"])
import zimg_gb300 as zg

out = sys.argv[1]
lib = zg.load()
lib.zg_pipeline_status(1)
src = np.load(os.path.join(out, "src.npy"))
conv = zg.ResizeConversion(1920, 1080, "word").set_depth(10).set_filter("lanczos", 3) \
    .set_dst_width(3840).set_dst_height(2160).create()
d_src = torch.from_numpy(src.view(np.int16)).cuda()
d_dst = torch.zeros((2160, 3840), dtype=torch.int16, device="cuda")
res = {"engine": conv.info["engine"]}
conv.process(d_src, d_dst)  # warm: module loaded, plan uploaded
torch.cuda.synchronize()
res["status_before"] = int(lib.zg_pipeline_status(1))
assert lib.zg_debug_pipeline_fault(0, 1000000) == 0
t0 = time.time()
conv.process(d_src, d_dst)
torch.cuda.synchronize()
res["fault_seconds"] = time.time() - t0
res["status_fault"] = int(lib.zg_pipeline_status(1))
res["status_after_reset"] = int(lib.zg_pipeline_status(0))
assert lib.zg_debug_pipeline_fault(-1, 0) == 0
d_dst.zero_()
conv.process(d_src, d_dst)
torch.cuda.synchronize()
res["status_clean"] = int(lib.zg_pipeline_status(1))
np.save(os.path.join(out, "got.npy"), d_dst.cpu().numpy().view(np.uint16))
json.dump(res, open(os.path.join(out, "res.json"), "w"))
"""


def test_bounded_wait_runs_out(cuda, oracle, tmp_path):
    rng = np.random.default_rng(0x7B)
    src = rng.integers(0, 1024, size=(1080, 1920), dtype=np.uint16)
    np.save(tmp_path / "src.npy", src)
    env = dict(os.environ, ZG_CHAIN_TMA="1", ZG_ROOT=ROOT)
    child = subprocess.run([sys.executable, "-c", FAULT_CHILD, str(tmp_path)], env=env, capture_output=True,
                           text=True, timeout=600)
    assert child.returncode == 0, child.stderr[-3000:]
    res = json.load(open(tmp_path / "res.json"))
    assert res["engine"] == "tensor"
    assert res["status_before"] == 0
    # the consumer's wait for the dropped group (1) or the producer's wait for
    # that stage's release (2), whichever gave up first
    assert res["status_fault"] in (1, 2), res
    assert res["status_after_reset"] == 0
    assert res["fault_seconds"] < 5.0, res
    assert res["status_clean"] == 0
    want = oracle.resize_plane(src, 3840, 2160, "lanczos", 3, depth=10, mode="c", nthreads=16)
    np.testing.assert_array_equal(np.load(tmp_path / "got.npy"), want)
