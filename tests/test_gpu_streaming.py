"""The CUDA-core streaming kernel (fused_kernel.cuh) over work items of many
steps: batches in which a CTA takes long runs of a strip's steps, so that rings
wrap, records alternate and lines are loaded beside or after the pass that
reads the ring. Bit for bit against the oracle (u16: the C path; f32: one fused
multiply-add per tap in its order), launched repeatedly."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def check_batch(oracle, sw, sh, dw, dh, kind, a, sample, planes=24):
    """`planes` planes of one conversion at alternating alignments, the same
    few contents in turn."""
    import torch
    import zimg_gb300 as zg
    from test_gpu_resize import empty, to_dev
    depth = {"word10": 10, "word16": 16}.get(sample)
    rng = np.random.default_rng(sw * 7919 + dw * 31 + dh)
    contents, want = [], []
    for _ in range(3):
        if depth:
            src = rng.integers(0, 1 << depth, size=(sh, sw), dtype=np.uint16)
            want.append(oracle.resize_plane(src, dw, dh, kind, a, depth=depth, mode="c", nthreads=16))
        else:
            src = rng.random((sh, sw), dtype=np.float32)
            want.append(oracle.resize_plane(src, dw, dh, kind, a, mode="fma", nthreads=16))
        contents.append(src)
    conv, srcs, dsts = [], [], []
    for k in range(planes):
        c = zg.ResizeConversion(sw, sh, "word" if depth else "float").set_filter(kind, a).set_dst_width(dw) \
            .set_dst_height(dh).set_engine("cuda")
        conv.append(c.set_depth(depth) if depth else c)
        src = contents[k % 3]
        srcs.append(empty(sh, sw, src.dtype, pad=k % 4, offset=k % 5))
        srcs[-1].copy_(to_dev(src))
        dsts.append(empty(dh, dw, src.dtype, pad=k % 3, offset=k % 4))
    assert conv[0].create().info["engine"] == "cuda"
    b = zg.Batch(conv)
    b.set_io(srcs, dsts)
    for run in (b.process, b.process, b.process_graph, b.process):
        for d in dsts:
            d.zero_()
        run()
        torch.cuda.synchronize()
        for k, d in enumerate(dsts):
            got = d.cpu().numpy()
            np.testing.assert_array_equal(got.view(np.uint16) if depth else got.view(np.uint32),
                                          want[k % 3] if depth else want[k % 3].view(np.uint32), err_msg="plane %d" % k)


@pytest.mark.parametrize("sample", ["word10", "word16", "float"])
@pytest.mark.parametrize("sw,sh,dw,dh,kind,a", [
    (96, 250, 300, 1000, "lanczos", 3.0),        # H first: records replaced a step ahead of their readers
    (65, 1100, 263, 1401, "spline64", math.nan),  # H first, odd sizes
    (40, 1500, 200, 900, "bilinear", math.nan),   # H first, lines down
    (515, 1300, 257, 650, "spline36", math.nan),  # V first
    (260, 1400, 129, 175, "bilinear", math.nan)])  # V first, 8x down: lines loaded late
def test_streaming_many_steps(cuda, oracle, sw, sh, dw, dh, kind, a, sample):
    check_batch(oracle, sw, sh, dw, dh, kind, a, sample)


@pytest.mark.parametrize("sample", ["word10", "word16", "float"])
@pytest.mark.parametrize("sw,sh,dw,dh", [
    (1920, 1080, 320, 180),   # 6x
    (1927, 1267, 275, 181),   # 7x, odd sizes
    (700, 3001, 129, 251),    # 12x, steps' windows far apart
    (900, 1500, 450, 125),    # 12x down the columns, 2x along the lines
    (300, 1400, 43, 800)])    # 7x along the lines only
def test_point_filter_gaps(cuda, oracle, sw, sh, dw, dh, sample):
    """One tap an output: where rows lie far apart, so do the steps' windows,
    and a step brings in more lines than its windows hold."""
    check_batch(oracle, sw, sh, dw, dh, "point", math.nan, sample, planes=12)


@pytest.mark.parametrize("sample", ["word16", "float"])
@pytest.mark.parametrize("planes", [1, 2, 5, 9, 20])
@pytest.mark.parametrize("sw,sh,dw,dh", [(257, 420, 101, 169), (515, 1300, 257, 650), (65, 600, 263, 1401)])
def test_small_batches_in_short_chunks(cuda, oracle, sw, sh, dw, dh, planes, sample):
    """Chunks of one step to eight, some of them across strips and planes."""
    check_batch(oracle, sw, sh, dw, dh, "bicubic", math.nan, sample, planes=planes)
