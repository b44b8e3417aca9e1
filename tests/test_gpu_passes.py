"""Separate passes with the width built in (pass_kernels.cu): every width the
kernels are built for and the first that they are not, lines and columns around
their batches, against the oracle bit for bit (u16: the C path; f32: one fused
multiply-add per tap in its order)."""
import numpy as np
import pytest

from test_gpu_resize import run_conversion

pytestmark = pytest.mark.gpu


def case_of_width(width):
    """A conversion of one direction whose filter has `width` taps."""
    import zimg_gb300 as zg
    for kind, a in [("point", np.nan), ("bilinear", np.nan), ("bicubic", np.nan), ("lanczos", 3.0), ("lanczos", 4.0)]:
        for sw in (131, 67, 211):
            for dw in range(12, 260):
                if dw != sw and zg.compute_filter(kind, sw, dw, a=a).filter_width == width:
                    return kind, a, sw, dw
    pytest.fail("no conversion with %d taps" % width)


@pytest.mark.parametrize("width", [*range(1, 18), 24, 31, 32, 34])
def test_horizontal_taps_in_registers(cuda, oracle, width):
    kind, a, sw, dw = case_of_width(width)
    rng = np.random.default_rng(width)
    for h, pad, offset in [(1, 0, 0), (7, 1, 1), (8, 3, 2), (13, 0, 5)]:
        for depth in (10, 16):
            src = rng.integers(0, 1 << depth, size=(h, sw), dtype=np.uint16)
            got, _ = run_conversion(src, dw, h, kind, a, depth=depth, pad=pad, offset=offset)
            np.testing.assert_array_equal(got, oracle.resize_plane(src, dw, h, kind, a, depth=depth, mode="c"))
        if width >= 32:  # the wide passes
            continue
        src = rng.standard_normal((h, sw)).astype(np.float32)
        got, _ = run_conversion(src, dw, h, kind, a, pad=pad, offset=offset)
        np.testing.assert_array_equal(got, oracle.resize_plane(src, dw, h, kind, a, mode="fma"))


@pytest.mark.parametrize("width", [*range(1, 18), 24, 31, 32, 34])
def test_vertical_window_in_flight(cuda, oracle, width):
    kind, a, sh, dh = case_of_width(width)
    rng = np.random.default_rng(100 + width)
    for w, pad, offset in [(1, 0, 0), (8, 0, 0), (19, 5, 0), (21, 3, 8), (1030, 2, 0), (130, 0, 1)]:
        for depth in (10, 16):
            src = rng.integers(0, 1 << depth, size=(sh, w), dtype=np.uint16)
            got, _ = run_conversion(src, w, dh, kind, a, depth=depth, pad=pad, offset=offset)
            np.testing.assert_array_equal(got, oracle.resize_plane(src, w, dh, kind, a, depth=depth, mode="c"))
        if width >= 32:
            continue
        src = rng.standard_normal((sh, w)).astype(np.float32)
        got, _ = run_conversion(src, w, dh, kind, a, pad=pad, offset=offset)
        np.testing.assert_array_equal(got, oracle.resize_plane(src, w, dh, kind, a, mode="fma"))


@pytest.mark.parametrize("planes", [1, 2, 16, 17, 35])
def test_batch_of_separate_passes(cuda, oracle, planes):
    """Jobs of separate passes, those of one conversion in the same launches:
    around the planes a launch takes, two conversions and one of a single
    pass interleaved, planes of different alignment."""
    import torch
    import zimg_gb300 as zg
    from test_gpu_resize import empty, to_dev
    rng = np.random.default_rng(planes)
    kinds = [(97, 61, 33, 20, "word", 16, "lanczos"), (64, 50, 24, 19, "float", None, "spline36"),
             (40, 30, 40, 51, "word", 10, "bicubic")]
    jobs, srcs, dsts, want = [], [], [], []
    for k in range(planes):
        for sw, sh, dw, dh, t, depth, kind in kinds:
            conv = zg.ResizeConversion(sw, sh, t).set_filter(kind).set_dst_width(dw).set_dst_height(dh).set_fusion(False)
            if depth:
                conv.set_depth(depth)
                src = rng.integers(0, 1 << depth, size=(sh, sw), dtype=np.uint16)
            else:
                src = rng.standard_normal((sh, sw)).astype(np.float32)
            s = empty(sh, sw, src.dtype, pad=k % 3, offset=k % 5)
            s.copy_(to_dev(src))
            jobs.append(conv)
            srcs.append(s)
            dsts.append(empty(dh, dw, src.dtype, pad=k % 2, offset=k % 4))
            want.append(oracle.resize_plane(src, dw, dh, kind, depth=depth, mode="c") if depth else
                        oracle.resize_plane(src, dw, dh, kind, mode="fma"))
    b = zg.Batch(jobs)
    b.set_io(srcs, dsts)
    for run in (b.process, b.process_graph):
        for d in dsts:
            d.zero_()
        run()
        torch.cuda.synchronize()
        for d, w in zip(dsts, want):
            got = d.cpu().numpy()
            np.testing.assert_array_equal(got.view(np.uint16) if w.dtype == np.uint16 else got, w)


@pytest.mark.parametrize("sample", ["word", "float"])
@pytest.mark.parametrize("odd", [(0,), (2,), (0, 2, 3), (0, 1, 2, 3)])
def test_large_planes_of_mixed_alignment(cuda, oracle, odd, sample):
    """Vertical passes of planes in 16-byte accesses beside those that cannot
    go so, in the order of the batch."""
    import torch
    import zimg_gb300 as zg
    from test_gpu_resize import empty, to_dev
    w, sh, dh = 3848, 1500, 771
    depth = 16 if sample == "word" else None
    rng = np.random.default_rng(len(odd))
    jobs, srcs, dsts, want = [], [], [], []
    for k in range(4):
        conv = zg.ResizeConversion(w, sh, sample).set_filter("bicubic").set_dst_height(dh)
        jobs.append(conv.set_depth(depth) if depth else conv)
        src = rng.integers(0, 1 << 16, size=(sh, w), dtype=np.uint16) if depth else \
            rng.standard_normal((sh, w)).astype(np.float32)
        off = k in odd
        srcs.append(empty(sh, w, src.dtype, pad=off, offset=off))
        srcs[-1].copy_(to_dev(src))
        dsts.append(empty(dh, w, src.dtype, pad=8 * (k % 2), offset=0))
        want.append(oracle.resize_plane(src, w, dh, "bicubic", depth=depth, mode="c", nthreads=16) if depth else
                    oracle.resize_plane(src, w, dh, "bicubic", mode="fma", nthreads=16))
    b = zg.Batch(jobs)
    b.set_io(srcs, dsts)
    b.process()
    torch.cuda.synchronize()
    for d, x in zip(dsts, want):
        got = d.cpu().numpy()
        np.testing.assert_array_equal(got.view(np.uint16) if depth else got, x)
