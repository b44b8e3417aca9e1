"""Horizontal passes with the taps in registers (pass_kernels.cu): every width
the kernel is built for and the first that it is not, line counts around its
batches, against the oracle bit for bit (u16: the C path; f32: one fused
multiply-add per tap in its order)."""
import numpy as np
import pytest

from test_gpu_resize import run_conversion

pytestmark = pytest.mark.gpu


def case_of_width(width):
    """A conversion of one direction whose filter has `width` taps."""
    import zimg_gb300 as zg
    for kind, a in [("point", np.nan), ("bilinear", np.nan), ("bicubic", np.nan), ("lanczos", 3.0), ("lanczos", 4.0)]:
        for sw in (131, 67):
            for dw in range(12, 260):
                if dw != sw and zg.compute_filter(kind, sw, dw, a=a).filter_width == width:
                    return kind, a, sw, dw
    pytest.fail("no conversion with %d taps" % width)


@pytest.mark.parametrize("width", range(1, 18))
def test_horizontal_taps_in_registers(cuda, oracle, width):
    kind, a, sw, dw = case_of_width(width)
    rng = np.random.default_rng(width)
    for h, pad, offset in [(1, 0, 0), (7, 1, 1), (8, 3, 2), (13, 0, 5)]:
        for depth in (10, 16):
            src = rng.integers(0, 1 << depth, size=(h, sw), dtype=np.uint16)
            got, _ = run_conversion(src, dw, h, kind, a, depth=depth, pad=pad, offset=offset)
            np.testing.assert_array_equal(got, oracle.resize_plane(src, dw, h, kind, a, depth=depth, mode="c"))
        src = rng.standard_normal((h, sw)).astype(np.float32)
        got, _ = run_conversion(src, dw, h, kind, a, pad=pad, offset=offset)
        np.testing.assert_array_equal(got, oracle.resize_plane(src, dw, h, kind, a, mode="fma"))
