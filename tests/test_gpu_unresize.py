"""GPU parity of unresize (zimg's UnresizeConversion) through the C ABI:
bit-exact against the oracle's restatement of zimg's C path (pinned against
zimg's own code by tests/test_oracle_unresize.py), on the cases and golden
planes, a full-HD plane, and a bottom-up source."""
import numpy as np
import pytest

from test_oracle_unresize import CASES, GOLDEN, make_src

pytestmark = pytest.mark.gpu


def run(src, ow, oh, sw=0.0, sh=0.0):
    import torch
    import zimg_gb300 as zg
    uh, uw = src.shape
    u = zg.UnresizeConversion(uw, uh).set_orig_width(ow).set_orig_height(oh).set_shift_w(sw).set_shift_h(sh).create()
    s = torch.from_numpy(np.ascontiguousarray(src)).cuda()
    d = torch.zeros((oh, ow), dtype=torch.float32, device="cuda")
    u.process(s, d)
    torch.cuda.synchronize()
    return d.cpu().numpy()


@pytest.mark.parametrize("case", range(len(CASES)))
def test_unresize_bitexact(cuda, oracle, case):
    uw, uh, ow, oh, sw, sh = CASES[case]
    src = make_src(np.random.default_rng(950 + case), uh, uw)
    np.testing.assert_array_equal(run(src, ow, oh, sw, sh).view(np.uint32),
                                  oracle.unresize_plane(src, ow, oh, sw, sh).view(np.uint32), err_msg=str(CASES[case]))


def test_unresize_golden(cuda):
    data = np.load(GOLDEN)
    for k in range(int(data["n"])):
        uw, uh, ow, oh, sw, sh = CASES[int(data[f"case{k}"])]
        np.testing.assert_array_equal(run(data[f"src{k}"], ow, oh, sw, sh).view(np.uint32),
                                      data[f"out{k}"].view(np.uint32), err_msg=f"golden {k}")


def test_unresize_full_hd(cuda, oracle):
    src = make_src(np.random.default_rng(99), 1080, 1920)
    np.testing.assert_array_equal(run(src, 1280, 720).view(np.uint32),
                                  oracle.unresize_plane(src, 1280, 720).view(np.uint32))


@pytest.mark.parametrize("uw,uh,ow,oh,sw,sh", [
    (31, 45, 30, 31, 0.0, 0.0), (64, 64, 63, 33, 0.0, 0.0), (200, 130, 150, 65, 0.3, -0.2),
    (1733, 97, 1301, 70, 0.0, 0.0), (97, 1733, 70, 1301, 0.0, 0.0), (600, 400, 600, 400, 0.25, -0.25),
    (600, 400, 600, 400, 0.5, 0.5), (1, 9, 1, 5, 0.0, 0.0), (40000, 6, 30000, 4, 0.0, 0.0)])
@pytest.mark.parametrize("content", ["noise", "black", "special"])
def test_unresize_chunks(cuda, oracle, uw, uh, ow, oh, sw, sh, content):
    """Lines cut into chunks that run side by side: around the chunk's length
    and the block's lines and columns, contexts whose recurrences do not die
    out (half-sample shifts), lines beyond shared memory; noise, black borders
    (where the recurrence dies out through the denormals, sample after
    sample), and NaN, infinities and huge values that reach the whole line."""
    rng = np.random.default_rng(uw * 131 + oh)
    src = rng.random((uh, uw), dtype=np.float32) - 0.25
    if content == "black":
        src[:, uw // 4:uw * 7 // 8] = 0.0
        src[uh // 3:uh * 5 // 6, :] = 0.0
    elif content == "special":
        for v in (np.nan, np.inf, -np.inf, 3e38, -0.0):
            src[rng.integers(0, uh), rng.integers(0, uw)] = v
    got, want = run(src, ow, oh, sw, sh), oracle.unresize_plane(src, ow, oh, sw, sh)
    nan = np.isnan(want)
    np.testing.assert_array_equal(np.isnan(got), nan)
    np.testing.assert_array_equal(got[~nan].view(np.uint32), want[~nan].view(np.uint32))


@pytest.mark.parametrize("ratio", [14.0, 15.0, 15.5, 16.0, 16.5, 17.0, 30.0])
def test_unresize_long_rows(cuda, oracle, ratio):
    """Rows around the number of taps from which the chunks give way."""
    rng = np.random.default_rng(int(ratio * 2))
    for ow, oh in ((37, 21), (130, 3), (5, 70)):
        uw, uh = int(ow * ratio), int(oh * ratio)
        src = make_src(rng, uh, uw)
        np.testing.assert_array_equal(run(src, ow, oh).view(np.uint32), oracle.unresize_plane(src, ow, oh).view(np.uint32))
