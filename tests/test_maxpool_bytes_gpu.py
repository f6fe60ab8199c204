"""Max pooling on the bytes themselves (equal quantisation of input and output): blocks of taps that the window ends inside of,
windows in the padding, and every pair of neighbouring bytes that could disturb a 16-bit maximum."""
import numpy as np
import pytest

from cases import S8, U8, SimpleCase, _abi, qt, qt_out, run_case

pytestmark = pytest.mark.gpu


def _pool(dtype, n, h, w, c, ph, pw, sh, sw, pads):
    def build(mem):
        rng = np.random.default_rng(ph * 10 + pw)
        lo, hi = (0, 256) if dtype == U8 else (-128, 128)
        x = rng.integers(lo, hi, size=(n, h, w, c))
        x[:, ::2] = rng.choice([lo, lo + 1, -1 if lo else 127, 0 if lo else 128, hi - 1], size=x[:, ::2].shape)    # ends and middle of the range side by side
        x = x.astype(np.uint8 if dtype == U8 else np.int8)
        p = _abi.Pool2dParams()
        p.x = qt(mem, x, dtype, 0.05, 7)
        oh, ow = (h + pads[0] + pads[1] - ph) // sh + 1, (w + pads[2] + pads[3] - pw) // sw + 1
        p.y, y = qt_out(mem, (n, oh, ow, c), dtype, 0.05, 7)
        p.n, p.h, p.wd, p.c, p.oh, p.ow = n, h, w, c, oh, ow
        p.pool_type, p.pool_h, p.pool_w, p.stride_h, p.stride_w = 0, ph, pw, sh, sw
        p.pad_top, p.pad_bottom, p.pad_left, p.pad_right = pads
        p.padding_method = 1
        return p, [y]
    return SimpleCase("pool2d_q8", build)


# (enough outputs for the 16-channel kernel: 148 SMs x 1024 threads x 16 channels)
@pytest.mark.parametrize("dtype", [S8, U8])
@pytest.mark.parametrize("ph,pw,sh,sw,pads", [(3, 3, 2, 2, (1, 0, 1, 0)), (2, 2, 2, 2, (0, 0, 0, 0)), (1, 1, 2, 2, (0, 0, 0, 0)), (2, 3, 1, 2, (1, 1, 1, 1)),
                                              (5, 4, 2, 2, (2, 2, 1, 1)), (1, 4, 1, 2, (0, 0, 1, 1)), (1, 5, 1, 2, (0, 0, 2, 2)), (4, 1, 2, 1, (1, 1, 0, 0)), (5, 1, 2, 1, (2, 2, 0, 0)), (7, 7, 2, 3, (3, 3, 3, 3)), (2, 2, 2, 2, (3, 3, 3, 3))])
def test_exact(built, dtype, ph, pw, sh, sw, pads):
    outputs = ((56 + pads[0] + pads[1] - ph) // sh + 1) * ((50 + pads[2] + pads[3] - pw) // sw + 1) * 4
    case = _pool(dtype, -(-148 * 1024 // outputs) + 1, 56, 50, 64, ph, pw, sh, sw, pads)
    want, got = run_case(case, "oracle"), run_case(case, "gpu")
    assert np.array_equal(want[0], got[0]), int((want[0] != got[0]).sum())
