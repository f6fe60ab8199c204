"""Quantisation scales at the ends of the float range.  The reference divides by the output scale, so a value whose quotient
overflows saturates and one that underflows becomes the zero point; the kernels' division-free quotients have to do the same.
Sparse operands with values of 0 and +-1 put zero and overflowing quotients side by side in every group of outputs."""
import numpy as np
import pytest

from cases import S8, SimpleCase, _abi, qt, qt_out, run_case

pytestmark = pytest.mark.gpu

# input scale, weight (second operand) scale, output scale
ELT_SCALES = {"overflow": (1e20, 1e20, 1e-20), "half_way": (1e16, 1e3, 1e-16), "ordinary": (0.02, 0.03, 0.05), "tiny": (1e-20, 1e-20, 1e-20),
              "near_the_bound": (3e9, 3e9, 1e-20), "output_huge": (1e19, 1e18, 1e20)}


def _sparse(rng, shape):
    return (rng.integers(0, 3, size=shape) == 0).astype(np.int8) * np.where(rng.integers(0, 2, size=shape) == 0, -1, 1).astype(np.int8)


def _bytes(rng, shape):
    v = rng.integers(-128, 128, size=shape).astype(np.int8)
    return np.where(rng.integers(0, 3, size=shape) == 0, np.int8(5), v).astype(np.int8)      # a third are the zero point


def _eltwise(op, scales, n=4099):
    def build(mem):
        rng = np.random.default_rng(op)
        p = _abi.EltwiseParams()
        p.a, p.b = qt(mem, _bytes(rng, (n,)), S8, scales[0], 5), qt(mem, _bytes(rng, (n,)), S8, scales[1], 5)
        p.out, out = qt_out(mem, (n,), S8, scales[2], 3)
        p.rank, p.op = 1, op
        p.shape_a[0] = p.shape_b[0] = p.shape_out[0] = n
        p.clamp_lo, p.clamp_hi = -128, 127
        return p, [out]
    return SimpleCase("eltwise_q8", build)


def _resize(method, scales):
    def build(mem):
        rng = np.random.default_rng(method)
        p = _abi.ResizeParams()
        p.x = qt(mem, _bytes(rng, (2, 5, 6, 7)), S8, scales[0], 5)
        p.y, y = qt_out(mem, (2, 17, 20, 7), S8, scales[2], 3)
        p.n, p.c, p.in_h, p.in_w, p.out_h, p.out_w = 2, 7, 5, 6, 17, 20
        p.method, p.half_pixel_centers = method, 1
        return p, [y]
    return SimpleCase("resize_q", build)


def _bmm(scales, ty):
    def build(mem):
        rng = np.random.default_rng(9)
        p = _abi.BmmParams()
        p.x, p.y = qt(mem, _sparse(rng, (2, 70, 40)), S8, scales[0], 0), qt(mem, _sparse(rng, (2, 72, 40) if ty else (2, 40, 72)), S8, scales[1], 0)
        p.out, out = qt_out(mem, (2, 70, 72), S8, scales[2], 3)
        p.batch, p.m, p.k, p.n, p.transpose_y = 2, 70, 40, 72, int(ty)
        p.batch_stride_x, p.batch_stride_y = 70 * 40, 40 * 72
        return p, [out]
    return SimpleCase("batch_matmul_q8", build)


@pytest.mark.parametrize("scales", ELT_SCALES)
@pytest.mark.parametrize("name,case", [("op%d" % op, lambda s, op=op: _eltwise(op, s)) for op in (0, 2, 3, 4, 5)] +
                         [("bilinear", lambda s: _resize(0, s)), ("nearest", lambda s: _resize(1, s)), ("bmm", lambda s: _bmm(s, False)), ("bmm_t", lambda s: _bmm(s, True))])
def test_values(built, name, case, scales):
    if name.startswith("bmm") and scales == "overflow":
        scales = "near_the_bound"                            # (the product of the scales is not a float)
    want, got = run_case(case(ELT_SCALES[scales]), "oracle"), run_case(case(ELT_SCALES[scales]), "gpu")
    assert np.array_equal(want[0], got[0]), (name, scales, int((want[0] != got[0]).sum()), want[0].size)
