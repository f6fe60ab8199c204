"""Quantisation scales at the ends of the float range.  The reference divides by the output scale, so a value whose quotient
overflows saturates and one that underflows becomes the zero point; the kernels' division-free quotients have to do the same.
Sparse operands with values of 0 and +-1 put zero and overflowing quotients side by side in every group of outputs."""
import numpy as np
import pytest

from cases import S8, U8, SimpleCase, _abi, qt, qt_out, run_case
from q8util import ConvCase, FcCase, diff_stats, random_qlstm_case
from test_shape_edges_gpu import softmax

pytestmark = pytest.mark.gpu

# input scale, weight (second operand) scale, output scale
ELT_SCALES = {"overflow": (1e20, 1e20, 1e-20), "half_way": (1e16, 1e3, 1e-16), "ordinary": (0.02, 0.03, 0.05), "tiny": (1e-20, 1e-20, 1e-20),
              "near_the_bound": (3e9, 3e9, 1e-20), "output_huge": (1e19, 1e18, 1e20)}
MAC_SCALES = {"overflow": (1e20, 1.0, 1e-20), "some_overflow": (1e18, 1e18, 1.0), "tiny": (1e-15, 1e-15, 2e-30), "subnormal": (1e-20, 1e-19, 3e-39),
              "output_huge": (1e16, 1e19, 1e35), "output_beyond_normal_reciprocals": (1e18, 2e19, 2e38), "ordinary": (0.02, 0.03, 0.002), "by_channel": (1e15, [1e15, 3e-35, 2e-35], 1e-20)}


def _sparse(rng, shape, lo=-1):
    return (rng.integers(0, 3, size=shape) == 0).astype(np.int8) * np.where(rng.integers(0, 2, size=shape) == 0, lo, 1).astype(np.int8)


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


def _conv(scales, c, oc, k, n=2, h=9, stride=1, depthwise=False, weights_u8=False, relu=False, add=False):
    rng = np.random.default_rng(c * 100 + k)
    x = _sparse(rng, (n, h, h, c))
    w = _sparse(rng, (1, k, k, oc) if depthwise else (oc, k, k, c), lo=1 if weights_u8 else -1)
    pad = (k // 2,) * 4
    case = ConvCase(x, w.astype(np.uint8) if weights_u8 else w, None, (scales[0], 0), (scales[1], 0), (scales[2], 3), stride=(stride, stride), pad=pad,
                    act=(1, 0., 0.) if relu else (0, 0., 0.), depthwise=depthwise, w_dtype=U8 if weights_u8 else S8)
    if isinstance(scales[1], list):                          # by channel: next to each other a scale that overflows and one that does not
        case.w_scales, case.w_q = np.resize(np.asarray(scales[1], np.float32), oc), (1.0, 0)
    if add:
        other = rng.integers(-128, 128, size=(n, case.oh, case.ow, oc)).astype(np.int8)
        case.add = (other, (scales[2] * 0.8, -3), (scales[2], 1))
    return case


def _fc(scales, m, k, n):
    rng = np.random.default_rng(m + n)
    return FcCase(_sparse(rng, (m, k)), _sparse(rng, (n, k)), None, (scales[0], 0), (scales[1], 0), (scales[2], 3))


MACS = {
    "conv_tc": lambda s: _conv(s, 64, 64, 1), "conv_tc_3x3_relu": lambda s: _conv(s, 64, 64, 3, relu=True), "conv_tc_add": lambda s: _conv(s, 64, 128, 1, add=True),
    "conv_grouped": lambda s: _conv(s, 16, 32, 1, n=8, h=8), "conv_stem": lambda s: _conv(s, 3, 64, 7, h=32, stride=2), "conv_dp4a": lambda s: _conv(s, 5, 7, 3),
    "dw_rows": lambda s: _conv(s, 32, 32, 3, depthwise=True), "dw_rows_relu": lambda s: _conv(s, 32, 32, 3, stride=2, depthwise=True, relu=True),
    "dw3x3": lambda s: _conv(s, 32, 32, 3, depthwise=True, weights_u8=True),
    "fc_stream": lambda s: _fc(s, 4, 64, 48), "fc_rows": lambda s: _fc(s, 2, 48, 33), "fc_mma": lambda s: _fc(s, 40, 51, 33),
}


@pytest.mark.parametrize("scales", ELT_SCALES)
@pytest.mark.parametrize("name,case", [("op%d" % op, lambda s, op=op: _eltwise(op, s)) for op in (0, 2, 3, 4, 5)] +
                         [("bilinear", lambda s: _resize(0, s)), ("nearest", lambda s: _resize(1, s)), ("bmm", lambda s: _bmm(s, False)), ("bmm_t", lambda s: _bmm(s, True))])
def test_values(built, name, case, scales):
    if name.startswith("bmm") and scales == "overflow":
        scales = "near_the_bound"                            # (the product of the scales is not a float)
    want, got = run_case(case(ELT_SCALES[scales]), "oracle"), run_case(case(ELT_SCALES[scales]), "gpu")
    assert np.array_equal(want[0], got[0]), (name, scales, int((want[0] != got[0]).sum()), want[0].size)


@pytest.mark.parametrize("name,scales", [(n, s) for n in MACS for s in MAC_SCALES if s != "by_channel" or n[:3] in ("con", "dw_")])
def test_contractions(built, name, scales):
    case = MACS[name](MAC_SCALES[scales])
    want, got = case.run_oracle(), case.run_gpu()
    assert np.array_equal(want[1], got[1])
    assert np.array_equal(want[0], got[0]), (name, scales, int((want[0] != got[0]).sum()), want[0].size)


@pytest.mark.parametrize("rows,axis", [(2100, 64), (2100, 63), (3, 64)])
def test_softmax_exponentials_that_overflow(built, rows, axis):
    """beta < 0: the reference's exponentials and their sum are infinite, and infinity over infinity is not a number."""
    case = softmax(rows, rows, axis, S8, beta=-40.0)
    want, got = run_case(case, "oracle"), run_case(case, "gpu")
    assert set(np.unique(want[0])) == {-128}
    assert np.array_equal(want[0], got[0]), int((want[0] != got[0]).sum())


@pytest.mark.parametrize("scale,zp", [(0.05, 7), (3e37, 0), (0.05, 300), (1e-39, -4)])
def test_max_pooling_without_requantisation(built, scale, zp):
    """Values that overflow when dequantised, and a zero point outside the type's range in windows that lie in the padding."""
    def build(mem):
        rng = np.random.default_rng(5)
        p = _abi.Pool2dParams()
        n, h, oh, c = 8, 284, 144, 16
        p.x = qt(mem, rng.integers(0, 256, size=(n, h, h, c)).astype(np.uint8), U8, scale, zp)
        p.y, y = qt_out(mem, (n, oh, oh, c), U8, scale, zp)
        p.n, p.h, p.wd, p.c, p.oh, p.ow = n, h, h, c, oh, oh
        p.pool_h = p.pool_w = p.stride_h = p.stride_w = 2
        p.pad_top = p.pad_bottom = p.pad_left = p.pad_right = 2
        p.pool_type, p.padding_method = 0, 1
        return p, [y]
    case = SimpleCase("pool2d_q8", build)
    want, got = run_case(case, "oracle"), run_case(case, "gpu")
    assert np.array_equal(want[0], got[0]), int((want[0] != got[0]).sum())


@pytest.mark.parametrize("projection", [False, True])
@pytest.mark.parametrize("batch", [2, 90])
def test_qlstm_products_that_overflow(built, batch, projection):
    """A product over the gate's scale is infinite: the step saturates, in the direction of its sign."""
    case = random_qlstm_case(batch, batch, 16, 20, 12 if projection else 20, layer_norm=False, projection=projection)
    case.x, case.h = _sparse(np.random.default_rng(1), case.x.shape), _sparse(np.random.default_rng(2), case.h.shape)
    case.s["input_scale"] = case.s["output_state_scale"] = 1e17
    for g in "ifco":
        case.s["s_i2" + g] = case.s["s_r2" + g] = 1e17
        for k in ("w_i2" + g, "w_r2" + g):
            case.w[k] = _sparse(np.random.default_rng(ord(g)), case.w[k].shape)
    for g in ("input", "forget", "cell", "output"):
        case.s[g + "_intermediate_scale"] = 2.0 ** -18
    want, got = case.run_oracle(), case.run_gpu()
    for w, g in zip(want, got):
        st = diff_stats(w, g)                  # (exp and tanh: see test_shape_edges_gpu.py)
        assert st["max_abs"] <= (2 if w.dtype == np.int16 else 1) and st["mismatch_frac"] <= 0.01, st
