"""Sizes where a kernel or its dispatch changes what it does: tile edges and remainders, the smallest and the largest of a
variant's range, every data type it takes.  Compared with the CPU oracle like tests/test_kernels_gpu.py does."""
import numpy as np
import pytest

from cases import F32, S8, U8, SimpleCase, _abi, _rand, qt, qt_out, run_case
from q8util import activation_clamp, diff_stats, random_qlstm_case, random_fc_case

pytestmark = pytest.mark.gpu


def _f32(rng, mem, shape, scale=1.0):
    return qt(mem, (rng.standard_normal(shape) * scale).astype(np.float32), F32)


def conv_f32(seed, n, h, w, c, oc, k, stride=1, pad=0, dil=1, depthwise=False):
    def build(mem):
        rng = np.random.default_rng(seed)
        oh, ow = ((e + 2 * pad - dil * (k - 1) - 1) // stride + 1 for e in (h, w))
        p = _abi.Conv2dParams()
        p.x, p.w = _f32(rng, mem, (n, h, w, c)), _f32(rng, mem, (1, k, k, oc) if depthwise else (oc, k, k, c), 0.2)
        p.bias = _f32(rng, mem, (oc,))
        p.y, y = qt_out(mem, (n, oh, ow, oc), F32)
        p.n, p.h, p.wd, p.c, p.oh, p.ow, p.oc, p.kh, p.kw = n, h, w, c, oh, ow, oc, k, k
        p.stride_h = p.stride_w = stride
        p.pad_top = p.pad_left = pad
        p.dil_h = p.dil_w = dil
        return p, [y]
    return SimpleCase("dwconv2d_f32" if depthwise else "conv2d_f32", build)


def fc_f32(seed, m, k, n, transpose):
    def build(mem):
        rng = np.random.default_rng(seed)
        p = _abi.FcParams()
        p.x, p.w, p.bias = _f32(rng, mem, (m, k)), _f32(rng, mem, (n, k) if transpose else (k, n), 0.1), _f32(rng, mem, (n,))
        p.y, y = qt_out(mem, (m, n), F32)
        p.m, p.k, p.n, p.transpose_w = m, k, n, int(transpose)
        return p, [y]
    return SimpleCase("fully_connected_f32", build)


def bmm_f32(seed, batch, m, k, n, tx, ty):
    def build(mem):
        rng = np.random.default_rng(seed)
        p = _abi.BmmParams()
        p.x, p.y = _f32(rng, mem, (batch, k, m) if tx else (batch, m, k)), _f32(rng, mem, (batch, n, k) if ty else (batch, k, n))
        p.out, out = qt_out(mem, (batch, m, n), F32)
        p.batch, p.m, p.k, p.n, p.transpose_x, p.transpose_y = batch, m, k, n, int(tx), int(ty)
        p.batch_stride_x, p.batch_stride_y = m * k, k * n
        return p, [out]
    return SimpleCase("batch_matmul_f32", build)


F32_CASES = {
    # 32 x 32 and 64 x 64 tiles, rows / columns / channels just below, at and above a tile or a chunk
    "conv3x3_tile32_c5": lambda: conv_f32(1, 1, 9, 7, 5, 33, 3, pad=1), "conv3x3_tile64_c4": lambda: conv_f32(2, 6, 42, 40, 4, 64, 3, pad=1),
    "conv3x3_tile64_c9_oc65": lambda: conv_f32(3, 4, 41, 31, 9, 65, 3, pad=1), "conv1x1_c33": lambda: conv_f32(4, 2, 65, 64, 33, 66, 1),
    "conv5x5_s2_dil2": lambda: conv_f32(5, 1, 23, 19, 3, 8, 5, stride=2, pad=4, dil=2), "conv8x8_most_taps": lambda: conv_f32(6, 1, 16, 16, 2, 6, 8, pad=3),
    "conv9x9_beyond_the_tap_mask": lambda: conv_f32(7, 1, 12, 12, 2, 5, 9, pad=4), "conv2x2_even_taps": lambda: conv_f32(8, 2, 12, 11, 16, 20, 2),
    "dw_vec4_s2": lambda: conv_f32(9, 2, 15, 14, 12, 12, 3, stride=2, pad=1, depthwise=True),
    "dw_odd_channels": lambda: conv_f32(10, 1, 9, 9, 7, 7, 5, pad=2, depthwise=True),
    "fc_1x1x1": lambda: fc_f32(11, 1, 1, 1, True), "fc_m65_k31_n129": lambda: fc_f32(12, 65, 31, 129, True),
    "fc_kn_m33_k70_n34": lambda: fc_f32(13, 33, 70, 34, False), "fc_tile64": lambda: fc_f32(14, 900, 40, 700, True),
    "bmm_nn": lambda: bmm_f32(15, 3, 33, 65, 31, False, False), "bmm_tt": lambda: bmm_f32(16, 2, 70, 9, 66, True, True),
    "bmm_tn_tile64": lambda: bmm_f32(17, 5, 384, 33, 385, True, False), "bmm_nt": lambda: bmm_f32(18, 2, 64, 32, 64, False, True),
}


def softmax(seed, rows, axis, dtype, beta=1.0, spread=None):
    def build(mem):
        rng = np.random.default_rng(seed)
        p = _abi.SoftmaxParams()
        x = _rand(rng, dtype, (rows, axis)) if spread is None else np.clip(rng.normal(0, spread, (rows, axis)), -128, 127).astype(np.int8)
        p.x = qt(mem, x, dtype, 0.05, 3 if dtype == S8 else 130)
        p.y, y = qt_out(mem, (rows, axis), dtype, 1 / 256., -128 if dtype == S8 else 0)
        p.outer, p.axis_size, p.inner, p.beta = rows, axis, 1, beta
        return p, [y]
    return SimpleCase("softmax_q8", build)


SOFTMAX_CASES = {
    # one row per CTA / eight rows per warp, word and byte access, every number of words per lane, rows left over
    "one_row_of_15": lambda: softmax(1, 1, 15, S8), "rows_257_axis_16": lambda: softmax(2, 257, 16, S8),
    "rows_2048_axis_2000": lambda: softmax(3, 2048, 2000, S8), "rows_4097_axis_1000": lambda: softmax(4, 4097, 1000, U8),
    "rows_8195_axis_512": lambda: softmax(5, 8195, 512, S8, spread=20.0), "rows_8193_axis_33": lambda: softmax(6, 8193, 33, U8, beta=0.5),
    "rows_9000_axis_1": lambda: softmax(7, 9000, 1, S8), "rows_2049_axis_128": lambda: softmax(9, 2049, 128, S8), "rows_2050_axis_130": lambda: softmax(10, 2050, 130, U8), "rows_2060_axis_1021": lambda: softmax(11, 2060, 1021, S8), "rows_2047_axis_4": lambda: softmax(12, 2047, 4, S8), "rows_2064_axis_2048": lambda: softmax(13, 2064, 2048, U8), "longest_axis": lambda: softmax(8, 2, 12272, S8, beta=0.1),
}


def eltwise(seed, count, op, ta, tb, to, act=(0, 0., 0.)):
    def build(mem):
        rng = np.random.default_rng(seed)
        p = _abi.EltwiseParams()
        zero = {S8: -3, U8: 121}
        p.a, p.b = qt(mem, _rand(rng, ta, (count,)), ta, 0.031, zero[ta]), qt(mem, _rand(rng, tb, (count,)), tb, 0.017, zero[tb])
        oscale = {0: 0.05, 2: 0.03, 3: 0.03, 4: 0.06, 5: 0.05}[op]
        p.out, out = qt_out(mem, (count,), to, oscale, 7)
        p.rank, p.op = 1, op
        p.shape_a[0] = p.shape_b[0] = p.shape_out[0] = count
        p.clamp_lo, p.clamp_hi = activation_clamp(act[0], act[1], act[2], oscale, 7, to)
        return p, [out]
    return SimpleCase("eltwise_q8", build)


ELTWISE_CASES = {"op%d_n%d" % (op, n): (lambda op=op, n=n, t=t: eltwise(op * 100 + n, n, op, *t))
                 for op, n, t in ((0, 1, (S8, S8, S8)), (0, 4095, (U8, U8, U8)), (0, 65536, (S8, U8, S8)), (2, 4111, (S8, S8, U8)),
                                  (3, 16, (U8, S8, U8)), (4, 100003, (S8, S8, S8)), (4, 65536, (U8, U8, U8)), (5, 4113, (U8, U8, S8)))}
ELTWISE_CASES["add_relu"] = lambda: eltwise(9, 5000, 0, S8, S8, S8, act=(1, 0, 0))


def resize(seed, n, c, ih, iw, oh, ow, method, align=0, half=0, nchw=0, dtype=U8):
    def build(mem):
        rng = np.random.default_rng(seed)
        p = _abi.ResizeParams()
        p.x = qt(mem, _rand(rng, dtype, (n, c, ih, iw) if nchw else (n, ih, iw, c)), dtype, 0.05, 11)
        p.y, y = qt_out(mem, (n, c, oh, ow) if nchw else (n, oh, ow, c), dtype, 0.045, 9)
        p.n, p.c, p.in_h, p.in_w, p.out_h, p.out_w = n, c, ih, iw, oh, ow
        p.method, p.align_corners, p.half_pixel_centers, p.nchw = method, align, half, nchw
        return p, [y]
    return SimpleCase("resize_q", build)


RESIZE_CASES = {
    "up4_c21": lambda: resize(1, 2, 21, 9, 10, 36, 40, 0, half=1), "up_row_of_bytes": lambda: resize(2, 1, 3, 5, 5, 17, 11, 0, dtype=S8),
    "down_odd": lambda: resize(3, 2, 5, 40, 33, 13, 7, 0), "one_pixel": lambda: resize(4, 1, 1, 1, 1, 33, 3, 0, half=1),
    "align_rows_past_a_block": lambda: resize(5, 1, 4, 8, 9, 35, 37, 0, align=1), "nchw_up3": lambda: resize(6, 2, 3, 6, 7, 18, 21, 0, half=1, nchw=1),
    "nearest_up": lambda: resize(7, 1, 19, 6, 6, 23, 25, 1), "nearest_align": lambda: resize(8, 1, 2, 9, 9, 17, 4, 1, align=1, dtype=S8),
}


def argminmax(seed, rows, axis, function, dtype, wide=False):
    def build(mem):
        rng = np.random.default_rng(seed)
        p = _abi.ArgMinMaxParams()
        p.x = qt(mem, rng.integers(100, 104, size=(rows, axis)).astype(np.uint8 if dtype == U8 else np.int8), dtype, 0.1, 5)
        out, ptr = mem.out((rows,), np.int64 if wide else np.int32)
        p.y = ptr
        p.outer, p.axis_size, p.inner, p.function, p.out_int64 = rows, axis, 1, function, int(wide)
        return p, [out]
    return SimpleCase("arg_min_max_q", build)


ARG_CASES = {"max_rows1_axis1": lambda: argminmax(1, 1, 1, 1, S8), "max_rows257_axis21": lambda: argminmax(2, 257, 21, 1, U8),
             "min_rows300_axis63": lambda: argminmax(3, 300, 63, 0, S8), "max_rows511_axis64": lambda: argminmax(4, 511, 64, 1, U8),
             "min_rows1000_axis2_int64": lambda: argminmax(5, 1000, 2, 0, U8, wide=True)}


def mean(seed, n, h, w, c, dtype):
    def build(mem):
        rng = np.random.default_rng(seed)
        p = _abi.MeanParams()
        p.x = _f32(rng, mem, (n, h, w, c)) if dtype == F32 else qt(mem, _rand(rng, dtype, (n, h, w, c)), dtype, 0.05, 3)
        p.y, y = qt_out(mem, (n, c), dtype, *(() if dtype == F32 else (0.02, 1)))
        p.n, p.h, p.wd, p.c = n, h, w, c
        return p, [y]
    return SimpleCase("mean_hw_q8", build)


MEAN_CASES = {"f32_1x1_c1": lambda: mean(1, 2, 1, 1, 1, F32), "f32_28x28_c33": lambda: mean(2, 2, 28, 28, 33, F32), "s8_128_pixels_c132": lambda: mean(3, 2, 8, 16, 132, S8),
              "u8_129_pixels_c5": lambda: mean(4, 1, 3, 43, 5, U8)}

U8_HEAD = dict(x_dtype=U8, w_dtype=U8, y_dtype=U8, per_axis=False, x_q=(0.03, 119))
FC_CASES = {
    # 32 x 32 tiles with remainders; K below a slice, beyond one pass, odd and at odd addresses; every signedness
    "m5_k1_n1": lambda: random_fc_case(1, 5, 1, 1), "m33_k31_n33": lambda: random_fc_case(2, 33, 31, 33),
    "m200_k1280_n1001_u8": lambda: random_fc_case(3, 200, 1280, 1001, **U8_HEAD), "m32_k2049_n40": lambda: random_fc_case(4, 32, 2049, 40),
    "m64_k4101_n65_u8": lambda: random_fc_case(5, 64, 4101, 65, **U8_HEAD), "m17_k130_n2033_u8x": lambda: random_fc_case(6, 17, 130, 2033, x_dtype=U8, y_dtype=U8, x_q=(0.03, 100)),
    "m6_k2080_n31_u8w": lambda: random_fc_case(7, 6, 2080, 31, w_dtype=U8, per_axis=False), "m1_k451_n77": lambda: random_fc_case(8, 1, 451, 77),
}


def bmm(seed, batch, m, k, n, tx, ty, xt=S8, yt=S8, ot=S8, bcast=False):
    def build(mem):
        rng = np.random.default_rng(seed)
        p = _abi.BmmParams()
        p.x = qt(mem, _rand(rng, xt, (batch, k, m) if tx else (batch, m, k)), xt, 0.02, 3 if xt == S8 else 126)
        p.y = qt(mem, _rand(rng, yt, ((1,) if bcast else (batch,)) + ((n, k) if ty else (k, n))), yt, 0.03, -2 if yt == S8 else 131)
        p.out, out = qt_out(mem, (batch, m, n), ot, 0.02 * 0.03 * 74 * 74 * float(k) ** 0.5 / 30, 4 if ot == S8 else 120)
        p.batch, p.m, p.k, p.n, p.transpose_x, p.transpose_y = batch, m, k, n, int(tx), int(ty)
        p.batch_stride_x, p.batch_stride_y = m * k, 0 if bcast else k * n
        return p, [out]
    return SimpleCase("batch_matmul_q8", build)


# tiles of 128 x 64 and 128 x 128 with remainders, fewer steps than stages, every layout, odd row lengths, every signedness
BMM_CASES = {"%s%s_b%d_m%d_k%d_n%d" % ("T" if tx else "N", "T" if ty else "N", b, m, k, n):
             (lambda i=i, b=b, m=m, k=k, n=n, tx=tx, ty=ty, t=t: bmm(40 + i, b, m, k, n, tx, ty, *t))
             for i, (b, m, k, n, tx, ty, t) in enumerate((
                 (1, 1, 1, 1, 0, 0, (S8, S8, S8)), (3, 129, 64, 64, 0, 1, (S8, S8, S8)), (2, 128, 65, 128, 0, 1, (U8, U8, U8)), (2, 130, 200, 65, 0, 0, (S8, U8, S8)),
                 (2, 17, 512, 33, 0, 0, (U8, S8, S8)), (1, 64, 333, 129, 1, 0, (S8, S8, U8)), (2, 136, 128, 48, 1, 1, (S8, S8, S8)), (5, 96, 17, 17, 1, 1, (U8, U8, S8)),
                 (2, 256, 256, 256, 1, 0, (S8, S8, S8)), (3, 77, 96, 77, 0, 1, (S8, S8, S8)), (3, 77, 77, 32, 0, 0, (S8, S8, S8)), (1, 128, 192, 20, 0, 0, (S8, S8, S8))))}
BMM_CASES["broadcast"] = lambda: bmm(60, 4, 40, 72, 80, 0, 0, bcast=True)

def qlstm(seed, batch, i, u, o, gate_scale=None, weight_scale=None, **kw):
    """gate_scale 2^-7 with 2^-7 weights and inputs: products that fall on exact halves; larger weight scales: chains that
    saturate"""
    case = random_qlstm_case(seed, batch, i, u, o, **kw)
    for g in "ifco":
        if weight_scale is not None:
            for k in ("s_i2" + g, "s_r2" + g):
                if k in case.s:
                    case.s[k] = weight_scale
    if gate_scale is not None:
        for g in ("input", "forget", "cell", "output"):
            case.s[g + "_intermediate_scale"] = gate_scale
    return case


QLSTM_CASES = {
    # clusters of one, two (one and two rows), four and eight CTAs; more units than threads; more steps than are staged
    "batch1_u512": lambda: qlstm(1, 1, 40, 512, 64), "batch20_u130": lambda: qlstm(2, 20, 33, 130, 24), "batch60": lambda: qlstm(3, 60, 16, 64, 32),
    "batch89_two_rows_odd": lambda: qlstm(4, 89, 24, 48, 16), "batch150_two_rows": lambda: qlstm(5, 150, 16, 32, 16),
    "units_600_staged_in_two": lambda: qlstm(6, 2, 1100, 600, 32), "tiny": lambda: qlstm(7, 3, 1, 1, 1),
    "exact_halves": lambda: qlstm(8, 4, 64, 48, 32, gate_scale=2.0 ** -7, weight_scale=2.0 ** -7),
    "halves_everywhere": lambda: qlstm(9, 2, 64, 48, 32, gate_scale=2.0 ** -13, weight_scale=2.0 ** -7),
    "saturating": lambda: qlstm(10, 4, 64, 48, 32, weight_scale=1.5), "large_accumulators": lambda: qlstm(11, 90, 256, 96, 64, weight_scale=0.05),
    "no_projection_odd": lambda: qlstm(12, 5, 19, 37, 37, projection=False), "cifg_two_rows": lambda: qlstm(13, 90, 16, 40, 24, cifg=True, peephole=True),
    "one_tile_of_a_large_layer": lambda: qlstm(14, 1, 24, 6000, 16), "projection_not_staged": lambda: qlstm(15, 1, 16, 700, 320),
}

EXACT = {"bmm": BMM_CASES, "fc": FC_CASES, "f32": F32_CASES, "eltwise": ELTWISE_CASES, "resize": RESIZE_CASES, "arg": ARG_CASES, "mean": MEAN_CASES}
ROUNDED = {"softmax": SOFTMAX_CASES, "qlstm": QLSTM_CASES}


@pytest.mark.parametrize("group,name", [(g, n) for g, c in EXACT.items() for n in c])
def test_exact(built, group, name):
    want, got = run_case(EXACT[group][name](), "oracle"), run_case(EXACT[group][name](), "gpu")
    for w, g in zip(want, got):
        assert w.shape == g.shape and np.array_equal(w, g), (group, name, int((w != g).sum()))


@pytest.mark.parametrize("group,name", [(g, n) for g, c in ROUNDED.items() for n in c])
def test_within_one_unit(built, group, name):
    """exp and tanh: the device's against the host's, +-1 on at most 1 % of the elements"""
    want, got = run_case(ROUNDED[group][name](), "oracle"), run_case(ROUNDED[group][name](), "gpu")
    for w, g in zip(want, got):
        st = diff_stats(w, g)
        # (the int16 cell state goes through two of them)
        assert st["max_abs"] <= (2 if w.dtype == np.int16 else 1) and st["mismatch_frac"] <= 0.01, (group, name, st)
