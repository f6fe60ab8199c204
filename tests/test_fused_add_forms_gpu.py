"""A convolution with a fused Add: the Add as arithmetic where that gives its table's every entry, by the table elsewhere."""
import numpy as np
import pytest

from armnn_b200 import lib
from cases import S8, U8, run_case
from q8util import Cuda, gpu_pack, random_conv_case

pytestmark = pytest.mark.gpu

# (type, convolution's output, other operand, Add's output, fused ReLU).  Scales in powers of two put sums on exact halves, which
# no linear form rounds away from zero on both sides; 1e-3 for the output saturates most sums; 40.0 leaves a few output values.
QUANT = {
    "s8": (S8, (0.02, 3), (0.031, -7), (0.043, 5), 0), "s8_relu": (S8, (0.02, 3), (0.031, -7), (0.043, -20), 1),
    "u8": (U8, (0.017, 121), (0.029, 140), (0.033, 118), 0), "u8_relu": (U8, (0.017, 0), (0.029, 255), (0.033, 9), 1),
    "halves": (S8, (2.0 ** -6, 0), (2.0 ** -6, 1), (2.0 ** -5, 0), 0), "saturating": (S8, (0.02, 0), (0.03, 0), (1e-3, 0), 0),
    "coarse": (U8, (0.02, 100), (0.03, 90), (40.0, 7), 0), "other_dominates": (S8, (1e-4, 0), (0.5, 0), (0.51, 0), 0),
    "one_value_left": (S8, (0.02, 3), (0.031, -7), (0.043, 127), 1),
}
# one tile per CTA with constants in shared memory; the first number of row tiles beyond two per SM (148); narrow and ragged n-tiles
SHAPES = {"small": (1, 9, 15, 64, 128), "many_tiles": (1, 2, 148 * 128 + 1, 32, 256), "ragged": (2, 31, 33, 48, 176), "narrow": (3, 16, 16, 128, 64)}


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("quant", QUANT)
def test_exact(built, quant, shape):
    dtype, y_q, other_q, out_q, relu = QUANT[quant]
    n, h, w, c, oc = SHAPES[shape]
    u8 = dict(x_dtype=U8, w_dtype=U8, y_dtype=U8, x_q=(0.02, 128)) if dtype == U8 else {}

    def case():
        k = random_conv_case(31, n, h, w, c, oc, 1, 1, act=(1, 0, 0) if relu else (0, 0, 0), fused_add=True, **u8)
        k.y_q, k.add = y_q, (k.add[0], other_q, out_q)
        return k
    want, got = run_case(case(), "oracle"), run_case(case(), "gpu")
    for a, b in zip(want, got):
        assert a.shape == b.shape and np.array_equal(a, b), (quant, shape, int((a != b).sum()))


# Without packed tables (which input zero point 0 does not need), and with a table that was made for another output scale: every
# value takes the reference arithmetic, and shared memory holds no table to look anything up in.
@pytest.mark.parametrize("table", ["none", "made_for_another_scale"])
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("quant", ["s8_relu", "u8"])
def test_no_usable_table(built, quant, shape, table):
    dtype, y_q, other_q, out_q, relu = QUANT[quant]
    n, h, w, c, oc = SHAPES[shape]
    u8 = dict(x_dtype=U8, y_dtype=U8) if dtype == U8 else {}
    case = random_conv_case(33, n, h, w, c, oc, 1, 1, act=(1, 0, 0) if relu else (0, 0, 0), fused_add=True, x_q=(0.02, 0), **u8)
    case.y_q, case.add = y_q, (case.add[0], other_q, out_q)
    want, got = case.run_oracle()[0], _without_table(case, table)
    assert np.array_equal(want, got), (quant, shape, int((want != got).sum()))


def _without_table(case, table):
    if table == "none":
        return case.run_gpu(want_acc=False, algo=2, pack=False)[0]
    mem = Cuda()
    p, y, _ = case.params(mem, False, 2)
    scale, p.add_out.scale = p.add_out.scale, p.add_out.scale * 1.5
    p.packed = gpu_pack(mem, p)
    p.add_out.scale = scale
    lib.call("conv2d_q8", p)
    return mem.fetch(y)


# Which of the two a launch takes: with every entry of its packed table inverted, only the arithmetic still gives the oracle's bytes.
@pytest.mark.parametrize("shape", ["small", "many_tiles"])
@pytest.mark.parametrize("quant", ["s8", "s8_relu", "u8", "u8_relu", "halves"])
def test_which_form_runs(built, quant, shape):
    dtype, y_q, other_q, out_q, relu = QUANT[quant]
    n, h, w, c, oc = SHAPES[shape]
    u8 = dict(x_dtype=U8, w_dtype=U8, y_dtype=U8, x_q=(0.02, 128)) if dtype == U8 else {}
    case = random_conv_case(31, n, h, w, c, oc, 1, 1, act=(1, 0, 0) if relu else (0, 0, 0), fused_add=True, **u8)
    case.y_q, case.add = y_q, (case.add[0], other_q, out_q)
    mem = Cuda()
    p, y, _ = case.params(mem, False, 2)
    p.packed = gpu_pack(mem, p)
    words = [t for t in mem.keep if t.data_ptr() == p.packed][0]
    tag = int(np.flatnonzero(words.cpu().numpy() == 0x4C555431)[0])                # the table's 256 rows of 260 bytes end here
    words[tag - 256 * 65:tag].bitwise_not_()
    lib.call("conv2d_q8", p)
    same = np.array_equal(case.run_oracle()[0], mem.fetch(y))
    assert same == (quant != "halves")
