"""Wide contractions with many rows: two CTAs on one 256 x 256 tile.  Odd numbers of row tiles (a pair's second tile beyond the
matrix), ragged rows and columns, few and many K-slices, taps outside the image, strides, both operand types and zero points."""
import numpy as np
import pytest

from cases import S8, U8, run_case
from q8util import Cuda, gpu_pack, random_conv_case, random_fc_case

pytestmark = pytest.mark.gpu

U8X = dict(x_dtype=U8, y_dtype=U8, x_q=(0.02, 117))
CASES = {
    "fc_74_pairs": lambda: random_fc_case(1, 74 * 256, 2048, 256), "fc_odd_tiles": lambda: random_fc_case(2, 149 * 128 - 5, 2064, 256),
    "fc_two_column_tiles": lambda: random_fc_case(3, 75 * 128 + 1, 2048, 512), "fc_ragged_columns": lambda: random_fc_case(4, 80 * 128 + 77, 2160, 272),
    "fc_several_tiles_per_pair": lambda: random_fc_case(5, 2500, 2048, 2048), "fc_one_row_in_the_last_tile": lambda: random_fc_case(6, 148 * 128 + 1, 2064, 256),
    "conv_3x3": lambda: random_conv_case(7, 25, 28, 28, 256, 256, 3, 3, pad=(1, 1, 1, 1), act=(1, 0, 0)),
    "conv_3x3_u8_input": lambda: random_conv_case(8, 49, 20, 20, 144, 320, 3, 3, pad=(1, 1, 1, 1), **U8X),
    "conv_stride_2": lambda: random_conv_case(9, 100, 28, 28, 256, 256, 3, 3, stride=(2, 2), pad=(0, 1, 0, 1)),
    "conv_1x1_stride_2": lambda: random_conv_case(10, 100, 28, 27, 2048, 256, 1, 1, stride=(2, 2)),
    "conv_1x1": lambda: random_conv_case(11, 97, 14, 14, 2048, 272, 1, 1, act=(1, 0, 0)),
    # 149 row tiles: the second tile of the last pair lies wholly beyond the last image
    "conv_3x3_odd_tiles": lambda: random_conv_case(13, 97, 14, 14, 256, 256, 3, 3, pad=(1, 1, 1, 1), act=(1, 0, 0)),
    "conv_3x3_odd_tiles_no_padding": lambda: random_conv_case(14, 132, 14, 14, 256, 256, 3, 3),
    "conv_stride_2_odd_tiles_u8_input": lambda: random_conv_case(15, 97, 28, 28, 240, 256, 3, 3, stride=(2, 2), pad=(0, 1, 0, 1), **U8X),
    "conv_1x1_stride_2_odd_tiles": lambda: random_conv_case(16, 97, 28, 27, 2048, 272, 1, 1, stride=(2, 2)),
    # one K-slice short of a pair's
    "fc_15_slices": lambda: random_fc_case(12, 74 * 256, 1920, 256),
}


@pytest.mark.parametrize("name", CASES)
def test_exact(built, name):
    case = CASES[name]()
    want, got = case.run_oracle(), case.run_gpu()
    for a, b in zip(want, got):
        assert a.shape == b.shape and np.array_equal(a, b), (name, int((np.asarray(a) != np.asarray(b)).sum()), np.asarray(a).size)


def test_bounded_waits_give_up(built):
    """Loads that never arrive (no load is issued at all): every wait of both CTAs runs into its limit, the launch returns and says so."""
    from armnn_b200 import _abi, lib
    l = lib.load_library()
    case = random_conv_case(17, 97, 14, 14, 256, 256, 3, 3, pad=(1, 1, 1, 1))
    mem = Cuda()
    p, _, _ = case.params(mem, False, 2)
    p.packed = gpu_pack(mem, p)
    p.selftest_us = 3000
    lib.call("conv2d_q8", p)
    assert l.b200k_poll_status() == _abi.E_TIMEOUT
    assert l.b200k_poll_status() == 0
    want, got = case.run_oracle(want_acc=False)[0], case.run_gpu(want_acc=False, algo=2)[0]
    assert np.array_equal(want, got)
