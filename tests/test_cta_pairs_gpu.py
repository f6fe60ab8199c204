"""Wide contractions with many rows: two CTAs on one 256 x 256 tile.  Odd numbers of row tiles (a pair's second tile beyond the
matrix), ragged rows and columns, few and many K-slices, taps outside the image, strides, both operand types and zero points."""
import numpy as np
import pytest

from cases import S8, U8, run_case
from q8util import random_conv_case, random_fc_case

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
    # one K-slice short of a pair's
    "fc_15_slices": lambda: random_fc_case(12, 74 * 256, 1920, 256),
}


@pytest.mark.parametrize("name", CASES)
def test_exact(built, name):
    case = CASES[name]()
    want, got = case.run_oracle(), case.run_gpu()
    for a, b in zip(want, got):
        assert a.shape == b.shape and np.array_equal(a, b), (name, int((np.asarray(a) != np.asarray(b)).sum()), np.asarray(a).size)
