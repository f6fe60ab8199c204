"""Few-channel stems with many tiles per CTA: one new row per tile (stride 1), more output channels than four accumulators hold."""
import ctypes as C

import numpy as np
import pytest

from cases import U8
from q8util import Host, random_conv_case

pytestmark = pytest.mark.gpu

U8X = dict(x_dtype=U8, y_dtype=U8, x_q=(0.02, 117))
CASES = {
    "3x3_oc16": lambda: random_conv_case(1, 256, 32, 32, 3, 16, 3, 3, pad=(1, 1, 1, 1), act=(1, 0, 0)), "3x3_oc144_u8": lambda: random_conv_case(2, 64, 48, 48, 3, 144, 3, 3, pad=(1, 1, 1, 1), **U8X),
    "5x5_c1": lambda: random_conv_case(3, 64, 64, 64, 1, 32, 5, 5, pad=(2, 2, 2, 2)), "7x7_no_padding": lambda: random_conv_case(4, 60, 70, 80, 3, 16, 7, 7),
    "3x3_stride_2": lambda: random_conv_case(5, 128, 96, 96, 3, 32, 3, 3, stride=(2, 2), pad=(0, 1, 0, 1), act=(1, 0, 0)), "7x7_stride_2_oc256": lambda: random_conv_case(6, 32, 64, 64, 3, 256, 7, 7, stride=(2, 2), pad=(3, 2, 3, 2)),
    "11x11_stride_4_rows": lambda: random_conv_case(7, 40, 200, 64, 3, 64, 11, 3, stride=(4, 2), pad=(2, 2, 1, 0)), "3x3_stride_3_rows": lambda: random_conv_case(8, 64, 96, 64, 4, 48, 3, 3, stride=(3, 1), pad=(0, 0, 1, 1)),
    # strides above the filter's height: rows between two tiles that none reads
    "1x1_stride_2_rows": lambda: random_conv_case(9, 400, 15, 32, 3, 16, 1, 1, stride=(2, 1)), "2x2_stride_3_rows": lambda: random_conv_case(10, 400, 23, 32, 3, 16, 2, 2, stride=(3, 2), **U8X),
    "3x3_stride_4_rows": lambda: random_conv_case(11, 400, 31, 48, 1, 32, 3, 3, stride=(4, 1), act=(1, 0, 0)), "1x3_stride_4_rows": lambda: random_conv_case(12, 600, 18, 32, 2, 48, 1, 3, stride=(4, 1), pad=(1, 0, 1, 1)),
    # tall filters with one or two output rows: tiles of different images share no rows
    "11_rows_one_output_row": lambda: random_conv_case(13, 3000, 11, 16, 3, 16, 11, 3), "9_rows_one_output_row": lambda: random_conv_case(14, 2500, 9, 16, 4, 32, 9, 3, pad=(0, 0, 1, 1)),
    "8_rows_one_output_row": lambda: random_conv_case(15, 2500, 8, 16, 3, 16, 8, 3, **U8X), "11_rows_stride_4_two_output_rows": lambda: random_conv_case(16, 1600, 14, 16, 3, 32, 11, 3, stride=(4, 1), pad=(1, 0, 0, 0)),
}


@pytest.mark.parametrize("name", CASES)
def test_exact(built, name):
    from armnn_b200 import lib
    case = CASES[name]()
    p, _, _ = case.params(Host())
    assert lib.load_library().b200k_conv2d_scratch_bytes(C.byref(p)) == 0            # (the kernel that reads the input where it lies)
    want, got = case.run_oracle(), case.run_gpu(algo=2)
    for a, b in zip(want, got):
        assert a.shape == b.shape and np.array_equal(a, b), (name, int((np.asarray(a) != np.asarray(b)).sum()), np.asarray(a).size)
