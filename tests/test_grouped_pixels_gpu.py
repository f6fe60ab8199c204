"""1x1 convolutions whose input channels are a multiple of 8 only: groups of two and four pixels, and the padded copy where the
pixels do not divide or the columns would not fill their tiles."""
import numpy as np
import pytest

from cases import U8
from q8util import random_conv_case

pytestmark = pytest.mark.gpu

U8W = dict(x_dtype=U8, w_dtype=U8, y_dtype=U8, x_q=(0.02, 120))
CASES = {
    "c24_oc144": lambda: random_conv_case(1, 3, 16, 18, 24, 144, 1, 1, act=(1, 0, 0)), "c24_oc144_u8": lambda: random_conv_case(2, 2, 14, 14, 24, 144, 1, 1, **U8W),
    "c24_oc144_pixels_left_over": lambda: random_conv_case(3, 1, 15, 17, 24, 144, 1, 1), "c40_oc240": lambda: random_conv_case(4, 2, 9, 14, 40, 240, 1, 1, **U8W),
    "c24_oc16": lambda: random_conv_case(5, 1, 12, 12, 24, 16, 1, 1), "c56_oc96": lambda: random_conv_case(6, 1, 12, 13, 56, 96, 1, 1), "c72_oc432": lambda: random_conv_case(7, 1, 10, 10, 72, 432, 1, 1, act=(1, 0, 0)),
    "c24_oc144_many": lambda: random_conv_case(8, 8, 56, 56, 24, 144, 1, 1, **U8W),
}


@pytest.mark.parametrize("name", CASES)
def test_exact(built, name):
    case = CASES[name]()
    want, got = case.run_oracle(), case.run_gpu()
    for a, b in zip(want, got):
        assert a.shape == b.shape and np.array_equal(a, b), (name, int((np.asarray(a) != np.asarray(b)).sum()), np.asarray(a).size)
