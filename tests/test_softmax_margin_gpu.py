"""Softmax over many short rows, whose requantisation takes a margin from the output's zero point: the same bytes as the kernel with
one CTA per row, which divides every value."""
import numpy as np
import pytest

from cases import S8, U8, SimpleCase, _abi, _rand, qt, qt_out, run_case

pytestmark = pytest.mark.gpu


def _case(x, dtype, scale, beta, y_q):
    def build(mem):
        p = _abi.SoftmaxParams()
        p.x = qt(mem, x, dtype, scale, 3)
        p.y, y = qt_out(mem, x.shape, dtype, *y_q)
        p.outer, p.axis_size, p.inner, p.beta = x.shape[0], x.shape[1], 1, beta
        return p, [y]
    return SimpleCase("softmax_q8", build)


# the usual output, zero points at the ends of the type, one far outside it, outputs that mostly saturate, and scales that put
# many quotients near a half
@pytest.mark.parametrize("y_q", [(1 / 256, -128), (0.001, 127), (0.003, 0), (1 / 256, -90000), (1e-4, -128), (1 / 384, -127), (1 / 1024, 5)])
@pytest.mark.parametrize("axis", [512, 511, 36, 129])
def test_the_same_bytes_as_one_row_per_block(built, axis, y_q):
    rows = 2048 + 13
    rng = np.random.default_rng(axis)
    dtype = S8 if axis != 36 else U8
    if dtype == U8:
        y_q = (y_q[0], y_q[1] + 128)
    x = _rand(rng, dtype, (rows, axis))
    many = run_case(_case(x, dtype, 0.02, 1.3, y_q), "gpu")[0]
    few = [run_case(_case(x[i:i + 1031], dtype, 0.02, 1.3, y_q), "gpu")[0] for i in (0, 1031)]
    assert np.array_equal(many, np.concatenate(few)[:rows])
