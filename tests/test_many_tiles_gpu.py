"""Counts beyond what one launch's grid holds, and FullyConnected with odd extents over many row tiles."""
import numpy as np
import pytest

from cases import S8, U8, run_case
from q8util import random_fc_case
from test_shape_edges_gpu import U8_HEAD, bmm_f32, fc_f32, mean, resize

pytestmark = pytest.mark.gpu

CASES = {
    # 65535 images, batches or column tiles are one launch
    "mean_65536_images": lambda: mean(1, 65536, 1, 1, 1, S8), "mean_131071_images_c4": lambda: mean(2, 131071, 2, 1, 4, U8),
    "bmm_f32_65537_batches": lambda: bmm_f32(3, 65537, 1, 1, 1, False, False), "bmm_f32_131071_batches": lambda: bmm_f32(4, 131071, 2, 3, 1, True, True),
    "fc_f32_65536_column_tiles": lambda: fc_f32(5, 1, 1, 65535 * 64 + 1, True), "fc_f32_kn_65536_column_tiles": lambda: fc_f32(6, 1, 2, 65535 * 64 + 3, False),
    "resize_65536_images": lambda: resize(7, 65536, 1, 1, 2, 2, 3, 0), "resize_65535_images": lambda: resize(8, 65535, 1, 2, 1, 3, 2, 1),
    # fc_mma_kernel: several passes over K in each of many row tiles, and its last number of rows and the one after
    "fc_1025_rows": lambda: random_fc_case(9, 1025, 4101, 70), "fc_777_rows_u8": lambda: random_fc_case(10, 777, 2064, 49, **U8_HEAD),
    "fc_4097_rows": lambda: random_fc_case(11, 4097, 80, 33), "fc_most_rows": lambda: random_fc_case(12, 65535 * 32, 3, 2), "fc_more_rows": lambda: random_fc_case(13, 65535 * 32 + 1, 3, 2),
}


@pytest.mark.parametrize("name", CASES)
def test_exact(built, name):
    want, got = run_case(CASES[name](), "oracle"), run_case(CASES[name](), "gpu")
    for w, g in zip(want, got):
        assert w.shape == g.shape and np.array_equal(w, g), (name, int((w != g).sum()))
