"""Row offsets of the device's row-major copy at the edges of the scan's tiles
(4,096 rows) and of the tiles that a scanning CTA adds up (1,024 of them)."""
import numpy as np
import pytest

from ccd_b200 import native, synthetic
from ccd_b200.data import MODEL_LOGISTIC

from .test_gpu_row_major import expected_row_major

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,P", [(1, 3), (4095, 5), (4096, 5), (4097, 5), (8193, 5), (4096 * 1025 + 1, 2)])
def test_row_offsets_at_tile_edges(gpu_ctx, K, P):
    d = synthetic.small(MODEL_LOGISTIC, seed=K % 1000, K=K, P=P, density=0.3, formats=("indicator", "sparse"))
    m = native.Matrix(gpu_ctx, d)
    try:
        got = m.row_major()
    finally:
        m.close()
    for a, b in zip(got, expected_row_major(d)):
        assert np.array_equal(a, b)
