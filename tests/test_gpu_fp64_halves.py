"""FP64 block products on both sides of the number of tiles (152) up to which tiles of more than 128 elements are
halved, against the products in extended precision.  Tolerance: an inner product of length K in FP64 is off by at
most K u sum |a||b| (u = 2^-53)."""
import numpy as np
import pytest

from vmps_gb300.blocks import Blocks, Symmetry
from vmps_gb300.enrich import _block_products

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(16, 16), (16, 9), (9, 16), (13, 11), (192, 192), (128, 304), (192, 208), (145, 270)])
def test_block_products_with_halved_tiles(gpu_ctx, m, n):
    k = 37
    rng = np.random.default_rng(m * n)
    A, B, C = (Blocks(1, [0], [0], [0], [r], [c]) for r, c in ((m, k), (k, n), (m, n)))
    A.data[:] = rng.standard_normal(A.data.size)
    B.data[:] = rng.standard_normal(B.data.size)
    C.data[:] = np.nan
    _block_products(gpu_ctx, Symmetry(("U1",)), A, B, C, [(0, 0, 0)], np.ones(1))
    ref = A.block(0).astype(np.longdouble) @ B.block(0).astype(np.longdouble)
    size = np.abs(A.block(0)) @ np.abs(B.block(0))
    assert np.all(np.abs(C.block(0) - ref) <= (k + 2) * 2.0 ** -53 * size)
