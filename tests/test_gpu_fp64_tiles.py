"""FP64 grouped GEMM at the edges of its tiles (16 x 16), K chunks (16) and staged segment lists (32
segments), through vmps_block_products, against the products in extended precision.

Tolerance: an inner product of length K in FP64 is off by at most K u sum |a||b| (u = 2^-53); segments add
their lengths."""
import numpy as np
import pytest

from vmps_gb300.blocks import Blocks, Symmetry
from vmps_gb300.enrich import _block_products

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,k,n,segs", [(1, 1, 1, 1), (15, 16, 17, 1), (16, 17, 16, 2), (17, 33, 31, 3), (11, 11, 11, 4),
                                        (16, 8, 8, 33), (33, 15, 1, 64), (5, 3, 7, 100), (70, 129, 65, 2)])
def test_block_products_at_tile_edges(gpu_ctx, m, k, n, segs):
    sym = Symmetry(("U1",))
    rng = np.random.default_rng(100 * m + k + n + segs)
    A = Blocks(1, np.arange(segs), np.zeros(segs), np.zeros(segs), [m] * segs, [k] * segs)
    B = Blocks(1, np.arange(segs), np.zeros(segs), np.zeros(segs), [k] * segs, [n] * segs)
    C = Blocks(1, [0, 1], [0, 0], [0, 0], [m, m], [n, n])   # block 1 has no product: zeros
    A.data[:] = rng.standard_normal(A.data.size)
    B.data[:] = rng.standard_normal(B.data.size)
    C.data[:] = np.nan
    coef = rng.standard_normal(segs)
    _block_products(gpu_ctx, sym, A, B, C, [(0, i, i) for i in range(segs)], coef)
    ref = sum(c * A.block(i).astype(np.longdouble) @ B.block(i).astype(np.longdouble) for i, c in enumerate(coef))
    size = sum(abs(c) * np.abs(A.block(i)) @ np.abs(B.block(i)) for i, c in enumerate(coef))
    assert np.all(np.abs(C.block(0) - ref) <= (segs * k + 2) * 2.0 ** -53 * size)
    assert not np.any(C.block(1))
