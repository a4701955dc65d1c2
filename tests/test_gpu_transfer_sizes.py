"""The device GMRES of the transfer operator at vector lengths around its reduction chunks (8192 elements: one chunk,
two, some, more than the 32 that a block sums itself): the solution's residual by the operator meets the tolerance
asked for, up to the rounding of both, and a run gives the same bits again."""
import numpy as np
import pytest

from vmps_gb300 import models
from vmps_gb300.blocks import Blocks
from vmps_gb300.uniform import UniformMPS, bond_bases_su2
from vmps_gb300.vumps import MpoTransferMatrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,chunks", [(40, 1), (250, 2), (700, 12), (1300, 33)])
def test_transfer_solve_at_vector_lengths(gpu_ctx, D, chunks):
    m = models.heisenberg_su2(8)
    u = UniformMPS(m, bond_bases_su2(D, 14), seed=2)
    rng = np.random.default_rng(D)
    A = u.A
    for t in A:   # a contraction: the cell's transfer operator stays far below 1
        for i in range(t.n):
            t.block(i)[...] = rng.standard_normal((t.rows[i], t.cols[i])) * 0.05 / np.sqrt(D)
    order, W, nq = m.basis_order_map(4), [m.W[4], m.W[5]], m.sym.nq
    slot = max(p for (q, _), p in order.items() if tuple(q) == m.sym.vacuum())
    q0, a = next(k for k, p in order.items() if p == slot)
    dims = sorted(u.dims[0].items())
    LR = Blocks.from_entries(nq, [(0, q, q, rng.standard_normal((n, n)) / n ** 2) for q, n in dims])
    Y = Blocks.from_entries(nq, [(a, q, q, tuple(q0), rng.standard_normal((n, n))) for q, n in dims], tripod=True)
    T = MpoTransferMatrix(gpu_ctx, m.sym, "L", A, A, W, LR, slot, order, Y.like())
    n = Y.data.size
    assert (n + 8191) // 8192 >= chunks
    b = Y.data * T.slot_mask()
    x, info = T.solve_device(b, tol=1e-11, dimK=60)
    r = (b - T.hxv(x)) * T.slot_mask()
    assert info["iterations"] > 1
    # the operator's own rounding: sums of at most a few thousand products, 1e-12 of |x|
    assert np.sqrt(T.dot(r, r)) <= 1e-11 * np.sqrt(T.dot(b, b)) + 1e-12 * np.sqrt(T.dot(x, x))
    assert np.array_equal(T.solve_device(b, tol=1e-11, dimK=60)[0], x)
    T.close()
