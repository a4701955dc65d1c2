"""Columns with special values or far exponents in tiles of the FP64 slice engine whose last 32 rows hold only a few rows
of the block: every column is recognised whichever rows the tile has, in each of the eight columns a flush warp
holds, for tiles of one segment (contraction length up to 64, up to 192, longer) and of several.

out = sum_s A_s^T E B_s through contract_L.  A column of the second operand of either phase that holds an Inf or NaN
makes its results NaN.  Otherwise the bound is that of FP64 inner products of length K, K u sum |a||b| (u = 2^-53) per
product, and 8 u for the two roundings per 64 columns and the rounding of the result, or half a subnormal unit."""
import os

import numpy as np
import pytest

from vmps_gb300.blocks import Blocks, MpoSite, Symmetry
from vmps_gb300.pivot import EnvUpdate

pytestmark = pytest.mark.gpu
SYM = Symmetry(("U1",))


def tables(ka, m, kb, n, states):
    s = range(states)
    E = Blocks(1, [0], [0], [0], [ka], [kb], qmid=[0])
    A = Blocks(1, [0] * states, [1] * states, s, [ka] * states, [m] * states)
    B = Blocks(1, [0] * states, [1] * states, s, [kb] * states, [n] * states)
    W = MpoSite(1, [(1,)] * states, [(0,)])
    for i in s:
        W.add(i, i, 0, (0,), (0,), 0, 0, 1.0)
    return E, A, B, W


def run(ctx, E, A, B, W):
    os.environ["VMPS_FP64_ENGINE"] = "slices"
    try:
        e = EnvUpdate(ctx, SYM, "L", E, A, W, B)
        out = e.run(E, A, B)
        e.close()
    finally:
        del os.environ["VMPS_FP64_ENGINE"]
    return out.block(0)


def exact(E, A, B):
    y = E.block(0).astype(np.longdouble)
    ref = size = 0
    for i in range(A.n):
        x, z = A.block(i).astype(np.longdouble), B.block(i).astype(np.longdouble)
        ref, size = ref + x.T @ y @ z, size + np.abs(x).T @ np.abs(y) @ np.abs(z)
    return ref, size


# (ka, m, kb, n, states); n > m: T = A^T E first (tiles of m rows), n < m: U = E B first (tiles of ka rows)
SHAPES = [(40, m, 40, 100, 1) for m in (1, 3, 33, 37, 65, 97)] + [
    (150, 33, 150, 60, 1), (300, 3, 200, 60, 1), (50, 37, 50, 60, 3), (130, 35, 200, 60, 3),
    (33, 100, 40, 20, 1), (37, 100, 150, 20, 3)]


def fill(E, A, B, seed):
    rng = np.random.default_rng(seed)
    for t in (E, A, B):
        t.data[:] = rng.standard_normal(t.data.size)


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_special_columns(gpu_ctx, shape, bad):
    E, A, B, W = tables(*shape)
    for c in range(8):
        fill(E, A, B, c)
        B.block(shape[4] - 1)[1, c] = bad
        nan = np.isnan(run(gpu_ctx, E, A, B, W))
        assert nan[:, c].all() and nan.sum() == shape[1], c
        fill(E, A, B, c)
        E.block(0)[1, c] = bad   # a column of the first product: every result holds it
        assert np.isnan(run(gpu_ctx, E, A, B, W)).all(), c


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("column,rows", [(2.0 ** -900, 1.0), (2.0 ** 600, 1.0), (2.0 ** -800, 2.0 ** -300),
                                         (2.0 ** -1015, 2.0 ** -20)])
def test_far_columns(gpu_ctx, shape, column, rows):
    E, A, B, W = tables(*shape)
    for c in range(8):
        for first in (False, True):
            fill(E, A, B, c)
            A.data *= rows
            if first:
                E.block(0)[:, c] *= column
            else:
                for i in range(B.n):
                    B.block(i)[:, c] *= column
            ref, size = exact(E, A, B)
            got = run(gpu_ctx, E, A, B, W)
            assert np.all(np.abs(got - ref) <= (shape[0] + shape[2] + 8) * 2.0 ** -53 * size + 2.0 ** -1073), (c, first)
