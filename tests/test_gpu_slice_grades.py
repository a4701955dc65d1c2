"""The FP64 slice engine on operands graded along the contracted index.

A rescaling G of a bond (A G times G^-1 B) changes no FP64 inner product of FMAs beyond their bound, K u sum |a||b|
(u = 2^-53), whatever its range; nor does it here: the digits of the second factor are taken relative to the first
one's columns.  Bounds: K u sum |a||b| per product and 8 u for the roundings of the sums, and for whole HxVs the
repository's 1e-12 in the norm."""
import os

import numpy as np
import pytest

from vmps_gb300.pivot import PivotMatrix1, PivotMatrix2

from helpers import pivot1_case, pivot2_case
from test_gpu_slice_columns import exact, fill, run, tables

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("decades", [0, 4, 8, 16, 60, 250])
@pytest.mark.parametrize("shape", [(64, 40, 64, 100, 1), (200, 33, 150, 60, 1), (300, 130, 260, 140, 2),
                                   (70, 100, 150, 20, 3)])
def test_opposite_grades_along_k(gpu_ctx, shape, decades):
    ka, m, kb, n, states = shape
    E, A, B, W = tables(*shape)
    rng = np.random.default_rng(decades)
    for left, right in ((1, 0), (0, 1), (1, 1), (-1, -1)):
        fill(E, A, B, decades)
        g = 10.0 ** rng.uniform(-decades / 2, decades / 2, ka) if left else np.ones(ka)
        h = 10.0 ** rng.uniform(-decades / 2, decades / 2, kb) if right else np.ones(kb)
        if left < 0:   # in order of the index
            g, h = np.sort(g), np.sort(h)[::-1]
        for i in range(states):
            A.block(i)[...] *= g[:, None]
            B.block(i)[...] *= h[:, None]
        E.block(0)[...] /= np.outer(g, h)
        ref, size = exact(E, A, B)
        got = run(gpu_ctx, E, A, B, W)
        assert np.all(np.abs(got - ref) <= (ka + kb + 8) * 2.0 ** -53 * size), (left, right)


@pytest.mark.parametrize("decades", [0, 8, 16, 40])
@pytest.mark.parametrize("sites,kind,L,D,profile", [(1, "heis", 12, 40, "even"), (1, "hubb", 8, 90, "gaussian"),
                                                    (2, "hubb", 10, 200, "even")])
def test_apply_in_any_gauge(gpu_ctx, sites, kind, L, D, profile, decades):
    """H |v> with the bonds rescaled, G L and G^-1 V (and so on the right), by each engine, is H |v> as it stands"""
    case = (pivot1_case if sites == 1 else pivot2_case)(kind, L=L, D=D, site=L // 2 - 1, seed=5, profile=profile)
    model, Lenv, Renv, ops, V = case[0], case[2], case[3], case[4:-1], case[-1]
    rng = np.random.default_rng(7)
    v = rng.standard_normal(V.data.size)

    def apply(engine):
        os.environ["VMPS_FP64_ENGINE"] = engine
        try:
            H = (PivotMatrix1 if sites == 1 else PivotMatrix2)(gpu_ctx, model.sym, Lenv, Renv, *ops, V)
            return H.apply(V.data.copy(), "fp64")
        finally:
            del os.environ["VMPS_FP64_ENGINE"]

    V.data[:] = v
    want = apply("fma")
    # the ket index of an L block is its columns, that of an R block its rows
    g = {q: 10.0 ** rng.uniform(-decades / 2, decades / 2, V.rows[i]) for i, q in enumerate(map(tuple, V.qin))}
    h = {q: 10.0 ** rng.uniform(-decades / 2, decades / 2, V.cols[i]) for i, q in enumerate(map(tuple, V.qout))}
    for i in range(V.n):
        V.block(i)[...] /= np.outer(g[tuple(V.qin[i])], h[tuple(V.qout[i])])
    for i, q in enumerate(map(tuple, Lenv.qout)):
        if q in g:
            Lenv.block(i)[...] *= g[q][None, :]
    for i, q in enumerate(map(tuple, Renv.qin)):
        if q in h:
            Renv.block(i)[...] *= h[q][:, None]
    for engine in ("fma", "slices"):
        assert np.linalg.norm(apply(engine) - want) <= 2e-12 * np.linalg.norm(want), engine


@pytest.mark.parametrize("zero_column", [False, True])
@pytest.mark.parametrize("bits", [3, 4, 12, 53])   # alike columns (up to 3 bits), unlike ones
@pytest.mark.parametrize("sites,kind,L,D,profile", [(1, "hubb", 8, 90, "gaussian"), (2, "heis", 12, 60, "even")])
def test_blocks_of_one_bond_with_unlike_columns(gpu_ctx, sites, kind, L, D, profile, bits, zero_column):
    """every second L block rescaled along its columns against V, the others far smaller and as they were: no block's
    products lose what another's columns would have them rounded to"""
    case = (pivot1_case if sites == 1 else pivot2_case)(kind, L=L, D=D, site=L // 2 - 1, seed=5, profile=profile)
    model, Lenv, Renv, ops, V = case[0], case[2], case[3], case[4:-1], case[-1]
    rng = np.random.default_rng(11)
    V.data[:] = rng.standard_normal(V.data.size)
    Lenv.data[:] = rng.standard_normal(Lenv.data.size)
    Renv.data[:] = rng.standard_normal(Renv.data.size)
    g = {q: 2.0 ** rng.integers(0, bits + 1, V.rows[i]) for i, q in enumerate(map(tuple, V.qin))}
    for i in range(V.n):
        V.block(i)[...] /= g[tuple(V.qin[i])][:, None]
        if zero_column:
            V.block(i)[0, :] = 1e16
    for i, q in enumerate(map(tuple, Lenv.qout)):
        if i % 2:
            Lenv.block(i)[...] *= 1e-40
        elif q in g:
            Lenv.block(i)[...] *= g[q][None, :]
            if zero_column:
                Lenv.block(i)[:, 0] = 0.0

    def apply(engine):
        os.environ["VMPS_FP64_ENGINE"] = engine
        try:
            H = (PivotMatrix1 if sites == 1 else PivotMatrix2)(gpu_ctx, model.sym, Lenv, Renv, *ops, V)
            return H.apply(V.data.copy(), "fp64")
        finally:
            del os.environ["VMPS_FP64_ENGINE"]

    want = apply("fma")
    assert np.linalg.norm(apply("slices") - want) <= 2e-12 * np.linalg.norm(want)
