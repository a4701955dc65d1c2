"""The FP64 slice engine (VMPS_FP64_ENGINE=slices) at the edges of its tiles (128 x 32, 16 columns for
narrow ones), K steps (16, 32), flushes (64), integer sums (192) and shared-memory buffer (256), through
contract_L of one block, out = A^T E B, against the products in extended precision.

Tolerance: an FP64 inner product of length K is off by at most K u sum |a||b| (u = 2^-53).  The slices' error is
bounded by 2^-60 K max|a| max|b| and two roundings per 64 columns of K, which for entries of one
magnitude per row is below that bound plus 8 u."""
import os

import numpy as np
import pytest

from vmps_gb300.blocks import Blocks, MpoSite, Symmetry
from vmps_gb300.pivot import Context, EnvUpdate, PivotMatrix1, PivotMatrix2

from helpers import pivot1_case, pivot2_case

SYM = Symmetry(("U1",))


def tables(ka, m, kb, n):
    E = Blocks(1, [0], [0], [0], [ka], [kb], qmid=[0])
    A = Blocks(1, [0], [1], [0], [ka], [m])
    B = Blocks(1, [0], [1], [0], [kb], [n])
    W = MpoSite(1, [(1,)], [(0,)])
    W.add(0, 0, 0, (0,), (0,), 0, 0, 1.0)
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
    x, y, z = (t.block(0).astype(np.longdouble) for t in (A, E, B))
    return x.T @ y @ z, np.abs(x).T @ np.abs(y) @ np.abs(z)


SHAPES = [(1, 1, 1, 1), (16, 127, 17, 16), (15, 128, 33, 17), (33, 129, 16, 32), (63, 5, 64, 33), (65, 130, 128, 31),
          (129, 16, 192, 64), (193, 257, 200, 65), (256, 33, 257, 3), (300, 2, 520, 40)]


@pytest.mark.gpu
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("graded", [False, True])
def test_slices_at_tile_edges(gpu_ctx, shape, graded):
    E, A, B, W = tables(*shape)
    rng = np.random.default_rng(sum(shape))
    for t in (E, A, B):
        t.data[:] = rng.standard_normal(t.data.size)
    if graded:   # rows and columns of the result over sixty decades
        A.block(0)[...] *= 10.0 ** rng.integers(-30, 30, A.cols[0])[None, :]
        B.block(0)[...] *= 10.0 ** rng.integers(-30, 30, B.cols[0])[None, :]
    ref, size = exact(E, A, B)
    got = run(gpu_ctx, E, A, B, W)
    assert np.all(np.abs(got - ref) <= (shape[0] + shape[2] + 8) * 2.0 ** -53 * size)


@pytest.mark.gpu
def test_slices_are_exact_on_integers_and_keep_special_values(gpu_ctx):
    E, A, B, W = tables(70, 40, 90, 35)
    rng = np.random.default_rng(3)
    for t in (E, A, B):
        t.data[:] = rng.integers(-1000, 1000, t.data.size)
    A.block(0)[:, 7] = 0.0
    ref, size = exact(E, A, B)
    assert np.array_equal(run(gpu_ctx, E, A, B, W), ref.astype(float))   # below 2^53, a zero row among them
    for scale in (2.0 ** -530, 2.0 ** 500):   # subnormal and overflowing results
        for t, f in ((A, scale), (E, 1.0), (B, scale)):
            t.data *= f
        with np.errstate(over="ignore", invalid="ignore"):
            want = (ref * np.longdouble(scale) ** 2).astype(float)
            ok = np.isfinite((size * np.longdouble(scale) ** 2).astype(float))   # no partial sum can overflow
        got = run(gpu_ctx, E, A, B, W)
        assert np.all(np.isinf(got[np.isinf(want)])) and np.all(np.abs(got[ok] - want[ok]) <= 2.0 ** -1073)
        for t, f in ((A, scale), (B, scale)):
            t.data /= f
    B.block(0)[3, 5] = np.inf
    A.block(0)[2, 1] = np.nan
    got = run(gpu_ctx, E, A, B, W)
    bad = np.zeros_like(got, dtype=bool)
    bad[1, :] = bad[:, 5] = True
    assert np.array_equal(np.isnan(got), bad) and np.array_equal(got[~bad], ref.astype(float)[~bad])


@pytest.mark.gpu
@pytest.mark.parametrize("sites,kind,L,D,profile", [(1, "heis", 12, 40, "even"), (1, "hubb", 8, 90, "gaussian"),
                                                    (2, "heis", 16, 250, "gaussian"), (2, "hubb", 10, 200, "even")])
def test_both_engines_apply_the_same_operator(gpu_ctx, sites, kind, L, D, profile):
    """sums over many segments; the repository's bound for FP64 (1e-12 in the norm) holds for each engine"""
    case = (pivot1_case if sites == 1 else pivot2_case)(kind, L=L, D=D, site=L // 2 - 1, seed=5, profile=profile)
    model, L_, R_, ops, V = case[0], case[2], case[3], case[4:-1], case[-1]
    out = {}
    for engine in ("fma", "slices"):
        os.environ["VMPS_FP64_ENGINE"] = engine
        try:
            H = (PivotMatrix1 if sites == 1 else PivotMatrix2)(gpu_ctx, model.sym, L_, R_, *ops, V)
            v = np.random.default_rng(6).standard_normal(V.data.size)
            out[engine] = H.apply(v, "fp64")
        finally:
            del os.environ["VMPS_FP64_ENGINE"]
    d = np.linalg.norm(out["slices"] - out["fma"])
    assert 0 < d <= 2e-12 * np.linalg.norm(out["fma"])


@pytest.mark.parametrize("shape", SHAPES)
def test_slice_plans_are_valid(shape):
    """the invariants of tiles, steps, flush groups and boxes are checked when a plan is made"""
    ctx = Context(-1)
    os.environ["VMPS_FP64_ENGINE"] = "slices"
    try:
        E, A, B, W = tables(*shape)
        st = EnvUpdate(ctx, SYM, "L", E, A, W, B).stats("fp64")
    finally:
        del os.environ["VMPS_FP64_ENGINE"]
    assert st["n_tiles_phase1"] > 0 and st["n_tiles_phase2"] == -(-shape[1] // 128) * -(-shape[3] // 32)
