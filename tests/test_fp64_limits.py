"""FP64 plans beyond the slice engine's limits run by FMAs: no pivot is refused for them."""
import numpy as np
import pytest

from vmps_gb300.blocks import Blocks, MpoSite, Symmetry
from vmps_gb300.pivot import Context, EnvUpdate, PivotMatrix1

# one contraction length per padded length of the panels
LENGTHS = [32 * i for i in range(1, 9)] + [256 + 128 * i for i in range(1, 7)] + [1024 + 512 * i for i in range(1, 7)]


def tables(lengths):
    """sectors of the given sizes among small ones, each coupled to itself and its neighbours"""
    sizes = [s for n in lengths for s in (8, n, 24, 48, n, 100)]
    pairs = [(i, j) for i in range(len(sizes)) for j in range(max(i - 1, 0), min(i + 2, len(sizes)))]
    i, j = np.array(pairs).T
    d = np.array(sizes)
    L = Blocks(1, i, j, [0] * len(pairs), d[i], d[j], qmid=i - j)
    R = Blocks(1, i, j, [0] * len(pairs), d[i], d[j], qmid=j - i)
    V = Blocks(1, range(len(sizes)), range(len(sizes)), [0] * len(sizes), sizes, sizes)
    W = MpoSite(1, [(0,)], [(0,)])
    for m in (-1, 0, 1):
        W.add(0, 0, 0, (m,), (m,), 0, 0, 1.0)
    return L, R, V, W


def stats(lengths, engine, monkeypatch):
    monkeypatch.setenv("VMPS_FP64_ENGINE", engine)
    L, R, V, W = tables(lengths)
    sym, ctx = Symmetry(("U1",)), Context(-1)
    H = PivotMatrix1(ctx, sym, L, R, W, V)
    return H.stats("fp64")["n_tiles_phase1"], EnvUpdate(ctx, sym, "L", L, V, W, V).stats("fp64")["n_tiles_phase1"]


@pytest.mark.parametrize("lengths,fits", [(LENGTHS[:8], True), (LENGTHS, False)])
def test_more_descriptors_than_a_phase_holds(lengths, fits, monkeypatch):
    """4 box heights by 20 padded lengths of the first operand are more than its 64 descriptors"""
    fma, slices = (stats(lengths, engine, monkeypatch) for engine in ("fma", "slices"))
    assert (slices[0] < fma[0] and slices[1] < fma[1]) if fits else slices == fma
