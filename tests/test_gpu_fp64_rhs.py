"""FP64 HxVs of several vectors in one launch: every vector's result is the bits of the HxV of that vector alone, for
one vector, a few, and a projector on the pivot (applied vector by vector)."""
import numpy as np
import pytest

from vmps_gb300.pivot import PivotMatrix1, PivotMatrix2

from helpers import pivot1_case, pivot2_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nrhs", [1, 2, 3, 17])
@pytest.mark.parametrize("projector", [False, True])
@pytest.mark.parametrize("sites", [1, 2])
def test_vectors_of_a_launch_are_independent(gpu_ctx, nrhs, projector, sites):
    case = pivot1_case("heis", L=10, D=24, site=4, seed=8) if sites == 1 else pivot2_case("hubb", L=8, D=40, site=3, seed=8)
    model, Lenv, Renv, ops, V = case[0], case[2], case[3], case[4:-1], case[-1]
    H = (PivotMatrix1 if sites == 1 else PivotMatrix2)(gpu_ctx, model.sym, Lenv, Renv, *ops, V)
    rng = np.random.default_rng(nrhs)
    n = V.data.size
    if projector:
        x = rng.standard_normal(n)
        H.set_projector(x[None, :] / np.linalg.norm(x), 3.0)
    X = rng.standard_normal((nrhs, n))
    one = np.array([H.apply(x, "fp64") for x in X])
    many = H.apply_multi(X, "fp64")
    assert np.array_equal(one, many)
    mu = H.chebyshev_moments(X, 8, 40.0, 0.0, "fp64")[0]
    each = np.array([H.chebyshev_moments(x[None, :], 8, 40.0, 0.0, "fp64")[0][0] for x in X])
    assert np.array_equal(mu, each)
