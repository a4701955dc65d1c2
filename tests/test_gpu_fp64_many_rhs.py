"""More FP64 vectors in one call than one launch holds (65535): each vector's result is the bits of its own HxV."""
import numpy as np
import pytest

from vmps_gb300.pivot import PivotMatrix1

from helpers import pivot1_case

pytestmark = pytest.mark.gpu


def test_more_vectors_than_a_launch_holds(gpu_ctx):
    model, _, Lenv, Renv, W, V = pivot1_case("heis", L=4, D=2, site=1, seed=8)
    H = PivotMatrix1(gpu_ctx, model.sym, Lenv, Renv, W, V)
    X = np.random.default_rng(1).standard_normal((65537, V.data.size))
    many = H.apply_multi(X, "fp64")
    for k in (0, 1, 65534, 65535, 65536):
        assert np.array_equal(many[k], H.apply(X[k], "fp64")), k
