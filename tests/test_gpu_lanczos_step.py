"""The device Lanczos step where its work changes shape: basis rows per warp (eight rows a block; one, two, four
and eight a warp; more than 64), a last chunk that is not full, one and two elements per thread (up to and above
311,296).

FP64 against a Lanczos run on the host with two orthogonalisation passes on the same operator, and split precision
against FP64 after refinement: the repository's bound for energies, 1e-10 relative."""
import numpy as np
import pytest

from vmps_gb300.pivot import PivotMatrix1, PivotMatrix2

from helpers import pivot1_case, pivot2_case

pytestmark = pytest.mark.gpu
TOL = 1e-10


def host_ritz(H, v, m):
    K, alpha, beta = [v / np.linalg.norm(v)], [], []
    for j in range(m):
        w = H.apply(K[j], "fp64")
        alpha.append(float(K[j] @ w))
        for _ in range(2):
            B = np.array(K)
            w = w - B.T @ (B @ w)
        beta.append(float(np.linalg.norm(w)))
        K.append(w / beta[-1])
    return float(np.linalg.eigvalsh(np.diag(alpha) + np.diag(beta[:-1], 1) + np.diag(beta[:-1], -1))[0])


@pytest.mark.parametrize("kind,L,D", [("heis", 16, 120), ("hubb", 10, 200)])
def test_ritz_values_at_row_counts(gpu_ctx, kind, L, D):
    model, _, Lenv, Renv, W, V = pivot1_case(kind, L=L, D=D, site=L // 2 - 1, seed=4)
    H = PivotMatrix1(gpu_ctx, model.sym, Lenv, Renv, W, V)
    v = np.random.default_rng(3).standard_normal(V.data.size)
    for m in (1, 2, 8, 9, 16, 17, 32, 33, 64, 65, 80):
        e = H.lanczos(v, "fp64", max_iter=m, tol_eigval=0, tol_state=0)[0]
        want = host_ritz(H, v, m)
        assert abs(e - want) <= TOL * max(1.0, abs(want)), m


def test_long_vectors(gpu_ctx):
    model, _, Lenv, Renv, W1, W2, V = pivot2_case("hubb", L=14, D=860, site=6, seed=4, profile="gaussian")
    assert V.data.size > 311296 and V.data.size % 512
    H = PivotMatrix2(gpu_ctx, model.sym, Lenv, Renv, W1, W2, V)
    v = V.data
    for m in (3, 18):
        want = host_ritz(H, v, m)
        assert abs(H.lanczos(v, "fp64", max_iter=m, tol_eigval=0, tol_state=0)[0] - want) <= TOL * max(1.0, abs(want)), m
    kw = dict(max_iter=300, tol_eigval=1e-12, tol_state=1e-8)
    e64 = H.lanczos(v, "fp64", **kw)[0]
    es = H.lanczos(v, "bf16x3", refine_iters=12, **kw)[0]
    assert abs(es - e64) <= TOL * max(1.0, abs(e64))
