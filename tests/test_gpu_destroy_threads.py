"""Objects of a context released on another thread, as a garbage collector may, while the context's stream is captured
(Lanczos, Chebyshev, the timed HxV graph): every result keeps its bits, as if they had been released before."""
import threading

import numpy as np
import pytest

from vmps_gb300.pivot import PivotMatrix1

from helpers import pivot1_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp64", "bf16x3"])
def test_release_during_captures(gpu_ctx, prec):
    model, _, Lenv, Renv, W, V = pivot1_case("heis", L=8, D=16, site=3, seed=4)

    def pivot():
        return PivotMatrix1(gpu_ctx, model.sym, Lenv, Renv, W, V)

    H = pivot()
    X = np.random.default_rng(2).standard_normal((2, V.data.size))
    want = H.apply(X[0], prec)
    moments = H.chebyshev_moments(X, 6, 40.0, 0.0, prec)[0]
    ground = H.lanczos(X[0].copy(), precision=prec, max_iter=4, refine_iters=0)[0]
    others = [pivot() for _ in range(400)]
    for o in others:
        o.apply(X[1], prec)

    def release():
        while others:
            others.pop().close()

    t = threading.Thread(target=release)
    t.start()
    rounds = 0
    while t.is_alive() or rounds < 20:
        assert np.array_equal(H.chebyshev_moments(X, 6, 40.0, 0.0, prec)[0], moments)
        assert H.lanczos(X[0].copy(), precision=prec, max_iter=4, refine_iters=0)[0] == ground
        assert np.array_equal(H.apply(X[0], prec), want)
        rounds += 1
    t.join()
    assert not others
