"""Trials of large blocks beside many small ones: the small matrices are factored in a launch of
their own where that frees CTAs for the large ones, and every result finds its place.

The bounds of a bisection and the steps of a backtracking search against the eigenvalues of
L⁻¹·dM·L⁻ᵀ; κ(M) = 100, so the bounds are within a few k·eps·κ·1e3 of them, and no candidate
step lies that close."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


# small blocks first, last and between; two CTAs for 460 in one launch; orders at the limit of
# one tile
@pytest.mark.parametrize("ks", [[460, 10], [10, 460], [5, 300, 5, 8, 5], [200] + [8] * 12, [64, 330, 65, 3], [70, 64]])
def test_searches(ks):
    from sdpx_b200.cuda_backend import CudaBackend
    from sdpx_b200.problem import ingest
    rng = np.random.default_rng(sum(ks))

    def spd(k):
        q, _ = np.linalg.qr(rng.standard_normal((k, k)))
        x = (q * np.logspace(-1, 1, k)) @ q.T
        return 0.5 * (x + x.T)
    A = [rng.standard_normal((3, k, k)) for k in ks]
    A = [a + a.transpose(0, 2, 1) for a in A]
    X, Y = [spd(k) for k in ks], [spd(k) for k in ks]
    with CudaBackend(ingest(rng.standard_normal(3), A, [np.eye(k) for k in ks])) as be:
        be.set_iterate(np.zeros(3), X, Y)
        assert be.compute_residuals([0.0] * len(ks), True, True)[2]
        be.schur_build()
        assert be.factorize()["ok"]
        be.predictor_rhs()
        be.solve_direction()
        be.direction_blocks()
        _, dX, dY = be.get_direction()
        bounds = be.line_search("fraction_to_boundary", 1.0, 1.0, 0.9, 1e-10, 0.0)
        steps = be.line_search("backtrack", 1.0, 1.0, 0.9, 1e-10, 0.0)
    for bound, step, M, dM in zip(bounds, steps, (X, Y), (dX, dY)):
        low = min(np.linalg.eigvalsh(W @ d @ W.T)[0]
                  for W, d in ((np.linalg.inv(np.linalg.cholesky(a)), d) for a, d in zip(M, dM)))
        top = -1.0 / low if low < -1.0 else 1.0
        assert abs(bound - top) <= 8 * max(ks) * EPS * 1e5 * top
        want = 1.0
        while want > top or (want == 1.0 and low <= -1.0):
            want *= 0.9
        assert step == pytest.approx(want, rel=1e-14)
