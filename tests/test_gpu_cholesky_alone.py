"""The tile-flag Cholesky (csrc/potrf_flow.cu) with one CTA a matrix and several tile rows:
more matrices of order above 128 than half the SMs (the factors of X and Y in one launch,
or the trials of a line search), and more than there are SMs.

Margins: pivots are accurate to about k·eps·κ.  The whole factor: dY = sym(X⁻¹(R − dX·Y)),
R = −XY, is within 16·k·eps·κ(X)·‖X⁻¹‖(‖X‖ + ‖dX‖)‖Y‖ (the products and the two
triangular factors are each backward stable)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


def _backend(ks, seed):
    from sdpx_b200.cuda_backend import CudaBackend
    from sdpx_b200.problem import ingest
    rng = np.random.default_rng(seed)

    def spd(k):
        q, _ = np.linalg.qr(rng.standard_normal((k, k)))
        x = (q * np.logspace(-1, 1, k)) @ q.T
        return 0.5 * (x + x.T)
    A = [rng.standard_normal((2, k, k)) for k in ks]
    A = [a + a.transpose(0, 2, 1) for a in A]
    be = CudaBackend(ingest(rng.standard_normal(2), A, [np.eye(k) for k in ks]))
    return be, [spd(k) for k in ks], [spd(k) for k in ks]


# 76 matrices of three tile rows, of four; orders at the edges of tiles side by side (82);
# 160 matrices: some CTAs take two
@pytest.mark.parametrize("ks", [[130] * 38, [200] * 38, [129, 192, 193, 256, 320, 40] * 7, [129] * 80])
def test_factors_and_directions(ks):
    be, X, Y = _backend(ks, len(ks))
    with be:
        be.set_iterate(np.zeros(2), X, Y)
        assert be.compute_residuals([0.0] * len(ks), True, True)[2]
        for got, M in zip(be.block_margins(), (X, Y)):
            margin = min(np.diag(c).min() / np.diag(c).max() for c in map(np.linalg.cholesky, M))
            assert abs(got - margin) <= 4 * max(ks) * EPS * 100 * margin
        be.schur_build()
        be.factorize()
        be.predictor_rhs()
        be.solve_direction()
        be.direction_blocks()
        _, dX, dY = be.get_direction()
    n = lambda a: np.linalg.norm(a, 2)  # noqa: E731
    for k, Xb, Yb, dXb, dYb in zip(ks, X, Y, dX, dY):
        Z = np.linalg.solve(Xb, -Xb @ Yb - dXb @ Yb)
        bound = 16 * k * EPS * np.linalg.cond(Xb) * n(np.linalg.inv(Xb)) * n(Yb) * (n(Xb) + n(dXb))
        assert n(dYb - (Z + Z.T) / 2) <= bound


@pytest.mark.parametrize("bad", [0, 63, 64, 127, 128, 150, 199])
def test_indefinite_block_is_reported(bad):
    ks = [200] * 38
    be, X, _ = _backend(ks, 1)
    with be:
        Y = [x.copy() for x in X]
        L = np.linalg.cholesky(X[17])
        Y[17][bad, bad] -= 1.5 * L[bad, bad] ** 2  # the leading minors before it stay positive
        be.set_iterate(np.zeros(2), X, Y)
        assert not be.compute_residuals([0.0] * len(ks), True, True)[2]
        be.set_iterate(np.zeros(2), X, X)  # nothing of the failure stays behind
        assert be.compute_residuals([0.0] * len(ks), True, True)[2]


# eight candidates of five blocks and two sides: 80 trials of three to five tile rows
def test_line_search_trials():
    ks = [130, 200, 193, 257, 300]
    be, X, Y = _backend(ks, 2)
    with be:
        be.set_iterate(np.zeros(2), X, Y)
        assert be.compute_residuals([0.0] * len(ks), True, True)[2]
        be.schur_build()
        be.factorize()
        be.predictor_rhs()
        be.solve_direction()
        be.direction_blocks()
        _, dX, dY = be.get_direction()
        got = be.line_search("backtrack", 0.9, 0.9, 0.9, 1e-10, 0.0)
    for t, M, dM in zip(got, (X, Y), (dX, dY)):
        top = 1.0
        for a, d in zip(M, dM):
            W = np.linalg.inv(np.linalg.cholesky(a))
            low = np.linalg.eigvalsh(W @ d @ W.T)[0]
            top = min(top, -1.0 / low) if low < 0 else top
        want = 1.0
        while want >= top:
            want *= 0.9
        assert t == pytest.approx(want, rel=1e-14)
