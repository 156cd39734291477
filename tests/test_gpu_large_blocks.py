"""Right-hand sides and directions with dense blocks whose k×k products fill the GPU on
their own (orders above 768 on 148 SMs): such a product leaves the grouped launch, and with
it every product of its group.

r = −(d + 𝒜ᵀvec(X⁻¹(P·Y − R))) with R = −XY (d, P from the data), and
dY = sym(X⁻¹(R − dX·Y)) from the dX the solver returns.  The products and the triangular
factors of X⁻¹ are each backward stable: every entry of X⁻¹T is within
16·k·eps·κ(X)·‖X⁻¹‖‖T‖ of the exact one, T bounded by the norms of its terms."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


# alone; beside small blocks (which then leave the grouped launch too); two of them; just
# below the limit
@pytest.mark.parametrize("ks", [[800], [800, 40], [30, 769, 5], [770, 800], [768, 65]])
def test_rhs_and_direction(ks):
    from sdpx_b200 import generators as G
    from sdpx_b200.cuda_backend import CudaBackend
    m = 4
    rng = np.random.default_rng(sum(ks))
    prob = G.sdpa_dense(m=m, blocks=ks, seed=3)

    def spd(k):
        a = rng.standard_normal((k, k))
        return a @ a.T / k + np.eye(k)
    X, Y, x = [spd(k) for k in ks], [spd(k) for k in ks], rng.standard_normal(m)
    with CudaBackend(prob) as be:
        be.set_iterate(x, X, Y)
        be.compute_residuals(np.zeros(len(ks)), True, True)
        be.schur_build()
        be.factorize()
        be.predictor_rhs()
        r = be.get_rhs()
        be.solve_direction()
        be.direction_blocks()
        dx, dX, dY = be.get_direction()

    n = lambda a: np.linalg.norm(a, 2)  # noqa: E731
    want, slack = np.zeros(m), np.zeros(m)
    for l, k in enumerate(ks):
        A = prob.Av[l].reshape(m, k, k)
        bound = 16 * k * EPS * np.linalg.cond(X[l]) * n(np.linalg.inv(X[l]))
        P = np.tensordot(x, A, 1) - X[l] - prob.C[l]
        R = -X[l] @ Y[l]
        V = np.linalg.solve(X[l], P @ Y[l] - R)
        want += A.reshape(m, -1) @ (Y[l] - V).reshape(-1)
        size = n(Y[l]) * (n(P) + n(X[l]))
        slack += np.linalg.norm(A.reshape(m, -1), axis=1) * (bound * size * np.sqrt(k) + k * EPS * np.linalg.norm(Y[l] - V))
        dZ = np.linalg.solve(X[l], R - dX[l] @ Y[l])
        assert n(dY[l] - (dZ + dZ.T) / 2) <= bound * n(Y[l]) * (n(X[l]) + n(dX[l]))
    assert (np.abs(r - (want - prob.c)) <= slack + 4 * EPS * np.abs(prob.c)).all()
