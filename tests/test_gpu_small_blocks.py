"""Block products of small dense blocks in one launch, at the edges of their 8-row strips
and of the 64-tile (and just above, where grouped products take over).

dY = sym(X⁻¹(R − dX·Y)) with R = −XY of the affine direction, from the dX the solver
returns; the products and the two triangular factors of X⁻¹ are each backward stable, so
|ΔdY| ≤ 16·k·eps·κ(X)·‖X⁻¹‖(‖X‖‖Y‖ + ‖dX‖‖Y‖)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


@pytest.mark.parametrize("ks", [[2], [3, 2], [7, 8, 9], [16, 17], [31, 64], [63], [65, 5], [5] * 20])
def test_direction_blocks(ks):
    from sdpx_b200 import generators as G
    from sdpx_b200.cuda_backend import CudaBackend
    rng = np.random.default_rng(sum(ks))
    prob = G.sdpa_dense(m=4, blocks=ks, seed=3)

    def spd(k):
        a = rng.standard_normal((k, k))
        return a @ a.T / k + np.eye(k)
    X, Y, x = [spd(k) for k in ks], [spd(k) for k in ks], rng.standard_normal(4)
    with CudaBackend(prob) as be:
        be.set_iterate(x, X, Y)
        be.compute_residuals(np.zeros(len(ks)), True, True)
        be.schur_build()
        be.factorize()
        be.predictor_rhs()
        be.solve_direction()
        be.direction_blocks()
        dx, dX, dY = be.get_direction()
    for k, Xb, Yb, dXb, dYb in zip(ks, X, Y, dX, dY):
        Z = np.linalg.solve(Xb, -Xb @ Yb - dXb @ Yb)
        want = (Z + Z.T) / 2
        n = lambda a: np.linalg.norm(a, 2)  # noqa: E731
        bound = 16 * k * EPS * np.linalg.cond(Xb) * n(np.linalg.inv(Xb)) * n(Yb) * (n(Xb) + n(dXb))
        assert n(dYb - want) <= bound
        assert np.array_equal(dYb, dYb.T)
