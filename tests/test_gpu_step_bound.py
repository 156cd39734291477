"""The eigenvalue step bounds (csrc/step_bound.cu) at the edges of its cluster sizes and
row shares, against NumPy's −1/λ_min, and where they must not be used."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


def _backend(ks, seed, scale=1.0):
    from sdpx_b200.cuda_backend import CudaBackend
    from sdpx_b200.problem import ingest
    rng = np.random.default_rng(seed)
    A = [scale * rng.standard_normal((3, k, k)) for k in ks]
    A = [a + a.transpose(0, 2, 1) for a in A]

    def spd(k):
        q, _ = np.linalg.qr(rng.standard_normal((k, k)))
        x = (q * np.logspace(-1, 1, k)) @ q.T
        return 0.5 * (x + x.T)
    X, Y = [spd(k) for k in ks], [spd(k) for k in ks]
    be = CudaBackend(ingest(rng.standard_normal(3), A, [np.eye(k) for k in ks]))
    return be, X, Y


def _direction(be, X, Y):
    be.set_iterate(np.zeros(3), X, Y)
    assert be.compute_residuals([0.0] * len(X), True, True)[2]
    be.schur_build()
    assert be.factorize()["ok"]
    be.predictor_rhs()
    be.solve_direction()
    be.direction_blocks()
    return be.get_direction()


def _exact(M, dM):
    t = 1.0
    for a, da in zip(M, dM):
        W = np.linalg.inv(np.linalg.cholesky(a))
        low = np.linalg.eigvalsh(W @ da @ W.T)[0]
        t = min(t, -1.0 / low) if low < -1.0 else t
    return t


# 3: the smallest; 64/65, 128/129, 256/257: one to eight CTAs; 439/447: the largest orders that
# fit, and 460 beyond them (bisection); mixed orders in one launch; 2 and 1 beside them
@pytest.mark.parametrize("ks", [[3], [4, 33], [64], [65], [128, 5], [129], [257, 40], [439], [460],
                                [3, 2, 70, 1]])
def test_affine_bounds_match_the_eigenvalues(ks):
    be, X, Y = _backend(ks, sum(ks))
    with be:
        _, dX, dY = _direction(be, X, Y)
        p = be.affine_diagnostics(True)
        # L⁻¹·dM·L⁻ᵀ is formed with errors of a few k·eps·κ(M), κ = 100, relative to
        # its norm, which is within 1e3 of |λ_min| for these directions
        for got, M, dM in ((p["tX"], X, dX), (p["tY"], Y, dY)):
            want = _exact(M, dM)
            assert abs(got - want) <= 4 * max(ks) * EPS * 1e2 * 1e3 * want
        # the bisection of the line search agrees to the same bound
        for got, t in zip(be.line_search("fraction_to_boundary", 1.0, 1.0, 0.9, 1e-10, 0.0),
                          (p["tX"], p["tY"])):
            assert abs(got - t) <= 8 * max(ks) * EPS * 1e5 * t


def test_full_step_inside_gives_one():
    be, X, Y = _backend([40, 7], 3)
    with be:
        _direction(be, X, [1e-3 * y for y in Y])
        dX = be.get_direction()[1]
        p = be.affine_diagnostics(True)
        assert (p["tX"] == 1.0) == (_exact(X, dX) == 1.0)


# After the iterate moved, the factors at hand belong to the old one: the bounds then come
# from the trial factorizations of the new iterate, as they always did.
def test_bounds_follow_a_changed_iterate():
    be, X, Y = _backend([30, 9], 5)
    with be:
        _, dX, dY = _direction(be, X, Y)
        p0 = be.affine_diagnostics(True)
        be.set_iterate(np.zeros(3), [4.0 * x for x in X], [4.0 * y for y in Y])
        p1 = be.affine_diagnostics(True)
        for key, M, dM in (("tX", X, dX), ("tY", Y, dY)):
            assert p1[key] == pytest.approx(_exact([4.0 * a for a in M], dM), rel=1e-10)
            assert p0[key] == pytest.approx(_exact(M, dM), rel=1e-10)


@pytest.mark.parametrize("ks", [[31], [32], [33, 3], [63], [100], [127, 65], [224, 3], [225], [320, 17, 4], [447], [448, 15]])
def test_affine_bounds_at_the_edges_of_the_clusters(ks):
    test_affine_bounds_match_the_eigenvalues(ks)
