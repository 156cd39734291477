"""The eigenvalue step bounds (csrc/step_bound.cu) of lists that hold a matrix with fewer
rows than its cluster has warps (such a cluster runs its reflections in lockstep), for
every cluster shape (largest order up to 32, 64, 128, 224, 448), and where the whole step
stays inside.

G = L⁻¹·dM·L⁻ᵀ is formed with errors of a few k·eps·κ(M), κ = 100, relative to its norm,
which is within 1e3 of |λ_min| for these directions."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


def _direction(ks, seed, scale_Y=1.0):
    from sdpx_b200.cuda_backend import CudaBackend
    from sdpx_b200.problem import ingest
    rng = np.random.default_rng(seed)

    def spd(k):
        q, _ = np.linalg.qr(rng.standard_normal((k, k)))
        x = (q * np.logspace(-1, 1, k)) @ q.T
        return 0.5 * (x + x.T)
    A = [rng.standard_normal((3, k, k)) for k in ks]
    A = [a + a.transpose(0, 2, 1) for a in A]
    X, Y = [spd(k) for k in ks], [scale_Y * spd(k) for k in ks]
    be = CudaBackend(ingest(rng.standard_normal(3), A, [np.eye(k) for k in ks]))
    be.set_iterate(np.zeros(3), X, Y)
    assert be.compute_residuals([0.0] * len(ks), True, True)[2]
    be.schur_build()
    assert be.factorize()["ok"]
    be.predictor_rhs()
    be.solve_direction()
    be.direction_blocks()
    return be, X, Y


def _exact(M, dM):
    t = 1.0
    for a, da in zip(M, dM):
        W = np.linalg.inv(np.linalg.cholesky(a))
        low = np.linalg.eigvalsh(W @ da @ W.T)[0]
        t = min(t, -1.0 / low) if low < -1.0 else t
    return t


# (32: one CTA, no cluster) 4 CTAs of 4 warps beside orders below 16; 8 of 4 below 32; 16
# of 4 below 64; 16 CTAs below 16; the smallest order beside each
@pytest.mark.parametrize("ks", [[32, 3], [64, 15, 3], [61, 16], [128, 31, 7], [100, 3], [200, 40], [224, 63, 3],
                                [300, 15], [448, 3, 16]])
def test_small_orders_beside_large_ones(ks):
    be, X, Y = _direction(ks, sum(ks))
    with be:
        _, dX, dY = be.get_direction()
        p = be.affine_diagnostics(True)
        for got, M, dM in ((p["tX"], X, dX), (p["tY"], Y, dY)):
            want = _exact(M, dM)
            assert abs(got - want) <= 4 * max(ks) * EPS * 1e2 * 1e3 * want
        for _ in range(3):
            q = be.affine_diagnostics(True)
            assert (q["tX"], q["tY"]) == (p["tX"], p["tY"])


# 8 blocks: the inverse factors of both sides in one list; 9 and more: those of Y are made
# when the bounds are asked for, once for an iterate
@pytest.mark.parametrize("ks", [[20, 70] * 4, [20, 70, 3] * 3, [9] * 40])
def test_many_blocks(ks):
    be, X, Y = _direction(ks, len(ks))
    with be:
        _, dX, dY = be.get_direction()
        for scale in (1.0, 3.0):
            p = [be.affine_diagnostics(True) for _ in range(2)]
            for key, M, dM in (("tX", X, dX), ("tY", Y, dY)):
                want = _exact([scale * a for a in M], dM)
                assert abs(p[0][key] - want) <= 4 * max(ks) * EPS * 1e2 * 1e3 * want
                assert p[1][key] == p[0][key]
            be.set_iterate(np.zeros(3), [3.0 * x for x in X], [3.0 * y for y in Y])
            assert be.compute_residuals([0.0] * len(ks), True, True)[2]


# The clusters of every order limit have a place on a whole GPU (where one has not, larger
# orders take the bisection).
def test_every_cluster_shape_runs():
    from sdpx_b200.cuda_backend import load_library
    import torch
    torch.cuda.init()
    assert load_library()["_ZN4sdpx20step_bound_max_orderEv"]() == 448


# A centring direction from a nearly central, feasible iterate: X + dX and Y + dY are inside.
@pytest.mark.parametrize("ks", [[3], [20, 32], [64], [40, 7], [128], [200], [300, 5], [460]])
def test_full_step_inside(ks):
    from sdpx_b200.cuda_backend import CudaBackend
    from sdpx_b200.problem import ingest
    rng = np.random.default_rng(len(ks) + ks[0])

    def sym(k):
        a = rng.standard_normal((k, k))
        return (a + a.T) / np.linalg.norm(a + a.T, 2)
    X = [np.eye(k) + 0.1 * sym(k) for k in ks]
    Y = [np.linalg.inv(x) + 0.05 * sym(len(x)) for x in X]
    Y = [(y + y.T) / 2 for y in Y]
    A = [np.array([sym(k) for _ in range(3)]) for k in ks]
    c = sum(np.einsum("ijk,jk->i", a, y) for a, y in zip(A, Y))
    with CudaBackend(ingest(c, A, [-x for x in X])) as be:
        be.set_iterate(np.zeros(3), X, Y)
        assert be.compute_residuals([1.0] * len(ks), False, True)[2]
        be.schur_build()
        assert be.factorize()["ok"]
        be.predictor_rhs()
        be.solve_direction()
        be.direction_blocks()
        _, dX, dY = be.get_direction()
        assert _exact(X, dX) == 1.0 and _exact(Y, dY) == 1.0
        p = be.affine_diagnostics(True)
        assert p["tX"] == 1.0 and p["tY"] == 1.0


# Late iterates: κ(X) = κ(Y) far above the 100 of the other tests.  A Cholesky test decides on
# M + t·dM up to k·eps·‖M‖, that is up to k·eps·κ(M) of the smallest eigenvalue, and the
# eigenvalue bound is formed with errors of the same size (κ enters once: W and Wᵀ bring its
# square root each); the direction's own scale adds the 1e3 of the tests above.
@pytest.mark.parametrize("ks", [[12], [61, 17], [130], [300, 40]])
@pytest.mark.parametrize("kappa", [1e6, 1e9])
def test_ill_conditioned_iterates_match_the_bisection(ks, kappa):
    from sdpx_b200.cuda_backend import CudaBackend
    from sdpx_b200.problem import ingest
    rng = np.random.default_rng(sum(ks))
    half = np.log10(kappa) / 2

    def spd(k, sign):
        q, _ = np.linalg.qr(rng.standard_normal((k, k)))
        x = (q * np.logspace(-sign * half, sign * half, k)) @ q.T
        return 0.5 * (x + x.T)
    A = [rng.standard_normal((3, k, k)) for k in ks]
    A = [a + a.transpose(0, 2, 1) for a in A]
    X, Y = [spd(k, 1) for k in ks], [spd(k, -1) for k in ks]
    with CudaBackend(ingest(rng.standard_normal(3), A, [np.eye(k) for k in ks])) as be:
        be.set_iterate(np.zeros(3), X, Y)
        assert be.compute_residuals([0.0] * len(ks), True, True)[2]
        be.schur_build()
        assert be.factorize()["ok"]
        be.predictor_rhs()
        be.solve_direction()
        be.direction_blocks()
        p = be.affine_diagnostics(True)
        for key, t in zip(("tX", "tY"), be.line_search("fraction_to_boundary", 1.0, 1.0, 0.9, 1e-300, 0.0)):
            assert abs(p[key] - t) <= 8 * max(ks) * EPS * kappa * 1e3 * t
