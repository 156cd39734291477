"""Small results that the kernels write straight to the host, and the lists that travel
with a launch (up to 16 matrices, shifts or trials; more go through device memory).

* Norms: vectors of 1 entry to several blocks, NaN counting as +inf, exact.
* Newton residuals, dot products and traces of problems with 1, 8, 9, 16, 17 blocks:
  sums of n products within n·eps of the sum of magnitudes.
* Gram matrices of the digit products over one or many K chunks: within the digits'
  truncation and the sum's rounding of numpy's product.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


def _backend(m, blocks, seed=1, lp=0):
    from sdpx_b200 import generators as G
    from sdpx_b200.cuda_backend import CudaBackend
    prob = G.sdpa_dense(m=m, blocks=blocks, lp=lp, seed=seed)
    return prob, CudaBackend(prob)


@pytest.mark.parametrize("m", [1, 31, 1023, 1024, 1025, 3000])
def test_norms_are_exact(m):
    prob, be = _backend(m, [4])
    maxC, cnorm = be.data_norms()[:2]
    assert maxC == max(np.abs(c).max() for c in prob.C)
    assert cnorm == np.abs(prob.c).max()
    be.close()


@pytest.mark.parametrize("nb", [1, 8, 9, 16, 17])
def test_block_lists(nb):
    ks = [3 + (i % 5) for i in range(nb)]
    prob, be = _backend(6, ks, seed=nb)
    rng = np.random.default_rng(nb)

    def spd(k):
        a = rng.standard_normal((k, k))
        return a @ a.T + k * np.eye(k)
    X, Y = [spd(k) for k in ks], [spd(k) for k in ks]
    x = rng.standard_normal(6)
    be.set_iterate(x, X, Y)
    xg, Xg, _, Yg = be.get_iterate()
    assert np.array_equal(xg, x)
    assert all(np.array_equal(a, b) for a, b in zip(Xg, X)) and all(np.array_equal(a, b) for a, b in zip(Yg, Y))
    dots, tX, tY = be.block_dots()
    for l, k in enumerate(ks):
        assert abs(dots[l] - np.sum(X[l] * Y[l])) <= 2 * k * k * EPS * np.sum(np.abs(X[l] * Y[l]))
        assert abs(tX[l] - np.trace(X[l])) <= 2 * k * EPS * np.trace(X[l])
        assert abs(tY[l] - np.trace(Y[l])) <= 2 * k * EPS * np.trace(Y[l])
    # factors of 2·nb blocks and the shifted residual R = μI − XY
    _, _, ok = be.compute_residuals(np.full(nb, 0.5), False, True)
    assert ok
    p, d = be.block_margins()
    q = [min(min(np.diag(np.linalg.cholesky(M))) / max(np.diag(np.linalg.cholesky(M))) for M in Ms) for Ms in (X, Y)]
    assert abs(p - q[0]) <= 1e-12 * q[0] and abs(d - q[1]) <= 1e-12 * q[1]
    be.close()


@pytest.mark.parametrize("m, k", [(1, 4), (63, 10), (64, 12), (65, 25), (129, 40), (300, 30)])
def test_digit_gram_chunks(m, k):
    prob, be = _backend(m, [k], seed=3)
    be.schur_build(identity=True)
    S = be.schur_matrix()
    A = np.asarray(prob.Av[0])
    ref = A @ A.T
    col = np.abs(A).max(axis=1)
    bound = k * k * 2.0 ** -51 * np.outer(col, col) + 64 * EPS * np.abs(A) @ np.abs(A).T
    assert np.all(np.abs(np.tril(S - ref)) <= bound)
    be.close()
