"""The tile-flag Cholesky (csrc/potrf_flow.cu) at the edges of its 64-tiles, its 8-row
strips and its groups of CTAs, against the factored matrix itself and NumPy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


# one matrix: strips (1, 7, 8, 9), one tile, two tiles (the chain alone), more tiles
# (other CTAs take part), a last tile of one row
@pytest.mark.parametrize("m", [1, 7, 8, 9, 63, 64, 65, 121, 128, 129, 193, 449, 1025])
def test_factor_of_one_matrix(m):
    from sdpx_b200.normal import NormalSystem
    rng = np.random.default_rng(m)
    n = 2 * m + 3
    with NormalSystem(rng.standard_normal((n, m)), n) as ns:
        ok, _, _ = ns.factor_reduced(rng.uniform(0.5, 1.5, n), 1e-10)
        Q, L = ns.matrix(0), ns.matrix(1)
    assert ok
    assert not np.triu(L, 1).any()
    # Higham, Accuracy and Stability, thm 10.3: |LLᵀ − Q| ≤ γ_{m+1}|L||Lᵀ|
    assert (np.abs(L @ L.T - Q) <= (m + 2) * EPS * 1.01 * (np.abs(L) @ np.abs(L).T)).all()


def _backend(ks, seed):
    from sdpx_b200.cuda_backend import CudaBackend
    from sdpx_b200.problem import ingest
    rng = np.random.default_rng(seed)
    A = [rng.standard_normal((2, k, k)) for k in ks]
    A = [a + a.transpose(0, 2, 1) for a in A]
    X = []
    for k in ks:
        q, _ = np.linalg.qr(rng.standard_normal((k, k)))
        x = (q * np.logspace(-1, 1, k)) @ q.T
        X.append(0.5 * (x + x.T))
    prob = ingest(rng.standard_normal(2), A, [np.eye(k) for k in ks])
    return CudaBackend(prob), X


# several orders in one launch; more matrices than the GPU has SMs
@pytest.mark.parametrize("ks", [[3, 65, 130, 64, 200], [320, 4], [5 + i % 13 for i in range(90)]])
def test_factors_of_many_blocks(ks):
    be, X = _backend(ks, len(ks))
    with be:
        be.set_iterate(np.zeros(2), X, X)
        _, _, ok = be.compute_residuals([0.0] * len(ks), True, True)
        assert ok
        margin = min(np.diag(c).min() / np.diag(c).max() for c in map(np.linalg.cholesky, X))
        # pivots are accurate to about k·eps·κ; κ = 100
        for got in be.block_margins():
            assert abs(got - margin) <= 4 * max(ks) * EPS * 100 * margin


@pytest.mark.parametrize("k,bad", [(8, 0), (8, 7), (64, 9), (65, 64), (130, 70), (200, 199)])
def test_indefinite_block_is_reported(k, bad):
    be, X = _backend([k, 70], k)
    with be:
        Y = [x.copy() for x in X]
        be.set_iterate(np.zeros(2), X, Y)
        assert be.compute_residuals([0.0, 0.0], True, True)[2]
        # pivot `bad` becomes negative: the leading minors up to it stay positive
        L = np.linalg.cholesky(X[0])
        Y[0][bad, bad] -= 1.5 * L[bad, bad] ** 2
        be.set_iterate(np.zeros(2), X, Y)
        assert not be.compute_residuals([0.0, 0.0], True, True)[2]
        be.set_iterate(np.zeros(2), X, X)  # nothing of the failure stays behind
        assert be.compute_residuals([0.0, 0.0], True, True)[2]
