"""Rounding of the FP64 Gram products (csrc/blas_f64.cu): no running sum is longer than 256
rows of K or a sixteenth of it, however few chunks K is split into.

Off the diagonal, with N(0,1) entries, the partial sums grow as √k and each is rounded with
an rms error of u/√3 of its size, u = eps/2.  A running sum of n products thus has an rms
error of at most (u/√6)·n, and the sum of C of them (u/√6)·√(C·n² + C²·n); Σ|products| is
2K/π.  A single sum over K = 3500 would be 3.2 times the bound."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


# one 64-tile chunk, 32-tiles, several chunks, an odd number of rows (8-byte copies)
@pytest.mark.parametrize("m,n", [(500, 3500), (1000, 3000), (700, 2101), (1300, 1302), (317, 6340)])
def test_rms_error(m, n):
    from sdpx_b200.normal import NormalSystem
    rng = np.random.default_rng(m + n)
    B = np.asfortranarray(rng.standard_normal((n, m)))
    with NormalSystem(B, n) as ns:
        Q = ns.assemble_reduced_schur(np.ones(n), 0.0)
    rows, cols = rng.integers(0, m, 100), rng.integers(0, m, 20)
    L = B.astype(np.longdouble)
    exact = L[:, rows].T @ L[:, cols]
    off = rows[:, None] != cols[None, :]
    err = np.asarray(Q[np.ix_(rows, cols)] - exact, dtype=np.float64)[off]
    run = max(256, n // 16)
    C = -(-n // run)
    bound = EPS / 2 / np.sqrt(6) * np.sqrt(C * run ** 2 + C ** 2 * run)
    assert np.sqrt(np.mean(err ** 2)) <= bound
