"""Normal system: calls whose vectors just fit the pinned staging, and the next larger ones.

The staging holds 2^20 − 64 bytes: a solve stages n + m ≤ 131064 numbers, the weights n_lp,
a scaling 4·nq + 3·ncones.  Both routes run the same kernels, so scalings agree bit for bit;
solves stay within the forward-error bound of the reduced system's formulas.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


def _normal():
    from sdpx_b200 import normal
    return normal


@pytest.mark.parametrize("n", [1, 7, 131062, 131063, 131064, 131065])
def test_solve_at_the_staging_limit(n):
    m, reg = min(n, 2), 0.5
    rng = np.random.default_rng(n)
    B, w = rng.standard_normal((n, m)), rng.uniform(0.5, 2.0, n)
    rhs = rng.standard_normal(n + m)
    with _normal().NormalSystem(B, n, []) as ns:
        Di = ns.lp_standard_pack(w, reg)[1]
        assert ns.factor_reduced(w, reg)[0]
        got = ns.solve_factor(rhs)
    Q = B.T @ (Di[:, None] * B) + reg * np.eye(m)
    t, Qi, aB = Di * rhs[:n], np.linalg.inv(Q), np.abs(B)
    dy = Qi @ (rhs[n:] - B.T @ t)
    e = 4 * (n + m) * EPS * np.abs(Qi) @ (aB.T @ np.abs(t) + np.abs(rhs[n:]) + np.abs(Q) @ np.abs(dy)
                                          + aB.T @ (Di * (aB @ np.abs(dy))))
    dx = t + Di * (B @ dy)
    assert np.all(np.abs(got[n:] - dy) <= e)
    assert np.all(np.abs(got[:n] - dx) <= 8 * EPS * (np.abs(t) + Di * (aB @ np.abs(dy))) + Di * (aB @ e))


@pytest.mark.parametrize("bad", [None, 3])
def test_scaling_at_the_staging_limit(bad):
    k = 131064 // 11  # cones of order 2: 4·2 + 3 numbers each
    rng = np.random.default_rng(5)
    u, v = rng.standard_normal((2, k + 1))
    s = np.column_stack([1.5 * np.abs(u) + 1.0, u])
    z = np.column_stack([1.2 * np.abs(v) + 0.5, v])
    if bad is not None:
        s[bad, 0] = -1.0
    out = []
    for c in (k, k + 1):
        with _normal().NormalSystem(np.zeros((2 * c, 1)), 0, [2] * c) as ns:
            out.append(ns.soc_nt_scaling(s[:c].ravel(), z[:c].ravel()))
    assert out[0][:2] == out[1][:2] == ((True, -1) if bad is None else (False, bad))
    fine = np.arange(k) != (-1 if bad is None else bad)
    for q in ("w", "lambda"):
        a, b = out[0][2][q].reshape(-1, 2), out[1][2][q].reshape(-1, 2)[:k]
        assert np.array_equal(a[fine], b[fine])
    for q in ("eta", "eta_squared", "ok"):
        assert np.array_equal(out[0][2][q], out[1][2][q][:k])
