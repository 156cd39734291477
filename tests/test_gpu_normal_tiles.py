"""The reduced normal system at the edges of its kernels' tiles.

* Gram product: tiles of 32 and 64, K steps of 16, rows of odd and even stride;
  within the forward-error bound (n + 2)·eps·|B|ᵀ|B|.
* Cone scaling: row tiles of 64 with whole cones, cones that span several tiles,
  column tiles of 32.  The reference scales each column with the W⁻¹ map, which is
  bit-identical to the oracle's.
* NT scaling with 4, 8, 16 and 32 lanes per cone (by the mean order): bit for bit.
* Triangular solve over row blocks of 64, also with more blocks than SMs.
"""
import numpy as np
import pytest

from oracle import cone_oracle as O

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


def _normal():
    from sdpx_b200 import normal
    return normal


def _interior(rng, q):
    u = rng.standard_normal(q - 1)
    return np.concatenate([[1.5 * np.linalg.norm(u) + 1.0], u])


@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 129, 300, 1000])
@pytest.mark.parametrize("m", [1, 31, 32, 33, 64, 65, 200])
def test_gram_tile_edges(n, m):
    B = np.random.default_rng(n * 1000 + m).standard_normal((n, m))
    with _normal().NormalSystem(B, n, []) as ns:
        Q = ns.assemble_reduced_schur(np.ones(n), 0.0)
    bound = (n + 2) * EPS * (np.abs(B).T @ np.abs(B))
    assert np.all(np.abs(Q - B.T @ B) <= 2 * bound)


@pytest.mark.parametrize("dims", [[1], [63, 1], [64], [65], [30, 30, 5], [3] * 30, [1, 2, 200, 7, 64, 129]])
@pytest.mark.parametrize("m", [1, 31, 33])
def test_cone_scaling_tile_edges(dims, m):
    rng = np.random.default_rng(len(dims) * 100 + m)
    nq, n_lp = sum(dims), 5
    s = np.concatenate([_interior(rng, q) for q in dims])
    z = np.concatenate([_interior(rng, q) for q in dims])
    B = rng.standard_normal((n_lp + nq, m))
    with _normal().NormalSystem(B, n_lp, dims) as ns:
        assert ns.soc_nt_scaling(s, z)[0]
        Q = ns.assemble_reduced_schur(np.ones(n_lp), 0.0)
        Bh = np.vstack([B[:n_lp], np.column_stack([ns.soc_nt_apply_winv(B[n_lp:, j].copy()) for j in range(m)])])
    bound = (n_lp + nq + 2) * EPS * (np.abs(Bh).T @ np.abs(Bh))
    assert np.all(np.abs(Q - Bh.T @ Bh) <= 2 * bound)


@pytest.mark.parametrize("dims", [[2] * 9, [5] * 7, [9] * 3 + [1], [17, 16], [40, 3, 33, 32]])
def test_nt_scaling_lanes_bit_exact(dims):
    rng = np.random.default_rng(sum(dims))
    s = [_interior(rng, q) for q in dims]
    z = [_interior(rng, q) for q in dims]
    with _normal().NormalSystem(np.zeros((sum(dims), 1)), 0, dims) as ns:
        ok, _, out = ns.soc_nt_scaling(np.concatenate(s), np.concatenate(z))
    assert ok
    ref = [O.nt_scaling(list(a), list(b)) for a, b in zip(s, z)]
    assert np.array_equal(out["w"], np.concatenate([r[1] for r in ref]))
    assert np.array_equal(out["lambda"], np.concatenate([r[2] for r in ref]))
    assert np.array_equal(out["eta"], [r[3] for r in ref])


@pytest.mark.parametrize("m", [1, 63, 64, 65, 128, 129, 640, 9537])
def test_triangular_solve_block_edges(m):
    """Q = BᵀB + δI of low rank: the residual of dy is formed without Q.  Cholesky solves are backward stable:
    ‖Q·dy − g‖ ≤ c·m·eps·‖Q‖‖dy‖ with c of a few units (here 8)."""
    n, delta = 8, 1.0
    rng = np.random.default_rng(m)
    B = rng.standard_normal((n, m)) / np.sqrt(m)
    rhs = rng.standard_normal(n + m)
    with _normal().NormalSystem(B, n, []) as ns:
        assert ns.factor_reduced(np.ones(n), delta)[0]
        d = ns.solve_factor(rhs)
    D = 1.0 + delta                     # LP pack: weight·c² + δ
    dy = d[n:]
    g = rhs[n:] - B.T @ (rhs[:n] / D)
    r = B.T @ (B @ dy) / D + delta * dy - g
    normQ = np.linalg.norm(B, 2) ** 2 / D + delta
    assert np.linalg.norm(r) <= 8 * (m + n) * EPS * (normQ * np.linalg.norm(dy) + np.linalg.norm(g))
