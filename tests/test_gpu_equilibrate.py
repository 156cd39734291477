"""Device equilibration against the oracle's: blocks around a warp's and a tile's size, 1×1
blocks, a row that is zero everywhere, badly scaled rows (more passes), and a second
solve on the same data.  Both multiply at most eight factors of a few roundings each into
E, so E, s and the scaled data agree to 1e-13; the pass counts are equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-13


@pytest.mark.parametrize("blocks, lp, spread", [([2], 0, 0), ([33], 3, 2), ([64, 31], 0, 4), ([65, 2, 3], 300, 1),
                                                ([3] * 17, 1, 3), ([130], 0, 6)])
def test_equilibrate_matches_oracle(blocks, lp, spread):
    from oracle.sdpx_oracle import equilibrate_problem
    from sdpx_b200 import generators as G
    from sdpx_b200.cuda_backend import CudaBackend
    prob = G.sdpa_dense(m=9, blocks=blocks, lp=lp, seed=5)
    rng = np.random.default_rng(6)
    for l, k in enumerate(prob.k):
        d = 10.0 ** (spread * rng.uniform(-1, 1, k))
        if l == 0:
            d[0] = 0.0  # a row and column of zeros
        prob.Av[l] = np.ascontiguousarray((prob.Av[l].reshape(-1, k, k) * np.outer(d, d)).reshape(-1, k * k))
        prob.C[l] = prob.C[l] * np.outer(d, d)
    _, _, _, E, s, osc, passes = equilibrate_problem([a.copy() for a in prob.Av], [c.copy() for c in prob.C],
                                                     prob.c.copy(), prob.k)
    with CudaBackend(prob) as be:
        q = be.equilibrate()
    assert list(q.ruiz_passes) == list(passes)
    for a, b in zip(q.E, E):
        np.testing.assert_allclose(a, b, rtol=TOL, atol=0)
    np.testing.assert_allclose(q.s, s, rtol=TOL, atol=0)
    np.testing.assert_allclose(q.objective_scale, osc, rtol=TOL, atol=0)
