"""Pinned blocks of the process cache under handles that live and die side by side: every
thread's results are those of the same calls one after the other."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_handles_side_by_side():
    from sdpx_b200 import generators as G
    from sdpx_b200.batch import BatchSolver, batch_options
    from sdpx_b200.cuda_backend import CudaBackend
    from sdpx_b200.normal import NormalSystem
    opts = batch_options(1e-8, iter_max=3)

    def dense(seed):
        p = G.sdpa_dense(m=8, blocks=[10 + seed % 5, 4], lp=3, seed=seed)
        with CudaBackend(p) as be:
            r = be.optimize(opts)
        return [r.x.tobytes()] + [b.tobytes() for b in r.X + r.Y]

    def normal(seed):
        rng = np.random.default_rng(seed)
        m, n = 20 + seed, 60 + seed
        with NormalSystem(rng.standard_normal((n, m)), n) as ns:
            ns.factor_reduced(rng.uniform(0.5, 2.0, n), 1e-8)
            return [ns.solve_factor(rng.standard_normal(n + m)).tobytes()]

    def batch(seed):
        with BatchSolver([G.sdpa_dense(m=4, blocks=[3 + i % 4], seed=seed + i) for i in range(9)]) as bs:
            return [r.x.tobytes() for r in bs.optimize(opts)]
    jobs = [(f, s) for s in range(12) for f in (dense, normal, batch)]
    want = [f(s) for f, s in jobs]
    for threads in (2, 8):
        with ThreadPoolExecutor(max_workers=threads) as pool:
            for _ in range(3):
                assert list(pool.map(lambda j: j[0](j[1]), jobs)) == want
