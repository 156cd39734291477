"""The batched line search: orders at the edges of its rules (8, 32), searches of many trials,
and its kernels for small, mixed, few and many instances, which have to agree exactly."""
import pytest

pytestmark = pytest.mark.gpu


def _problem(n, m, seed):
    from sdpx_b200 import generators as G
    return G.sdpa_dense(m=m, blocks=[n], seed=seed)


# As the single solves: status, iterations and objectives to the tolerance of the solve.
def test_orders_at_the_edges_match_single_solves():
    from sdpx_b200 import solve
    from sdpx_b200.batch import BATCH_OPTIONS, BatchSolver, batch_options
    probs = [_problem(n, 5, seed) for n in (3, 7, 8, 9, 16, 17, 31, 32, 33, 40) for seed in (1, 2)]
    with BatchSolver(probs) as bs:
        batch = bs.optimize(batch_options(1e-8))
    for p, r in zip(probs, batch):
        one = solve(p, tolerance=1e-8, **BATCH_OPTIONS)
        assert r.status == one.status and abs(r.iterations - one.iterations) <= 1
        assert abs(r.pObj - one.pObj) <= 1e-7 * (1 + abs(one.pObj))


# (27, 7, 500) stalls: its last searches go through hundreds of trials.
@pytest.mark.parametrize("inst", [(27, 7, 500), (6, 4, 1), (8, 9, 2), (32, 20, 3)])
def test_kernels_agree(inst):
    from sdpx_b200.batch import BatchSolver, batch_options
    p, opts = _problem(*inst), batch_options(1e-8)

    def first(others):
        with BatchSolver([p] + others) as bs:
            r = bs.optimize(opts)[0]
        return r.status, r.iterations, r.pObj, r.x.tolist()
    alone = first([])
    small = [_problem(4 + i % 9, 3, i) for i in range(160)]
    assert first(small) == alone          # more instances than SMs
    assert first([_problem(40, 6, 1)]) == alone   # beside a larger order
    assert first(small + [_problem(40, 6, 1)]) == alone
