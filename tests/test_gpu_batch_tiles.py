"""The batched engine at the edges of its tiles: block orders around the strips of eight
and the 64×64 tile, constraint counts around the Schur tiles, more instances than read
their inputs in place, and two engines of different orders alive at once.

One interior-point iteration decides nothing by rounding, so an instance solved in a
batch agrees with the same instance in a batch of its own to the rounding of sums taken in
another order (1e-10 of the largest entry at the start's conditioning)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problems(shapes):
    from sdpx_b200 import generators as G
    return [G.sdpa_dense(m=m, blocks=[k], seed=17 * k + m) for k, m in shapes]


def _solve(probs, iters=1):
    from sdpx_b200.batch import BatchSolver, batch_options
    with BatchSolver(probs) as bs:
        return bs.optimize(batch_options(1e-8, iter_max=iters))


def _close(a, b):
    for p, q in ((a.x, b.x), (a.X[0], b.X[0]), (a.Y[0], b.Y[0])):
        assert np.max(np.abs(p - q)) <= 1e-10 * max(1.0, np.max(np.abs(q)))


@pytest.mark.parametrize("shapes", [[(3, 1)], [(8, 9), (9, 1), (7, 28)], [(16, 63), (17, 64), (15, 65)],
                                    [(32, 128), (33, 129), (31, 3)], [(63, 200), (64, 256), (3, 6)]])
def test_batch_matches_instances_alone(shapes):
    probs = _problems(shapes)
    both = _solve(probs)
    for p, r in zip(probs, both):
        _close(r, _solve([p])[0])


def test_more_instances_than_are_read_in_place():
    probs = _problems([(3 + i % 6, 2 + i % 5) for i in range(130)])
    res = _solve(probs)
    for i in (0, 64, 127, 128, 129):
        _close(res[i], _solve([probs[i]])[0])


def test_a_smaller_engine_does_not_lower_the_limits_of_a_larger():
    from sdpx_b200.batch import BatchSolver, batch_options
    big, small = _problems([(64, 100), (60, 40)]), _problems([(4, 3)])
    with BatchSolver(big) as a:
        first = a.optimize(batch_options(1e-8, iter_max=1))
        with BatchSolver(small) as b:
            b.optimize(batch_options(1e-8, iter_max=1))
            again = a.optimize(batch_options(1e-8, iter_max=1))
    for p, q in zip(first, again):
        assert np.array_equal(p.x, q.x)
