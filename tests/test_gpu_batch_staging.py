"""More instances than the batched engine has input slots for at its full count of slots
(16 up to about 5000 instances): the phases then share fewer, here 5, and every instance
gets the same answer as in a small batch."""
import pytest

pytestmark = pytest.mark.gpu


def test_many_instances_share_fewer_slots():
    from sdpx_b200 import generators as G
    from sdpx_b200.batch import BatchSolver, batch_options
    base = [G.sdpa_dense(m=3 + i % 3, blocks=[3 + i % 4], seed=i) for i in range(60)]
    opts = batch_options(1e-8, iter_max=4)
    with BatchSolver(base) as bs:
        few = [(r.status, r.iterations, r.pObj, r.dObj) for r in bs.optimize(opts, solutions=False)]
    with BatchSolver(base * 250) as bs:
        many = [(r.status, r.iterations, r.pObj, r.dObj) for r in bs.optimize(opts, solutions=False)]
    assert many == few * 250
