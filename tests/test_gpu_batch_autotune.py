"""The autotuner of the batched engine times the launch shape an engine starts with, so that
calling it never leaves a slower one."""
import pytest

pytestmark = pytest.mark.gpu


def test_default_shape_is_a_candidate():
    from sdpx_b200 import batch_instances
    from sdpx_b200.batch import BatchSolver, batch_options
    probs = batch_instances(24, seed=5, n_range=(4, 16), m_cap=30)
    opts = batch_options(1e-8)
    with BatchSolver(probs) as bs:
        before = [r.pObj for r in bs.optimize(opts)]
        table = bs.autotune(opts, cache=False)
        assert (128, 64, -1.0) in [row[:3] for row in table]
        bs.set_schur_shape(128, 64, -1.0)
        assert [r.pObj for r in bs.optimize(opts)] == before  # the shape it started with
