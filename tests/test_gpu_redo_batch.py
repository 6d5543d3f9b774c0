"""Right-hand sides of a mixed batch that are solved again in FP64: one at a time while
they are fewer than a 32-slot iteration costs one-slot ones at the operator's size,
else as a batch.  Every solve hits its limit of three iterations; a one-slot solve is
told apart by its barrier, which gives up at once."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NOT_CONVERGED, TIMEOUT = -5, -9


@pytest.mark.parametrize("k,status", [(2, TIMEOUT), (10, NOT_CONVERGED)])
def test_redo_follows_the_batch_cost(k, status):
    import cpm_gb300 as cg

    op = cg.OpSet(cg.Tube(cg.desc(cg.SPHERE, [1.0]), 3, 0.1), [])
    assert 2 < cg.batch_cost(op.D, cg.BATCH_FP64) < 10
    b = np.cos(op.rows()["point"] @ np.array([0.9, -0.5, 2.0])) * np.arange(1, k + 1)[:, None]
    s = cg.Solver(op, 1.0, -1.0, kslots=32)
    s.set_one_kernel(wait_polls=0)
    _, st = s.solve(b, tol=1e-10, precision=1, max_iters=3, raise_on_error=False)
    assert [q["status"] for q in st] == [status] * k
    assert all(q["fp64_fallback"] == 1 for q in st)
