"""One-vector FP64 solves whose grid barrier gives up at once (no poll of its wait): the
kernel ends, the right-hand side reports a timeout with its statistics, other
right-hand sides keep their results and the solver's next solve is unharmed."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TIMEOUT = -9


def _system():
    import cpm_gb300 as cg

    op = cg.OpSet(cg.Tube(cg.desc(cg.SPHERE, [1.0]), 3, 0.1), [])
    return op, np.cos(op.rows()["point"] @ np.array([0.9, -0.5, 2.0]))


@pytest.mark.parametrize("precond,sweeps", [(1, 0), (2, 4)])
def test_a_wait_that_runs_out_is_reported(precond, sweeps):
    import cpm_gb300 as cg

    op, b = _system()
    kw = dict(tol=1e-12, precond=precond, precond_iters=sweeps)
    s = cg.Solver(op, 1.0, -1.0)
    want = s.solve(b, **kw)
    s.set_one_kernel(wait_polls=0)
    x, st = s.solve(b, raise_on_error=False, **kw)
    assert st[0]["status"] == TIMEOUT and st[0]["iterations"] == 0
    with pytest.raises(cg.CpmError):
        s.solve(b, **kw)
    s.set_one_kernel()
    again = s.solve(b, **kw)
    assert np.array_equal(again[0], want[0]) and again[1][0]["iterations"] == want[1][0]["iterations"]


def test_statistics_are_written():
    """the C entry fills the caller's entry, whatever it held"""
    import cpm_gb300 as cg

    op, b = _system()
    s = cg.Solver(op, 1.0, -1.0)
    s.set_one_kernel(wait_polls=0)
    o = cg.SolveOpts(tol=1e-12, max_iters=1000, precision=0, precond=1)
    st = (cg.SolveStats * 1)()
    ctypes.memset(st, 0x5A, ctypes.sizeof(st))
    x = np.zeros_like(b)
    rc = cg.lib().cpm_solve(s.h, 1, b.ctypes.data_as(ctypes.c_void_p), x.ctypes.data_as(ctypes.c_void_p), ctypes.byref(o), st)
    assert rc == TIMEOUT and st[0].status == TIMEOUT and st[0].iterations == 0 and st[0].restarts == 0


def test_a_batch_keeps_the_results_of_its_other_slots():
    """a right-hand side of a mixed batch that is solved again alone: only that one times out
    (three iterations are too few for b, and none are needed for 0)"""
    import cpm_gb300 as cg

    op, b = _system()
    s = cg.Solver(op, 1.0, -1.0, kslots=32)
    s.set_one_kernel(wait_polls=0)
    x, st = s.solve(np.stack([0.0 * b, b, 0.0 * b]), tol=1e-10, precision=1, max_iters=3, raise_on_error=False)
    assert [q["status"] for q in st] == [0, TIMEOUT, 0]
    assert st[1]["fp64_fallback"] == 1 and st[1]["iterations"] == 3
    assert not np.any(x[[0, 2]])
