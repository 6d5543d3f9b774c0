"""A one-vector FP64 solve that restarts: each breakdown of rho leaves the kernel, the
true residual replaces the recursive one and the kernel is launched again.  With a
tolerance that no residual meets the recursive residual falls to rounding level over
and over, so a cycle takes some tens of iterations; the solve has to go on to its
iteration limit, as the kernels of a graph do."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _system(dx):
    import cpm_gb300 as cg

    op = cg.OpSet(cg.Tube(cg.desc(cg.SPHERE, [1.0]), 3, dx), [])
    return op, np.cos(3.0 * op.rows()["point"] @ np.array([0.3, -0.5, 0.8]))


@pytest.mark.parametrize("precond,sweeps", [(1, 0), (2, 3)])
def test_restarts_up_to_the_iteration_limit(precond, sweeps):
    import cpm_gb300 as cg

    op, b = _system(0.2)
    kw = dict(precond=precond, precond_iters=sweeps, raise_on_error=False)
    x, st = cg.Solver(op, 1.0, -1.0).solve(b, tol=1e-300, max_iters=4000, max_refine=1, **kw)
    assert st[0]["restarts"] > 0
    assert st[0]["status"] == -5 and st[0]["iterations"] == 4000, st
    # the solution stays the solution: smallest eigenvalue 1, as in the one-kernel solves' test
    ref, s2 = cg.Solver(op, 1.0, -1.0, kslots=32).solve(b, tol=1e-12, **kw)
    assert s2[0]["status"] == 0
    assert np.max(np.abs(x - ref)) <= 1e-9 * np.max(np.abs(ref))


def test_two_threads_solve_at_once():
    """each solver on its own stream, both in one kernel: neither waits for blocks of the other"""
    import threading

    import cpm_gb300 as cg

    op, b = _system(0.05)
    ref = cg.Solver(op, 1.0, -1.0).solve(b, tol=1e-12)[0]
    out, errors = {}, []

    def work(i):
        try:
            s = cg.Solver(op, 1.0, -1.0)
            out[i] = [s.solve(b, tol=1e-12)[0] for _ in range(20)]
        except Exception as e:
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    assert all(np.array_equal(x, ref) for xs in out.values() for x in xs)
