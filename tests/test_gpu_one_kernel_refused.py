"""One-vector FP64 solves where the one-kernel launch is refused: the solve and those
after it iterate by graphs, from the state the kernel would have started from."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precond,sweeps", [(1, 0), (2, 4)])
def test_refused_launch_goes_on_by_graphs(precond, sweeps):
    import cpm_gb300 as cg

    op = cg.OpSet(cg.Tube(cg.desc(cg.SPHERE, [1.0]), 3, 0.1), [])
    b = np.cos(op.rows()["point"] @ np.array([0.9, -0.5, 2.0]))
    kw = dict(tol=1e-12, precond=precond, precond_iters=sweeps)
    graph = cg.Solver(op, 1.0, -1.0)
    graph.set_one_kernel(0)
    want = graph.solve(b, **kw)
    s = cg.Solver(op, 1.0, -1.0)
    s.set_one_kernel(60000)  # more blocks than any device holds: the launch is refused on the host
    for _ in range(2):
        got = s.solve(b, **kw)
        assert got[1][0]["status"] == 0
        assert np.array_equal(got[0], want[0]) and got[1][0]["iterations"] == want[1][0]["iterations"]
    s.set_one_kernel()
    x = s.solve(b, **kw)[0]  # the kernel again; the smallest eigenvalue is 1
    assert np.max(np.abs(x - want[0])) <= 1e-9 * np.max(np.abs(x))


def test_shapes_out_of_range_are_rejected():
    import cpm_gb300 as cg

    s = cg.Solver(cg.OpSet(cg.Tube(cg.desc(cg.SPHERE, [1.0]), 3, 0.2), []), 1.0, -1.0)
    for blocks in (-2, 65536):
        with pytest.raises(cg.CpmError):
            s.set_one_kernel(blocks)
