"""E x of 32 slots with the groups' tables read one group ahead, from one block
per SM (many groups a warp) to one group a warp, against the exported Efull rows
in extended precision: small operators with groups of one row, of more rows than
are taken at a time, and with moved columns.

Tolerance, in units of the sum of |weight x value| of a row: the three FP32
weights are rounded once each, the sums over z and y at most four times and the
one over x five times, a further entry and the sign at most three: 20 units of
2^-24.  FP64 rows: as in test_gpu_fixed_point, 4 units of 2^-52 of the largest
value read."""
import numpy as np
import pytest

from test_gpu_fixed_point import _circle, _reference

pytestmark = pytest.mark.gpu

CURVES = {"plain": ((), 1), "order1": ((0.3,), 1), "order2": ((0.3, -0.5), 2)}


def _apply(op, x, fp32):
    import torch

    import cpm_gb300 as cg

    d = torch.from_numpy(x).cuda()
    t, y = torch.full_like(d, float("nan")), torch.empty_like(d)
    torch.cuda.synchronize()
    op.apply_device(0.0, -1.0, 32, fp32, d.data_ptr(), t.data_ptr(), y.data_ptr())
    torch.cuda.synchronize()
    cg.sync()
    return t.cpu().numpy()


@pytest.mark.parametrize("curves", list(CURVES))
@pytest.mark.parametrize("dx", [0.35, 0.2, 0.1])
def test_rows_at_every_launch_shape(curves, dx):
    import cpm_gb300 as cg

    zs, order = CURVES[curves]
    op = cg.OpSet(cg.Tube(cg.desc(cg.SPHERE, [1.0]), 3, dx), [_circle(cg, z, order) for z in zs])
    ptr, idx, val = op.csr(1)
    if curves == "plain":  # rows with the same columns: some stencils have more of them than a chunk
        sets = {}
        for r in range(op.D):
            key = idx[ptr[r]:ptr[r + 1]].tobytes()
            sets[key] = sets.get(key, 0) + 1
        assert max(sets.values()) > 10
    x = np.random.default_rng(11).uniform(-1, 1, (op.D, 32)).astype(np.float32)
    cols = [0, 13, 31]
    ref, big = _reference((ptr, idx, val), x[:, cols].astype(np.float64))
    size = np.stack([np.add.reduceat(np.abs(val * x[idx, s]), ptr[:-1]) for s in cols], axis=1)
    first = None
    for shape in (0, 1, 2, 64):
        op.set_launch(shape, shape, shape)
        t32, t64 = _apply(op, x, True), _apply(op, x.astype(np.float64), False)
        if first is None:
            first = t32, t64
            assert np.all(np.abs(t32[:, cols] - ref) <= 20 * 2.0 ** -24 * size)
            assert np.all(np.abs(t64[:, cols] - ref) <= 4 * 2.0 ** -52 * big)
        assert np.array_equal(t32, first[0]) and np.array_equal(t64, first[1])
