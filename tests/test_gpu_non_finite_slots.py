"""Infinities and NaN in one slot of a 32-slot FP64 apply, in either half of a warp's
slots: they reach the rows that read them and no other, the slot's other rows are the
clean run's within what either sum may be off (30 units of 2^-53 of its terms), and every other slot is the
clean run's bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DX = 0.1


@pytest.fixture(scope="module", params=[0, 2])
def op(request):
    import cpm_gb300 as cg

    ibcs = [cg.desc(cg.CIRCLE3D, [np.sqrt(1 - z * z), 0, 0, z, 0, 0, 1], (-1.0, 1.0), boundary_order=2,
                    on_ibc_tolerance=0.1 * DX * DX) for z in (0.3, 0.36)[:request.param]]
    op = cg.OpSet(cg.Tube(cg.desc(cg.SPHERE, [1.0]), 3, DX), ibcs)
    return op, op.csr(1)


def _e(op, x):
    import torch

    import cpm_gb300 as cg

    d = torch.from_numpy(np.ascontiguousarray(x)).cuda()
    t, y = torch.zeros_like(d), torch.zeros_like(d)
    torch.cuda.synchronize()
    op.apply_device(0.0, -1.0, 32, False, d.data_ptr(), t.data_ptr(), y.data_ptr())
    cg.sync()
    return t.cpu().numpy()


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("slot", [0, 15, 20, 31])
def test_non_finite_values_stay_in_their_slot_and_rows(op, bad, slot):
    op, (ptr, idx, val) = op
    rng = np.random.default_rng(7)
    x = rng.standard_normal((op.D, 32))
    where = rng.integers(0, op.D, 5)
    clean = x.copy()
    clean[where, slot] = 0.0
    x[where, slot] = bad
    t, tc = _e(op, x), _e(op, clean)
    hit = np.add.reduceat(np.abs(val) * np.isin(idx, where), ptr[:-1]) > 0
    assert not np.any(np.isfinite(t[hit, slot]))
    assert np.all(np.isfinite(t[~hit, slot]))
    size = np.add.reduceat(np.abs(val * clean[idx, slot]), ptr[:-1])
    assert np.all(np.abs(t - tc)[~hit, slot] <= 2 * 30 * 2.0 ** -53 * size[~hit])
    others = np.arange(32) != slot
    assert np.array_equal(t[:, others], tc[:, others])
