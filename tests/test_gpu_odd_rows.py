"""A(-x) = -A(x) and E(-x) = -E(x) bit for bit for FP64 vectors, as FP64 arithmetic
has it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DX = 0.1


@pytest.fixture(scope="module")
def op():
    import cpm_gb300 as cg

    z = 0.3
    return cg.OpSet(cg.Tube(cg.desc(cg.SPHERE, [1.0]), 3, DX),
                    [cg.desc(cg.CIRCLE3D, [np.sqrt(1 - z * z), 0, 0, z, 0, 0, 1], (-1.0, 1.0), boundary_order=2,
                             on_ibc_tolerance=0.1 * DX * DX)])


def _apply(op, x, m, n):
    import torch

    import cpm_gb300 as cg

    d = torch.from_numpy(np.ascontiguousarray(x)).cuda()
    t, y = torch.zeros_like(d), torch.zeros_like(d)
    torch.cuda.synchronize()
    op.apply_device(m, n, x.shape[1], False, d.data_ptr(), t.data_ptr(), y.data_ptr())
    cg.sync()
    return t.cpu().numpy(), y.cpu().numpy()


@pytest.mark.parametrize("kind", ["rough", "dyadic", "sparse", "decay", "tiny"])
@pytest.mark.parametrize("k", [1, 32])
def test_applies_are_odd(op, kind, k):
    rng = np.random.default_rng(4)
    x = rng.standard_normal((op.D, k))
    if kind == "dyadic":  # few bits, both signs: sums that end half way between two units
        x = rng.integers(-8, 9, x.shape) / 8.0
    elif kind == "sparse":
        x[rng.random(x.shape) < 0.9] = 0.0
    elif kind == "decay":
        x *= np.exp(-12.0 * np.linalg.norm(op.rows()["point"] - np.array([0.0, 0.6, 0.8]), axis=1))[:, None]
    elif kind == "tiny":
        x *= np.exp2(rng.integers(-905, -885, x.shape).astype(float))
    for m, n in ((0.0, -1.0), (1.0, -0.37)):
        t, y = _apply(op, x, m, n)
        tn, yn = _apply(op, -x, m, n)
        assert np.array_equal(tn, -t) and np.array_equal(yn, -y)

