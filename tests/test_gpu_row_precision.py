"""E x of FP64 vectors against the exported Efull rows in extended precision, row by
row and relative to the row's own terms sum |w x|, on fields whose values differ
widely within a stencil (fixed-point sums are accurate relative to the largest
value of the 64, so such rows have to take the FP64 sum).

Tolerance, in units of 2^-53 sum |w x|: a term of the FP64 sum is rounded at most
12 times; a fixed-point row is off by at most 25 2^(e - 60) with its terms at
least 2^(e - 7), so by 25, and rounded once more; the exported weight products are
rounded twice, sign and extra entries add two roundings.  30 in all.  Products
below 2^-1074 in the sum are lost to either: a few of the smallest numbers."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DX = 0.1


@pytest.fixture(scope="module", params=["plain", "order1", "order2"])
def op(request):
    import cpm_gb300 as cg

    zs, order = {"plain": ((), 1), "order1": ((0.3, -0.5), 1), "order2": ((0.3, 0.36), 2)}[request.param]
    op = cg.OpSet(cg.Tube(cg.desc(cg.SPHERE, [1.0]), 3, DX),
                  [cg.desc(cg.CIRCLE3D, [np.sqrt(1 - z * z), 0, 0, z, 0, 0, 1], (-1.0, 1.0), boundary_order=order,
                           on_ibc_tolerance=0.1 * DX * DX) for z in zs])
    return op, op.csr(1)


def _field(kind, op, k, rng):
    d = np.linalg.norm(op.rows()["point"] - np.array([0.6, 0.0, 0.8]), axis=1)[:, None] / DX
    rough = rng.standard_normal((op.D, k))
    if kind == "noise":
        return rough
    if kind == "decay1":
        return np.exp(-d) * (1.0 + 0.0 * rough)
    if kind == "decay0.3":
        return np.exp(-d / 0.3) * (1.0 + 1e-3 * rough)
    if kind == "steep":  # a factor 1e-4 a cell, the first iterates of a solve from a point source
        return np.maximum(10.0 ** (-4.0 * d), 1e-290) * rough
    if kind == "spread":
        return rough * np.exp2(rng.integers(-60, 60, rough.shape).astype(float))
    if kind == "sparse":
        return np.where(rng.random(rough.shape) < 0.97, 0.0, rough)
    lone = np.zeros((op.D, k))  # one value far above the others
    lone[rng.integers(0, op.D, 40)] = 1e8
    return lone + rough


@pytest.mark.parametrize("kind", ["noise", "decay1", "decay0.3", "steep", "spread", "sparse", "lone"])
@pytest.mark.parametrize("k", [1, 32])
def test_e_rows_relative_to_their_terms(op, kind, k):
    import torch

    import cpm_gb300 as cg

    op, (ptr, idx, val) = op
    x = _field(kind, op, k, np.random.default_rng(2))
    d = torch.from_numpy(np.ascontiguousarray(x)).cuda()
    t, y = torch.zeros_like(d), torch.zeros_like(d)
    torch.cuda.synchronize()
    op.apply_device(0.0, -1.0, k, False, d.data_ptr(), t.data_ptr(), y.data_ptr())
    cg.sync()
    t = t.cpu().numpy()
    for s in [0] if k == 1 else [0, 20, 31]:
        term = val.astype(np.longdouble) * x[idx, s]
        ref, size = np.add.reduceat(term, ptr[:-1]), np.add.reduceat(np.abs(term), ptr[:-1])
        err = np.abs(t[:, s] - ref)
        tol = 30 * np.longdouble(2.0) ** -53 * size + 64 * np.longdouble(2.0) ** -1074
        worst = float(np.max(err / np.maximum(size, np.longdouble(2.0) ** -1020)) * 2.0 ** 53)
        assert np.all(err <= tol), (worst, np.count_nonzero(err > tol))
