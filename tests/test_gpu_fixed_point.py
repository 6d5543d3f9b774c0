"""E x of FP64 vectors (summed in 64-bit fixed point aligned to each stencil)
against the exported Efull rows in extended precision, for one vector and for
32 slots, at the ranges of values where alignment can go wrong.

Tolerance, in units of 2^-52 of the largest value a row reads: the fixed-point
row is off by at most 1.5 units of its last bit, 2^-54 (0.4), and its conversion
to FP64 by 2^-53 of a sum of at most 1.95 (1.0); the exported weight products
are rounded twice (2.0).  Rows that take the FP64 sum (values outside the
exponent range, 2^-895 to 2^1023) round at most 12 times (12)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DX = 0.1


def _circle(cg, z, order):
    return cg.desc(cg.CIRCLE3D, [np.sqrt(1 - z * z), 0, 0, z, 0, 0, 1], (-1.0, 1.0), boundary_order=order,
                   on_ibc_tolerance=0.1 * DX * DX)


CURVES = {"plain": ((), 1), "order1": ((0.3, -0.5), 1), "order2": ((0.3, -0.5), 2), "close": ((0.3, 0.36), 2)}


def _inputs(kind, n, k, rng):
    x = rng.standard_normal((n, k))
    if kind == "smooth":
        x = np.cos(np.linspace(0, 6, n))[:, None] + 0.01 * np.arange(k)
    elif kind == "spread":
        x *= np.exp2(rng.integers(-60, 60, (n, k)).astype(float))
    elif kind == "sparse":
        x[rng.random((n, k)) < 0.97] = 0.0
    elif kind == "huge":
        x *= 2.0 ** 1018
    elif kind == "tiny":
        x *= 2.0 ** -1030
    elif kind == "edge":  # around the smallest exponent that is aligned to
        x *= np.exp2(rng.integers(-905, -885, (n, k)).astype(float))
    elif kind == "one":
        x = np.zeros((n, k))
        x[rng.integers(0, n, k), np.arange(k)] = 1.0
    return x


def _e(op, x, m=0.0, n=-1.0, whole=False):
    """E~x of [D][k] (whole: and A x) through the device apply"""
    import torch

    import cpm_gb300 as cg

    d = torch.from_numpy(np.ascontiguousarray(x)).cuda()
    t, y = torch.zeros_like(d), torch.zeros_like(d)
    torch.cuda.synchronize()
    op.apply_device(m, n, x.shape[1], False, d.data_ptr(), t.data_ptr(), y.data_ptr())
    torch.cuda.synchronize()
    cg.sync()
    return (t.cpu().numpy(), y.cpu().numpy()) if whole else t.cpu().numpy()


def _reference(rows, x):
    """per row: the sum in extended precision, and the largest value read"""
    ptr, idx, val = rows
    ref = np.empty((len(ptr) - 1, x.shape[1]), np.longdouble)
    big = np.empty(ref.shape)
    for s in range(x.shape[1]):
        v = x[idx, s]
        ref[:, s] = np.add.reduceat(val.astype(np.longdouble) * v, ptr[:-1])
        big[:, s] = np.maximum.reduceat(np.abs(v), ptr[:-1])
    return ref, big


@pytest.fixture(scope="module", params=list(CURVES))
def op(request):
    import cpm_gb300 as cg

    zs, order = CURVES[request.param]
    op = cg.OpSet(cg.Tube(cg.desc(cg.SPHERE, [1.0]), 3, DX), [_circle(cg, z, order) for z in zs])
    return op, op.csr(1)


@pytest.mark.parametrize("kind", ["smooth", "rough", "spread", "sparse", "one", "huge", "tiny", "edge"])
@pytest.mark.parametrize("k", [1, 32])
def test_e_rows(op, kind, k):
    op, rows = op
    x = _inputs(kind, op.D, k, np.random.default_rng(3))
    cols = [0] if k == 1 else [0, 31]
    t = _e(op, x)[:, cols]
    ref, big = _reference(rows, x[:, cols])
    units = 16.0 if kind in ("huge", "tiny", "edge") else 4.0
    tol = units * 2.0 ** -52 * big + (2.0 ** -1070 if kind == "tiny" else 0.0)  # subnormal results: a few of the smallest
    err = np.abs((t - ref).astype(np.float64))
    assert np.all(err <= tol), (np.max(err / np.maximum(tol, 5e-324)), np.count_nonzero(err > tol))


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("k", [1, 32])
def test_non_finite_values_stay_in_their_rows(op, bad, k):
    op, (ptr, idx, val) = op
    rng = np.random.default_rng(7)
    x = rng.standard_normal((op.D, k))
    where = rng.integers(0, op.D, 5)
    clean = x.copy()
    clean[where, 0] = 0.0
    x[where, 0] = bad
    t, tc = _e(op, x), _e(op, clean)
    hit = np.add.reduceat(np.abs(val) * np.isin(idx, where), ptr[:-1]) > 0
    assert not np.any(np.isfinite(t[hit, 0]))
    fine = np.isfinite(t[:, 0])
    # the batched pass corrects its bulk sums for moved columns: there a row may read a replaced one
    assert k == 32 or np.all(fine[~hit])
    assert np.allclose(t[fine, 0], tc[fine, 0], rtol=0, atol=64 * 2.0 ** -52 * 5)
    assert np.array_equal(t[:, 1:], tc[:, 1:])


@pytest.mark.parametrize("kind", ["smooth", "rough", "spread", "sparse", "large", "tiny", "low"])
@pytest.mark.parametrize("k", [1, 32])
@pytest.mark.parametrize("m,n", [(0.0, -1.0), (1.0, -0.37), (0.5, 0.0), (0.0, 2.0 ** -80)])
def test_l_rows(op, kind, k, m, n):
    """A x from the device's own E~x.  The two coefficients, the product with x, the sum's
    conversion and the result are rounded once each, the FP64 sum of six at most five times:
    4 units of 2^-52 of |c0 x| + |c1| sum |t|."""
    op, _ = op
    rng = np.random.default_rng(5)
    x = _inputs(kind if kind not in ("large", "low") else "rough", op.D, k, rng)
    if kind == "large":
        x *= 2.0 ** 960
    if kind == "low":  # around the smallest exponent that the row's sum is aligned to
        x *= np.exp2(rng.integers(-835, -810, x.shape).astype(float))
    t, y = _e(op, x, m, n, whole=True)
    ptr, idx, val = op.csr(0)
    row = np.repeat(np.arange(op.D), np.diff(ptr))
    ident = op.rows()["identity"]
    for s in ([0] if k == 1 else [0, 17]):
        xs, ts = x[:, s].astype(np.longdouble), t[:, s].astype(np.longdouble)
        diag = idx == row
        term = np.where(diag, (m + n * val) * xs[idx], n * val * ts[idx])  # m on the diagonal
        ref = np.where(ident, xs, np.add.reduceat(term, ptr[:-1]))
        big = np.add.reduceat(np.abs(term), ptr[:-1]).astype(float)
        err = np.abs((y[:, s] - ref).astype(float))
        assert np.all(err <= 4 * 2.0 ** -52 * big + 2.0 ** -1070), np.max(err / np.maximum(big, 5e-324)) * 2.0 ** 52


@pytest.mark.parametrize("k", [1, 32])
def test_l_rows_pass_on_non_finite_values(op, k):
    op, _ = op
    x = np.random.default_rng(9).standard_normal((op.D, k))
    x[op.D // 3, 0] = np.inf
    t, y = _e(op, x, whole=True)
    ptr, idx, val = op.csr(0)
    row = np.repeat(np.arange(op.D), np.diff(ptr))
    ident = op.rows()["identity"]
    reads = np.where(idx == row, x[idx, 0], t[idx, 0])
    bad = (np.add.reduceat((~np.isfinite(reads)).astype(int), ptr[:-1]) > 0) & ~ident
    assert np.array_equal(~np.isfinite(y[:, 0]), bad | (ident & ~np.isfinite(x[:, 0])))
