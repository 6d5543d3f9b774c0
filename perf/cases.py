"""The work that a user of this framework has it do, as cases to be timed.

Each case goes through the package's public classes (Tube, OpSet, Solver,
Server, Geodesic): applies of the closest-point operator (one vector or a
32-slot batch, FP32 or FP64, device arrays), solves of one or 32 right-hand
sides (plain FP64 or FP32 with FP64 reliable updates), requests through the
continuous-batching server, a heat-method geodesic, implicit heat steps on host
vectors, and the set-up of a new geometry.  Sizes are those of the tests and of
the benchmark: the unit sphere (two circles), the torus R = 1, r = 0.4 (outer
and inner equators) and a perturbed icosphere (parallel plane cuts).
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "cpm-ibc_gb300", "python"))

import cpm_gb300 as cg  # noqa: E402
from cpm_gb300 import workloads  # noqa: E402

TOL = 1e-10


# ---------------------------------------------------------------- the cases

def listed():
    return [
        # the smallest call: one operator product on a coarse tube, as an explicit loop of a user's own makes it
        dict(name="apply_f64_1_sphere_0.1", kind="apply", surface="sphere", dx=0.1, curves=2, order=2, slots=1, f32=False),
        # one vector on the largest tube of the configurations (1.4 M rows)
        dict(name="apply_f64_1_torus_0.01", kind="apply", surface="torus", dx=0.01, curves=2, order=2, slots=1, f32=False),
        # the inner operator of the served batches at the benchmark's size
        dict(name="apply_f32_32_sphere_0.025", kind="apply", surface="sphere", dx=0.025, curves=2, order=2, slots=32, f32=True),
        # the same on the largest tube, first-order IBCs
        dict(name="apply_f32_32_torus_0.01", kind="apply", surface="torus", dx=0.01, curves=2, order=1, slots=32, f32=True),
        # the FP64 batch: true residuals of the mixed path, the FP64 server and batched geodesics
        dict(name="apply_f64_32_sphere_0.025", kind="apply", surface="sphere", dx=0.025, curves=2, order=2, slots=32, f32=False),
        # a small solve: implicit heat steps from and to host vectors, where latency and launches count
        dict(name="heat_sphere_0.1", kind="heat", surface="sphere", dx=0.1, curves=2, order=2),
        # one request alone in FP64 (the reference's algorithm; the benchmark's plain path)
        dict(name="solve_f64_1_sphere_0.025", kind="solve", surface="sphere", dx=0.025, curves=2, order=2, slots=1, k=1, mixed=False),
        # a batch that FP32 inner iterations cannot follow at its finer sizes: FP64 throughout
        dict(name="solve_f64_32_torus_0.04", kind="solve", surface="torus", dx=0.04, curves=2, order=2, slots=32, k=32, mixed=False),
        # a ragged static batch, FP32 with FP64 reliable updates
        dict(name="solve_mixed_27_sphere_0.05", kind="solve", surface="sphere", dx=0.05, curves=2, order=2, slots=32, k=27, mixed=True),
        # the headline: requests through the continuous-batching server, two batches, device-resident
        dict(name="serve_mixed_64_sphere_0.025", kind="serve", surface="sphere", dx=0.025, curves=2, order=2, k=64, batches=2),
        # one heat-method geodesic: 2000 Jacobi sweeps per preconditioner call, then three Poisson solves
        dict(name="geodesic_sphere_0.05", kind="geodesic", surface="sphere", dx=0.05),
        # a new geometry: tube and operator of a triangle mesh with four polyline IBCs, and the rows that plot a
        # solution at the mesh's vertices
        dict(name="setup_mesh_0.02", kind="setup", surface="mesh", dx=0.02, curves=4, order=2, level=5),
    ]


def _log(rng, lo, hi):
    return round(math.exp(rng.uniform(math.log(lo), math.log(hi))), 5)


def draw(rng):
    kind = rng.choice(["apply"] * 5 + ["solve"] * 4 + ["heat", "serve", "geodesic", "setup"])
    if kind == "apply":
        surface = rng.choice(["sphere", "torus"])
        return dict(kind=kind, surface=surface, dx=_log(rng, 0.0125 if surface == "sphere" else 0.011, 0.12),
                    curves=rng.choice([0, 1, 2]), order=rng.choice([1, 2]), slots=rng.choice([1, 32]), f32=rng.random() < 0.5)
    if kind == "solve":
        surface = rng.choice(["sphere", "torus"])
        slots = rng.choice([1, 32])
        # the torus is left to FP64, as the serving rules do
        return dict(kind=kind, surface=surface, dx=_log(rng, 0.03 if slots == 1 else 0.045, 0.12), curves=2,
                    order=rng.choice([1, 2]), slots=slots, k=1 if slots == 1 else rng.randint(2, 32),
                    mixed=surface == "sphere" and rng.random() < 0.6)
    if kind == "heat":
        return dict(kind=kind, surface="sphere", dx=_log(rng, 0.04, 0.15), curves=rng.choice([1, 2]), order=2)
    if kind == "serve":
        return dict(kind=kind, surface="sphere", dx=_log(rng, 0.04, 0.1), curves=2, order=2, k=rng.randint(33, 90),
                    batches=rng.choice([1, 2]))
    if kind == "geodesic":
        return dict(kind=kind, surface="sphere", dx=_log(rng, 0.055, 0.15))
    return dict(kind=kind, surface="mesh", dx=_log(rng, 0.02, 0.05), curves=rng.randint(1, 4), order=2, level=rng.choice([4, 5]))


# ---------------------------------------------------------------- geometry

def _curves(case):
    """(centre height, radius) of the circles: parallels of the sphere, equators of the torus"""
    if case["surface"] == "sphere":
        c = [(z, math.sqrt(1 - z * z)) for z in (0.3, -0.5)]
    else:
        c = [(0.0, 1.4), (0.0, 0.6)]
    return c[:case.get("curves", 0)]


def _surface(case):
    if case["surface"] == "sphere":
        return cg.desc(cg.SPHERE, [1.0]), (-1.0, 1.0)
    bb = (-1.4, 1.4)
    return cg.desc(cg.TORUS, [1.0, 0.4], bb), bb


def _operator(case):
    dx = case["dx"]
    s, bb = _surface(case)
    tube = cg.Tube(s, 3, dx)
    ibcs = [cg.desc(cg.CIRCLE3D, [R, 0, 0, z, 0, 0, 1], bb, boundary_order=case["order"], on_ibc_tolerance=0.1 * dx * dx)
            for z, R in _curves(case)]
    return cg.OpSet(tube, ibcs)


def _dirichlet(rows):
    """rows that carry a curve's value: the Dirichlet value rows of second-order IBCs, the DOF rows of first-order ones"""
    return (rows["kind"] == 2) if (rows["kind"] == 2).any() else ((rows["kind"] > 0) & rows["identity"])


def _laplace_rhs(rows, vals):
    """Laplace with the value vals[c] on curve c"""
    b = np.zeros(len(rows["kind"]))
    d = _dirichlet(rows)
    b[d] = vals[rows["ibc"][d]]
    return b


def _rng(seed):
    return np.random.default_rng(seed)


def _field(points, k, seed, dtype):
    """[D][k] vectors as a Krylov iteration meets them: a smooth field of each slot and a rough part"""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    p = torch.from_numpy(points).cuda()
    wave = 2.0 * torch.randn((3, k), generator=g, device="cuda", dtype=torch.float64)
    phase = 6.0 * torch.rand((1, k), generator=g, device="cuda", dtype=torch.float64)
    x = torch.sin(p @ wave + phase) + 0.1 * torch.randn((len(points), k), generator=g, device="cuda", dtype=torch.float64)
    return x.to(dtype).contiguous()


def _source(seed):
    v = _rng(seed).standard_normal(3)
    return v / np.linalg.norm(v)


def _mesh(case, seed):
    v, f = workloads.perturbed_icosphere(case["level"], seed=seed)
    curves, _ = workloads.parallel_plane_curves(v, f, case["curves"], seed=seed + 1)
    return v, f, curves


def _heat_rhs(case, rows, seed):
    """a smooth temperature on every row, the curves' values on theirs"""
    r = _rng(seed)
    b = np.cos(rows["point"] @ (2.0 * r.standard_normal(3)) + 6.0 * r.random())
    d = _dirichlet(rows)
    b[d] = r.uniform(0, 1, 2)[rows["ibc"][d]]
    return b


def _heat_dt(case):
    return 0.1 * case["dx"]


def _values(case, seed):
    return _rng(seed).uniform(0, 1, size=(case["k"], 2))


# ---------------------------------------------------------------- one case

def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind == "setup":
        dx = case["dx"]
        v, f, curves = _mesh(case, seed)
        bb = workloads.mesh_bbox(v)
        s["surface"] = cg.desc(cg.TRIANGULATION, (), bb, verts=v, prims=f)
        s["vertices"] = v
        s["ibcs"] = [cg.desc(cg.POLYLINE, (), bb, boundary_order=case["order"], on_ibc_tolerance=0.1 * dx * dx, verts=p, prims=q)
                     for p, q in curves]
        return s
    if kind == "geodesic":
        s["tube"] = cg.Tube(_surface(case)[0], 3, case["dx"])
        s["geodesic"] = cg.Geodesic(s["tube"], _source(seed))
        return s
    op = s["op"] = _operator(case)
    rows = op.rows()
    if kind == "apply":
        s["x"] = _field(rows["point"], case["slots"], seed, torch.float32 if case["f32"] else torch.float64)
        s["t"], s["y"] = torch.empty_like(s["x"]), torch.empty_like(s["x"])
    elif kind == "heat":
        s["solver"] = cg.Solver(op, 1.0, -_heat_dt(case))
        s["b"] = _heat_rhs(case, rows, seed)
    elif kind == "solve":
        s["solver"] = cg.Solver(op, 0.0, -1.0, kslots=case["slots"])
        b = np.zeros((op.D, case["slots"]))
        for j, v in enumerate(_values(case, seed)):
            b[:, j] = _laplace_rhs(rows, v)
        s["b"] = torch.from_numpy(b).cuda()
        s["x"] = torch.zeros_like(s["b"])
    else:
        s["server"] = cg.Server(op, 0.0, -1.0, tol=TOL, batches=case["batches"])
        s["b"] = torch.from_numpy(np.stack([_laplace_rhs(rows, v) for v in _values(case, seed)])).cuda()
        s["x"] = torch.zeros_like(s["b"])
    torch.cuda.synchronize()  # the library's stream does not wait for torch's
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "apply":
        s["op"].apply_device(0.0, -1.0, case["slots"], case["f32"], s["x"].data_ptr(), s["t"].data_ptr(), s["y"].data_ptr())
        return s["y"]
    if kind == "heat":
        return s["solver"].solve(s["b"], tol=TOL)[0]
    if kind == "solve":
        s["solver"].solve_device(s["b"].data_ptr(), s["x"].data_ptr(), case["k"], tol=TOL, precision=int(case["mixed"]))
        return s["x"][:, :case["k"]]
    if kind == "serve":
        for j in range(case["k"]):
            s["server"].submit_device(s["b"][j].data_ptr(), s["x"][j].data_ptr(), j)
        s["server"].drain(want_x=False)
        return s["x"]
    if kind == "geodesic":
        # the distance on the tube's rows (the DOF rows behind them differ in number from source to source)
        return s["geodesic"].run(case["dx"] ** 2, tol=TOL)[0][:s["tube"].N]
    tube = cg.Tube(s["surface"], 3, case["dx"])
    op = cg.OpSet(tube, s["ibcs"])
    return [*tube.interp_query(s["vertices"]), op.D, op.N, op.n_patched, op.n_moved, op.n_patch_entries]


# ---------------------------------------------------------------- what a pass cannot do without

def _rows(case):
    """rows of the operator: the tube band is 8.25 dx wide (radius 4.123 dx), an IBC's band has radius 4.123 dx
    about the curve; second-order IBCs add a value row to every DOF row"""
    dx, band = case["dx"], 4.1235
    area = {"sphere": 4 * math.pi, "torus": 4 * math.pi ** 2 * 0.4, "mesh": 3.1}[case["surface"]]
    length = 2.2 * case.get("curves", 0) if case["surface"] == "mesh" else sum(2 * math.pi * R for _, R in _curves(case))
    return 2 * band * area / dx ** 2 + case.get("order", 1) * math.pi * band ** 2 * length / dx


APPLY_FLOPS = 2 * 84 + 18  # a row: tricubic interpolation (64 + 16 + 4 multiply-adds), seven-point row
VECTOR_FLOPS = 22          # a row of the Krylov vector updates and dots


def work(case):
    D, kind = _rows(case), case["kind"]
    if kind == "apply":
        e = 4 if case["f32"] else 8
        return dict(bytes=D * (4 + 12 * e + 2 * e * case["slots"]), flops=D * case["slots"] * APPLY_FLOPS)
    if kind == "setup":
        return dict(bytes=D * (24 + 8 + 96 + 4 + 24), flops=D * 400)
    k = case.get("k", 1)
    if kind == "geodesic":  # heat: two iterations of 2 x 2000 sweeps; three Poisson solves; products of the rounds
        iters = 2 * 2000 + 3 * 10 / case["dx"]
    elif kind == "heat":
        iters = 0.8 / math.sqrt(case["dx"]) + 10
    else:
        iters = 6.1 / case["dx"]
    return dict(bytes=D * (4 + 96 + 16 * k), flops=iters * k * D * (2 * APPLY_FLOPS + VECTOR_FLOPS))


# ---------------------------------------------------------------- 64-bit values

class _Rows:
    """The operator's rows (its exported Lfull and Efull matrices) as data, and A x = m x + n (diag(L) x + offdiag(L) E x),
    identity rows A x = x, in plain torch."""

    def __init__(self, op, m, n):
        ident = torch.from_numpy(op.rows()["identity"]).cuda()
        ptr, idx, val = (torch.from_numpy(a).cuda() for a in op.csr(0))
        row = torch.repeat_interleave(torch.arange(op.D, device="cuda"), ptr[1:] - ptr[:-1])
        diag = torch.zeros(op.D, dtype=torch.float64, device="cuda")
        diag[row[idx == row]] = val[idx == row]
        val = torch.where((idx == row) | ident[row], 0.0, val)
        self.off = torch.sparse_csr_tensor(ptr, idx, n * val, (op.D, op.D))
        self.diag = torch.where(ident, 1.0, m + n * diag)[:, None]
        ptr, idx, val = (torch.from_numpy(a).cuda() for a in op.csr(1))
        self.e = torch.sparse_csr_tensor(ptr, idx, val, (op.D, op.D))

    def __call__(self, x):
        return self.diag * x + self.off @ (self.e @ x)

    def solve(self, b):
        """BiCGStab with the inverse diagonal, repeated on the true residual until it stays"""
        x, last = torch.zeros_like(b), math.inf
        for _ in range(6):
            r = b - self(x)
            now = float(r.norm() / b.norm())
            if now > 0.2 * last or now == 0.0:
                break
            last = now
            x = x + self._bicgstab(r, 1e-9)
        return x

    def _bicgstab(self, b, tol, most=2000):
        def dot(u, v):
            return (u * v).sum(0, keepdim=True)

        def div(u, v):
            return torch.where(v == 0, 0.0, u / torch.where(v == 0, 1.0, v))

        x, r, p, v = torch.zeros_like(b), b.clone(), torch.zeros_like(b), torch.zeros_like(b)
        r0 = r.clone()
        rho = alpha = omega = torch.ones((1, b.shape[1]), dtype=b.dtype, device=b.device)
        goal = (tol * tol) * dot(b, b)
        for _ in range(most):
            new = dot(r0, r)
            fresh = new.abs() < 1e-28 * dot(r0, r0)
            r0 = torch.where(fresh, r, r0)
            new = torch.where(fresh, dot(r, r), new)
            p = torch.where(fresh, r, r + div(new, rho) * div(alpha, omega) * (p - omega * v))
            rho = new
            y = p / self.diag
            v = self(y)
            alpha = div(rho, dot(r0, v))
            s = r - alpha * v
            z = s / self.diag
            t = self(z)
            omega = div(dot(t, s), dot(t, t))
            live = dot(r, r) > goal
            x = torch.where(live, x + alpha * y + omega * z, x)
            r = torch.where(live, s - omega * t, r)
            if not bool(live.any()):
                break
        return x


def exact(case, seed):
    kind = case["kind"]
    if kind in ("setup", "geodesic") or _rows(case) > 6e5:  # no closed value, or the exported rows alone take too long
        return None
    op = _operator(case)
    rows = op.rows()
    if kind == "apply":
        return _Rows(op, 0.0, -1.0)(_field(rows["point"], case["slots"], seed, torch.float32 if case["f32"] else torch.float64).double())
    if kind == "heat":
        b = torch.from_numpy(_heat_rhs(case, rows, seed)).cuda()[:, None]
        return _Rows(op, 1.0, -_heat_dt(case)).solve(b).T
    # the right-hand sides are combinations of the curves' own
    b = np.stack([_laplace_rhs(rows, e) for e in np.eye(2)], axis=1)
    x = _Rows(op, 0.0, -1.0).solve(torch.from_numpy(b).cuda()) @ torch.from_numpy(_values(case, seed)).cuda().T
    return x if kind == "solve" else x.T
