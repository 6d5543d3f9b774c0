"""Closest points on meshes and polylines, whose search passes primitives over by
FP32 spheres, against an FP64 scan of every primitive: points on vertices, edges
and the surface (equally near primitives), near it, far outside, bounded and
unbounded searches, and a mesh far from the origin, where FP32 has few bits left."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _distance(v, f, x):
    """|x - nearest point| of every point to the triangles or segments f, exact up to FP64 rounding"""
    best = np.full(len(x), np.inf)
    for t in f:
        p = v[t]
        edges = [(0, 1)] if len(t) == 2 else [(0, 1), (1, 2), (2, 0)]
        for a, b in edges:
            d = p[b] - p[a]
            s = np.clip(((x - p[a]) @ d) / (d @ d), 0.0, 1.0)
            best = np.minimum(best, np.linalg.norm(x - (p[a] + s[:, None] * d), axis=1))
        if len(t) == 3:
            n = np.cross(p[1] - p[0], p[2] - p[0])
            h = ((x - p[0]) @ n) / (n @ n)
            q = x - h[:, None] * n
            inside = np.ones(len(x), bool)
            for a, b in edges:
                inside &= np.cross(p[b] - p[a], q - p[a]) @ n >= 0
            best = np.where(inside, np.minimum(best, np.abs(h) * np.linalg.norm(n)), best)
    return best


@pytest.mark.parametrize("shift", [0.0, 300.0])
@pytest.mark.parametrize("shape", ["mesh", "curve"])
def test_culled_search_finds_the_nearest(shape, shift):
    import cpm_gb300 as cg
    from cpm_gb300 import workloads

    v, f = workloads.perturbed_icosphere(2, seed=4)
    rng = np.random.default_rng(8)
    if shape == "curve":
        v, f = workloads.parallel_plane_curves(v, f, 1, seed=2)[0][0]
    kind = cg.TRIANGULATION if shape == "mesh" else cg.POLYLINE
    mid = v[f].mean(axis=1)
    x = np.concatenate([v[:40], mid[:40], 0.5 * (v[f[:40, 0]] + v[f[:40, 1]]), mid[:60] + 0.02 * rng.standard_normal((len(mid[:60]), 3)),
                        1.5 * rng.standard_normal((60, 3)), np.zeros((1, 3))])
    want = _distance(v, f, x)
    bb = workloads.mesh_bbox(v + shift)
    for max_dist in (0.0, 0.1):
        d = cg.desc(kind, (), bb, verts=v + shift, prims=f)
        cp, dist = cg.closest_points(d, x + shift, max_dist)
        # more points than are searched by a warp each: near each other 32 at a time, then scattered
        for many in (np.repeat(np.arange(len(x)), 160), np.tile(np.arange(len(x)), 160)):
            cpm, distm = cg.closest_points(d, (x + shift)[many], max_dist)
            ok = dist[many] <= (max_dist or np.inf)
            assert np.array_equal(distm[ok], dist[many][ok]) and np.array_equal(cpm[ok], cp[many][ok])
            assert np.all(distm[~ok] > max_dist)
        near = np.ones(len(x), bool) if max_dist == 0.0 else want <= max_dist
        tol = 1e-13 + 4 * shift * 2.0 ** -52 * 4
        assert np.all(np.abs(dist - want)[near] <= tol), np.max(np.abs(dist - want)[near])
        assert np.all(dist[~near] > max_dist)
        assert np.all(np.abs(np.linalg.norm(x + shift - cp, axis=1) - dist)[near] <= tol)
