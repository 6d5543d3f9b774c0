"""A tube around a mesh of few large triangles: its candidate bricks are those along
the faces, as around the same surface in small triangles, so the two builds give
the same tube and take comparable times.  (Bricks picked by the triangles' bounding
spheres alone fill the inside: five times as long for the tetrahedron.)"""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _split(v, f, times):
    for _ in range(times):
        a, b, c = v[f[:, 0]], v[f[:, 1]], v[f[:, 2]]
        n, m = len(v), len(f)
        i = np.arange(m)
        v = np.concatenate([v, 0.5 * (a + b), 0.5 * (b + c), 0.5 * (c + a)])
        ab, bc, ca = n + i, n + m + i, n + 2 * m + i
        f = np.concatenate([np.stack(t, 1) for t in ((f[:, 0], ab, ca), (ab, f[:, 1], bc), (ca, bc, f[:, 2]), (ab, bc, ca))])
    return v, f


def test_coarse_and_split_mesh_alike():
    import cpm_gb300 as cg

    v = np.array([[1, 1, 1], [1, -1, -1], [-1, 1, -1], [-1, -1, 1]], float)
    f = np.array([[0, 1, 2], [0, 3, 1], [0, 2, 3], [1, 3, 2]])
    tubes, best = [], []
    for times in (0, 4):
        vv, ff = _split(v, f, times)
        d = cg.desc(cg.TRIANGULATION, (), (-1.0, 1.0), verts=vv, prims=ff)
        t = []
        for _ in range(4):
            t0 = time.perf_counter()
            tube = cg.Tube(d, 3, 0.015)
            cg.sync()
            t.append(time.perf_counter() - t0)
        tubes.append(tube.export())
        best.append(min(t))
    assert np.array_equal(tubes[0]["x"], tubes[1]["x"])
    assert np.max(np.abs(tubes[0]["dist"] - tubes[1]["dist"])) <= 1e-13  # coordinates of order 1, some 100 roundings
    assert best[0] <= 2.0 * best[1], best
