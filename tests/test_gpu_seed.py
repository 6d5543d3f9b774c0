"""The seed node of a tube on a triangle mesh: the grid node nearest the closest
point of the grid's first corner, which scans the whole mesh (fewer primitives
than a block, more than the grid of blocks, in between), against the closest
point query of that corner."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("level,dx", [(0, 0.05), (2, 0.04), (3, 0.05), (5, 0.04), (6, 0.03)])
def test_seed_is_the_node_nearest_the_corners_closest_point(level, dx):
    import cpm_gb300 as cg
    from cpm_gb300 import workloads

    v, f = workloads.perturbed_icosphere(level, seed=level)
    d = cg.desc(cg.TRIANGULATION, (), workloads.mesh_bbox(v), verts=v, prims=f)
    tube = cg.Tube(d, 3, dx)
    cp, _ = cg.closest_points(d, np.full((1, 3), tube.xstart))
    want = np.rint((cp[0] - tube.xstart) / dx)
    seed = tube.export()["x"][tube.reference_order()[0]]
    assert np.array_equal(np.rint((seed - tube.xstart) / dx), want)
