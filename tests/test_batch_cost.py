"""The costs that decide between one by one and a batch follow the surface's size
(no GPU: the function is host code), and the serving rules read them."""
import numpy as np
import pytest

MEASURED = {  # kind: (rows, cost of 32 in units of one)
    0: [(14626, 4.71), (39153, 7.11), (106926, 10.17), (215662, 14.45), (762158, 21.57)],
    1: [(14626, 2.72), (39153, 2.81), (106926, 3.31), (215662, 3.91), (762158, 4.77)],
    2: [(10906, 8.8), (41870, 10.6), (166390, 13.8), (260062, 18.8), (1300000, 31.7)],
}


@pytest.mark.parametrize("kind", list(MEASURED))
def test_costs_follow_the_measurements(kind):
    import cpm_gb300 as cg

    for rows, cost in MEASURED[kind]:
        assert abs(cg.batch_cost(rows, kind) - cost) <= 0.2 * cost
    sizes = [cg.batch_cost(int(n), kind) for n in np.geomspace(1, 1e8, 60)]
    assert all(a <= b for a, b in zip(sizes, sizes[1:])) and sizes[0] >= 1.0
    assert cg.batch_cost(1000, 3) == 0.0


def test_geodesics_wait_for_their_surfaces_break_even():
    from cpm_gb300 import serving as SV

    small, large = object.__new__(SV.ServedSurface), object.__new__(SV.ServedSurface)
    small.geo_batch_min, large.geo_batch_min = 9, 32
    loop = object.__new__(SV.ServingLoop)
    loop.geodesic_batch_min = None
    waiting = list(range(20))
    assert loop._geo_take(small, waiting) == waiting and loop._geo_take(large, waiting) == [0]
    loop.geodesic_batch_min = 4
    assert loop._geo_take(large, waiting) == waiting
