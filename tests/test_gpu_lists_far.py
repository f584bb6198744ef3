"""Neighbor lists of a network far from the origin, where single-precision midpoints are coarser than the slack of the
single-precision decisions: beads on a grid, many midpoint distances exactly at the cutoff, lists integer-exact against
the oracle."""
import numpy as np
import pytest

import oracle
from picgo_gb300 import Engine
from test_gpu_lists import snapped

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("offset", [0.0, 13_500.0, 900_000.0, -90_000_000.0])
@pytest.mark.parametrize("axes", [(1, 0, 0), (0, 1, 1)])
def test_pairs_far_from_the_origin(precision, offset, axes):
    net = snapped(41, 25, seed=3)
    net.coord = net.coord + offset * np.array(axes, float)
    with Engine(precision) as eng:
        eng.set_network(net)
        x = eng.coords()
        assert np.array_equal(x, net.coord)
        want = oracle.cyl_pairs(net, x)
        assert len(want) == 95
        assert np.array_equal(eng.pairs(), want)
