"""Neighbor lists where their kernels' edges lie: distances and plane distances exactly at the cutoff, cylinders with
more neighbors than are kept from the count, entry counts around the boundary tiles, replicas that share tiles.
Lists are integer-exact against the oracle."""
import numpy as np
import pytest

import oracle
from picgo_gb300 import Engine, make_network

pytestmark = pytest.mark.gpu


def snapped(n_filaments, n_cyl, seed, grid=9.0):
    """A network whose beads sit on a grid: many midpoint distances of exactly 27 nm and plane distances of exactly 100."""
    net = make_network(dict(n_filaments=n_filaments, n_cyl_per_filament=n_cyl, box=900.0, n_linkers=0,
                            shape="chain"), seed=seed)
    net.coord = np.round(net.coord / grid) * grid
    rng = np.random.default_rng(seed)
    net.coord = net.coord + 0.0
    net.cyl_id = rng.permutation(net.n_cyl).astype(np.int64) * 3 + 7
    net.planes[:, 3] -= np.sign(net.planes[:, :3].sum(1)) * 2.0   # planes at 27 nm and box - 23 nm
    return net


def check(eng, net, r=0):
    x = eng.coords(r)
    assert np.array_equal(eng.pairs(r), oracle.cyl_pairs(net, x))
    flat, count = oracle.boundary_list(net, x)
    plane = np.repeat(np.arange(len(count)), count)
    assert np.array_equal(eng.boundary_list(r), np.stack([plane, flat], 1))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("shape", [(1, 1), (17, 10), (32, 16), (41, 25), (205, 20)])
@pytest.mark.parametrize("cutoff,cell", [(27.0, 0.0), (27.0, 27.0), (140.0, 0.0)])
def test_lists_at_ties_and_tile_edges(precision, shape, cutoff, cell):
    net = snapped(*shape, seed=3)
    net.exvol_cutoff = cutoff
    with Engine(precision) as eng:
        eng.set_network(net)
        eng.rebuild(cell)
        check(eng, net)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_lists_of_replicas_sharing_tiles(precision):
    nets = [snapped(*s, seed=20 + k) for k, s in enumerate([(3, 5), (17, 10), (1, 1), (52, 20)])]
    nets[1].exvol_cutoff = 81.0
    with Engine(precision) as eng:
        eng.set_networks(nets)
        for r, net in enumerate(nets):
            check(eng, net, r)
