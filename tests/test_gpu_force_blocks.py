"""Filament forces are formed in blocks of 253 (FP64) or 254 (mixed) beads, cut wherever they fall: computed for a single
network, listed for the replicas of an ensemble.  Every bead's force is the same operations in both, so the forces agree
bit for bit."""
import numpy as np
import pytest

from picgo_gb300 import Engine, jitter, make_network

pytestmark = pytest.mark.gpu


# (filaments, cylinders per filament): 2, 252 .. 257, 506 .. 512 and 1,265 beads
@pytest.mark.parametrize("filaments,cylinders", [(1, 1), (2, 125), (11, 22), (2, 126), (15, 16), (4, 63), (1, 256),
                                                 (22, 22), (13, 38), (2, 253), (8, 63), (55, 22)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_cut_anywhere_keeps_every_bit(precision, filaments, cylinders):
    cfg = dict(n_filaments=filaments, n_cyl_per_filament=cylinders, box=3000.0, n_linkers=0, shape="chain")
    net = jitter(make_network(cfg, seed=filaments), 0.5, seed=8)
    with Engine(precision) as eng:
        eng.set_network(net)
        alone = eng.forces()
    with Engine(precision) as eng:
        eng.set_networks([net, net])
        both = [eng.forces(replica=r) for r in (0, 1)]
    assert np.isfinite(alone).all() and np.abs(alone).max() > 0
    assert np.array_equal(alone, both[0]) and np.array_equal(alone, both[1])
