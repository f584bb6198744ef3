"""Hessian-vector products where the filament part's blocks of 253 beads begin and end: against central differences of the
forces.  The forces are smooth at these states and of magnitude up to F; with a step h of 1e-4 nm the differences err by
about h^2 |F'''| / 6 and eps F / h: 1e-5 of the largest product leaves a factor of ten."""
import numpy as np
import pytest

from picgo_gb300 import Engine, jitter, make_network

pytestmark = pytest.mark.gpu


# 2, 252 .. 257, 506, 507 and 1,265 beads
@pytest.mark.parametrize("filaments,cylinders", [(1, 1), (2, 125), (11, 22), (2, 126), (15, 16), (4, 63), (1, 256), (22, 22),
                                                 (13, 38), (55, 22)])
def test_hvp_at_block_edges(filaments, cylinders):
    cfg = dict(n_filaments=filaments, n_cyl_per_filament=cylinders, box=6000.0, n_linkers=0, shape="chain")
    net = jitter(make_network(cfg, seed=filaments), 0.5, seed=8)
    net.exvol_cutoff = 1.0   # filament terms (and the boundary's) only
    rng = np.random.default_rng(filaments)
    v = rng.normal(size=net.coord.shape)
    with Engine("fp64") as eng:
        eng.set_network(net)
        hv = eng.hvp(v).reshape(net.coord.shape)
        h = 1e-4
        fp, fm = eng.forces(net.coord + h * v), eng.forces(net.coord - h * v)
    want = -(np.asarray(fp) - np.asarray(fm)).reshape(net.coord.shape) / (2 * h)
    assert np.abs(hv - want).max() <= 1e-5 * np.abs(want).max()
