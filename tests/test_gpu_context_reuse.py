"""One context used for call after call: buffers, the iteration graph and the host's mirror of the states are kept
between calls, and every call gives bit for bit what a fresh context gives."""
import numpy as np
import pytest

from picgo_gb300 import Engine, cg_params, jitter, make_network
from picgo_gb300.network import make_ensemble

pytestmark = pytest.mark.gpu

PARAMS = cg_params(energy_rel_tol=0.0, energy_call_limit=37)


def networks():
    # other sizes, and other graph shapes: no linkers, motors too
    a = jitter(make_network("c1", n_filaments=60, n_cyl_per_filament=12, box=1500.0, n_linkers=80, n_motors=40, seed=3),
               0.3, seed=1)
    b = jitter(make_network("c1", n_filaments=7, n_cyl_per_filament=9, box=1500.0, n_linkers=0, seed=4), 0.3, seed=2)
    c = jitter(make_network("c1", seed=5), 0.3, seed=3)
    return [a, b, c]


def minimized(eng, n=1):
    res = eng.minimize(PARAMS)
    return ([(r["num_iter"], r["num_energy_call"], list(r["energies_before"]), list(r["energies_after"])) for r in res],
            [eng.coords(r) for r in range(n)], [eng.last_forces(r) for r in range(n)])


def same(a, b):
    assert a[0] == b[0]
    for u, v in zip(a[1] + a[2], b[1] + b[2]):
        assert np.array_equal(u, v)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_minimizations_of_one_context_equal_fresh_ones(precision):
    nets = networks()
    fresh = []
    for net in nets:
        with Engine(precision) as eng:
            eng.set_network(net)
            fresh.append(minimized(eng))
    with Engine(precision) as eng:
        for k in (0, 1, 2, 2, 0, 1):
            eng.set_network(nets[k])
            same(minimized(eng), fresh[k])
            eng.reset_coords()
            same(minimized(eng), fresh[k])
            eng.set_graph_mode("conditional" if k else "unrolled")


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_evaluations_after_a_minimization_equal_fresh_ones(precision):
    nets = make_ensemble(3, seed=9, fil_range=(20, 60), cyl_range=(10, 14))
    with Engine(precision) as eng:
        eng.set_networks(nets)
        minimized(eng, 3)
        for r in (2, 0, 0, 1):
            per, total, _ = eng.energies(nets[r].coord, replica=r)
            f = eng.forces(replica=r)
            x = eng.coords(r)
            eng.energies(replica=(r + 1) % 3)
            assert np.array_equal(f, eng.last_forces(r))
            with Engine(precision) as one:
                one.set_network(nets[r])
                want, wtotal, _ = one.energies()
                assert np.allclose(per, want, rtol=1e-12, atol=1e-10) and abs(total - wtotal) <= 1e-12 * abs(wtotal)
                assert np.allclose(f, one.forces(), rtol=1e-12, atol=1e-9)
                assert np.array_equal(x, one.coords())
