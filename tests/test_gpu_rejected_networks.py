"""A network that mech_set_networks rejects leaves its context without one: nothing may run on the buffers of the
network before it, whose sizes the rejected one has replaced, and the next network is as good as in a fresh context."""
import copy

import numpy as np
import pytest

from picgo_gb300 import Engine, _lib, cg_params, jitter, make_network

pytestmark = pytest.mark.gpu

ERR_ARG, ERR_TOPOLOGY, ERR_STATE = -1, -2, -9


def small():
    return jitter(make_network("c1", n_filaments=24, n_cyl_per_filament=10, box=1400.0, n_linkers=40), 0.3,
                  seed=1)


def rejected(what):
    big = make_network("c1", n_filaments=300, n_cyl_per_filament=20, box=3000.0, n_linkers=100, n_motors=10, seed=2)
    linker = copy.deepcopy(big)
    linker.lk_cyl[3, 1] = big.n_cyl
    motor = copy.deepcopy(big)
    motor.mt_cyl[0, 0] = -1
    chain = copy.deepcopy(big)
    chain.cyl_b1[5] = big.cyl_b1[25]
    return {"linker": [linker], "motor": [motor], "chain": [chain], "last of more replicas": [small()] * 40 + [linker]}[what]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("what", ["linker", "motor", "chain", "last of more replicas"])
def test_context_after_a_rejected_network(precision, what):
    p = cg_params(energy_rel_tol=0.0, energy_call_limit=30)
    with Engine(precision) as fresh:
        fresh.set_network(small())
        want = fresh.minimize(p)[0], fresh.coords()
    with Engine(precision) as eng:
        eng.set_network(small())
        eng.minimize(p)
        with pytest.raises(_lib.MechError) as e:
            eng.set_networks(rejected(what))
        assert e.value.code in (ERR_ARG, ERR_TOPOLOGY)
        x = np.zeros((10_000, 3))
        calls = [lambda: eng.energies(), lambda: eng.energies(x), lambda: eng.forces(x), lambda: eng.coords(),
                 lambda: eng.set_coords(x), lambda: eng.rebuild(), lambda: eng.pairs(), lambda: eng.minimize(p),
                 lambda: eng.last_forces(), lambda: eng.stretch_forces(), lambda: eng.reset_coords(),
                 lambda: eng.hvp(x), lambda: eng.adjoint(x), lambda: eng.newton_refine(), lambda: eng.autotune(),
                 lambda: eng.profile(1), lambda: eng.load_forces(), lambda: eng.energy_terms(),
                 lambda: eng.set_linker_params(k=np.ones(40)), lambda: eng.boundary_list()]
        for call in calls:
            with pytest.raises(_lib.MechError) as e:
                call()
            assert e.value.code == ERR_STATE
        eng.set_network(small())
        got = eng.minimize(p)[0], eng.coords()
        assert got[0]["num_iter"] == want[0]["num_iter"] and list(got[0]["energies_after"]) == list(want[0]["energies_after"])
        assert np.array_equal(got[1], want[1])
