"""The two forms of the FP64 force gather (a bead per thread; the components of the beads with contributions spread over
a warp) add the same contributions in the same order: a network's forces and the reductions over them keep every bit when
it is evaluated alone and as one of replicas with 608 tiles or more between them."""
import numpy as np
import pytest

from picgo_gb300 import Engine, cg_params, jitter, make_network

pytestmark = pytest.mark.gpu

LIMIT = 608   # tiles from which the spread form is taken


def network(n_filaments, seed, linkers):
    cfg = dict(n_filaments=n_filaments, n_cyl_per_filament=12, box=520.0, n_linkers=linkers, shape="chain")
    net = jitter(make_network(cfg, seed=seed), 0.3, seed=2)
    net.exvol_cutoff = 70.0
    return net


@pytest.mark.parametrize("replicas", [LIMIT - 1, LIMIT, LIMIT + 3])
def test_gather_forms_agree_bit_for_bit(replicas):
    # no contribution at all, some beads with a few, beads with more than are loaded together
    nets = [network(1, 31, 0), network(6, 32, 2), network(16, 33, 40)]
    params = cg_params(energy_rel_tol=0.0, energy_call_limit=6, force_call_limit=6)
    alone = []
    for net in nets:
        with Engine("fp64") as eng:
            eng.set_network(net)
            f = eng.forces()
            alone.append((f, eng.minimize(params)[0], eng.coords()))
    with Engine("fp64") as eng:
        eng.set_networks([nets[r % 3] for r in range(replicas)])
        first = [eng.forces(replica=r) for r in (0, 1, 2, replicas - 1)]
        res = eng.minimize(params)
        for k, r in enumerate((0, 1, 2, replicas - 1)):
            f, want, x = alone[r % 3]
            assert np.array_equal(first[k], f)
            assert res[r]["grad_inf_norm"] == want["grad_inf_norm"]
            assert list(res[r]["energies_after"]) == list(want["energies_after"])
            assert np.array_equal(eng.coords(r), x)
