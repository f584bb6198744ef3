"""The kernels of the mixed engine's excluded-volume chain are released before or at the end of their predecessor,
according to the network's bead tiles; inside a conditional graph they follow one another without programmatic launch.
The same kernels do the same work, so on both sides of the rule's limit a minimization, with pairs in the extended pass,
and a plain evaluation after it agree bit for bit."""
import numpy as np
import pytest

from picgo_gb300 import Engine, cg_params, jitter, make_network

pytestmark = pytest.mark.gpu

LIMIT = 608   # tiles of 256 beads
PER_TILE = 8  # filaments of 31 cylinders (32 beads)


def _run(net, mode):
    with Engine("mixed") as eng:
        eng.set_graph_mode(mode)
        eng.set_network(net)
        first = eng.energies()
        f0 = eng.forces()
        res = eng.minimize(cg_params(energy_rel_tol=0.0, energy_call_limit=30, force_call_limit=60))[0]
        return first, f0, res, eng.coords(), eng.energies(), eng.forces(), len(eng.pairs())


@pytest.mark.parametrize("filaments", [8, PER_TILE * LIMIT, PER_TILE * LIMIT + 1])
def test_chain_release_keeps_every_bit(filaments):
    cfg = dict(n_filaments=filaments, n_cyl_per_filament=31, box=700.0 * (filaments / 8.0) ** (1.0 / 3.0), n_linkers=0,
               shape="chain")
    net = jitter(make_network(cfg, seed=4), 0.3, seed=6)
    net.exvol_cutoff = 60.0
    a, b = _run(net, "conditional"), _run(net, "unrolled")
    assert a[6] == b[6] and a[6] > 0
    for k in ("num_iter", "num_energy_eval", "num_line_search_trials", "grad_inf_norm"):
        assert a[2][k] == b[2][k]
    assert np.array_equal(a[0][0], b[0][0]) and np.array_equal(a[4][0], b[4][0])
    for k in (1, 3, 5):
        assert np.array_equal(a[k], b[k])


def _flat(filaments, seed):
    cfg = dict(n_filaments=filaments, n_cyl_per_filament=12, box=520.0, n_linkers=0, shape="chain")
    net = jitter(make_network(cfg, seed=seed), 0.2, seed=2)
    net.exvol_cutoff = 60.0
    net.coord[:, 2] = 260.0 + 0.2 * (net.coord[:, 2] - 260.0)   # nearly coplanar pairs
    return net


@pytest.mark.parametrize("replicas", [1, 5])
def test_pairs_listed_at_the_trial(replicas):
    """An unrolled graph lists the pairs of the extended force pass at the line search's trials, a conditional one in the
    force pass itself: the same pairs, the same forces, whichever trial each replica accepts."""
    nets = [_flat(8 + 3 * k, 60 + k) for k in range(replicas)]
    out = []
    for mode in ("conditional", "unrolled"):
        with Engine("mixed") as eng:
            eng.set_graph_mode(mode)
            eng.set_networks(nets)
            assert eng.profile(1)["n_exvol_ext_force"] > 0
            eng.reset_coords()
            res = eng.minimize(cg_params(energy_rel_tol=0.0, energy_call_limit=60, force_call_limit=200))
            out.append((res, [eng.coords(r) for r in range(replicas)]))
    assert sum(r["num_line_search_trials"] - r["num_iter"] for r in out[0][0]) > 0   # some trials were rejected
    for a, b in zip(*(o[0] for o in out)):
        for k in ("num_iter", "num_force_call", "num_energy_eval", "num_line_search_trials", "grad_inf_norm"):
            assert a[k] == b[k]
        assert list(a["energies_after"]) == list(b["energies_after"])
    for u, v in zip(*(o[1] for o in out)):
        assert np.array_equal(u, v)
