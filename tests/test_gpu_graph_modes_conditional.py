"""The unrolled graph against the conditional one where they differ most: the minimum-energy backup and the force-call
limit that ends such a run, recovery moves, lost conjugacy in most searches, and replicas that finish one after another
(compacted in between).

The conditional graph runs without programmatic dependent launch, without pairs listed at the trial and without idle
passes, so a kernel that reads what it has not waited for shows as a difference.  Bit for bit: counts, energies,
coordinates, forces."""
import numpy as np
import pytest

from picgo_gb300 import Engine, cg_params, jitter, make_network
from picgo_gb300.network import make_ensemble

pytestmark = pytest.mark.gpu


def run(precision, nets, mode, params):
    with Engine(precision) as eng:
        eng.set_graph_mode(mode)
        eng.set_networks(nets)
        res = eng.minimize(params)
        return (res, [(eng.coords(r), eng.last_forces(r), *eng.stretch_forces(r)) for r in range(len(nets))],
                eng.timing()["launches"])


def same(precision, nets, params):
    (ra, xa, la), (rb, xb, lb) = (run(precision, nets, m, params) for m in ("conditional", "unrolled"))
    assert la != lb      # other launches: the two did not run the same graph
    for x, y in zip(ra, rb):
        for k in ("status", "error_flags", "num_iter", "num_energy_call", "num_force_call", "num_energy_eval",
                  "num_line_search_trials", "num_safe_mode", "num_recover", "grad_inf_norm"):
            assert x[k] == y[k], (k, x[k], y[k])
        assert list(x["energies_before"]) == list(y["energies_before"])
        assert list(x["energies_after"]) == list(y["energies_after"])
    for u, v in zip(xa, xb):
        assert all(np.array_equal(p, q) for p, q in zip(u, v))
    return ra


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_backup_at_the_call_limit(precision):
    net = make_network("c1", n_filaments=3, n_cyl_per_filament=5, box=1500.0, n_linkers=0, seed=11)
    net.coord = net.coord + np.random.default_rng(0).normal(0, 1e-2, net.coord.shape)
    same(precision, [net], cg_params(grad_tol=1e-3, energy_rel_tol=0.0, report_on_call_limit=1, energy_call_limit=0,
                                     force_call_limit=0))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_lost_conjugacy_and_recovery(precision):
    net = make_network("c1", seed=20261204)
    r = same(precision, [net], cg_params(energy_rel_tol=0.0, energy_call_limit=3000))[0]
    assert r["num_safe_mode"] > 0


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_replicas_finishing_one_after_another(precision):
    nets = make_ensemble(8, seed=3, fil_range=(20, 200), cyl_range=(10, 20))
    r = same(precision, nets, cg_params(energy_rel_tol=0.0, energy_call_limit=2000))
    assert len({x["num_iter"] for x in r}) > 4


def test_failing_line_searches():
    net = jitter(make_network("c1", n_filaments=60, n_cyl_per_filament=12, box=1500.0, n_linkers=80, n_motors=40, seed=3),
                 0.3, seed=7)
    r = same("mixed", [net], cg_params(lambda_max=1e-9, energy_call_limit=40, try_to_recover=1))[0]
    assert r["num_recover"] >= 5
