"""Evaluations of a minimization in which most searches lose conjugacy.

A pass whose new direction turns out not to descend is thrown away, so it shows as an energy evaluation without a
trial.  After a search along the forces themselves the slope of the next direction is known beforehand and no such
pass is made.  What remains: the evaluations before and after the iterations, one per recovery move, a thrown-away
pass where the lost direction followed another one, and in mixed precision a second trial that was not needed: together
well under one per ten iterations, where a pass thrown away in every search would make it nearly one per iteration."""
import pytest

from picgo_gb300 import Engine, cg_params, make_network

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_lost_conjugacy_spends_no_pass(precision):
    net = make_network("c1", seed=20261204)
    with Engine(precision) as eng:
        eng.set_network(net)
        r = eng.minimize(cg_params(energy_rel_tol=0.0, energy_call_limit=4000))[0]
    assert r["num_iter"] >= 500
    assert 2 <= r["num_energy_eval"] - r["num_line_search_trials"] <= 2 + r["num_iter"] // 10, r
