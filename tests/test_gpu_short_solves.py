"""Solves of few iterations, on both sides of the line where they begin to set up the Hessian's blocks: a conjugate
gradient on the host with the products of mech_hvp gives the same truncated solution.  Eight iterations at a condition
number under 2 keep a rounding of 1e-15 below 1e-11 of the solution; 1e-9 of the largest gradient."""
import numpy as np
import pytest

from picgo_gb300 import Engine, jitter, make_network

pytestmark = pytest.mark.gpu

SHIFT = 1e5


def host_cg(eng, b, m):
    x, r, p = np.zeros_like(b), b.copy(), b.copy()
    rr = (r * r).sum()
    for _ in range(m):
        Ap = eng.hvp(p) + SHIFT * p
        alpha = rr / (p * Ap).sum()
        x += alpha * p
        r -= alpha * Ap
        new = (r * r).sum()
        p = r + new / rr * p
        rr = new
    return x


@pytest.mark.parametrize("cutoff", [27.0, 150.0])
def test_truncated_solutions(cutoff):
    cfg = dict(n_filaments=200, n_cyl_per_filament=20, box=2000.0, n_linkers=500, linker_k=8.0, n_motors=50, shape="chain")
    net = jitter(make_network(cfg, seed=3), 0.2, seed=1)
    net.exvol_cutoff = cutoff
    net.cyl_kexvol = 1e-4 * net.cyl_kexvol
    g = np.random.default_rng(2).normal(size=net.coord.shape)
    s1, s2 = net.lk_pos[:, :1], net.lk_pos[:, 1:]
    a, b = net.lk_cyl[:, 0], net.lk_cyl[:, 1]
    at = lambda v: ((1 - s2) * v[net.cyl_b1[b]] + s2 * v[net.cyl_b2[b]]) - ((1 - s1) * v[net.cyl_b1[a]] + s1 * v[net.cyl_b2[a]])   # noqa: E731
    l = at(net.coord)
    d = np.linalg.norm(l, axis=1)
    with Engine("fp64") as eng:
        eng.set_network(net)
        for m in (1, 2, 5, 6, 8):
            dk, dl0, info = eng.adjoint(g, 0.0, rel_tol=1e-300, max_iter=m, shift=SHIFT)
            assert info["iterations"] == m and not info["negative_curvature"]
            gl = (l * at(host_cg(eng, g, m))).sum(1) / d
            assert np.abs(dk + (d - net.lk_l0) * gl).max() <= 1e-9 * np.abs(dk).max()
            assert np.abs(dl0 - net.lk_k * gl).max() <= 1e-9 * np.abs(dl0).max()
