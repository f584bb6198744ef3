"""The block form of the Hessian that a solve applies, against the dual-number products it stands for: the adjoint's
parameter gradients equal those of a dense solve with the Hessian assembled from products with the unit vectors.

Tolerance: the solve stops at a relative residual of 1e-12, so the solution is off by at most the condition number
(largest eigenvalue over the shift, under 1e4 here) times that, and the dense side by as much of 1e-15: 1e-7 of the
largest gradient leaves a factor of ten."""
import numpy as np
import pytest

from picgo_gb300 import Engine, jitter, make_network

pytestmark = pytest.mark.gpu

SHIFT = 200.0


def network(n_filaments, n_cyl, seed, theta0):
    cfg = dict(n_filaments=n_filaments, n_cyl_per_filament=n_cyl, box=700.0, n_linkers=2 * n_filaments,
               linker_k=(4.0, 12.0), linker_l0=(20.0, 40.0), n_motors=n_filaments, shape="chain")
    net = jitter(make_network(cfg, seed=seed), 0.2, seed=2)
    net.cyl_kexvol = 1e-4 * net.cyl_kexvol
    if theta0:   # on every other triple that is bent: a straight one has no Hessian at theta0 != 0
        r = net.coord[net.cyl_b2] - net.coord[net.cyl_b1]
        u = r / np.linalg.norm(r, axis=1)[:, None]
        bent = np.zeros(net.n_cyl, bool)
        bent[1:] = (u[1:] * u[:-1]).sum(1) < 0.98
        bent[1::2] = False
        net.cyl_theta0[bent] = theta0
    return net


# (filaments, cylinders, seed): 12, 15, 255, 256 and 272 beads; blocks hold 256
@pytest.mark.parametrize("shape", [(6, 1, 9), (3, 4, 30), (17, 14, 1), (16, 15, 1), (8, 33, 6)])
@pytest.mark.parametrize("theta0", [0.0, 0.4])
def test_solve_applies_the_hessian_of_the_products(shape, theta0):
    net = network(*shape, theta0)
    n = net.coord.size
    g = np.random.default_rng(5).normal(size=net.coord.shape)
    with Engine("fp64") as eng:
        eng.set_network(net)
        H = np.empty((n, n))
        for j in range(n):
            e = np.zeros(n)
            e[j] = 1.0
            H[:, j] = eng.hvp(e.reshape(-1, 3)).reshape(-1)
        dk, dl0, info = eng.adjoint(g, 0.25, rel_tol=1e-12, max_iter=2000, shift=SHIFT)
    eig = np.linalg.eigvalsh(0.5 * (H + H.T))
    assert eig[0] + SHIFT > 1.0 and eig[-1] < 1e4, (eig[0], eig[-1])   # the case is the one the tolerance is for
    assert info["converged"] == 1 and info["negative_curvature"] == 0
    lam = np.linalg.solve(H + SHIFT * np.eye(n), g.reshape(-1)).reshape(-1, 3)
    x = net.coord
    s1, s2 = net.lk_pos[:, :1], net.lk_pos[:, 1:]
    a, b = net.lk_cyl[:, 0], net.lk_cyl[:, 1]
    at = lambda v: ((1 - s2) * v[net.cyl_b1[b]] + s2 * v[net.cyl_b2[b]]) - ((1 - s1) * v[net.cyl_b1[a]] + s1 * v[net.cyl_b2[a]])
    l = at(x)
    d = np.linalg.norm(l, axis=1)
    gl = (l * at(lam)).sum(1) / d
    dd = d - net.lk_l0
    want_k, want_l = 0.25 * 0.5 * dd * dd - dd * gl, -0.25 * net.lk_k * dd + net.lk_k * gl
    assert np.abs(dk - want_k).max() <= 1e-7 * np.abs(want_k).max()
    assert np.abs(dl0 - want_l).max() <= 1e-7 * np.abs(want_l).max()
