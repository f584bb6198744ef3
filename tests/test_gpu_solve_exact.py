"""Solves whose residual reaches zero between two looks of the host at it (every 16 iterations).

A constant vector is an eigenvector of H + shift I, with the eigenvalue shift, away from the walls: one iteration
solves it to rounding, and a few more reduce r.r until it underflows.  The solution is uniform, so no linker's length
changes along it and the gradients of the linker parameters are zero to its rounding: lambda = g / shift with a relative
rounding of a few eps, times k and the extension, under 1e3 each."""
import numpy as np
import pytest

from picgo_gb300 import Engine, make_network

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [1.0, 0.37, 20.0, 1e-5])
@pytest.mark.parametrize("scale", [1.0, 1e-140])
def test_adjoint_of_a_uniform_gradient(shift, scale):
    net = make_network("c1", n_filaments=30, n_cyl_per_filament=8, box=1500.0, n_linkers=60, seed=21)
    net.planes[:, 3] += 1e5 * np.linalg.norm(net.planes[:, :3], axis=1)   # walls out of reach
    g = np.tile(scale * np.array([1.0, -2.0, 0.5]), (net.n_beads, 1))
    with Engine("fp64") as eng:
        eng.set_network(net)
        assert eng.rebuild()["n_boundary_beads"] == 0
        dk, dl0, info = eng.adjoint(g, 0.0, rel_tol=1e-10, max_iter=64, shift=shift)
        dk2, dl02, _ = eng.adjoint(g, 1.0, rel_tol=1e-10, max_iter=64, shift=shift)
        zk, zl, _ = eng.adjoint(0 * g, 1.0, rel_tol=1e-10, max_iter=64, shift=shift)
    assert info["converged"] and not info["negative_curvature"] and info["rel_residual"] <= 1e-10, info
    tol = 1e-9 * scale / shift
    assert np.all(np.abs(dk) <= tol) and np.all(np.abs(dl0) <= tol), (np.abs(dk).max(), np.abs(dl0).max())
    # with the energy's own share beside it
    assert np.allclose(dk2, zk, rtol=1e-12, atol=tol) and np.allclose(dl02, zl, rtol=1e-12, atol=tol)
