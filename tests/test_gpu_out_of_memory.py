"""Device allocations that fail, by a build of the library whose device buffers refuse more than a limit that the test
sets (no memory is filled): a call that fails on one leaves its context usable, and nothing runs on lists that are new
in part."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from picgo_gb300 import Engine, _lib, build, cg_params, jitter, make_network

pytestmark = pytest.mark.gpu

ERR_CUDA = -3
NO_LIMIT = 1 << 62


@pytest.fixture(scope="module")
def limited_library(tmp_path_factory):
    """The library with mech_nl.cu (which allocates) compiled for a limit, and its other objects as they are."""
    d = tmp_path_factory.mktemp("limited")
    nl, out = str(d / "mech_nl.o"), str(d / build.LIBNAME)
    subprocess.run([build.nvcc(), *build.ARCH, *build.COMMON, f"-DMECH_ALLOC_LIMIT={NO_LIMIT}ull", "-c",
                    os.path.join(build.CSRC, "mech_nl.cu"), "-o", nl], check=True)
    objs = [nl if o == "mech_nl.o" else os.path.join(build.OUTDIR, o) for _, o, _ in build.UNITS]
    subprocess.run([build.nvcc(), *build.ARCH, "-shared", "-o", out, *objs, "-Xcompiler", "-fPIC"], check=True)
    return out


@pytest.fixture
def limit(limited_library, monkeypatch):
    """Contexts made in the test use that library; the fixture sets the limit in bytes."""
    monkeypatch.setattr(_lib, "_lib", None)
    monkeypatch.setattr(build, "lib_path", lambda: limited_library)
    value = C.c_size_t.in_dll(_lib.load(), "mech_alloc_limit")

    def set_limit(n):
        value.value = n
    set_limit(NO_LIMIT)
    yield set_limit
    set_limit(NO_LIMIT)


def chain_net(n_filaments=200):
    return make_network("c1", n_filaments=n_filaments, n_linkers=0, seed=4)


def crowded(net):
    """The same filaments, all of them within the pair cutoff of one another."""
    x = net.coord.reshape(net.n_filaments, -1, 3)
    rng = np.random.default_rng(1)
    return (x[:1] + rng.normal(0, 2.0, (net.n_filaments, 1, 3))).reshape(-1, 3)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_lists_after_a_rebuild_that_fails(precision, limit):
    net = chain_net()
    with Engine(precision) as eng:
        eng.set_network(net)
        want, pairs, f = eng.energies(), eng.pairs().copy(), eng.forces()
        n_full = 0
        with Engine(precision) as other:
            other.set_network(net)
            other.set_coords(crowded(net))
            n_full = other.rebuild()["n_exvol_pairs"]
        assert n_full > 50 * net.n_cyl
        limit(16 * n_full // 2)          # the pair list fits (8 bytes a pair), the beads of the pairs (16) do not
        eng.set_coords(crowded(net))
        for call in (lambda: eng.rebuild(), lambda: eng.energies(), lambda: eng.forces(), lambda: eng.minimize()):
            with pytest.raises(_lib.MechError) as e:
                call()
            assert e.value.code == ERR_CUDA
        with pytest.raises(_lib.MechError):
            eng.pairs()
        eng.set_coords(net.coord)        # what fitted fits again, by the lists that the evaluation builds
        got = eng.energies()
        assert np.array_equal(got[0], want[0]) and got[1:] == want[1:]
        assert np.array_equal(eng.pairs(), pairs) and np.array_equal(eng.forces(), f)
        limit(NO_LIMIT)
        eng.set_coords(crowded(net))
        assert eng.rebuild()["n_exvol_pairs"] == n_full


@pytest.mark.parametrize("forces", [False, True])
def test_coordinates_of_a_failed_evaluation_have_been_read(forces, limit):
    """An evaluation that fails before its first wait (no room for the lists) has read the caller's pinned coordinates
    when it returns: they can be overwritten at once."""
    torch = pytest.importorskip("torch")
    net = make_network("c1", n_filaments=10000, n_cyl_per_filament=50, box=10000.0, n_linkers=0, seed=4)
    moved = net.coord + 1.0
    with Engine("mixed") as eng:
        limit(28 * net.n_beads)          # positions (24 bytes a bead) fit, the neighbors kept from the count (32) do not
        with pytest.raises(_lib.MechError):
            eng.set_network(net)
        eng.nbeads, eng.nlinkers, eng.nmotors = [net.n_beads], [0], [0]
        pinned = torch.empty((net.n_beads, 3), dtype=torch.float64, pin_memory=True)
        pinned.copy_(torch.from_numpy(moved))
        x = pinned.numpy()
        with pytest.raises(_lib.MechError) as e:
            eng.forces(x) if forces else eng.energies(x)
        x[:] = -1e6
        assert e.value.code == ERR_CUDA
        # positions are held to 48 bits
        assert np.abs(eng.coords() - moved).max() <= 1e-10


@pytest.mark.parametrize("what", ["filaments", "pairs"])
def test_solves_without_room_for_the_hessian(what, limit):
    """A solve that finds no room for the Hessian's blocks applies it by duals: the same Hessian, rounded differently.
    The eigenvalues of this network's (central differences of the oracle's forces) plus the shift lie between 160 and
    1,900, so a relative residual of 1e-12 leaves the solutions within 1e-10 of their size; 1e-8 of the gradients."""
    cfg = dict(n_filaments=17, n_cyl_per_filament=14, box=700.0, n_linkers=34, linker_k=(4.0, 12.0),
               linker_l0=(20.0, 40.0), n_motors=17, shape="chain")
    net = jitter(make_network(cfg, seed=1), 0.2, seed=2)
    net.cyl_kexvol = 1e-4 * net.cyl_kexvol
    net.exvol_cutoff = 100.0
    g = np.random.default_rng(3).normal(size=net.coord.shape)
    kw = dict(rel_tol=1e-12, max_iter=2000, shift=200.0)
    with Engine("fp64") as eng:
        eng.set_network(net)
        n = eng.rebuild()["n_exvol_pairs"]
        assert 648 * n > 400 * net.n_beads
        want = eng.adjoint(g, 0.5, **kw)
    with Engine("fp64") as eng:
        eng.set_network(net)
        limit({"filaments": 100, "pairs": 300}[what] * net.n_beads)
        got = eng.adjoint(g, 0.5, **kw)
        flat = eng.adjoint(np.ones_like(g), 0.5, rel_tol=1e-10, max_iter=200, shift=200.0)
        limit(NO_LIMIT)
        after = eng.adjoint(g, 0.5, **kw)
    assert want[2]["converged"] and got[2]["converged"] and flat[2]["converged"] and after[2]["converged"]
    assert got[2]["launches"] != want[2]["launches"] and after[2]["launches"] == want[2]["launches"]
    for a, b, c in zip(want[:2], got[:2], after[:2]):
        assert np.abs(a - b).max() <= 1e-8 * np.abs(a).max() and np.array_equal(a, c)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_repeated_calls_allocate_nothing(precision, limit):
    net = jitter(make_network("c1", n_filaments=60, n_cyl_per_filament=12, box=1500.0, n_linkers=80, n_motors=40, seed=3),
                 0.3, seed=7)
    p = cg_params(energy_rel_tol=0.0, energy_call_limit=300)
    v = np.random.default_rng(1).normal(size=net.coord.shape)
    with Engine(precision) as eng:
        calls = [lambda: eng.set_network(net), lambda: eng.energies(net.coord)[0], lambda: eng.forces(),
                 lambda: eng.energy_terms(), lambda: eng.load_forces(), lambda: eng.rebuild()["n_exvol_pairs"],
                 lambda: list(eng.minimize(p)[0]["energies_after"]), lambda: eng.coords(), lambda: eng.stretch_forces(),
                 lambda: eng.set_coords(net.coord)]
        if precision == "fp64":
            calls += [lambda: eng.hvp(v), lambda: eng.adjoint(v, max_iter=32, shift=1e4)[0]]
        first = [call() for call in calls]
        limit(0)
        for call, want in zip(calls, first):
            got = call()
            if isinstance(want, tuple):
                assert all(np.array_equal(a, b) for a, b in zip(want, got))
            else:
                assert want is None or np.array_equal(want, got)
