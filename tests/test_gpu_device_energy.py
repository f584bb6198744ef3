"""mech_filament_energy_device where its block logic can go wrong: filaments that start, end or span at the edges of its
256-cylinder blocks, one-cylinder filaments, a filament count past one search step, theta0 != 0.

Against numpy in FP64: every term is a handful of rounded operations, so a sum of n terms differs by less than
(n + 20) eps of the sum of their magnitudes; 1e-12 of it leaves a factor of ten at the largest size here."""
import ctypes as C

import numpy as np
import pytest

from picgo_gb300 import _lib

pytestmark = pytest.mark.gpu


def reference(fcs, x, ks, l0, kb, t0):
    n = int(fcs[-1])
    fil = np.repeat(np.arange(len(fcs) - 1), np.diff(fcs))
    b = np.arange(n) + fil
    r = x[b + 1] - x[b]
    L = np.sqrt((r * r).sum(1))
    stretch = 0.5 * ks * (L - l0) ** 2
    k = np.nonzero(fil[1:] == fil[:-1])[0] + 1
    cosine = np.clip((r[k - 1] * r[k]).sum(1) / (L[k - 1] * L[k]), -1, 1)
    bend = kb[k] * (1 - np.where(np.abs(t0[k]) < 1e-6, cosine,
                                 cosine * np.cos(t0[k]) + np.sqrt(1 - cosine ** 2) * np.sin(t0[k])))
    return np.array([stretch.sum(), bend.sum()]), np.array([stretch.sum(), (kb[k] * 2).sum()])


LENGTHS = {
    "one": [1], "exactly a block": [256], "over a block": [257], "ends at the edge": [100, 156, 3],
    "starts at the edge": [255, 1, 40], "spans blocks": [5, 700, 2], "all of one cylinder": [1] * 700,
    "many": [2 + (7 * k) % 41 for k in range(1500)], "past a search step": [1 + k % 2 for k in range(40000)],
}


@pytest.mark.parametrize("name", LENGTHS)
@pytest.mark.parametrize("theta0", [0.0, 0.3])
def test_device_energy_at_block_edges(name, theta0):
    torch = pytest.importorskip("torch")
    fcs = np.concatenate([[0], np.cumsum(LENGTHS[name])]).astype(np.int32)
    n, nfil = int(fcs[-1]), len(fcs) - 1
    rng = np.random.default_rng(n)
    x = np.cumsum(rng.normal(0, 60, (n + nfil, 3)) + [40, 0, 0], axis=0)
    ks, l0, kb = rng.uniform(50, 150, n), rng.uniform(80, 130, n), rng.uniform(300, 900, n)
    t0 = np.where(rng.random(n) < 0.5, theta0, 0.0)
    dev = [torch.from_numpy(a).cuda() for a in (fcs, x, ks, l0, kb, t0)]
    out = torch.zeros(2, dtype=torch.float64, device="cuda")
    p = lambda t: C.c_void_p(t.data_ptr())   # noqa: E731
    _lib.check(_lib.load().mech_filament_energy_device(nfil, n, *[p(t) for t in dev], p(out),
                                                       C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    want, scale = reference(fcs, x, ks, l0, kb, t0)
    assert np.all(np.abs(out.cpu().numpy() - want) <= 1e-12 * scale), (out, want)


SHARES = {
    "filaments without cylinders": [0, 0, 3, 0, 5, 0, 0, 40, 1, 0, 31, 0, 0, 0, 64, 0],
    "more of them than a read": [7] + [0] * 70 + [90, 0, 2],
    "a chunk": [32], "over a chunk": [33], "a chunk and a start": [32, 32, 1],
    "one share each": [17] * 9156, "two chunks in some": [40] * 3900, "long shares": [997] * 500, "one filament": [300001],
}


@pytest.mark.parametrize("name", SHARES)
def test_device_energy_at_share_edges(name):
    """The same where a warp's share of the 32-cylinder chunks begins, ends and passes from one chunk to the next."""
    torch = pytest.importorskip("torch")
    fcs = np.concatenate([[0], np.cumsum(SHARES[name])]).astype(np.int32)
    n, nfil = int(fcs[-1]), len(fcs) - 1
    rng = np.random.default_rng(n)
    x = np.cumsum(rng.normal(0, 60, (n + nfil, 3)) + [40, 0, 0], axis=0) % 5000.0
    ks, l0, kb = rng.uniform(50, 150, n), rng.uniform(80, 130, n), rng.uniform(300, 900, n)
    t0 = np.zeros(n)
    dev = [torch.from_numpy(a).cuda() for a in (fcs, x, ks, l0, kb, t0)]
    out = torch.zeros(2, dtype=torch.float64, device="cuda")
    p = lambda t: C.c_void_p(t.data_ptr())   # noqa: E731
    for _ in range(2):
        _lib.check(_lib.load().mech_filament_energy_device(nfil, n, *[p(t) for t in dev], p(out),
                                                           C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    want, scale = reference(fcs, x, ks, l0, kb, t0)
    assert np.all(np.abs(out.cpu().numpy() - want) <= 1e-11 * scale), (out, want)
