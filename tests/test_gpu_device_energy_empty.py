"""mech_filament_energy_device with filaments without cylinders behind 32 starts in one 32-cylinder chunk, where the
walk has read no start beyond them.  Tolerance as in test_gpu_device_energy: a sum of n terms of a handful of rounded
operations each."""
import ctypes as C

import numpy as np
import pytest

from picgo_gb300 import _lib
from test_gpu_device_energy import reference

pytestmark = pytest.mark.gpu

LENGTHS = {
    "one": [1] * 31 + [0, 40, 7], "several": [1] * 31 + [0, 0, 0, 40, 7], "in the second chunk": [32] + [1] * 31 + [0, 12, 5],
    "at the end of the array": [1] * 31 + [0, 1], "after the last cylinder": [1] * 32 + [0, 0],
    "every chunk": ([1] * 31 + [0, 1]) * 300 + [3], "long after": [1] * 31 + [0] + [45] * 4000,
}


@pytest.mark.parametrize("name", LENGTHS)
def test_filaments_without_cylinders_behind_a_full_read(name):
    torch = pytest.importorskip("torch")
    fcs = np.concatenate([[0], np.cumsum(LENGTHS[name])]).astype(np.int32)
    n, nfil = int(fcs[-1]), len(fcs) - 1
    rng = np.random.default_rng(n)
    x = np.cumsum(rng.normal(0, 60, (n + nfil, 3)) + [40, 0, 0], axis=0) % 5000.0
    ks, l0, kb, t0 = rng.uniform(50, 150, n), rng.uniform(80, 130, n), rng.uniform(300, 900, n), np.zeros(n)
    dev = [torch.from_numpy(a).cuda() for a in (fcs, x, ks, l0, kb, t0)]
    out = torch.zeros(2, dtype=torch.float64, device="cuda")
    p = lambda t: C.c_void_p(t.data_ptr())   # noqa: E731
    _lib.check(_lib.load().mech_filament_energy_device(nfil, n, *[p(t) for t in dev], p(out),
                                                       C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    want, scale = reference(fcs, x, ks, l0, kb, t0)
    assert np.all(np.abs(out.cpu().numpy() - want) <= 1e-11 * np.maximum(scale, 1e-30)), (out, want)
