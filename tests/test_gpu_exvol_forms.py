"""The two forms of the FP64 excluded-volume kernel (a pair per thread; a pair over the four warps of a block) make the
same operations in the same order: a network's energies and forces keep every bit when it is evaluated alone, where
its few tiles of pairs go split, and as one of many replicas, whose full rounds of tiles go unsplit."""
import numpy as np
import pytest

from picgo_gb300 import Engine, jitter, make_network

pytestmark = pytest.mark.gpu

ROUND, SPLIT = 76, 57   # tiles of a full round; most tiles that go split


def network(n_filaments, seed, flat=False):
    cfg = dict(n_filaments=n_filaments, n_cyl_per_filament=12, box=520.0, n_linkers=0, shape="chain")
    net = jitter(make_network(cfg, seed=seed), 0.2, seed=2)
    net.exvol_cutoff = 60.0    # many pairs, near and far
    if flat:
        net.coord[:, 2] = 260.0 + 0.5 * (net.coord[:, 2] - 260.0)
    return net


@pytest.mark.parametrize("flat", [False, True])
@pytest.mark.parametrize("replicas", [ROUND, ROUND + 1, ROUND + SPLIT + 1])
def test_split_and_unsplit_pairs_agree_bit_for_bit(replicas, flat):
    nets = [network(8 + k, 50 + k, flat) for k in range(4)]   # every one has a single tile of at most 256 pairs
    alone = []
    for net in nets:
        with Engine("fp64") as eng:
            eng.set_network(net)
            assert 32 < len(eng.pairs()) <= 256 and len(eng.pairs()) % 32
            alone.append((eng.energies()[0], eng.forces(), eng.energies()[2]))
    with Engine("fp64") as eng:
        eng.set_networks([nets[r % 4] for r in range(replicas)])
        for r in sorted({0, 1, 2, 3, ROUND - 2, ROUND - 1, replicas - 2, replicas - 1}):
            per, _, value = eng.energies(replica=r)
            f = eng.forces(replica=r)
            want = alone[r % 4]
            assert per[4] == want[0][4] and (value == want[2] or not np.isfinite(want[2]))
            assert np.array_equal(f, want[1], equal_nan=True)
