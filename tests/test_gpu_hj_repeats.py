"""GPU test of hash-join buckets whose keys repeat: numbers of tuples per key on
both sides of the line between the lists by places and the count table, one hot
key among distinct ones, and either side as the build side; unpartitioned
windows, partitioned ones and both in one call."""
import numpy as np
import pytest

from helpers import make_tuples

pytestmark = pytest.mark.gpu

SMALL = [(1, 1), (2, 5), (64, 4096), (511, 513), (4096, 4096), (3000, 5000), (5000, 900)]
LARGE = [(40_000, 30_000), (9_000, 120_000), (120_000, 9_000)]


def keys_of(kind, n, rng):
    if isinstance(kind, int):   # that many tuples per key
        k = rng.integers(0, max(1, n // kind), n, dtype=np.uint32)
    else:                       # distinct, but for one key of that many tuples
        k = rng.permutation(np.arange(1, n + 1, dtype=np.uint32))
        k[: min(n, int(kind[3:]))] = 7
    return k * np.uint32(0x9E3779B1)   # too far apart for direct tables


@pytest.mark.parametrize("part", ["PART_AUTO", "PART_RADIX"])
@pytest.mark.parametrize("sizes", [SMALL, LARGE, SMALL + LARGE], ids=["small", "large", "both"])
@pytest.mark.parametrize("kind", [1, 2, 3, 4, 5, 9, 40, 700, "hot19", "hot20", "hot21", "hot32", "hot300"])
def test_repeated_keys(lib, oracle, kind, sizes, part):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(17)
    lefts, rights, descs, lo, ro = [], [], [], 0, 0
    for nl, nr in sizes:
        lefts.append(keys_of(kind, nl, rng))
        rights.append(keys_of(kind, nr, rng))
        descs.append((lo, nl, ro, nr, 0, 0))
        lo, ro = lo + nl, ro + nr
    left, right = make_tuples(np.concatenate(lefts)), make_tuples(np.concatenate(rights))
    want, _ = oracle.join_windows(left, right, descs, enumerate_pairs=False)
    dl, dr = torch.from_numpy(left.view(np.uint8)).cuda(), torch.from_numpy(right.view(np.uint8)).cuda()
    with lib.Joiner(lib.ALG_HJ, lib.LAZY, partitioner=getattr(lib, part), max_tuples_per_window=1 << 17) as j:
        for _ in range(2):
            got = j.lazy_execute_batch(dl, dr, descs, mem=lib.MEM_DEVICE)
            for d, g, w in zip(descs, got, want):
                assert (g["count"], g["prod"]) == (w["count"], w["prod"]), d
