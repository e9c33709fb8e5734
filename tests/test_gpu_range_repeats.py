"""GPU test of hash ranges whose keys repeat: numbers of tuples per key around the
line to the table, more distinct keys than it has slots beside hot ones (sorted),
and the mark of its free slots among the keys."""
import numpy as np
import pytest

from helpers import make_tuples

pytestmark = pytest.mark.gpu

SIZES = [(70_000, 65_536), (3000, 9000), (1, 40_000), (100_001, 700), (700, 30_000)]


def keys_of(per, hot, mark, n, rng):
    k = rng.integers(0, max(1, int(n / per)), n, dtype=np.uint32) * np.uint32(0x9E3779B1)
    k[: min(n, hot)] = 77
    if mark:
        k[rng.integers(0, n, max(1, n // 50))] = 0xFFFFFFFF
    return rng.permutation(k)


@pytest.mark.parametrize("mark", [False, True])
@pytest.mark.parametrize("per,hot", [(0.25, 0), (1, 0), (2, 0), (3, 0), (4, 0), (8, 0), (60, 0), (900, 0), (0.25, 33),
                                     (0.25, 2000), (3, 300)])
def test_repeated_keys_by_ranges(lib, oracle, per, hot, mark):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(41)
    lefts, rights, descs, lo, ro = [], [], [], 0, 0
    for nl, nr in SIZES:
        lefts.append(keys_of(per, hot, mark, nl, rng))
        rights.append(keys_of(per, hot, mark, nr, rng))
        descs.append((lo, nl, ro, nr, 0, 0))
        lo, ro = lo + nl, ro + nr
    left, right = make_tuples(np.concatenate(lefts)), make_tuples(np.concatenate(rights))
    want, _ = oracle.join_windows(left, right, descs, enumerate_pairs=False)
    dl, dr = torch.from_numpy(left.view(np.uint8)).cuda(), torch.from_numpy(right.view(np.uint8)).cuda()
    with lib.Joiner(lib.ALG_HJ, lib.LAZY, flags=lib.F_PROFILE, max_tuples_per_window=1 << 17) as j:
        for _ in range(2):
            got = j.lazy_execute_batch(dl, dr, descs, mem=lib.MEM_DEVICE)
            for d, g, w in zip(descs, got, want):
                assert (g["count"], g["prod"]) == (w["count"], w["prod"]), d
        assert "range_join" in j.kernel_stats()
