"""GPU test of calls of small windows whose pieces make more than one wave of CTAs:
build sides up to a table's slots, probe sides of one piece to many."""
import numpy as np
import pytest

from helpers import make_tuples

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[(20_000, 5000)] * 32, [(5343, 5343)] * 120, [(2, 90_000), (90_000, 5343), (4097, 4096)] * 9,
                                   [(400_000, 5000)] * 2, [(400_000, 5344)] * 2])
def test_whole_build_sides(lib, oracle, sizes):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(len(sizes))
    lefts, rights, descs, lo, ro = [], [], [], 0, 0
    for nl, nr in sizes:
        for side, n in ((lefts, nl), (rights, nr)):
            side.append(rng.integers(0, 9000, n, dtype=np.uint32) * np.uint32(0x9E3779B1))
        descs.append((lo, nl, ro, nr, 0, 0))
        lo, ro = lo + nl, ro + nr
    left, right = make_tuples(np.concatenate(lefts)), make_tuples(np.concatenate(rights))
    want, _ = oracle.join_windows(left, right, descs, enumerate_pairs=False)
    dl, dr = torch.from_numpy(left.view(np.uint8)).cuda(), torch.from_numpy(right.view(np.uint8)).cuda()
    with lib.Joiner(lib.ALG_HJ, lib.LAZY, flags=lib.F_PROFILE, max_tuples_per_window=1 << 19) as j:
        for _ in range(2):
            got = j.lazy_execute_batch(dl, dr, descs, mem=lib.MEM_DEVICE)
            for d, g, w in zip(descs, got, want):
                assert (g["count"], g["prod"]) == (w["count"], w["prod"]), d
        assert ("raw_join" in j.kernel_stats()) == all(min(s) < 5344 for s in sizes)
