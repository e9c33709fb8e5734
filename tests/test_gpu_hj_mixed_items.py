"""GPU test of automatic hash joins whose join list mixes unpartitioned windows
with buckets of partitioned ones: a CTA takes items of both kinds in turn, dense
keys (direct tables) next to keys at the other end of the domain."""
import numpy as np
import pytest

from helpers import make_tuples

pytestmark = pytest.mark.gpu

SIZES = [(300_000, 280_000)] + [(3000, 2500), (40_000, 50_000), (1, 9000), (4096, 4096)] * 12


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("far", [False, True])
def test_raw_and_partitioned_windows(lib, oracle, far, graph):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(14)
    lefts, rights, descs, lo, ro = [], [], [], 0, 0
    for i, (nl, nr) in enumerate(SIZES):
        base = np.uint32(0xFFF00000 if far and i % 2 else 0)
        for side, n in ((lefts, nl), (rights, nr)):
            k = base + rng.integers(0, max(nl // 2, 1), n, dtype=np.uint32)
            if i == 0:
                k[:6000] = 11   # (does not fit its hash range: the call goes by buckets)
            side.append(k)
        descs.append((lo, nl, ro, nr, 0, 0))
        lo, ro = lo + nl, ro + nr
    left, right = make_tuples(np.concatenate(lefts)), make_tuples(np.concatenate(rights))
    want, _ = oracle.join_windows(left, right, descs, enumerate_pairs=False)
    dl, dr = torch.from_numpy(left.view(np.uint8)).cuda(), torch.from_numpy(right.view(np.uint8)).cuda()
    with lib.Joiner(lib.ALG_HJ, lib.LAZY, flags=lib.F_PROFILE | (lib.F_GRAPH if graph else 0),
                    max_tuples_per_window=1 << 19) as j:
        for _ in range(4):
            got = j.lazy_execute_batch(dl, dr, descs, mem=lib.MEM_DEVICE)
            for d, g, w in zip(descs, got, want):
                assert (g["count"], g["prod"]) == (w["count"], w["prod"]), d
        assert "bucket_join_count" in j.kernel_stats()
