"""GPU test of key ranges whose sample misses the ends of the keys' span: the sampled
positions of the larger side (one in 256) hold no key of the outer few distances
between sampled keys, at either end or both, and the window is joined by ranges."""
import numpy as np
import pytest

from helpers import make_tuples

pytestmark = pytest.mark.gpu

N, STEP = 1 << 20, 256
GAP = N // STEP   # samples of the side: a distance between sampled keys is 4 * N / GAP keys


@pytest.mark.parametrize("low,high", [(0, 0), (3, 0), (6, 0), (0, 6), (6, 6)])
@pytest.mark.parametrize("base", [0, 5_000_000, 0xFFFFFFFF - 4 * N + 1])
def test_keys_beyond_the_sample(lib, oracle, low, high, base):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(47)
    unit = 4 * N // GAP
    keys = rng.integers(0, 4 * N, N, dtype=np.int64)
    keys[::STEP] = rng.integers(low * unit, 4 * N - high * unit, N // STEP)
    others = rng.integers(max(low, 1) * unit, 4 * N - max(high, 1) * unit, 900)
    left = make_tuples((keys + base).astype(np.uint32))
    right = make_tuples((others + base).astype(np.uint32))
    descs = [(0, N, 0, len(others), 0, 0)]
    want, _ = oracle.join_windows(left, right, descs, enumerate_pairs=False)
    dl, dr = torch.from_numpy(left.view(np.uint8)).cuda(), torch.from_numpy(right.view(np.uint8)).cuda()
    with lib.Joiner(lib.ALG_SMJ, lib.LAZY, flags=lib.F_PROFILE, max_tuples_per_window=N) as j:
        got = j.lazy_execute_batch(dl, dr, descs, mem=lib.MEM_DEVICE)
        assert (got[0]["count"], got[0]["prod"]) == (want[0]["count"], want[0]["prod"])
        stats = j.kernel_stats()
        assert "range_join" in stats and "rs_downsweep" not in stats
