"""GPU tests of learned hash-join windows whose light tuples are compacted and
joined from sorted tiles: numbers of light tuples at the tile's edges, one
empty light side, buckets with more keys than the count table takes."""
import numpy as np
import pytest

from helpers import make_tuples

pytestmark = pytest.mark.gpu

HOT = np.array([3, 1 << 20, 0x12345678, 0xFFFFFFFE], np.uint32)


def side(n, light, rng):
    """n keys, the given light ones among them at random places."""
    k = HOT[rng.integers(0, len(HOT), n)]
    k[rng.choice(n, len(light), replace=False)] = light
    return k


def light_keys(kind, n, rng):
    if kind == "spread":   # the table's empty marker among them
        k = rng.integers(0, 1 << 32, n, dtype=np.uint32) & np.uint32(0xFFFFF00F)
        k[::31] = 0xFFFFFFFF
        return k
    if kind == "crowd":    # a dense run of keys and few far away: one line over their range puts the run in one bucket
        k = rng.integers(1000, 1000 + 50_000, n, dtype=np.uint32)
        k[::1000] = 0xF0000000
        return k
    return np.full(n, 99, np.uint32)


@pytest.mark.parametrize("leaves", [0, 1])
@pytest.mark.parametrize("kind", ["spread", "crowd", "one"])
def test_light_tuples_joined_from_sorted_tiles(lib, oracle, kind, leaves):
    rng = np.random.default_rng(23)
    W = 150_001
    lights = [(60_000, 60_000), (4096, 4097), (4095, 1), (0, 5000), (5000, 0), (8192, 60_001), (1, 1), (7000, 3000), (9000, 9000),
              (14_000, 2000)]
    lefts = [side(W, light_keys(kind, a, rng), rng) for a, _ in lights]
    rights = [side(W, light_keys(kind, b, rng), rng) for _, b in lights]
    descs = [(i * W, W, i * W, W, 0, 0) for i in range(len(lights))]
    left, right = make_tuples(np.concatenate(lefts)), make_tuples(np.concatenate(rights))
    want, _ = oracle.join_windows(left, right, descs, enumerate_pairs=False)
    with lib.Joiner(lib.ALG_HJ, lib.LAZY, partitioner=lib.PART_LEARNED, learned_leaves=leaves,
                    max_tuples_per_window=W) as j:
        for _ in range(2):
            got = j.lazy_execute_batch(left, right, descs)
            for d, g, w in zip(lights, got, want):
                assert (g["count"], g["prod"]) == (w["count"], w["prod"]), (d, g["partitioner_used"])
