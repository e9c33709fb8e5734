"""GPU test of large bucket targets (SJBG_BUCKET_TARGET): the count table then
takes up to all of the shared memory a CTA may have, with and without room for
the lists of the join from sorted tiles beside it."""
import numpy as np
import pytest

from helpers import make_tuples
from test_gpu_hj_compact import light_keys, side

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("part", ["PART_LEARNED", "PART_RADIX", "PART_AUTO"])
@pytest.mark.parametrize("target", [9000, 11_000, 16_384, 65_536])
def test_large_bucket_targets(lib, oracle, monkeypatch, part, target):
    torch = pytest.importorskip("torch")
    monkeypatch.setenv("SJBG_BUCKET_TARGET", str(target))
    rng = np.random.default_rng(31)
    W, n = 150_001, 3
    lights = [(60_000, 60_000), (9000, 40_000), (0, 5000)]
    left = make_tuples(np.concatenate([side(W, light_keys("spread", a, rng), rng) for a, _ in lights]))
    right = make_tuples(np.concatenate([side(W, light_keys("spread", b, rng), rng) for _, b in lights]))
    descs = [(w * W, W, w * W, W, 0, 0) for w in range(n)]
    want, _ = oracle.join_windows(left, right, descs, enumerate_pairs=False)
    dl, dr = torch.from_numpy(left.view(np.uint8)).cuda(), torch.from_numpy(right.view(np.uint8)).cuda()
    with lib.Joiner(lib.ALG_HJ, lib.LAZY, partitioner=getattr(lib, part), max_tuples_per_window=W) as j:
        for _ in range(2):
            got = j.lazy_execute_batch(dl, dr, descs, mem=lib.MEM_DEVICE)
            for d, g, w in zip(descs, got, want):
                assert (g["count"], g["prod"]) == (w["count"], w["prod"]), d
