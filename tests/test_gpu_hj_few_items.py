"""GPU test of radix joins with few buckets in use: one, fewer than SMs, as many,
one more, and about one for each join CTA."""
import numpy as np
import pytest

from helpers import make_tuples

pytestmark = pytest.mark.gpu

BITS = 9


@pytest.mark.parametrize("per", [40, 3000])
@pytest.mark.parametrize("used", [1, 2, 75, 76, 77, 151, 152, 153, 303, 304, 305, 512])
def test_few_buckets(lib, oracle, used, per):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(used)
    buckets = rng.permutation(1 << BITS)[:used].astype(np.uint32)

    def side(n):
        return make_tuples(rng.integers(0, n, n, dtype=np.uint32) << BITS | buckets[rng.integers(0, used, n)])

    left, right = side(used * per), side(used * per + 100)
    descs = [(0, len(left), 0, len(right), 0, 0)]
    want, _ = oracle.join_windows(left, right, descs, enumerate_pairs=False)
    dl, dr = torch.from_numpy(left.view(np.uint8)).cuda(), torch.from_numpy(right.view(np.uint8)).cuda()
    with lib.Joiner(lib.ALG_HJ, lib.LAZY, partitioner=lib.PART_RADIX, radix_bits=BITS,
                    max_tuples_per_window=len(right)) as j:
        for _ in range(2):
            got = j.lazy_execute_batch(dl, dr, descs, mem=lib.MEM_DEVICE)
            assert (got[0]["count"], got[0]["prod"]) == (want[0]["count"], want[0]["prod"])
