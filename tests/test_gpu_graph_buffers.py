"""GPU test of captured calls (F_GRAPH) on a handle whose workspaces grow: a call
that needs larger buffers frees those that the captured kernels hold the
addresses of, so the smaller call is captured again, on the new ones."""
import numpy as np
import pytest

from helpers import make_tuples

pytestmark = pytest.mark.gpu

SMALL, LARGE = [(3000, 2500), (700, 5000)], [(400_000, 300_000), (90_000, 150_001)]


def batch(torch, sizes, skewed, rng):
    """Device tensors of a batch and its windows, with room to be filled again in place."""
    nl, nr = sum(s[0] for s in sizes), sum(s[1] for s in sizes)
    descs, lo, ro = [], 0, 0
    for l, r in sizes:
        descs.append((lo, l, ro, r, 0, 0))
        lo, ro = lo + l, ro + r
    dev = [torch.empty(n * 16, dtype=torch.uint8, device="cuda") for n in (nl, nr)]

    def fill():
        host = []
        for d, n in zip(dev, (nl, nr)):
            k = rng.integers(0, 50_000, n, dtype=np.uint32)
            if skewed:
                k[rng.random(n) < 0.6] %= np.uint32(40)
            t = make_tuples(k)
            d.copy_(torch.from_numpy(t.view(np.uint8)))
            host.append(t)
        torch.cuda.synchronize()
        return host

    return dev, descs, fill


@pytest.mark.parametrize("grow", ["device", "host"])
@pytest.mark.parametrize("algo,part,skewed", [("HJ", "PART_AUTO", False), ("HJ", "PART_NONE", False),
                                              ("HJ", "PART_RADIX", False), ("HJ", "PART_LEARNED", True),
                                              ("SMJ", "PART_AUTO", False)])
def test_small_large_small(lib, oracle, algo, part, skewed, grow):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(21)
    small, large = batch(torch, SMALL, skewed, rng), batch(torch, LARGE, skewed, rng)
    with lib.Joiner(getattr(lib, "ALG_" + algo), lib.LAZY, partitioner=getattr(lib, part), flags=lib.F_GRAPH,
                    max_tuples_per_window=1 << 19) as j:
        for dev, descs, fill in (small, small, large, small, small, large, large, small):
            left, right = fill()
            want, _ = oracle.join_windows(left, right, descs, enumerate_pairs=False)
            if grow == "host" and dev is large[0]:
                got = j.lazy_execute_batch(left, right, descs, mem=lib.MEM_HOST)
            else:
                got = j.lazy_execute_batch(*dev, descs, mem=lib.MEM_DEVICE)
            for g, w in zip(got, want):
                assert (g["count"], g["prod"]) == (w["count"], w["prod"])
