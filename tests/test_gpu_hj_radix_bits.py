"""GPU test of radix handles with a given number of bits, few tuples per bucket to
many: the counting pass keeps its number of CTAs with many buckets, long and hot
buckets are cut into pieces, small ones come by the thousand."""
import numpy as np
import pytest

from helpers import make_tuples

pytestmark = pytest.mark.gpu


def keys_of(kind, n, rng):
    if kind == "sparse":
        return rng.integers(0, n, n, dtype=np.uint32) * np.uint32(0x9E3779B1)
    if kind == "dense":
        return rng.integers(0, n, n, dtype=np.uint32)
    if kind == "repeats":
        return rng.integers(0, n // 8, n, dtype=np.uint32) * np.uint32(0x9E3779B1)
    k = rng.integers(0, n, n, dtype=np.uint32)   # hot: a third of the tuples hold one key, a tenth another
    k[: n // 3] = 77
    k[n // 3: n // 3 + n // 10] = 0xFFFFFFFF
    return rng.permutation(k)


@pytest.mark.parametrize("bits", [1, 5, 7, 10, 12, 14])
@pytest.mark.parametrize("kind", ["sparse", "dense", "repeats", "hot"])
def test_bits(lib, oracle, kind, bits):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(bits)
    sizes = [(400_000, 500_003), (30_000, 9_000), (5, 7)]
    lefts, rights, descs, lo, ro = [], [], [], 0, 0
    for nl, nr in sizes:
        lefts.append(keys_of(kind, nl, rng) if nl > 100 else np.arange(nl, dtype=np.uint32))
        rights.append(keys_of(kind, nr, rng) if nr > 100 else np.arange(nr, dtype=np.uint32))
        descs.append((lo, nl, ro, nr, 0, 0))
        lo, ro = lo + nl, ro + nr
    left, right = make_tuples(np.concatenate(lefts)), make_tuples(np.concatenate(rights))
    want, _ = oracle.join_windows(left, right, descs, enumerate_pairs=False)
    dl, dr = torch.from_numpy(left.view(np.uint8)).cuda(), torch.from_numpy(right.view(np.uint8)).cuda()
    with lib.Joiner(lib.ALG_HJ, lib.LAZY, partitioner=lib.PART_RADIX, radix_bits=bits, max_tuples_per_window=1 << 19) as j:
        for _ in range(2):
            got = j.lazy_execute_batch(dl, dr, descs, mem=lib.MEM_DEVICE)
            for d, g, w in zip(descs, got, want):
                assert (g["count"], g["prod"]) == (w["count"], w["prod"]), d


def test_counting_pass_of_many_buckets(lib):
    """2^14 buckets: the pass over 512 tiles takes well under twice that of 2^12 buckets."""
    torch = pytest.importorskip("torch")
    n = 1 << 20
    t = torch.zeros((n, 4), dtype=torch.int32, device="cuda")
    t[:, 0] = torch.randperm(n, device="cuda", dtype=torch.int32)
    t[:, 1] = torch.arange(n, device="cuda", dtype=torch.int32)
    torch.cuda.synchronize()
    ms = {}
    for bits in (12, 14):
        with lib.Joiner(lib.ALG_HJ, lib.LAZY, partitioner=lib.PART_RADIX, radix_bits=bits, flags=lib.F_PROFILE,
                        max_tuples_per_window=n) as j:
            for k in range(6):
                if k == 2:
                    j.kernel_stats_reset()
                got = j.lazy_execute_batch(t, t, [(0, n, 0, n, 0, 0)], mem=lib.MEM_DEVICE)[0]
                assert got["count"] == n
            ms[bits] = j.kernel_stats()["part_hist"][1]
    assert ms[14] < 2 * ms[12]


@pytest.mark.parametrize("windows,n", [(1, 600_000), (3, 250_000), (40, 60_000)])
def test_hot_buckets_in_pieces(lib, oracle, windows, n):
    """One hot bucket of a call in many pieces, many of them in few or one."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(windows)
    left, right = [make_tuples(np.concatenate([keys_of("hot", n, rng) for _ in range(windows)])) for _ in range(2)]
    descs = [(w * n, n, w * n, n, 0, 0) for w in range(windows)]
    want, _ = oracle.join_windows(left, right, descs, enumerate_pairs=False)
    dl, dr = torch.from_numpy(left.view(np.uint8)).cuda(), torch.from_numpy(right.view(np.uint8)).cuda()
    for bits in (0, 2):
        with lib.Joiner(lib.ALG_HJ, lib.LAZY, partitioner=lib.PART_RADIX, radix_bits=bits, max_tuples_per_window=n) as j:
            got = j.lazy_execute_batch(dl, dr, descs, mem=lib.MEM_DEVICE)
            for d, g, w in zip(descs, got, want):
                assert (g["count"], g["prod"]) == (w["count"], w["prod"]), d
