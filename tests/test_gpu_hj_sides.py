"""GPU tests of the hash join's windows whose sides or buckets differ in size:
the join builds from the smaller side, cuts long probe runs into pieces, cuts
both runs of a bucket far longer than its table, and does not partition a
window whose smaller side is one bucket."""
import numpy as np
import pytest

from helpers import make_tuples

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (0, 70000), (4096, 4097), (4097, 4096), (4096, 300_000), (300_000, 3), (5000, 200_001),
         (200_001, 5000), (70_000, 70_001), (2_000, 24_576), (24_577, 2_000), (1, 100_000),
         (400_000, 300_000)]


def keys_of(kind, n, rng):
    if kind == "dense":
        return rng.integers(0, 5000, n, dtype=np.uint32)
    if kind == "wide":   # the table's empty marker among them
        k = rng.integers(0, 1 << 18, n, dtype=np.uint32) * np.uint32(0x9E3779B1)
        k[:: 97] = 0xFFFFFFFF
        return k
    k = rng.integers(0, 1 << 20, n, dtype=np.uint32)   # hot: a third of the tuples hold one key
    k[:: 3] = 77
    return k


@pytest.mark.parametrize("part,bits", [("PART_AUTO", 0), ("PART_RADIX", 0), ("PART_RADIX", 1)])
@pytest.mark.parametrize("flags", ["count", "xor"])
@pytest.mark.parametrize("kind", ["dense", "wide", "hot"])
def test_windows_of_different_sides(lib, oracle, kind, flags, part, bits):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(11)
    lefts, rights, descs, lo, ro = [], [], [], 0, 0
    for nl, nr in SIZES:
        if flags == "xor" and kind == "hot" and nl * nr > 1 << 31:
            continue   # the oracle visits every pair
        lefts.append(keys_of(kind, nl, rng))
        rights.append(keys_of(kind, nr, rng))
        descs.append((lo, nl, ro, nr, 0, 0))
        lo, ro = lo + nl, ro + nr
    left, right = make_tuples(np.concatenate(lefts)), make_tuples(np.concatenate(rights))
    want, _ = oracle.join_windows(left, right, descs, enumerate_pairs=flags == "xor")
    dl, dr = torch.from_numpy(left.view(np.uint8)).cuda(), torch.from_numpy(right.view(np.uint8)).cuda()
    f = lib.F_XOR if flags == "xor" else 0
    with lib.Joiner(lib.ALG_HJ, lib.LAZY, partitioner=getattr(lib, part), flags=f, radix_bits=bits,
                    max_tuples_per_window=1 << 19) as j:
        got = j.lazy_execute_batch(dl, dr, descs, mem=lib.MEM_DEVICE)
    # (automatic: radix, by the largest window)
    assert got[0]["partitioner_used"] == lib.PART_RADIX
    for d, g, w in zip(descs, got, want):
        assert (g["count"], g["prod"]) == (w["count"], w["prod"]), d
        if flags == "xor":
            assert g["xor"] == w["xor"], d


RAW = [(1, 1), (0, 5), (5, 0), (1535, 1537), (4096, 4096), (5343, 5343), (3, 100_000), (100_000, 3), (700, 40_000)]


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("kind", ["dense", "wide", "hot"])
@pytest.mark.parametrize("windows", [RAW[:1], RAW[1:2], RAW[3:4], RAW[4:5], RAW, RAW * 30, RAW * 120,
                                     [(11_727, 11_727)], [(65_536, 65_536)], [(9000, 30_001), (20_000, 6000)]])
def test_calls_of_small_windows_only(lib, oracle, windows, kind, graph):
    """One launch for the call: one item, items passed by value, items in a list,
    more windows than it takes; repeated calls (accumulators left zero)."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(len(windows))
    lefts, rights, descs, lo, ro = [], [], [], 0, 0
    for nl, nr in windows:
        lefts.append(keys_of(kind, nl, rng))
        rights.append(keys_of(kind, nr, rng))
        descs.append((lo, nl, ro, nr, 0, 0))
        lo, ro = lo + nl, ro + nr
    left, right = make_tuples(np.concatenate(lefts)), make_tuples(np.concatenate(rights))
    want, _ = oracle.join_windows(left, right, descs, enumerate_pairs=False)
    dl, dr = torch.from_numpy(left.view(np.uint8)).cuda(), torch.from_numpy(right.view(np.uint8)).cuda()
    with lib.Joiner(lib.ALG_HJ, lib.LAZY, flags=lib.F_GRAPH if graph else 0, max_tuples_per_window=1 << 17) as j:
        for _ in range(3):
            got = j.lazy_execute_batch(dl, dr, descs, mem=lib.MEM_DEVICE)
            for d, g, w in zip(descs, got, want):
                assert (g["count"], g["prod"]) == (w["count"], w["prod"]), d


MIDDLE = [(40_000, 30_001), (4096, 4097), (3328, 6657), (1, 70_000), (0, 9000), (100_000, 100), (65_536, 65_537)]


@pytest.mark.parametrize("where", ["device", "host", "graph"])
@pytest.mark.parametrize("kind", ["dense", "wide", "hot", "thick"])
def test_calls_of_the_middle_sizes(lib, oracle, kind, where):
    """Hash ranges finished in shared memory; keys whose ranges do not fit (hot, or
    each key a thousand times) send the call to the general path."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(8)
    lefts, rights, descs, lo, ro = [], [], [], 0, 0
    for nl, nr in MIDDLE:
        make = (lambda n: rng.integers(0, 90, n, dtype=np.uint32)) if kind == "thick" else \
            (lambda n: keys_of(kind, n, rng))
        lefts.append(make(nl))
        rights.append(make(nr))
        descs.append((lo, nl, ro, nr, 0, 0))
        lo, ro = lo + nl, ro + nr
    left, right = make_tuples(np.concatenate(lefts)), make_tuples(np.concatenate(rights))
    want, _ = oracle.join_windows(left, right, descs, enumerate_pairs=False)
    mem = lib.MEM_HOST if where == "host" else lib.MEM_DEVICE
    if where != "host":
        left, right = torch.from_numpy(left.view(np.uint8)).cuda(), torch.from_numpy(right.view(np.uint8)).cuda()
    with lib.Joiner(lib.ALG_HJ, lib.LAZY, flags=lib.F_GRAPH if where == "graph" else 0,
                    max_tuples_per_window=1 << 17) as j:
        for _ in range(3):
            got = j.lazy_execute_batch(left, right, descs, mem=mem)
            for d, g, w in zip(descs, got, want):
                assert (g["count"], g["prod"]) == (w["count"], w["prod"]), d
