"""GPU tests of the sort-merge join by key ranges: edges of tiles and ranges,
keys over the whole 32-bit domain, sides of different sizes, and keys whose
ranges do not fit (a hot key, a cluster with an outlier), which the full sort
takes - on a first call, in a graph replay and for host inputs."""
import numpy as np
import pytest

from helpers import make_tuples

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (0, 3000), (3000, 0), (4096, 4097), (4095, 1), (3072, 3073), (6145, 6144), (50_000, 700),
         (900, 130_000), (100_001, 99_999)]


def keys_of(kind, n, rng):
    if kind == "dense":
        return rng.integers(0, 60_000, n, dtype=np.uint32)
    if kind == "wide":
        k = rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32) & np.uint32(0xFFFFC000)
        k[:: 61] = 0xFFFFFFFF
        k[1:: 61] = 0
        return k
    if kind == "hot":
        k = rng.integers(0, 1 << 22, n, dtype=np.uint32)
        k[:: 2] = 12345
        return k
    k = rng.integers(1 << 20, (1 << 20) + 70_000, n, dtype=np.uint32)   # a cluster, and one key far off
    k[: 1] = 0xFFFFFFF0
    return k


def windows(kind, rng, sizes=SIZES):
    lefts, rights, descs, lo, ro = [], [], [], 0, 0
    for nl, nr in sizes:
        lefts.append(keys_of(kind, nl, rng))
        rights.append(keys_of(kind, nr, rng))
        descs.append((lo, nl, ro, nr, 0, 0))
        lo, ro = lo + nl, ro + nr
    return make_tuples(np.concatenate(lefts)), make_tuples(np.concatenate(rights)), descs


def check(got, want, descs):
    for d, g, w in zip(descs, got, want):
        assert (g["count"], g["prod"]) == (w["count"], w["prod"]), d


@pytest.mark.parametrize("where", ["device", "host", "graph"])
@pytest.mark.parametrize("kind", ["dense", "wide", "hot", "cluster"])
def test_windows_by_key_ranges(lib, oracle, kind, where):
    torch = pytest.importorskip("torch")
    left, right, descs = windows(kind, np.random.default_rng(5))
    want, _ = oracle.join_windows(left, right, descs, enumerate_pairs=False)
    mem = lib.MEM_HOST if where == "host" else lib.MEM_DEVICE
    if where != "host":
        left, right = torch.from_numpy(left.view(np.uint8)).cuda(), torch.from_numpy(right.view(np.uint8)).cuda()
    with lib.Joiner(lib.ALG_SMJ, lib.LAZY, flags=lib.F_GRAPH if where == "graph" else 0,
                    max_tuples_per_window=1 << 18) as j:
        for _ in range(3):
            check(j.lazy_execute_batch(left, right, descs, mem=mem), want, descs)
        # one window alone: host inputs take another way in
        one = j.lazy_execute_batch(left, right, descs[3:4], mem=mem)
        check(one, want[3:4], descs[3:4])


def test_graph_replay_meets_keys_that_do_not_fit(lib, oracle):
    """The buffers of a captured call get other tuples: the replay's status sends the call to the full sort."""
    torch = pytest.importorskip("torch")
    sizes = [(60_000, 50_000), (3000, 9000)]
    with lib.Joiner(lib.ALG_SMJ, lib.LAZY, flags=lib.F_GRAPH, max_tuples_per_window=1 << 16) as j:
        dl = torch.zeros(63_000 * 16, dtype=torch.uint8, device="cuda")
        dr = torch.zeros(59_000 * 16, dtype=torch.uint8, device="cuda")
        for kind in ("dense", "dense", "hot", "cluster", "dense"):
            left, right, descs = windows(kind, np.random.default_rng(6), sizes)
            want, _ = oracle.join_windows(left, right, descs, enumerate_pairs=False)
            dl.copy_(torch.from_numpy(left.view(np.uint8)))
            dr.copy_(torch.from_numpy(right.view(np.uint8)))
            torch.cuda.synchronize()
            check(j.lazy_execute_batch(dl, dr, descs, mem=lib.MEM_DEVICE), want, descs)
