"""GPU test of hash ranges whose keys repeat: numbers of tuples per key around the
line to the table, more distinct keys than it has slots beside hot ones (sorted),
and the mark of its free slots among the keys."""
import numpy as np
import pytest

from helpers import make_tuples, sorted_pairs

pytestmark = pytest.mark.gpu

SIZES = [(70_000, 65_536), (3000, 9000), (1, 40_000), (100_001, 700), (700, 30_000)]


def keys_of(per, hot, mark, n, rng):
    k = rng.integers(0, max(1, int(n / per)), n, dtype=np.uint32) * np.uint32(0x9E3779B1)
    k[: min(n, hot)] = 77
    if mark:
        k[rng.integers(0, n, max(1, n // 50))] = 0xFFFFFFFF
    return rng.permutation(k)


@pytest.mark.parametrize("mark", [False, True])
@pytest.mark.parametrize("per,hot", [(0.25, 0), (1, 0), (2, 0), (3, 0), (4, 0), (8, 0), (60, 0), (900, 0), (0.25, 33),
                                     (0.25, 2000), (3, 300)])
def test_repeated_keys_by_ranges(lib, oracle, per, hot, mark):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(41)
    lefts, rights, descs, lo, ro = [], [], [], 0, 0
    for nl, nr in SIZES:
        lefts.append(keys_of(per, hot, mark, nl, rng))
        rights.append(keys_of(per, hot, mark, nr, rng))
        descs.append((lo, nl, ro, nr, 0, 0))
        lo, ro = lo + nl, ro + nr
    left, right = make_tuples(np.concatenate(lefts)), make_tuples(np.concatenate(rights))
    want, _ = oracle.join_windows(left, right, descs, enumerate_pairs=False)
    dl, dr = torch.from_numpy(left.view(np.uint8)).cuda(), torch.from_numpy(right.view(np.uint8)).cuda()
    with lib.Joiner(lib.ALG_HJ, lib.LAZY, flags=lib.F_PROFILE, max_tuples_per_window=1 << 17) as j:
        for _ in range(2):
            got = j.lazy_execute_batch(dl, dr, descs, mem=lib.MEM_DEVICE)
            for d, g, w in zip(descs, got, want):
                assert (g["count"], g["prod"]) == (w["count"], w["prod"]), d
        assert "range_join" in j.kernel_stats()


@pytest.mark.parametrize("per", [1, 3, 12, 25])
def test_pairs_of_repeated_keys_by_hash_ranges(lib, oracle, per):
    """Lists and (12 and more tuples per key) sorted ranges; the second window's pairs are cut short."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(43)
    sizes = [(70_000, 60_001), (9_000, 20_000), (5, 1000)]
    lefts = [keys_of(per, 0, False, nl, rng) for nl, _ in sizes]
    rights = [keys_of(per * max(1.0, nr / nl), 0, False, nr, rng) for nl, nr in sizes]
    spans, lo, ro = [], 0, 0
    for nl, nr in sizes:
        spans.append((lo, nl, ro, nr))
        lo, ro = lo + nl, ro + nr
    left, right = make_tuples(np.concatenate(lefts)), make_tuples(np.concatenate(rights))
    want = [oracle.join(left[a:a + b], right[c:c + d], pairs_capacity=1 << 22) for a, b, c, d in spans]
    caps = [w["count"] for w in want]
    caps[1] //= 2
    offs = np.concatenate([[0], np.cumsum(caps)])
    descs = [s + (int(o), int(c)) for s, o, c in zip(spans, offs, caps)]
    l, r, p = [torch.from_numpy(x.view(np.uint8)).cuda() for x in (left, right, np.zeros(int(offs[-1]), lib.PAIR_DTYPE))]
    with lib.Joiner(lib.ALG_HJ, lib.LAZY, lib.RESULT_ATOMIC, flags=lib.F_PROFILE, max_tuples_per_window=1 << 17) as j:
        for _ in range(2):
            got = j.lazy_execute_batch(l, r, descs, mem=lib.MEM_DEVICE, pairs=p)
            out = p.cpu().numpy().view(lib.PAIR_DTYPE)
            for i, (g, w) in enumerate(zip(got, want)):
                assert (g["count"], g["xor"], g["prod"], g["n_pairs"]) == (w["count"], w["xor"], w["prod"], caps[i]), i
                have = sorted_pairs(out[offs[i]:offs[i] + caps[i]])
                if i != 1:
                    assert np.array_equal(have, sorted_pairs(w["pairs"])), i
                else:
                    assert len(np.unique(have)) == len(have) and np.isin(have, sorted_pairs(w["pairs"])).all()
        assert "range_join" in j.kernel_stats()


@pytest.mark.parametrize("per", [1, 4])
@pytest.mark.parametrize("sizes", [[(1 << 20, 1 << 20)], [(1_063_000, 900_000)], [(1_064_500, 1_000_000)], [(65_536, 65_536)] * 16,
                                   [(66_400, 66_400)] * 16])
def test_one_wave_of_ranges(lib, oracle, sizes, per):
    """Sizes around those whose ranges are filled up to make one wave of CTAs."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(47)
    lefts = [keys_of(per, 0, False, nl, rng) for nl, _ in sizes]
    rights = [keys_of(per, 0, False, nr, rng) for _, nr in sizes]
    descs, lo, ro = [], 0, 0
    for nl, nr in sizes:
        descs.append((lo, nl, ro, nr, 0, 0))
        lo, ro = lo + nl, ro + nr
    left, right = make_tuples(np.concatenate(lefts)), make_tuples(np.concatenate(rights))
    want, _ = oracle.join_windows(left, right, descs, enumerate_pairs=False)
    dl, dr = torch.from_numpy(left.view(np.uint8)).cuda(), torch.from_numpy(right.view(np.uint8)).cuda()
    with lib.Joiner(lib.ALG_HJ, lib.LAZY, flags=lib.F_PROFILE, max_tuples_per_window=1 << 21) as j:
        got = j.lazy_execute_batch(dl, dr, descs, mem=lib.MEM_DEVICE)
        assert "range_join" in j.kernel_stats()
    for d, g, w in zip(descs, got, want):
        assert (g["count"], g["prod"]) == (w["count"], w["prod"]), d


@pytest.mark.parametrize("hot", [16, 17, 40, 1500, 3900])
@pytest.mark.parametrize("keys", [1, 3, 60])
def test_hot_subranges(lib, oracle, keys, hot):
    """Some keys of `hot` tuples each among distinct ones: lists, and a table behind
    them that the fullest ranges leave little room for."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(hot + keys)
    W = 70_000
    sides = []
    for _ in range(2):
        k = rng.permutation(np.arange(1, 1 << 20, dtype=np.uint32))[:W]
        if keys * hot <= W:
            k[: keys * hot] = np.repeat(np.arange(keys, dtype=np.uint32) * np.uint32(9973) + np.uint32(1 << 21), hot)
        sides.append(make_tuples(rng.permutation(k * np.uint32(0x9E3779B1))))
    left, right = sides
    want = oracle.join(left, right, enumerate_pairs=False)
    dl, dr = torch.from_numpy(left.view(np.uint8)).cuda(), torch.from_numpy(right.view(np.uint8)).cuda()
    with lib.Joiner(lib.ALG_HJ, lib.LAZY, flags=lib.F_PROFILE, max_tuples_per_window=1 << 17) as j:
        for _ in range(2):
            got = j.lazy_execute_batch(dl, dr, [(0, W, 0, W, 0, 0)], mem=lib.MEM_DEVICE)[0]
            assert (got["count"], got["prod"]) == (want["count"], want["prod"])
        assert "range_join" in j.kernel_stats()
