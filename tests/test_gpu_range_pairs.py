"""GPU tests of pairs and xor checksums from joins by ranges (range_join.cu):
sorted pair lists against the oracle's, truncation, crowded ranges (each key a
dozen times), and keys whose ranges do not fit."""
import numpy as np
import pytest

from helpers import make_tuples, sorted_pairs

pytestmark = pytest.mark.gpu

SIZES = [(50_000, 41_000), (0, 100), (4096, 4097), (20_000, 9_000)]


def keys(kind, n, rng, hot):
    if kind == "sparse":
        return rng.integers(0, 200_000, n, dtype=np.uint32)
    if kind == "thick":
        return rng.integers(0, max(n // 12, 1), n, dtype=np.uint32)
    k = rng.integers(0, 1 << 20, n, dtype=np.uint32)
    k[: min(n, hot)] = 99   # one key fills a range of the left side
    return k


@pytest.mark.parametrize("where", ["device", "host"])
@pytest.mark.parametrize("kind", ["sparse", "thick", "hot"])
@pytest.mark.parametrize("algo,mode", [("HJ", "RESULT_ATOMIC"), ("SMJ", "RESULT_ATOMIC"), ("HJ", "RESULT_COUNT_KERNEL")])
def test_pairs_of_every_window(lib, oracle, algo, mode, kind, where):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(21)
    lefts, rights, spans, lo, ro = [], [], [], 0, 0
    for nl, nr in SIZES:
        lefts.append(keys(kind, nl, rng, 5000))
        rights.append(keys(kind, nr, rng, 100))
        spans.append((lo, nl, ro, nr))
        lo, ro = lo + nl, ro + nr
    left, right = make_tuples(np.concatenate(lefts)), make_tuples(np.concatenate(rights))
    want = [oracle.join(left[a:a + b], right[c:c + d], pairs_capacity=1 << 21) for a, b, c, d in spans]
    caps = [w["count"] for w in want]
    if mode == "RESULT_ATOMIC":
        caps[2] //= 2   # truncated
    offs = np.concatenate([[0], np.cumsum(caps)])
    descs = [s + (int(o), int(c)) for s, o, c in zip(spans, offs, caps)]
    pairs = np.zeros(max(int(offs[-1]), 1), lib.PAIR_DTYPE)
    mem, l, r, p = lib.MEM_HOST, left, right, pairs
    if where == "device":
        mem = lib.MEM_DEVICE
        l, r, p = [torch.from_numpy(x.view(np.uint8)).cuda() for x in (left, right, pairs)]
    with lib.Joiner(getattr(lib, "ALG_" + algo), lib.LAZY, getattr(lib, mode), max_tuples_per_window=1 << 16) as j:
        for _ in range(2):
            got = j.lazy_execute_batch(l, r, descs, mem=mem, pairs=p)
            out = p.cpu().numpy().view(lib.PAIR_DTYPE) if where == "device" else p
            for i, (g, w) in enumerate(zip(got, want)):
                assert (g["count"], g["xor"], g["prod"]) == (w["count"], w["xor"], w["prod"]), i
                assert g["n_pairs"] == caps[i]
                have = sorted_pairs(out[offs[i]:offs[i] + caps[i]])
                if caps[i] == w["count"]:
                    assert np.array_equal(have, sorted_pairs(w["pairs"])), i
                else:
                    assert len(np.unique(have)) == len(have) and np.isin(have, sorted_pairs(w["pairs"])).all()
                    assert g["flags"] & lib.WR_PAIRS_TRUNCATED
