"""GPU tests of recorded eager streams counted by buckets: batches of one tile,
of a ragged tile and of several, windows that open with either side, key groups
that are too large for it (sorted instead, and from then on), strided keys."""
import numpy as np
import pytest

from helpers import make_tuples
from test_gpu_eager import window_members

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("algo", ["HJ", "SMJ"])
@pytest.mark.parametrize("B,W,D,nb,stride", [(1024, 4096, 4096, 20, 1), (1500, 6000, 900, 11, 1), (5000, 20000, 20000, 13, 1),
                                             (4097, 5000, 1 << 12, 9, 1), (4096, 1 << 17, 1 << 17, 40, 1 << 14),
                                             (1023, 4000, 1000, 9, 1), (4096, 8192, 3, 7, 1), (2048, 1 << 16, 40, 40, 1)])
def test_batch_counts_and_totals(lib, oracle, algo, B, W, D, nb, stride):
    rng = np.random.default_rng(B + W)
    ranks = [rng.integers(0, D, nb * B, dtype=np.uint32) for _ in range(2)]
    # counts by rank (the oracle's keys must be dense), joined as rank * stride, one rank as 0xFFFFFFFF
    left, right = [make_tuples(np.where(r == D - 1, np.uint32(0xFFFFFFFF), r * np.uint32(stride))) for r in ranks]
    want_bc, want_wc = oracle.eager_hj(make_tuples(ranks[0]), make_tuples(ranks[1]), B, W, D)
    with lib.Joiner(getattr(lib, "ALG_" + algo), lib.EAGER, batch_size=B, window_size=W, max_tuples_per_window=W) as j:
        for _ in range(2):
            bc, wins = j.eager_run(left, right, nb)
            assert np.array_equal(bc, want_bc)
            members = window_members(nb, B, W)
            assert len(wins) == len(members) == len(want_wc)
            for w, (lb, rb), wc in zip(wins, members, want_wc):
                l = np.concatenate([left[b * B:(b + 1) * B] for b in lb]) if lb else left[:0]
                r = np.concatenate([right[b * B:(b + 1) * B] for b in rb]) if rb else right[:0]
                e = oracle.join(l, r, enumerate_pairs=False)
                assert (w["count"], w["prod"]) == (e["count"], e["prod"]) and w["count"] == int(wc)


@pytest.mark.parametrize("persistent", [False, True])
def test_a_recorded_stream_leaves_no_window_behind(lib, oracle, persistent):
    """eager_run between two windows of per-batch calls: the batches before it are gone."""
    B = 1024
    left = make_tuples(np.arange(2 * B, dtype=np.uint32) % 700)
    right = make_tuples(np.arange(2 * B, dtype=np.uint32) % 900)
    with lib.Joiner(lib.ALG_HJ, lib.EAGER, batch_size=B, window_size=2 * B, max_tuples_per_window=2 * B,
                    flags=lib.F_PERSISTENT if persistent else 0) as j:
        counts = []
        for _ in range(2):
            counts.append([j.eager_execute(left[:B], True), j.eager_execute(right[:B], False)])
            bc, _ = j.eager_run(left, right, 2)
            assert list(bc[:2]) == counts[-1] and counts[-1] == counts[0]
        assert counts[0][1] == oracle.join(left[:B], right[:B], enumerate_pairs=False)["count"]
