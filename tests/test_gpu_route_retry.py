"""GPU test of what a call whose keys do not fit leaves behind on its handle: the
next calls of its size take the general path, and later ones ranges or buckets
again; calls of other sizes are not concerned."""
import numpy as np
import pytest

from helpers import make_tuples

pytestmark = pytest.mark.gpu

WAIT = 16   # calls after the first miss


def window(n, hot, rng):
    k = rng.integers(0, 1 << 20, n, dtype=np.uint32)
    if hot:
        k[:6000] = 5
    return make_tuples(rng.permutation(k))


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("algo", ["HJ", "SMJ"])
def test_lazy_calls(lib, oracle, algo, graph):
    torch = pytest.importorskip("torch")
    W, other = 70_000, 300_000
    rng = np.random.default_rng(2)
    even, hot = [[window(W, h, rng) for _ in range(2)] for h in (False, True)]
    large = [torch.from_numpy(window(other, False, rng).view(np.uint8)).cuda() for _ in range(2)]
    want = {id(p): oracle.join(*p, enumerate_pairs=False) for p in (even, hot)}
    dev = [torch.empty(W * 16, dtype=torch.uint8, device="cuda") for _ in range(2)]
    with lib.Joiner(getattr(lib, "ALG_" + algo), lib.LAZY, flags=lib.F_GRAPH if graph else 0,
                    max_tuples_per_window=other) as j:
        def call(pair):
            for d, t in zip(dev, pair):
                d.copy_(torch.from_numpy(t.view(np.uint8)))
            torch.cuda.synchronize()
            before = j.launch_count()
            got = j.lazy_execute_batch(*dev, [(0, W, 0, W, 0, 0)], mem=lib.MEM_DEVICE)[0]
            assert (got["count"], got["prod"]) == (want[id(pair)]["count"], want[id(pair)]["prod"])
            return j.launch_count() - before

        ranges = call(even)
        assert call(even) == ranges
        assert call(hot) > ranges                     # ranges, then the general path
        general = call(hot)
        before = j.launch_count()
        j.lazy_execute_batch(*large, [(0, other, 0, other, 0, 0)], mem=lib.MEM_DEVICE)
        assert j.launch_count() - before == ranges    # another size
        assert general != ranges
        assert [call(even) for _ in range(WAIT - 1)] == [general] * (WAIT - 1)
        assert [call(even) for _ in range(3)] == [ranges] * 3
        assert call(hot) > max(ranges, general)
        assert [call(even) for _ in range(WAIT)] == [general] * WAIT   # (a hit lay between: 16 again)
        assert call(hot) > max(ranges, general)       # two misses without one
        assert [call(even) for _ in range(2 * WAIT)] == [general] * (2 * WAIT)
        assert call(even) == ranges


@pytest.mark.parametrize("algo", ["HJ", "SMJ"])
def test_recorded_streams(lib, oracle, algo):
    B, W, nb = 1024, 8192, 16
    rng = np.random.default_rng(3)
    even = [rng.integers(0, 4000, nb * B, dtype=np.uint32) for _ in range(2)]
    few = [rng.integers(0, 3, nb * B, dtype=np.uint32) for _ in range(2)]
    with lib.Joiner(getattr(lib, "ALG_" + algo), lib.EAGER, batch_size=B, window_size=W, max_tuples_per_window=W) as j:
        def call(keys, D):
            left, right = make_tuples(keys[0]), make_tuples(keys[1])
            before = j.launch_count()
            bc, _ = j.eager_run(left, right, nb)
            assert np.array_equal(bc, oracle.eager_hj(left, right, B, W, D)[0])
            return j.launch_count() - before

        grouped = call(even, 4000)
        assert call(few, 3) > grouped
        assert grouped not in [call(even, 4000) for _ in range(WAIT)]
        assert call(even, 4000) == grouped


def test_ring_windows(lib, oracle):
    W, nw = 70_000, WAIT + 6
    rng = np.random.default_rng(4)
    with lib.Joiner(lib.ALG_SMJ, lib.LAZY, max_tuples_per_window=W) as j:
        j.ring_open(W, 4)
        took = []
        for k in range(nw):
            pair = [window(W, k == 1, rng) for _ in range(2)]
            before = j.launch_count()
            for t, is_left in zip(pair, (True, False)):
                j.ring_push(t, is_left)
            got = []
            while not got:
                got = j.ring_poll()
            took.append(j.launch_count() - before)
            want = oracle.join(*pair, enumerate_pairs=False)
            assert (got[0]["count"], got[0]["prod"]) == (want["count"], want["prod"]), k
        j.ring_close()
    assert took[1] > took[0] and took[0] not in took[2:2 + WAIT - 1] and took[-3:] == [took[0]] * 3
