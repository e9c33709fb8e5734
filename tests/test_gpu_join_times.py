"""GPU test of the device times reported for joins that are made a second time
because a range of their keys does not fit: both passes are in them."""
import time

import numpy as np
import pytest

from helpers import make_tuples
from test_gpu_ring import expected

pytestmark = pytest.mark.gpu


def hot_window(n, rng):
    k = rng.integers(0, 1 << 22, n, dtype=np.uint32)
    k[:6000] = 5
    return rng.permutation(k)


@pytest.mark.parametrize("where", ["device", "host"])
def test_lazy_call(lib, oracle, where):
    torch = pytest.importorskip("torch")
    W, n = 400_000, 6
    rng = np.random.default_rng(8)
    left, right = [make_tuples(np.concatenate([hot_window(W, rng) for _ in range(n)])) for _ in range(2)]
    descs = [(w * W, W, w * W, W, 0, 0) for w in range(n)]
    want, _ = oracle.join_windows(left, right, descs, enumerate_pairs=False)
    mem = lib.MEM_HOST
    if where == "device":
        mem = lib.MEM_DEVICE
        left, right = [torch.from_numpy(t.view(np.uint8)).cuda() for t in (left, right)]
        torch.cuda.synchronize()
    with lib.Joiner(lib.ALG_SMJ, lib.LAZY, flags=lib.F_PROFILE, max_tuples_per_window=W) as j:
        got = j.lazy_execute_batch(left, right, descs, mem=mem)
        st = j.kernel_stats()
    for g, w in zip(got, want):
        assert (g["count"], g["prod"]) == (w["count"], w["prod"])
    assert "range_join" in st and "merge_join_count" in st   # (two passes)
    # the kernels of both passes ran one after another inside the reported time
    assert got[0]["ms"] >= sum(ms for _, ms in st.values())


def wait_one(j):
    for _ in range(5000):
        got = j.ring_poll()   # (does not wait)
        if got:
            return got[0]
        time.sleep(0.001)
    raise AssertionError("no window reported")


def test_ring_window(lib, oracle):
    """A hot window after an even one: its time is from the copies to the end of its second join."""
    W = 1 << 20
    rng = np.random.default_rng(9)
    even = [make_tuples(rng.integers(0, 1 << 22, W, dtype=np.uint32)) for _ in range(2)]
    hot = [make_tuples(hot_window(W, rng)) for _ in range(2)]
    with lib.Joiner(lib.ALG_SMJ, lib.LAZY, flags=lib.F_PROFILE, max_tuples_per_window=W) as j:
        j.lazy_execute(*hot)
        general = sum(ms for k, (_, ms) in j.kernel_stats().items() if not k.startswith("range_"))
    with lib.Joiner(lib.ALG_SMJ, lib.LAZY, max_tuples_per_window=W) as j:
        j.ring_open(W, 4)
        for window in (even, hot):   # (the even one sizes the first join's buffers)
            j.ring_push(window[0], True)
            j.ring_push(window[1], False)
            got = wait_one(j)
            want = expected(oracle, *window, W, False)[0]
            assert (got["status"], got["count"], got["prod"]) == (0, want["count"], want["prod"])
        j.ring_close()
    assert got["ms"] > 0.6 * general
