"""GPU test of the ingest ring's joins by ranges: several windows in flight when
one of them holds keys whose ranges do not fit."""
import numpy as np
import pytest

from helpers import make_tuples
from test_gpu_ring import expected, push_all

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("algo", ["HJ", "SMJ"])
@pytest.mark.parametrize("hot", [(), (0,), (2, 3), (5,)])
def test_windows_in_flight_with_hot_keys(lib, oracle, algo, hot):
    W, nw = 70_000, 6
    rng = np.random.default_rng(4)
    sides = [rng.integers(0, 1 << 18, nw * W, dtype=np.uint32) for _ in range(2)]
    for k in hot:
        for s in sides:
            s[k * W:k * W + 9000] = 5
    left, right = make_tuples(sides[0]), make_tuples(sides[1])
    with lib.Joiner(getattr(lib, "ALG_" + algo), lib.LAZY, max_tuples_per_window=W) as j:
        j.ring_open(W, 4)
        res = push_all(j, left, right, 35_000)
        j.ring_close()
        res += j.ring_poll()
    want = expected(oracle, left, right, W, False)
    assert [(r["status"], r["count"], r["prod"]) for r in res] == [(0, w["count"], w["prod"]) for w in want]
