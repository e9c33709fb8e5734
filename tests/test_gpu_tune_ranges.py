"""GPU test of the tuner on automatic handles: the untuned choice, which may go by
hash ranges, is among the settings it times, and its decision is kept."""
import numpy as np
import pytest

from helpers import make_tuples

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("xor", [False, True])
@pytest.mark.parametrize("hot", [False, True])
def test_tuned_call(lib, oracle, tmp_path, monkeypatch, hot, xor):
    torch = pytest.importorskip("torch")
    monkeypatch.setenv("SJBG_TUNE_CACHE", str(tmp_path / "tune.json"))
    W = 1_000_003
    rng = np.random.default_rng(6)
    keys = [rng.integers(0, 1 << 22, W, dtype=np.uint32) for _ in range(2)]
    if hot:   # does not fit its range
        keys[0][:6000] = 5
    left, right = make_tuples(keys[0]), make_tuples(keys[1])
    want = oracle.join(left, right, enumerate_pairs=xor)
    dl, dr = torch.from_numpy(left.view(np.uint8)).cuda(), torch.from_numpy(right.view(np.uint8)).cuda()
    torch.cuda.synchronize()
    flags = lib.F_AUTOTUNE | lib.F_PROFILE | (lib.F_XOR if xor else 0)
    for _ in range(2):   # the second handle reads the first one's decision
        with lib.Joiner(lib.ALG_HJ, lib.LAZY, flags=flags, max_tuples_per_window=W) as j:
            for k in range(3):
                if k == 1:
                    j.kernel_stats_reset()
                got = j.lazy_execute_batch(dl, dr, [(0, W, 0, W, 0, 0)], mem=lib.MEM_DEVICE)[0]
                assert (got["count"], got["prod"]) == (want["count"], want["prod"])
                if xor:
                    assert got["xor"] == want["xor"]
            # (ranges take some 55 us, the others 85 and more)
            assert ("range_join" in {k for k, v in j.kernel_stats().items() if v[0]}) == (not hot)
