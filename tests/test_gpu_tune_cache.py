"""GPU test of a tuning cache whose line names the learned partitioner for an
automatic handle: windows of one bucket among larger ones are partitioned as the
rest of the call is."""
import json
import math

import numpy as np
import pytest

from helpers import make_tuples

pytestmark = pytest.mark.gpu


def test_cached_learned_choice_with_windows_of_one_bucket(lib, oracle, tmp_path, monkeypatch):
    torch = pytest.importorskip("torch")
    sizes = [(3000, 2000), (60_000, 50_000), (4000, 9000), (0, 10), (1, 1), (100, 70_000)]
    rng = np.random.default_rng(5)
    lefts, rights, descs, lo, ro = [], [], [], 0, 0
    for nl, nr in sizes:
        for side, n in ((lefts, nl), (rights, nr)):
            k = rng.integers(0, 20_000, n, dtype=np.uint32)
            k[: n // 2] %= np.uint32(50)
            side.append(k)
        descs.append((lo, nl, ro, nr, 0, 0))
        lo, ro = lo + nl, ro + nr
    left, right = make_tuples(np.concatenate(lefts)), make_tuples(np.concatenate(rights))
    want, _ = oracle.join_windows(left, right, descs, enumerate_pairs=False)
    shape = "hj-part%d-enum0-t%d-w%d-sm%d" % (lib.PART_AUTO, int(math.log2(lo + ro)), int(math.log2(len(sizes))),
                                             torch.cuda.get_device_properties(0).multi_processor_count)
    cache = tmp_path / "tune.json"
    cache.write_text(json.dumps({"shape": shape, "bucket_target": 4096, "persistent": 1,
                                 "partitioner": lib.PART_LEARNED, "ms": 0.1}) + "\n")
    monkeypatch.setenv("SJBG_TUNE_CACHE", str(cache))
    dl, dr = torch.from_numpy(left.view(np.uint8)).cuda(), torch.from_numpy(right.view(np.uint8)).cuda()
    before = dl.clone(), dr.clone()
    torch.cuda.synchronize()
    with lib.Joiner(lib.ALG_HJ, lib.LAZY, flags=lib.F_AUTOTUNE | lib.F_PROFILE, max_tuples_per_window=1 << 17) as j:
        got = j.lazy_execute_batch(dl, dr, descs, mem=lib.MEM_DEVICE)
        assert "learned_sample" in j.kernel_stats()   # (the line was taken)
    for d, g, w in zip(descs, got, want):
        assert (g["count"], g["prod"]) == (w["count"], w["prod"]), d
    assert torch.equal(dl, before[0]) and torch.equal(dr, before[1])
