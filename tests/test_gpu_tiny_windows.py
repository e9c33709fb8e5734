"""GPU test of automatic hash joins over many tiny windows: tables in HBM rather
than hash ranges, whose tiles would take hundreds of times the tuples' space."""
import numpy as np
import pytest

from helpers import make_tuples

pytestmark = pytest.mark.gpu


def batch(sizes, rng, spread):
    lefts, rights, descs, lo, ro = [], [], [], 0, 0
    for nl, nr in sizes:
        lefts.append(rng.integers(0, spread * max(nl, nr, 1), nl, dtype=np.uint32))
        rights.append(rng.integers(0, spread * max(nl, nr, 1), nr, dtype=np.uint32))
        descs.append((lo, nl, ro, nr, 0, 0))
        lo, ro = lo + nl, ro + nr
    return make_tuples(np.concatenate(lefts)), make_tuples(np.concatenate(rights)), descs


@pytest.mark.parametrize("xor", [False, True])
@pytest.mark.parametrize("sizes,ranges", [([(16, 16)] * 20_000, False), ([(64, 70)] * 1100 + [(9000, 9000)], False),
                                          ([(0, 50), (300, 1)] * 700, False), ([(4000, 4000)] * 400 + [(9000, 9000)], True),
                                          ([(2000, 2500)] * 60 + [(70_000, 70_000)], True)])
def test_route_and_results(lib, oracle, sizes, ranges, xor):
    torch = pytest.importorskip("torch")
    left, right, descs = batch(sizes, np.random.default_rng(3), 2)
    want, _ = oracle.join_windows(left, right, descs, enumerate_pairs=xor)
    dl, dr = torch.from_numpy(left.view(np.uint8)).cuda(), torch.from_numpy(right.view(np.uint8)).cuda()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    with lib.Joiner(lib.ALG_HJ, lib.LAZY, flags=lib.F_PROFILE | (lib.F_XOR if xor else 0),
                    max_tuples_per_window=1 << 17) as j:
        got = j.lazy_execute_batch(dl, dr, descs, mem=lib.MEM_DEVICE)
        took = free - torch.cuda.mem_get_info()[0]
        assert any(k.startswith("range_join") for k in j.kernel_stats()) == ranges
    if not ranges:   # plans and tables: a few hundred bytes per window and some tens per tuple
        assert took < (64 << 20) + 1024 * len(sizes) + 64 * (len(left) + len(right))
    for d, g, w in zip(descs, got, want):
        assert (g["count"], g["prod"]) == (w["count"], w["prod"]), d
        if xor:
            assert g["xor"] == w["xor"], d
