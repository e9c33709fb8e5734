"""GPU tests of eager batches read where they lie: pageable, pinned and device
memory, and addresses that are not 16-byte aligned (those are copied first),
with and without pair enumeration, for batch sizes around a CTA's."""
import numpy as np
import pytest

from helpers import make_tuples

pytestmark = pytest.mark.gpu

SIZES = [1, 255, 256, 257, 0, 1000, 3000]


def place(torch, t, kind):
    """The tuples in memory of the given kind, as (array or tensor, mem name)."""
    raw = torch.from_numpy(t.view(np.uint8).copy())
    if kind == "pageable":
        return t, "MEM_HOST"
    if kind == "pinned":
        return raw.pin_memory(), "MEM_HOST"
    if kind == "device":
        return raw.cuda(), "MEM_DEVICE"
    buf = torch.zeros(raw.numel() + 16, dtype=torch.uint8, device="cuda" if kind == "device+8" else "cpu")
    buf[8:8 + raw.numel()] = raw.to(buf.device)
    if kind == "device+8":
        torch.cuda.synchronize()   # the copy above is on another stream than the handle's
    return buf[8:8 + raw.numel()], "MEM_DEVICE" if kind == "device+8" else "MEM_HOST"


@pytest.mark.parametrize("xor", [False, True])
@pytest.mark.parametrize("kind", ["pageable", "pinned", "device", "device+8", "host+8"])
@pytest.mark.parametrize("algo", ["HJ", "SMJ", "NLJ"])
def test_batches_in_place(lib, oracle, algo, kind, xor):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(3)
    sides = [make_tuples(rng.integers(0, 300, sum(SIZES), dtype=np.uint32)) for _ in range(2)]
    sides[0]["key"][::50] = 0xFFFFFFFF
    sides[1]["key"][::70] = 0xFFFFFFFF
    with lib.Joiner(getattr(lib, "ALG_" + algo), lib.EAGER, batch_size=3000, window_size=sum(SIZES),
                    max_tuples_per_window=sum(SIZES), flags=lib.F_XOR if xor else 0) as j:
        for _ in range(2):   # the second window starts from cleared states
            at = 0
            for n in SIZES:
                for side in (0, 1):   # left, then right: a left batch meets `at` right tuples, a right one `at + n` left
                    b, mem = place(torch, sides[side][at:at + n], kind)
                    got = j.eager_execute(b, side == 0, mem=getattr(lib, mem), n=n)
                    other = sides[1 - side]["key"][:at + (n if side else 0)]
                    own = sides[side]["key"][at:at + n]
                    keys, cnt = np.unique(other, return_counts=True)
                    i = np.minimum(np.searchsorted(keys, own), max(len(keys) - 1, 0))
                    want = int(cnt[i][keys[i] == own].sum()) if len(keys) and n else 0
                    assert got == want, (n, side)
                at += n
            want = oracle.join(sides[0], sides[1], enumerate_pairs=True)
            res = j.eager_window_result()
            assert (res["count"], res["prod"]) == (want["count"], want["prod"])
            if xor:
                assert res["xor"] == want["xor"]
            j.eager_clear_states()
