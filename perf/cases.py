"""Performance cases of the stream-join library: what its users have it do, through its public calls.

A case is a dict of plain values.  prepare() makes what a program has in hand before the call (the
streams, on the GPU or in pinned host memory as the call takes them, and the joiner that such a
program keeps for all its windows), run() is one pass through the public entry points, exact() the
same results from plain torch, and work() the bytes and compares that a pass cannot do without.
"""
import ctypes
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "gpu-stream-join-benchmark_gb300"))
import sjbg  # noqa: E402

ALGORITHMS = {"hj": sjbg.ALG_HJ, "smj": sjbg.ALG_SMJ, "nlj": sjbg.ALG_NLJ}
PARTITIONERS = {"auto": sjbg.PART_AUTO, "learned": sjbg.PART_LEARNED}


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # One small window per call, as a program that joins each window when it closes:
        # launches and the host's share of the call are what it costs.
        lazy("hj_window_4096", "hj", 1, 4096, 4096, 1.0),
        # One large window of an odd length with mostly distinct keys.
        lazy("hj_window_1m", "hj", 1, 1_000_003, 1_000_003, 4.0),
        # The uniform workload: 16 windows of 65,536 tuples per stream, keys in [0, 65,536).
        lazy("hj_uniform_16x65536", "hj", 16, 65536, 65536, 1.0),
        # A foreign-key join whose pairs are written and consumed (each right tuple's partner).
        pairs("hj_foreign_key_pairs", 500_009, 2_000_003),
        # The headline workload: 8 windows of 2^24 tuples per stream, Zipf 1.5, learned
        # partitioning, buffers kept by the program and the call replayed as a graph.
        lazy("hj_skewed_z1.5_8x2p24", "hj", 8, 1 << 24, 1 << 24, 1.0, zipf=1.5, partitioner="learned", graph=True),
        # Moderate skew, windows of an odd length, each call on its own (no replay).
        lazy("hj_skewed_z1.0_2x5m", "hj", 2, 5_000_011, 5_000_011, 1.0, zipf=1.0, partitioner="learned"),
        # Many uneven windows in one call, 2^10 to 2^20 tuples per stream, keys in [0, 4W).
        lazy("hj_batched_1024", "hj", 1024, 1 << 10, 1 << 20, 4.0),
        # The same kind of batch through the sort-merge join.
        lazy("smj_batched_128", "smj", 128, 1 << 10, 1 << 20, 4.0),
        # A recorded stream through the eager sort-merge join, windows of 2^20, batches of 4,096.
        eager_run("eager_run_smj_2p20", "smj", 1 << 20, 4096, 768),
        # The same through the eager nested-loop join, windows of 65,536.
        eager_run("eager_run_nlj_65536", "nlj", 65536, 4096, 32),
        # Batches joined as they arrive from pinned host memory: one window of an eager hash join.
        eager_batches("eager_hj_batches", "hj", 1 << 17, 4096, 32),
        # Count windows through the device-resident ring, fed batch by batch from pinned host memory.
        ring("ring_hj_65536", "hj", 65536, 4096, 8),
    ]


def lazy(name, algorithm, windows, lo, hi, keys_per_tuple, zipf=0.0, partitioner="auto", graph=False, xor=False):
    return {"name": name, "op": "lazy", "algorithm": algorithm, "windows": windows, "lo": lo, "hi": hi,
            "keys_per_tuple": keys_per_tuple, "zipf": zipf, "partitioner": partitioner, "graph": graph, "xor": xor}


def pairs(name, n_left, n_right):
    return {"name": name, "op": "pairs", "n_left": n_left, "n_right": n_right}


def eager_run(name, algorithm, window, batch, n_batches):
    return {"name": name, "op": "eager_run", "algorithm": algorithm, "window": window, "batch": batch,
            "n_batches": n_batches}


def eager_batches(name, algorithm, window, batch, n_batches):
    return {"name": name, "op": "eager_batches", "algorithm": algorithm, "window": window, "batch": batch,
            "n_batches": n_batches}


def ring(name, algorithm, window, batch, windows):
    return {"name": name, "op": "ring", "algorithm": algorithm, "window": window, "batch": batch, "windows": windows}


def _log_uniform(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["window", "windows", "skewed", "uneven", "smj", "pairs", "eager_smj", "eager_nlj",
                       "eager_batches", "ring"])
    per = rng.choice([0.5, 1.0, 4.0])
    if kind == "window":
        n = _log_uniform(rng, 1000, 1 << 24)
        c = lazy("", "hj", 1, n, n, per, xor=rng.random() < 0.2 and n < 1 << 21 and per >= 1.0)
    elif kind == "windows":
        n = _log_uniform(rng, 1000, 1 << 20)
        c = lazy("", "hj", _log_uniform(rng, 2, 64), n, n, per)
    elif kind == "skewed":
        n = _log_uniform(rng, 1 << 20, 1 << 24)
        c = lazy("", "hj", rng.randint(1, 4), n, n, 1.0, zipf=rng.choice([0.5, 1.0, 1.25, 1.5]), partitioner="learned",
                 graph=rng.random() < 0.5)
    elif kind == "uneven":
        lo = _log_uniform(rng, 1 << 10, 1 << 14)
        c = lazy("", "hj", _log_uniform(rng, 16, 512), lo, lo * rng.choice([8, 64]), per)
    elif kind == "smj":
        lo = _log_uniform(rng, 1 << 10, 1 << 18)
        c = lazy("", "smj", _log_uniform(rng, 1, 64), lo, min(1 << 21, lo * rng.choice([1, 8, 64])), per)
    elif kind == "pairs":
        c = pairs("", _log_uniform(rng, 10_000, 4_000_000), _log_uniform(rng, 10_000, 4_000_000))
    elif kind == "eager_smj":
        b = rng.choice([1024, 3000, 4096])
        w = b * _log_uniform(rng, 8, 512)
        c = eager_run("", rng.choice(["smj", "hj"]), w, b, max(2, _log_uniform(rng, 1 << 16, 1 << 22) // b))
    elif kind == "eager_nlj":
        b = rng.choice([1000, 4096])
        c = eager_run("", "nlj", b * rng.randint(4, 24), b, rng.randint(8, 32))
    elif kind == "eager_batches":
        b = rng.choice([512, 1000, 4096])
        n = rng.randint(4, 64)
        c = eager_batches("", rng.choice(["hj", "smj"]), b * n, b, n)
    else:
        w = _log_uniform(rng, 1 << 13, 1 << 19)
        c = ring("", rng.choice(["hj", "smj"]), w, min(w, rng.choice([4096, 10_000])), rng.randint(2, 8))
    del c["name"]
    return c


# ---------------------------------------------------------------- inputs
def _sizes(case):
    """Tuples of each window of a lazy case, (left, right); part of the case, not of the seed."""
    r = random.Random(case["windows"] * 1_000_003 + case["lo"])
    if case["lo"] == case["hi"]:
        return [(case["lo"], case["lo"])] * case["windows"]
    return [(_log_uniform(r, case["lo"], case["hi"]), _log_uniform(r, case["lo"], case["hi"]))
            for _ in range(case["windows"])]


def _gen(seed, side):
    g = torch.Generator(device="cuda")
    g.manual_seed(2 * seed + side)
    return g


def _tuples(keys):
    """16-byte tuples {key, val = index, ts = index} of a stream's keys (int64 on the GPU)."""
    n = keys.numel()
    t = torch.empty((n, 4), dtype=torch.int32, device="cuda")
    index = torch.arange(n, dtype=torch.int64, device="cuda")
    t[:, 0] = keys.to(torch.int32)
    t[:, 1] = index.to(torch.int32)
    t[:, 2] = index.to(torch.int32)
    t[:, 3] = 0
    return t


class _Zipf:
    """Zipf(z) ranks over [0, domain), mapped to keys by a permutation both streams share."""

    def __init__(self, domain, z, seed):
        w = torch.arange(1, domain + 1, dtype=torch.float64, device="cuda").pow_(-z)
        self.cdf = torch.cumsum(w, 0)
        self.cdf /= self.cdf[-1].clone()
        self.perm = torch.randperm(domain, device="cuda", generator=_gen(seed, 7))

    def keys(self, n, g):
        u = torch.rand(n, dtype=torch.float64, device="cuda", generator=g)
        return self.perm[torch.searchsorted(self.cdf, u).clamp_(max=self.perm.numel() - 1)]


def _domain(case, size):
    return max(1, int(max(size) * case["keys_per_tuple"]))


def _lazy_streams(case, seed):
    sides = []
    zipf = None
    sizes = _sizes(case)
    for side in (0, 1):
        g = _gen(seed, side)
        keys = torch.empty(sum(s[side] for s in sizes), dtype=torch.int64, device="cuda")
        at = 0
        for s in sizes:
            if case["zipf"]:
                zipf = zipf or _Zipf(_domain(case, s), case["zipf"], seed)
                keys[at:at + s[side]] = zipf.keys(s[side], g)
            else:
                keys[at:at + s[side]].random_(0, _domain(case, s), generator=g)
            at += s[side]
        sides.append(keys)
    return sides


def _foreign_key_streams(case, seed):
    """Left: distinct keys.  Right: references to a domain twice the left's, so half of them match."""
    domain = 2 * case["n_left"]
    left = torch.randperm(domain, device="cuda", generator=_gen(seed, 0))[:case["n_left"]]
    right = torch.randint(0, domain, (case["n_right"],), device="cuda", generator=_gen(seed, 1))
    return left, right


def _batch_streams(case, seed, tuples):
    return [torch.randint(0, case["window"], (tuples,), device="cuda", generator=_gen(seed, side)) for side in (0, 1)]


def _pinned(t):
    host = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    host.copy_(t)
    return host


# ---------------------------------------------------------------- joiners
_joiners = {}   # a program keeps one joiner for all windows of a kind, and the stream it runs on


def _joiner(key, make):
    if key not in _joiners:
        j, stream = make(), torch.cuda.Stream()
        j.set_stream(stream.cuda_stream)
        _joiners[key] = (j, stream)
    return _joiners[key]


def prepare(case, seed):
    op = case["op"]
    if op == "lazy":
        sizes = _sizes(case)
        left, right = [_tuples(k) for k in _lazy_streams(case, seed)]
        flags = (sjbg.F_GRAPH if case["graph"] else 0) | (sjbg.F_XOR if case["xor"] else 0)
        most = max(max(s) for s in sizes)
        key = (op, case["algorithm"], case["partitioner"], flags, most)
        joiner, stream = _joiner(key, lambda: sjbg.Joiner(
            ALGORITHMS[case["algorithm"]], sjbg.LAZY, partitioner=PARTITIONERS[case["partitioner"]],
            max_tuples_per_window=most, flags=flags))
        descs = (sjbg.WindowDesc * len(sizes))()
        lo = ro = 0
        for d, (nl, nr) in zip(descs, sizes):
            d.left_offset, d.n_left, d.right_offset, d.n_right = lo, nl, ro, nr
            lo, ro = lo + nl, ro + nr
        state = {"left": left, "right": right, "descs": descs, "results": (sjbg.WindowResult * len(sizes))()}
    elif op == "pairs":
        left, right = [_tuples(k) for k in _foreign_key_streams(case, seed)]
        joiner, stream = _joiner((op, case["n_left"], case["n_right"]), lambda: sjbg.Joiner(
            sjbg.ALG_HJ, sjbg.LAZY, sjbg.RESULT_ATOMIC, max_tuples_per_window=max(case["n_left"], case["n_right"])))
        state = {"left": left, "right": right,
                 "pairs": torch.empty((case["n_right"], 2), dtype=torch.int32, device="cuda"),
                 "partner": torch.empty(case["n_right"], dtype=torch.int32, device="cuda")}
    elif op == "eager_run":
        left, right = [_tuples(k) for k in _batch_streams(case, seed, case["batch"] * case["n_batches"])]
        joiner, stream = _joiner((op, case["algorithm"], case["window"], case["batch"]), lambda: _eager(case))
        state = {"left": left, "right": right}
    elif op == "eager_batches":
        streams = [_pinned(_tuples(k)) for k in _batch_streams(case, seed, case["batch"] * case["n_batches"])]
        joiner, stream = _joiner((op, case["algorithm"], case["window"], case["batch"]), lambda: _eager(case))
        state = {"left": streams[0].split(case["batch"]), "right": streams[1].split(case["batch"])}
    elif op == "ring":
        streams = [_pinned(_tuples(k)) for k in _batch_streams(case, seed, case["window"] * case["windows"])]
        joiner, stream = _joiner((op, case["algorithm"], case["window"]), lambda: _ring_joiner(case))
        state = {"left": streams[0].split(case["batch"]), "right": streams[1].split(case["batch"])}
    torch.cuda.synchronize()   # the joiner runs on a stream of its own
    return dict(state, case=dict(case), joiner=joiner, stream=stream)


def _eager(case):
    return sjbg.Joiner(ALGORITHMS[case["algorithm"]], sjbg.EAGER, batch_size=case["batch"],
                       window_size=case["window"], max_tuples_per_window=case["window"])


def _ring_joiner(case):
    j = sjbg.Joiner(ALGORITHMS[case["algorithm"]], sjbg.LAZY, max_tuples_per_window=case["window"])
    j.ring_open(case["window"], 4)
    return j


# ---------------------------------------------------------------- one pass
def run(state):
    case, j = state["case"], state["joiner"]
    op = case["op"]
    if op == "lazy":
        j.lazy_execute_batch_raw(state["left"].data_ptr(), state["right"].data_ptr(), state["descs"],
                                 state["results"])
        words = np.frombuffer(state["results"], dtype=np.int64).reshape(len(state["results"]), -1)
        out = {"count": words[:, 0].copy(), "prod": words[:, 2].copy()}
        if case["xor"]:
            out["xor"] = words[:, 1].copy()
        return out
    if op == "pairs":
        r = j.lazy_execute(state["left"], state["right"], mem=sjbg.MEM_DEVICE, pairs=state["pairs"])
        with torch.cuda.stream(state["stream"]):
            found = state["pairs"][:r["n_pairs"]]
            state["partner"].fill_(-1)
            state["partner"][found[:, 1].long()] = found[:, 0]
        return {"count": r["count"], "prod": _signed(r["prod"]), "xor": _signed(r["xor"]), "partner": state["partner"]}
    if op == "eager_run":
        counts, windows = j.eager_run(state["left"], state["right"], case["n_batches"], mem=sjbg.MEM_DEVICE)
        return {"batch_counts": counts.astype(np.int64), **_totals(windows)}
    if op == "eager_batches":
        counts = []
        for l, r in zip(state["left"], state["right"]):
            counts.append(j.eager_execute(l, True))
            counts.append(j.eager_execute(r, False))
        total = j.eager_window_result()
        j.eager_clear_states()
        return {"batch_counts": np.array(counts, np.int64), **_totals([total])}
    done = []
    for l, r in zip(state["left"], state["right"]):
        j.ring_push(l, True)
        j.ring_push(r, False)
    while len(done) < case["windows"]:
        done += j.ring_poll(64)
    return _totals(done)


def _signed(x):
    return ctypes.c_int64(x).value


def _totals(windows):
    return {"count": np.array([w["count"] for w in windows], np.int64),
            "prod": np.array([w["prod"] for w in windows], np.uint64).view(np.int64)}


# ---------------------------------------------------------------- the same in plain torch
def _mix(x, k):
    low = (1 << 32) - 1
    h1 = (x ^ k) * 0x9E3779B1
    h2 = ((h1 & low) ^ ((h1 >> 32) & low) ^ 0x7F4A7C15) * 0x85EBCA77
    return (h1 ^ (h2 << 32) ^ ((h2 >> 13) & ((1 << 51) - 1))) | 1


def _window_totals(kl, vl, kr, vr, domain):
    """(count, prod) of one window from per-key sums, mod 2^64."""
    sums = []
    for k, v, side in ((kl, vl, 0x243F6A88), (kr, vr, 0xB7E15162)):
        zero = torch.zeros(domain, dtype=torch.int64, device="cuda")
        sums.append((torch.bincount(k, minlength=domain), zero.index_add_(0, k, _mix(v, side))))
    (cl, fl), (cr, fr) = sums
    return int((cl * cr).sum()), int((fl * fr).sum())


def _batch_counts(kl, kr, batch, n_batches, windows):
    """Matches of each batch, in arrival order L0, R0, L1, ..., with the earlier batches of its window."""
    out = np.zeros(2 * n_batches, np.int64)
    for l0, l1, r0, r1 in windows:
        bl = torch.arange(l0 * batch, l1 * batch, device="cuda")
        br = torch.arange(r0 * batch, r1 * batch, device="cuda")
        key = torch.cat([kl[bl], kr[br]])
        tag = torch.cat([2 * (bl // batch), 2 * (br // batch) + 1])
        order = torch.argsort(key * (2 * n_batches) + tag)
        key, tag = key[order], tag[order]
        right = tag & 1
        before_r = torch.cumsum(right, 0) - right
        before_l = torch.cumsum(1 - right, 0) - (1 - right)
        start = torch.searchsorted(key, key)   # the first position of each key
        other = torch.where(right == 1, before_l - before_l[start], before_r - before_r[start])
        out += torch.zeros(2 * n_batches, dtype=torch.int64, device="cuda").index_add_(0, tag, other).cpu().numpy()
    return out


def _eager_windows(case):
    """Batch ranges of a stream's windows: one closes before a batch once either side holds `window` tuples."""
    wins, held, cur = [], [0, 0], None
    for b in range(case["n_batches"]):
        for side in (0, 1):
            if max(held) >= case["window"]:
                wins.append(cur)
                held, cur = [0, 0], None
            if cur is None:
                cur = [b + side, b + side, b, b]
            cur[1 + 2 * side] = b + 1
            held[side] += case["batch"]
    return wins + [cur]


def exact(case, seed):
    op = case["op"]
    if op == "pairs":
        left, right = _foreign_key_streams(case, seed)
        at = torch.full((2 * case["n_left"],), -1, dtype=torch.int32, device="cuda")
        at[left] = torch.arange(case["n_left"], dtype=torch.int32, device="cuda")
        partner = at[right]
        count, prod = _window_totals(left, torch.arange(left.numel(), device="cuda"), right,
                                     torch.arange(right.numel(), device="cuda"), 2 * case["n_left"])
        return {"count": count, "prod": prod, "xor": None, "partner": partner}
    if op == "lazy":
        kl, kr = _lazy_streams(case, seed)
        spans, domains, lo, ro = [], [], 0, 0
        for nl, nr in _sizes(case):
            spans.append((lo, lo + nl, ro, ro + nr))
            domains.append(_domain(case, (nl, nr)))
            lo, ro = lo + nl, ro + nr
    else:
        if op == "ring":
            w = case["window"]
            kl, kr = _batch_streams(case, seed, w * case["windows"])
            spans = [(i * w, i * w + w, i * w, i * w + w) for i in range(case["windows"])]
        else:
            b = case["batch"]
            kl, kr = _batch_streams(case, seed, b * case["n_batches"])
            wins = _eager_windows(case) if op == "eager_run" else [(0, case["n_batches"], 0, case["n_batches"])]
            spans = [tuple(x * b for x in w) for w in wins]
        domains = [case["window"]] * len(spans)
    totals = []
    for (l0, l1, r0, r1), domain in zip(spans, domains):
        totals.append(_window_totals(kl[l0:l1], torch.arange(l0, l1, device="cuda"), kr[r0:r1],
                                     torch.arange(r0, r1, device="cuda"), domain))
    out = {"count": np.array([c for c, _ in totals], np.int64), "prod": np.array([p for _, p in totals], np.int64)}
    if op in ("eager_run", "eager_batches"):
        out["batch_counts"] = _batch_counts(kl, kr, case["batch"], case["n_batches"], wins)
    elif op == "lazy" and case["xor"]:
        out["xor"] = None
    return out


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    op = case["op"]
    if op == "lazy":
        sizes = _sizes(case)
        return {"bytes": sum(16 * (a + b) + 48 for a, b in sizes), "flops": 0}
    if op == "pairs":   # the tuples, about n_right / 2 pairs of 8 bytes, and each right tuple's partner
        return {"bytes": 16 * (case["n_left"] + case["n_right"]) + 8 * case["n_right"], "flops": 0}
    if op == "ring":
        return {"bytes": 32 * case["window"] * case["windows"] + 48 * case["windows"], "flops": 0}
    moved = 32 * case["batch"] * case["n_batches"] + 16 * case["n_batches"]
    flops = 0
    if op == "eager_run" and case["algorithm"] == "nlj":   # one compare per pair of a window's tuples
        flops = sum((l1 - l0) * (r1 - r0) for l0, l1, r0, r1 in _eager_windows(case)) * case["batch"] ** 2
    return {"bytes": moved, "flops": flops}
