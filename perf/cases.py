"""The work a user of the search path has it do, as cases that can be timed.

Each case is one pass through the public Python face of the C ABI
(`wwcuda.py`): a plain range (clear, sieve, tests, read-back at every
checkpoint), the sieve's PRP list, the exact prime count, a list of primes
tested on the device or from host memory, per-prime digits, a batch of uneven
ranges, and a set of requests through the server.  Starts, lists, units and
requests come from the seed; the widths are the case's own.
"""
from __future__ import annotations

import math
import random
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "wwocl-boinc_b200"))

import wwcuda as ww  # noqa: E402

CHECKPOINT = 1 << 30  # numbers per checkpoint of the plain path
TOP = 2**64 - 2**35   # start of the 2^34-wide range below 2^64


def listed():
    return [
        # the smallest request a server or a script sends: launch and read-back latency
        {"name": "range 1e5", "kind": "range", "base": 10**12, "width": 100_000, "fused": True},
        # the reference's small published range [127, 5e7): small primes, p^2 below 2^64 at first, hits to report
        {"name": "range 127..5e7", "kind": "range", "base": 127, "width": 49_999_873, "fused": True},
        # a mid-domain work unit through the reference-shaped separate Wieferich and Wall-Sun-Sun kernels
        {"name": "range 2^28 separate", "kind": "range", "base": 10**17, "width": 1 << 28, "fused": False},
        # four checkpoint segments of the wide range at the top of the domain: the long production run
        {"name": "range 2^32 top", "kind": "range", "base": TOP, "width": 1 << 32, "fused": True},
        # the PRP list itself, for a caller that runs its own tests on it
        {"name": "prp list 1e6", "kind": "prps", "base": 2**62 + 12345, "width": 1_000_003},
        # an exact prime count that sizes the buffers of a run
        {"name": "count 2^31", "kind": "count", "base": 10**18, "width": (1 << 31) - 12_345},
        # a fixed prime list of [2^62, 2^64) resident on the device: both tests
        {"name": "list 2^24", "kind": "list", "n": 1 << 24, "how": "device"},
        # a ragged list from pinned host memory, copied inside the call
        {"name": "list 1000003 host", "kind": "list", "n": 1_000_003, "how": "host"},
        # a short list through the two separate test kernels
        {"name": "list 65537 separate", "kind": "list", "n": 65_537, "how": "separate"},
        # per-prime digits, as a verifier asks for them
        {"name": "digits 10007", "kind": "digits", "n": 10_007},
        # many uneven work units in one batched launch
        {"name": "batch 96", "kind": "batch", "units": 96, "wmin": 1e6, "wmax": 1e8},
        # requests of three decades of width served to completion, their PRP lists kept
        {"name": "serve 64", "kind": "serve", "requests": 64, "wmin": 1e5, "wmax": 1e8},
    ]


def _log_uniform(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    kind = rng.choice(["range", "range", "range", "prps", "count", "list", "list", "digits", "batch", "serve"])
    base = rng.choice([_log_uniform(rng, 10**3, 10**12), _log_uniform(rng, 10**12, 2**62), rng.randrange(2**62, TOP)])
    if kind == "range":
        return {"kind": kind, "base": base, "width": _log_uniform(rng, 10**5, 2**31), "fused": rng.random() < 0.7}
    if kind == "prps":
        return {"kind": kind, "base": base, "width": _log_uniform(rng, 10**5, 10**7)}
    if kind == "count":
        return {"kind": kind, "base": base, "width": _log_uniform(rng, 10**6, 2**32)}
    if kind == "list":
        return {"kind": kind, "n": _log_uniform(rng, 1000, 1 << 23), "how": rng.choice(["device", "host", "separate"])}
    if kind == "digits":
        return {"kind": kind, "n": _log_uniform(rng, 100, 200_000)}
    wmin = _log_uniform(rng, 10**5, 10**7)
    if kind == "batch":
        return {"kind": kind, "units": _log_uniform(rng, 4, 400), "wmin": float(wmin), "wmax": wmin * rng.uniform(2, 20)}
    return {"kind": kind, "requests": _log_uniform(rng, 4, 128), "wmin": float(wmin), "wmax": wmin * rng.uniform(2, 10)}


def _start(case, seed):
    """The case's range moved by a seeded offset of at most a thousandth of its start (or of its width)."""
    rng = np.random.default_rng(seed)
    return case["base"] + int(rng.integers(0, max(case["base"] // 1000 if case["base"] < TOP else 2**30, case["width"] // 1000)))


def _list_seed(seed):
    return random.Random(int(seed)).getrandbits(64)


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind in ("range", "prps", "count"):
        lo = _start(case, seed)
        st["lo"], st["hi"] = lo, lo + case["width"]
        prps = 1 << 12 if kind == "count" else ww.prp_count_bound(0, min(case["width"], CHECKPOINT)) + 1000
        st["ctx"] = ww.Context(0, max_prps=prps)
        st["most"] = prps
    elif kind in ("list", "digits"):
        st["primes"], _ = ww.random_primes(_list_seed(seed), case["n"])
        if kind == "list":
            st["ctx"] = ww.Context(0, max_prps=max(2, case["n"]))
            if case["how"] == "host":
                st["pinned"] = torch.from_numpy(st["primes"].view(np.int64)).pin_memory()
            else:
                st["ctx"].load_prps(st["primes"])
                st["ctx"].sync()
    elif kind == "batch":
        st["units"] = ww.uneven_units(seed, case["units"], case["wmin"], case["wmax"])
        st["ctx"] = ww.Context(0, max_prps=1 << 12)
        st["batch"] = ww.Batch(st["ctx"])
    elif kind == "serve":
        units = ww.uneven_units(seed, case["requests"], case["wmin"], case["wmax"], smin=10**12)
        st["requests"] = [(i, a, b) for i, (a, b) in enumerate(units)]
        st["ctx"] = ww.Context(0, max_prps=1 << 12)
        st["server"] = ww.Server(st["ctx"], prp_pool_bytes=1 << 30)
    return st


def _counters(st, c, hits):
    """Checksum, counts and the hit records in prime order (the list's own
    order is unspecified), in an array of the case's own length: small primes
    hit by the thousand, large ones hardly ever."""
    rows = np.zeros((15000 if st["case"].get("base", TOP) < 10**12 else 64, 4), np.uint64)
    hits = [[v % 2**64 for v in h] for h in sorted(hits)[: len(rows)]]
    if hits:
        rows[: len(hits)] = np.array(hits, np.uint64)
    return {"sums": np.array([c["checksum"], c["total_prp_count"], c["result_count"], c["overflow"]], np.uint64),
            "hits": rows}


def run(st):
    case = st["case"]
    kind = case["kind"]
    ctx = st.get("ctx")
    if kind == "range":
        c = ctx.run_range(st["lo"], st["hi"], fused=case["fused"], segment=CHECKPOINT)
        return _counters(st, c, c["hits"])
    if kind == "prps":
        ctx.clear_results()
        ctx.clear_segment()
        ctx.sieve_prp(st["lo"], st["hi"])
        prps = ctx.prps()
        prps.sort()  # the list's own order is unspecified
        out = np.zeros(st["most"], np.uint64)  # as long as any list of this width
        out[: prps.size] = prps
        return out
    if kind == "count":
        return ctx.count_prps(st["lo"], st["hi"])
    if kind == "list":
        ctx.clear_results()
        if case["how"] == "host":
            ctx.test_prps_host_ptr(st["pinned"].data_ptr(), case["n"])
        elif case["how"] == "device":
            ctx.test_prps()
        else:
            ctx.wieferich()
            ctx.wallsunsun()
        c = ctx.counters()
        return _counters(st, c, ctx.hits() if c["result_count"] else [])
    if kind == "digits":
        return ww.digits(st["primes"])
    if kind == "batch":
        got = st["batch"].run(st["units"])
        rows = np.array([(r["checksum"], r["prp_count"], r["hits"]) for r in got], np.uint64)
        return {"units": rows, "hits": st["batch"].hit_count}
    server = st["server"]
    server.submit(st["requests"])
    got = sorted(server.drain(), key=lambda r: r["id"])
    return np.array([(r["id"], r["checksum"], r["prp_count"], r["prps_stored"], r["hits"], -r["status"]) for r in got],
                    np.uint64)


# 32-bit multiplies of one prime's tests and one candidate's PRP test with
# k-bit numbers (a 64x64->128 product counts 8, its low half 4): k - 6 steps
# of three two-digit squarings, and k - 5 one-digit squarings
def _test_ops(k):
    return 114.0 * max(k - 6, 1) + 168.0


def _prp_ops(k):
    return 20.0 * max(k - 5, 1) + 12.0


def _density(x):
    return 1.0 / math.log(max(x, 10))


def _range_work(lo, width, tests):
    k = max(lo + width // 2, 2).bit_length()
    primes = width * _density(lo + width // 2)
    return primes * (_prp_ops(k) + (_test_ops(k) if tests else 0.0)), primes


def work(case):
    kind = case["kind"]
    if kind == "range":
        return {"bytes": 48.0, "flops": _range_work(case["base"], case["width"], True)[0]}
    if kind == "count":
        return {"bytes": 24.0, "flops": _range_work(case["base"], case["width"], False)[0]}
    if kind == "prps":
        ops, primes = _range_work(case["base"], case["width"], False)
        return {"bytes": 16.0 + 8.0 * primes, "flops": ops}
    if kind == "list":
        return {"bytes": 8.0 * case["n"] + 32.0, "flops": case["n"] * _test_ops(64)}
    if kind == "digits":
        return {"bytes": 40.0 * case["n"], "flops": case["n"] * _test_ops(64)}
    n = case["units"] if kind == "batch" else case["requests"]
    mean = (case["wmax"] - case["wmin"]) / math.log(case["wmax"] / case["wmin"])
    ops, primes = _range_work(2**63, int(mean), True)
    return {"bytes": n * (48.0 + (8.0 * primes if kind == "serve" else 0.0)), "flops": n * ops}


def _fib(n, m):
    """F_n mod m by doubling."""
    a, b = 0, 1
    for bit in bin(n)[2:]:
        a, b = a * (2 * b - a) % m, (a * a + b * b) % m
        if bit == "1":
            a, b = b, (a + b) % m
    return a


def exact(case, seed):
    """The digits in whole numbers: 2^((p-1)/2) and F_(p-(p|5)) mod p^2, low and high digit."""
    if case["kind"] != "digits" or case["n"] > 50_000:
        return None
    primes, _ = ww.random_primes(_list_seed(seed), case["n"])
    rows = np.empty((len(primes), 4), np.uint64)
    for i, p in enumerate(int(v) for v in primes):
        s = pow(2, (p - 1) // 2, p * p)
        c = _fib(p + 1 if p % 5 in (2, 3) else p - 1, p * p)
        rows[i] = (s % p, s // p, c % p, c // p)
    return rows
