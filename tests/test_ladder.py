"""The ladders of both tests (csrc/ww_ladder.cuh, csrc/ww_tests.cuh) against
whole-number arithmetic: the host twin on the CPU, and on the GPU with
numbers of every size in one warp, whose lanes take the same number of steps.
Nothing in the ladders needs a prime, so the numbers are any without a
factor 5.  All comparisons are exact."""
from __future__ import annotations

import random

import numpy as np
import pytest


def fib(n: int, m: int) -> int:
    a, b = 0, 1
    for bit in bin(n)[2:]:
        a, b = a * (2 * b - a) % m, (a * a + b * b) % m
        if bit == "1":
            a, b = b, (a + b) % m
    return a


def want(p: int) -> tuple[int, int, int, int]:
    s = pow(2, (p - 1) // 2, p * p)
    c = fib(p + 1 if p % 5 in (2, 3) else p - 1, p * p)
    return s % p, s // p, c % p, c // p


def numbers(bits: int) -> list[int]:
    """Odd numbers of the given length: both ends of it, and the exponent's
    extremes (long runs of ones and of zeros)."""
    rng = random.Random(bits)
    lo, hi = 1 << (bits - 1), 1 << bits
    out = [lo + d for d in range(1, 16, 2)] + [hi - d for d in range(1, 16, 2)]
    out += [rng.randrange(lo, hi) | 1 for _ in range(40)]
    out += [(hi - 1) ^ (1 << rng.randrange(1, bits - 1)) for _ in range(8)]
    return sorted({p for p in out if lo < p < hi and p % 5 and p >= 127})


@pytest.mark.parametrize("bits", list(range(7, 65)))
def test_host_ladders_match_whole_numbers(ww, bits):
    ps = numbers(bits)
    got = ww.selftest_digits(np.array(ps, np.uint64))
    assert [tuple(int(v) for v in row) for row in got] == [want(p) for p in ps]


@pytest.mark.gpu
@pytest.mark.parametrize("keep", [1, 31, 32, 33, 0])
def test_gpu_ladders_mixed_sizes(ww, keep):
    """Every length from 7 to 64 bits shuffled into the same warps (0: all of
    them), through the digits kernel and, as sums, the list kernels."""
    ps = [p for b in range(7, 65) for p in numbers(b)]
    random.Random(5).shuffle(ps)
    ps = ps[:keep] if keep else ps
    rows = [want(p) for p in ps]
    arr = np.array(ps, np.uint64)
    assert [tuple(int(v) for v in row) for row in ww.digits(arr)] == rows
    total = sum((r[1] & 0xFFFFFFFF) + (r[3] & 0xFFFFFFFF) for r in rows)
    with ww.Context(0, max_prps=1 << 13) as ctx:
        ctx.load_prps(arr)
        for fused in (True, False):
            ctx.clear_results()
            if fused:
                ctx.test_prps()
            else:
                ctx.wieferich()
                ctx.wallsunsun()
            assert ctx.counters()["checksum"] == total
