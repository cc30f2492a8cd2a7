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


SMALL = [3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37, 41, 43, 47, 53, 59, 61, 67, 71, 73, 79, 83, 89, 97, 101, 103, 107,
         109, 113]


def strong_prp2(n: int) -> bool:
    if any(n % r == 0 for r in SMALL):
        return False
    t = ((n - 1) & -(n - 1)).bit_length() - 1
    x = pow(2, (n - 1) >> t, n)
    if x in (1, n - 1):
        return True
    for _ in range(t - 1):
        x = x * x % n
        if x == n - 1:
            return True
    return False


@pytest.mark.gpu
@pytest.mark.parametrize("k", list(range(8, 65)))
def test_gpu_prp_test_around_powers_of_two(ww, k):
    """Both sides of 2^k: numbers of two lengths in one warp, and n - 1 with
    every 2-adic valuation up to k (2^32 + 1 is a strong pseudoprime)."""
    lo = max(127, 2**k - 2000)
    hi = min(2**64 - 1, 2**k + 2000)
    expect = [n for n in range(lo | 1, hi, 2) if strong_prp2(n)]
    with ww.Context(0, max_prps=1 << 12) as ctx:
        ctx.clear_segment()
        ctx.sieve_prp(lo, hi)
        assert sorted(int(v) for v in ctx.prps()) == expect


@pytest.mark.gpu
@pytest.mark.parametrize("width", [2**11 - 2, 2**11 + 2, 40_000, 1_212_416, 1_300_000, 9_700_000, 77_594_624,
                                   77_600_000, 2**26 - 1, 2**26 + 1, 310_400_000, 311_000_000, 620_000_000, 2**29])
@pytest.mark.parametrize("low", [127, 10**9 + 1, 2**64 - 2**31 + 3])
def test_gpu_small_segments_equal_fixed_ones(ww, low, width):
    """The segment size chosen by width against the fixed narrow segments, at
    the widths where the size, the rounds or the marks change: same list."""
    with ww.Context(0, max_prps=ww.prp_count_bound(low, low + width) + 1000) as ctx:
        lists = []
        for shape, depth in ((0, 28), (2, 20)):
            ctx.set_sieve_shape(shape)
            ctx.set_sieve_depth(depth)
            ctx.clear_segment()
            ctx.sieve_prp(low, low + width)
            lists.append(np.sort(ctx.prps()))
        assert np.array_equal(lists[0], lists[1])


@pytest.mark.gpu
@pytest.mark.parametrize("widths", [[1], [2**13 - 1, 2**13 + 1], [100_000], [300_001] * 5, [40_000_000, 999, 1_000_000],
                                    [50_000] * 300, [2**28 + 5, 7, 2**20]])
@pytest.mark.parametrize("cfg", [(16384, 512, 1, 0), (4096, 128, 1, 0), (16384, 1024, 1, 0), (8192, 256, 8, 0)])
def test_gpu_cut_tiles_equal_units_alone(ww, widths, cfg):
    """Batches whose tiles are cut small: each unit as alone on the plain path,
    and its tiles still counted in the configuration's full ones; the same
    ranges as requests (one step may take the first's last tile and the next
    one's) and through the allocation-free entry (tests/test_zz_no_alloc.py
    covers its own sizes)."""
    rng = random.Random(len(widths) + cfg[1])
    starts = [rng.randrange(127, 2**64 - 2**29) for _ in widths]
    units = [(a, a + w) for a, w in zip(starts, widths)]
    with ww.Context(0, max_prps=ww.prp_count_bound(0, max(widths)) + 1000) as ctx:
        batch = ww.Batch(ctx)
        batch.set_config(*cfg)
        got = batch.run(units)
        alone = [ctx.run_range(a, b) for a, b in units]
        want = [(r["checksum"], r["total_prp_count"], r["result_count"]) for r in alone]
        assert [(r["checksum"], r["prp_count"], r["hits"]) for r in got] == want
        assert [r["tiles_done"] for r in got] == [-(-w // (64 * cfg[0])) for w in widths]
        server = ww.Server(ctx, prp_pool_bytes=1 << 28, max_active=8)
        server.submit([(i, a, b) for i, (a, b) in enumerate(units)])
        done = sorted(server.drain(), key=lambda r: r["id"])
        assert [(r["checksum"], r["prp_count"], r["hits"]) for r in done] == want
        assert [r["prps_stored"] for r in done] == [w[1] for w in want]
        server.close()


@pytest.mark.gpu
@pytest.mark.parametrize("widths", [[1], [2**13 - 1, 2**13 + 1], [100_000], [300_001] * 5, [40_000_000, 999, 1_000_000],
                                    [50_000] * 300, [2**28 + 5, 7, 2**20]])
def test_gpu_cut_tiles_through_the_allocation_free_entry(ww, widths):
    """The same widths through ww_batch_run_noalloc: the batch's results in
    its configuration, and the finished tiles counted in full ones."""
    import ctypes as C

    import torch

    rng = random.Random(len(widths))
    units = [(a, a + w) for a, w in ((rng.randrange(127, 2**64 - 2**29), w) for w in widths)]
    with ww.Context(0, max_prps=1 << 12) as ctx:
        batch = ww.Batch(ctx)
        batch.set_config(8192, 256, 1)
        want = [(r["checksum"], r["prp_count"], r["hits"], r["tiles_done"]) for r in batch.run(units)]
    arr = (ww.Unit * len(units))()
    for i, (a, b) in enumerate(units):
        arr[i].start, arr[i].end = a, b
    out = torch.zeros(len(units) * C.sizeof(ww.UnitResult), dtype=torch.uint8, device="cuda")
    count = torch.zeros(1, dtype=torch.int32, device="cuda")
    ww.check(ww.lib().ww_batch_run_noalloc(arr, len(units), out.data_ptr(), None, None, 0, count.data_ptr(),
                                           torch.cuda.current_stream().cuda_stream), "ww_batch_run_noalloc")
    got = (ww.UnitResult * len(units)).from_buffer_copy(out.cpu().numpy().tobytes())
    assert [(r.checksum, r.prp_count, r.hits, r.tiles_done) for r in got] == want


@pytest.mark.gpu
@pytest.mark.parametrize("cfg", [(16384, 512, 1, 1), (8192, 256, 1, 1)])
@pytest.mark.parametrize("low", [127, 2**32 - 300_000, 2**32 + 1])
def test_gpu_joint_loop_around_one_word_primes(ww, cfg, low):
    """Both tests in one loop on whole warps of primes below 2^32, on warps
    that hold some of each, and above: each unit as alone on the plain path,
    where the tests run one after the other."""
    units = [(low, low + 600_000), (low + 600_000, low + 600_100), (2**40 + low, 2**40 + low + 50_000)]
    with ww.Context(0, max_prps=100_000) as ctx:
        batch = ww.Batch(ctx)
        batch.set_config(*cfg)
        got = batch.run(units)
        alone = [ctx.run_range(a, b) for a, b in units]
    assert [(r["checksum"], r["prp_count"], r["hits"]) for r in got] == [
        (r["checksum"], r["total_prp_count"], r["result_count"]) for r in alone]
