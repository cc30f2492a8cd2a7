"""Every operation of the ladders' arithmetic (csrc/ww_ladder.cuh) operand by
operand against whole numbers: its C forms on the host, and on the GPU the
instruction sequences that the test and PRP kernels run.  Operands are the
edges that whole ladders seldom meet: high digits from p to 2p, words of all
ones, sums that need each of the three corrections, a borrow out of a zero
high word.  All comparisons are exact."""
from __future__ import annotations

import random

import numpy as np
import pytest

R = 2**64
MODS = [127, 131, 65521, 2**31 - 1, 4294967291, 4294967311, 0xFFFFFFFF00000001, 0x80000000FFFFFFFF, 2**61 - 1,
        2**62 - 57, 2**62 + 135, 9223372036854775783, 2**63 + 29, 2**64 - 59, 2**64 - 1, 2**64 - 3,
        12297829382473034411, 16129, 4294967291**2, 0xFFFFFFFFFFFFFF01]


def _sets(p):
    """Low (below p) and high (below 2p and 2^64) digits, and any words."""
    rng = random.Random(p)
    top = min(2 * p, R)
    low = {0, 1, 2, p - 1, p - 2, p // 2, 2**32 % p, (2**32 - 1) % p} | {rng.randrange(p) for _ in range(2)}
    high = {0, 1, p - 1, p, min(p + 1, top - 1), top - 1, top - 2, top - 2**31 if top > 2**32 else p} | {rng.randrange(top)}
    words = [0, 1, 2**32 - 1, 2**32, 2**63, R - 1, R - 2, R - 2**32, 0xFFFFFFFF00000001, 0xFFFFFFFF, rng.randrange(R)]
    return sorted(low), sorted(high), words, rng


def _cases(op, p):
    """(operands, expected words) of op for the modulus p; a high digit of
    ops 0 to 3 may be any representative below 2p: those come as a residue."""
    low, high, words, rng = _sets(p)
    n, q = p * p, pow(p, -1, R)
    rinv_n, rinv_p = pow(R, -1, n), pow(R, -1, p)
    half_n, half_p = pow(2**32, -1, n), pow(2**32, -1, p)
    some = [(a, b) for a in low[:3] + low[-2:] for b in high[::2]]
    kk = [(0, 0), (1, 0), (p - 1, p - 1), (0, p - 1), (rng.randrange(p), rng.randrange(p))]
    two = lambda z: (z % n % p, z % n // p)  # noqa: E731
    out = []
    if op <= 3:
        for x0 in low:
            for x1 in high:
                x = x0 + p * x1
                if op == 0:
                    out.append(((x0, x1, 0, 0, 0, 0), two(x * x * rinv_n)))
                elif op == 1:
                    out += [((x0, x1, 0, 0, a, b), two((x * x + a + p * b) * rinv_n)) for a, b in kk]
                elif op == 2:
                    out += [((x0, x1, c, d, a, b), two((x * (c + p * d) + a + p * b) * rinv_n))
                            for c, d in some for a, b in kk[1:4]]
                else:
                    out += [((x0, x1, 0, 0, d, 0), two(x * 2**d * half_n))
                            for d in (0, 1, 5, 16, 30, 31)]
    elif op <= 7:
        for a in low:
            for b in low:
                if op == 4:
                    z = a * a * rinv_p
                elif op == 5:
                    d = b % 32
                    out.append(((a, 0, 0, 0, d, 0), (a * 2**d * half_p % p, 0, 0)))
                    continue
                elif op == 6:
                    for c in (0, 1, p - 1, low[len(low) // 2]):
                        out.append(((a, 0, b, 0, c, 0), ((a * b + c) * rinv_p % p, 0, 0)))
                    continue
                else:
                    z = (a * a + b) * rinv_p
                out.append(((a, 0, 0, 0, b if op == 7 else 0, 0), (z % p, 0, 0)))
    elif op <= 12:
        for a in words + low:
            for b in words + low[-3:]:
                if op in (8, 9):
                    w = a * b if op == 8 else a * b >> 64
                    out.append(((a, 0, b, 0, 0, 0), (w % R, w >> 64, 0)))
                elif op == 10:
                    for c in (0, R - 1, 2**32, b):
                        w = a * b + c
                        out.append(((a, 0, b, 0, c, 0), (w % R, w >> 64, 0)))
                else:
                    w = a * a + (b if op == 12 else 0)
                    out.append(((a, 0, 0, 0, b if op == 12 else 0, 0), (w % R, w >> 64, 0)))
    elif op == 13:
        for x0, x1 in [(a, b) for a in words[:8] for b in words[:7]]:
            for y0, y1 in [(a, b) for a in (0, 1, R - 1, 2**63) for b in (0, R - 1, 2**63)]:
                for u in (0, 1, R - 1):
                    for neg in (0, 1):
                        w = x0 + R * x1 + y0 + R * y1 + u - R * neg
                        out.append(((x0, x1, y0, y1, u, neg), (w % R, (w >> 64) % R, (w >> 128) % R)))
    else:
        for s in words + low:
            v = (s * q % R) * p >> 64
            for neg in (0, 1) if op == 15 else (0,):
                near = {-p, -p + 1, -1, 0, 1, p - 1, p, p + 1, 2 * p - 1, R - 1, R, R + 1,
                        -v, -v - 1, R - v, R - v - 1, R - v - 2} | {rng.randrange(-p, 2 * p)}
                for digit in near:
                    if not -p <= digit < 2 * p:
                        continue
                    total = digit + v + neg  # (k:h), the reduced part v and the borrow still in it
                    out.append(((s, total % R, (total >> 64) % 2**32, 0, 0, neg), (digit - (digit >> 64) * p, 0, 0)))
    return out


@pytest.mark.parametrize("side", ["host", pytest.param("device", marks=pytest.mark.gpu)])
@pytest.mark.parametrize("p", MODS)
def test_ladder_operations(ww, side, p):
    run = ww.selftest_ladder if side == "host" else ww.devtest_ladder
    top = min(2 * p, R)
    for op in range(16):
        cases = _cases(op, p)
        got = run(op, p, np.array([c for c, _ in cases], np.uint64))
        for (operands, want), row in zip(cases, got.tolist()):
            if op <= 3:
                assert row[1] < top, (op, hex(p), operands, row)
                row, want = (row[0], row[1] % p, row[2]), (*want, 0)
            assert tuple(row) == tuple(want), (op, hex(p), operands, row, want)


def test_ladder_operations_refuse_bad_arguments(ww):
    case = np.zeros(6, np.uint64)
    for op, p in ((-1, 127), (16, 127), (0, 128), (0, 1)):
        for run in (ww.selftest_ladder, ww.devtest_ladder):
            with pytest.raises(ww.WWError):
                run(op, p, case)
    assert ww.devtest_ladder(0, 127, np.zeros(0, np.uint64)).shape == (0, 3)
