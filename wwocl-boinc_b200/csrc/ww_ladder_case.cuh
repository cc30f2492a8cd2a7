// ww_ladder_case.cuh -- one operation of the ladders' arithmetic
// (ww_ladder.cuh) on given operands, for checking it operand by operand on
// the host and on the device: whole ladders seldom meet its rare carries (a
// sum of 2^64 or more before lz_fix, a borrow out of a zero high word, high
// digits of p or more).
#pragma once

#include "ww_ladder.cuh"

namespace ww {

constexpr int kLadderOps = 16;

// in: x0, x1, y0, y1, k0, k1; out: three words, unused ones zero.
WW_HD void ladder_case(int op, const LzMod &m, const u64 *in, u64 *out) {
    const D2 x = {in[0], in[1]}, y = {in[2], in[3]}, kk = {in[4], in[5]};
    const u32 d = (u32)kk.d0 & 31u;
    const u32 neg = 0u - ((u32)kk.d1 & 1u);
    D2 z = {0, 0};
    u128 w;
    u64 u, s, h;
    u32 borrow, k;
    out[2] = 0;
    switch (op) {
        // the two-digit steps mod p^2
        case 0: z = lz_sqr(x, m); break;
        case 1: z = lz_sqr_add(x, lz_halve(kk, m.p), m); break;
        case 2: z = lz_mul_add(x, y, kk, m); break;
        case 3: z = lz_shift(x, d, m); break;
        // the one-word steps mod p
        case 4: z.d0 = lz_sqr1(x.d0, m); break;
        case 5: z.d0 = lz_shift1(x.d0, d, m); break;
        case 6: z.d0 = lz_low(lz_mad(x.d0, y.d0, kk.d0), m, u, borrow); break;
        case 7: z.d0 = lz_low(lz_square_add(x.d0, kk.d0), m, u, borrow); break;
        // the products, any words
        case 8:
        case 10:
        case 11:
        case 12:
            w = op == 8 ? lz_mul(x.d0, y.d0) : op == 10 ? lz_mad(x.d0, y.d0, kk.d0)
                : op == 11 ? lz_square(x.d0) : lz_square_add(x.d0, kk.d0);
            z.d0 = (u64)w;
            z.d1 = (u64)(w >> 64);
            break;
        case 9: z.d0 = lz_hi(x.d0, y.d0); break;
        // the sum of a two-digit square's high half, x + y + k0 - 2^64 (k1 & 1)
        case 13:
            lz_sum(((u128)x.d1 << 64) | x.d0, ((u128)y.d1 << 64) | y.d0, kk.d0, neg, s, h, k);
            z.d0 = s;
            z.d1 = h;
            out[2] = (u64)(long long)(int)k;
            break;
        // the high digit from the sum (y0 : x1 : x0), y0 signed
        case 14: z.d0 = lz_high(x.d0, x.d1, (u32)y.d0, m); break;
        default: z.d0 = lz_high_less(x.d0, x.d1, (u32)y.d0, neg, m); break;
    }
    out[0] = z.d0;
    out[1] = z.d1;
}

}  // namespace ww
