// ww_ladder.cuh -- the two-digit arithmetic of the test ladders, with the
// corrections it does not need left out.
//
// A residue is X = x0 + p*x1 in Montgomery form, R = 2^64, as in
// ww_arith.cuh, but only x0 is canonical: x1 is any representative in
// [0, 2p) that fits 64 bits.  With x0 < p the low digit of a product needs
// one conditional addition of p, as there; its high digit
//     T = (C + u + k1) / 2^64 - v - borrow,   C = 2 x0 x1 (or x0 y1 + x1 y0)
// lies in [-p, 2p), and t = T >> 64 is -1, 0 or 1: T - t p fits 64 bits again
// and is below 2p, so one three-way correction replaces the two of the
// canonical form.  The constant of a ladder step (k0 + p k1 = c R^2 mod p^2)
// is added before the reduction, where it costs two additions and no
// correction.
//
// What bounds it (B200, cycles of one of an SM's four schedulers): a 32x32->64
// multiply holds the multiply pipe for 4 cycles and the ALU side for 2.3,
// any other integer instruction holds its pipe for 2, and the compiler
// spreads moves and carries over both, so the time is about 3.15 cycles a
// wide multiply and one for every other instruction, of which 87 % is
// reached; occupancy (48 to 80 registers) moves it by 1 %.  So what counts is
// the number of instructions: a ladder step was 319 (54 wide multiplies) with
// canonical digits, a pair of squarings and doublings bit by bit, 235 in this
// form on __int128 products, and some 215 on the products below.  Both tests
// over 2^24 primes of [2^62, 2^64): 12.33, 10.78 and 10.11 ms (1 360, 1 557 and
// 1 660 M primes/s).
#pragma once

#include "ww_arith.cuh"

namespace ww {

typedef unsigned __int128 u128;

struct LzMod {
    u64 p, q;      // q = p^-1 mod 2^64
    u32 npl, nph;  // -p = npl + 2^32 nph mod 2^64, npl signed
};

WW_HD LzMod lz_mod(u64 p, u64 q) {
    LzMod m;
    m.p = p;
    m.q = q;
    const u64 n = 0 - p;
    m.npl = (u32)n;
    m.nph = (u32)(n >> 32) + (m.npl >> 31);
    return m;
}

// r - t p mod 2^64 for t in {-1, 0, 1} (a word, -1 as 2^32 - 1): a signed
// wide multiply-add and a multiply-add, two instructions (by two selects and
// a predicated add: 1 433 against 1 504 M primes/s).
WW_HD u64 lz_fix(u64 r, u32 t, const LzMod &m) {
#if defined(__CUDA_ARCH__)
    u64 o;
    asm("{\n\t.reg .u32 l, h;\n\t"
        "mad.wide.s32 %0, %1, %2, %3;\n\t"
        "mov.b64 {l, h}, %0;\n\t"
        "mad.lo.u32 h, %1, %4, h;\n\t"
        "mov.b64 %0, {l, h};\n\t}"
        : "=l"(o) : "r"(t), "r"(m.npl), "l"(r), "r"(m.nph));
    return o;
#else
    return r - (u64)(long long)(int)t * m.p;
#endif
}
// r + (neg ? p : 0) for the mask neg (0 or 2^32 - 1), on the ALU: 1 504 M
// primes/s, against 1 492 M with the "& p" as two multiplies by the mask and
// 1 467 M as lz_fix.
WW_HD u64 lz_addp(u64 r, u32 neg, const LzMod &m) {
#if defined(__CUDA_ARCH__)
    u64 t;
    asm("{\n\t.reg .u32 a0, a1, r0, r1;\n\t"
        "mov.b64 {a0, a1}, %2;\n\t"
        "mov.b64 {r0, r1}, %3;\n\t"
        "and.b32 a0, a0, %1;\n\t"
        "and.b32 a1, a1, %1;\n\t"
        "add.cc.u32 r0, r0, a0;\n\t"
        "addc.u32 r1, r1, a1;\n\t"
        "mov.b64 %0, {r0, r1};\n\t}"
        : "=l"(t) : "r"(neg), "l"(m.p), "l"(r));
    return t;
#else
    return neg ? r + m.p : r;
#endif
}

// a - b mod 2^64 and the borrow as a mask
WW_HD u64 lz_sub(u64 a, u64 b, u32 &neg) {
#if defined(__CUDA_ARCH__)
    u64 r;
    asm("sub.cc.u64 %0, %2, %3;\n\t"
        "subc.u32 %1, 0, 0;"
        : "=&l"(r), "=r"(neg) : "l"(a), "l"(b));
    return r;
#else
    neg = a < b ? ~0u : 0u;
    return a - b;
#endif
}

// Products from four 32x32 ones (three for a square), each written so that
// the cross products' sum is the addend of the top one, a1 b1 + (y:z) with the
// carry of the word below: on the device a `mad.lo.cc` / `madc.hi.cc` pair on
// the same factors is one wide multiply-add with carry in and out, so an
// addend costs next to nothing.  A product is 6 instructions (7.4 as the
// unsigned __int128 one, whose last word is added after the multiply), a
// product plus a word 8 (11.4).  Over 2^24 primes: 10.78 ms with __int128
// products and added constants, 10.67 with the square's constant as its
// addend, 10.33 with the cross products', 10.11 ms in this form throughout.
WW_HD u128 lz_mul(u64 a, u64 b) {
#if defined(__CUDA_ARCH__)
    u64 lo, hi;
    asm("{\n\t.reg .u64 e, o;\n\t.reg .u32 r0, r1, r2, r3, x, y, z;\n\t"
        "mul.wide.u32 o, %2, %5;\n\t"
        "mov.b64 {x, y}, o;\n\t"
        "mad.lo.cc.u32 x, %3, %4, x;\n\t"
        "madc.hi.cc.u32 y, %3, %4, y;\n\t"
        "addc.u32 z, 0, 0;\n\t"
        "mul.wide.u32 e, %2, %4;\n\t"
        "mov.b64 {r0, r1}, e;\n\t"
        "add.cc.u32 r1, r1, x;\n\t"
        "madc.lo.cc.u32 r2, %3, %5, y;\n\t"
        "madc.hi.u32 r3, %3, %5, z;\n\t"
        "mov.b64 %0, {r0, r1};\n\t"
        "mov.b64 %1, {r2, r3};\n\t}"
        : "=l"(lo), "=l"(hi)
        : "r"((u32)a), "r"((u32)(a >> 32)), "r"((u32)b), "r"((u32)(b >> 32)));
    return ((u128)hi << 64) | lo;
#else
    return (u128)a * b;
#endif
}

// The high word.
WW_HD u64 lz_hi(u64 a, u64 b) {
#if defined(__CUDA_ARCH__)
    u64 hi;
    asm("{\n\t.reg .u64 e, o;\n\t.reg .u32 r0, r1, r2, r3, x, y, z;\n\t"
        "mul.wide.u32 o, %1, %4;\n\t"
        "mov.b64 {x, y}, o;\n\t"
        "mad.lo.cc.u32 x, %2, %3, x;\n\t"
        "madc.hi.cc.u32 y, %2, %3, y;\n\t"
        "addc.u32 z, 0, 0;\n\t"
        "mul.wide.u32 e, %1, %3;\n\t"
        "mov.b64 {r0, r1}, e;\n\t"
        "add.cc.u32 r1, r1, x;\n\t"
        "madc.lo.cc.u32 r2, %2, %4, y;\n\t"
        "madc.hi.u32 r3, %2, %4, z;\n\t"
        "mov.b64 %0, {r2, r3};\n\t}"
        : "=l"(hi)
        : "r"((u32)a), "r"((u32)(a >> 32)), "r"((u32)b), "r"((u32)(b >> 32)));
    return hi;
#else
    return mul_hi(a, b);
#endif
}

// a b + k
WW_HD u128 lz_mad(u64 a, u64 b, u64 k) {
#if defined(__CUDA_ARCH__)
    u64 lo, hi;
    asm("{\n\t.reg .u64 o;\n\t.reg .u32 r0, r1, r2, r3, x, y, z, kl, kh;\n\t"
        "mov.b64 {kl, kh}, %6;\n\t"
        "mul.wide.u32 o, %2, %5;\n\t"
        "mov.b64 {x, y}, o;\n\t"
        "mad.lo.cc.u32 x, %3, %4, x;\n\t"
        "madc.hi.cc.u32 y, %3, %4, y;\n\t"
        "addc.u32 z, 0, 0;\n\t"
        "mad.lo.cc.u32 r0, %2, %4, kl;\n\t"
        "madc.hi.cc.u32 r1, %2, %4, kh;\n\t"
        "addc.cc.u32 y, y, 0;\n\t"
        "addc.u32 z, z, 0;\n\t"
        "add.cc.u32 r1, r1, x;\n\t"
        "madc.lo.cc.u32 r2, %3, %5, y;\n\t"
        "madc.hi.u32 r3, %3, %5, z;\n\t"
        "mov.b64 %0, {r0, r1};\n\t"
        "mov.b64 %1, {r2, r3};\n\t}"
        : "=l"(lo), "=l"(hi)
        : "r"((u32)a), "r"((u32)(a >> 32)), "r"((u32)b), "r"((u32)(b >> 32)), "l"(k));
    return ((u128)hi << 64) | lo;
#else
    return (u128)a * b + k;
#endif
}

// a^2: a0 a1 is shifted in by 33 bits.
WW_HD u128 lz_square(u64 a) {
#if defined(__CUDA_ARCH__)
    u64 lo, hi;
    asm("{\n\t.reg .u64 e, o;\n\t.reg .u32 r0, r1, r2, r3, x, y, z;\n\t"
        "mul.wide.u32 o, %2, %3;\n\t"
        "mov.b64 {x, y}, o;\n\t"
        "shf.l.clamp.b32 z, x, y, 1;\n\t"
        "shl.b32 x, x, 1;\n\t"
        "shr.u32 y, y, 31;\n\t"
        "mul.wide.u32 e, %2, %2;\n\t"
        "mov.b64 {r0, r1}, e;\n\t"
        "add.cc.u32 r1, r1, x;\n\t"
        "madc.lo.cc.u32 r2, %3, %3, z;\n\t"
        "madc.hi.u32 r3, %3, %3, y;\n\t"
        "mov.b64 %0, {r0, r1};\n\t"
        "mov.b64 %1, {r2, r3};\n\t}"
        : "=l"(lo), "=l"(hi) : "r"((u32)a), "r"((u32)(a >> 32)));
    return ((u128)hi << 64) | lo;
#else
    return (u128)a * a;
#endif
}

// a^2 + k0 (below 2^128 for a^2 + k0 of the ladders: a < p, k0 < p)
WW_HD u128 lz_square_add(u64 a, u64 k0) {
#if defined(__CUDA_ARCH__)
    u64 lo, hi;
    asm("{\n\t.reg .u64 o;\n\t.reg .u32 r0, r1, r2, r3, x, y, z, kl, kh;\n\t"
        "mov.b64 {kl, kh}, %4;\n\t"
        "mul.wide.u32 o, %2, %3;\n\t"
        "mov.b64 {x, y}, o;\n\t"
        "shf.l.clamp.b32 z, x, y, 1;\n\t"
        "shl.b32 x, x, 1;\n\t"
        "shr.u32 y, y, 31;\n\t"
        "mad.lo.cc.u32 r0, %2, %2, kl;\n\t"
        "madc.hi.cc.u32 r1, %2, %2, kh;\n\t"
        "addc.cc.u32 z, z, 0;\n\t"
        "addc.u32 y, y, 0;\n\t"
        "add.cc.u32 r1, r1, x;\n\t"
        "madc.lo.cc.u32 r2, %3, %3, z;\n\t"
        "madc.hi.u32 r3, %3, %3, y;\n\t"
        "mov.b64 %0, {r0, r1};\n\t"
        "mov.b64 %1, {r2, r3};\n\t}"
        : "=l"(lo), "=l"(hi) : "r"((u32)a), "r"((u32)(a >> 32)), "l"(k0));
    return ((u128)hi << 64) | lo;
#else
    return (u128)a * a + k0;
#endif
}

// Low digit of T / R for T < p 2^64: the digit, u = T q mod 2^64 and the
// borrow mask that the high digit takes over.
WW_HD u64 lz_low(u128 T, const LzMod &m, u64 &u, u32 &neg) {
    u = (u64)T * m.q;
    const u64 r = lz_sub((u64)(T >> 64), lz_hi(u, m.p), neg);
    return lz_addp(r, neg, m);
}

// High digit from the sum (k:h:s), k signed: ((k:h) - hi(s q p)) in [-p, 2p).
WW_HD u64 lz_high(u64 s, u64 h, u32 k, const LzMod &m) {
    const u64 v = lz_hi(s * m.q, m.p);
#if defined(__CUDA_ARCH__)
    u64 r;
    u32 t;
    asm("sub.cc.u64 %0, %2, %3;\n\t"
        "subc.u32 %1, %4, 0;"
        : "=&l"(r), "=r"(t) : "l"(h), "l"(v), "r"(k));
    return lz_fix(r, t, m);
#else
    const __int128 T = (((__int128)(int)k) << 64) + h - v;
    return (u64)T - (u64)(long long)(T >> 64) * m.p;
#endif
}

// As lz_high for the sum (k:h:s) less 2^64 for the borrow mask neg.
WW_HD u64 lz_high_less(u64 s, u64 h, u32 k, u32 neg, const LzMod &m) {
#if defined(__CUDA_ARCH__)
    const u64 v = lz_hi(s * m.q, m.p);
    u64 r;
    u32 t;
    asm("{\n\t.reg .u32 z;\n\t"
        "sub.cc.u32 z, 0, %5;\n\t"
        "subc.cc.u64 %0, %2, %3;\n\t"
        "subc.u32 %1, %4, 0;\n\t}"
        : "=&l"(r), "=r"(t) : "l"(h), "l"(v), "r"(k), "r"(neg));
    return lz_fix(r, t, m);
#else
    if (neg) k -= h-- == 0;
    return lz_high(s, h, k, m);
#endif
}

// (k:h:s) = a + b + u + 2^64 neg, neg a borrow mask (0 or -1).
WW_HD void lz_sum(u128 a, u128 b, u64 u, u32 neg, u64 &s, u64 &h, u32 &k) {
#if defined(__CUDA_ARCH__)
    u64 neg2;
    asm("mov.b64 %0, {%1, %1};" : "=l"(neg2) : "r"(neg));
    asm("add.cc.u64 %0, %3, %5;\n\t"
        "addc.cc.u64 %1, %4, %6;\n\t"
        "addc.u32 %2, 0, %8;\n\t"
        "add.cc.u64 %0, %0, %7;\n\t"
        "addc.cc.u64 %1, %1, %9;\n\t"
        "addc.u32 %2, %2, 0;"
        : "=&l"(s), "=&l"(h), "=&r"(k)
        : "l"((u64)a), "l"((u64)(a >> 64)), "l"((u64)b), "l"((u64)(b >> 64)), "l"(u), "r"(neg), "l"(neg2));
#else
    u128 t = a + b;
    k = t < a;
    t += u;
    k += t < u;
    s = (u64)t;
    h = (u64)(t >> 64);
    if (neg) k -= h-- == 0;
#endif
}

// X^2 / R
WW_HD D2 lz_sqr(D2 x, const LzMod &m) {
    u64 u, s, h;
    u32 neg, k;
    D2 r;
    r.d0 = lz_low(lz_square(x.d0), m, u, neg);
    const u128 c = lz_mul(x.d0, x.d1);
    lz_sum(c, c, u, neg, s, h, k);
    r.d1 = lz_high(s, h, k, m);
    return r;
}
// (X^2 + K) / R for K = kh.d0 + 2 p kh.d1, both digits below p (lz_halve)
WW_HD D2 lz_sqr_add(D2 x, D2 kh, const LzMod &m) {
    u64 u, s, h;
    u32 neg, k;
    D2 r;
    r.d0 = lz_low(lz_square_add(x.d0, kh.d0), m, u, neg);
    const u128 c = lz_mad(x.d0, x.d1, kh.d1);
    lz_sum(c, c, u, neg, s, h, k);
    r.d1 = lz_high(s, h, k, m);
    return r;
}
// Canonical K as lz_sqr_add takes it: its high digit halved mod p
WW_HD D2 lz_halve(D2 kk, u64 p) {
    const u64 add = (kk.d1 & 1) ? p : 0;
    const u64 sum = kk.d1 + add;
    kk.d1 = (sum >> 1) | ((u64)(sum < add) << 63);
    return kk;
}
// (X Y + K) / R, K canonical
WW_HD D2 lz_mul_add(D2 x, D2 y, D2 kk, const LzMod &m) {
    u64 u, s, h;
    u32 neg, k;
    D2 r;
    r.d0 = lz_low(lz_mad(x.d0, y.d0, kk.d0), m, u, neg);
    const u128 a = lz_mad(x.d0, y.d1, u), b = lz_mad(x.d1, y.d0, kk.d1);
#if defined(__CUDA_ARCH__)
    asm("add.cc.u64 %0, %3, %5;\n\t"
        "addc.cc.u64 %1, %4, %6;\n\t"
        "addc.u32 %2, 0, 0;"
        : "=&l"(s), "=&l"(h), "=&r"(k)
        : "l"((u64)a), "l"((u64)(a >> 64)), "l"((u64)b), "l"((u64)(b >> 64)));
#else
    const u128 t = a + b;
    k = t < a;
    s = (u64)t;
    h = (u64)(t >> 64);
#endif
    r.d1 = lz_high_less(s, h, k, neg, m);
    return r;
}

// X 2^(d - 32) for 0 <= d < 32: each digit shifted left by d and reduced by
// one 32-bit Montgomery step.
WW_HD D2 lz_shift(D2 x, u32 d, const LzMod &m) {
    const u32 q0 = (u32)m.q, p0 = (u32)m.p, p1 = (u32)(m.p >> 32);
    D2 r;
    u32 neg, neg1;
    // low digit: T = x0 2^d, (T - w p) / 2^32 with w = T q mod 2^32
    const u64 h0 = x.d0 >> (32 - d);  // T >> 32 (d = 0: x0 >> 32)
    const u32 w = ((u32)x.d0 << d) * q0;
    const u64 v = (u64)w * p1 + (((u64)w * p0) >> 32);
    const u64 r0 = lz_sub(h0, v, neg);
    r.d0 = lz_addp(r0, neg, m);
    // high digit: x1 2^d + w the same way, less the borrow
    const u32 c0 = (u32)x.d1 << d;
    const u32 s0 = c0 + w;
    const u64 h1 = (x.d1 >> (32 - d)) + (u64)(s0 < w);
    const u32 w1 = s0 * q0;
    const u64 v1 = (u64)w1 * p1 + (((u64)w1 * p0) >> 32) + (u64)(neg & 1u);
    const u64 r1 = lz_sub(h1, v1, neg1);
    r.d1 = lz_addp(r1, neg1, m);
    return r;
}

// 2^e by left-to-right squaring, for the Wieferich test and the PRP test: the
// bits of e below its start are multiplied in five at a time as 2^(d-32),
// 0 <= d < 32 (one-word Montgomery steps: 6 instructions a bit for two digits
// where a conditional doubling takes 18, 3 against 11 for one).  With
// f = e + sum of 32^(w+1) over the windows w, e is the start f >> steps
// times 2^steps plus the sum of (d_w - 32) 32^w.  Where e >> steps is below
// 32 the start is at most 48 (steps = 5 w + 1 and an exponent of ones: 31,
// 16 from the top window's 32^w and a carry).
constexpr int kWinBits = 5;
WW_HD u64 power_windows(u64 e, int steps) {
    // 32 + 32^2 + ... for ceil(steps / 5) windows
    const int n = (steps + kWinBits - 1) / kWinBits;
    const u64 ones = 0x0842108421084210ull << 1;  // bits 5, 10, ..., 60
    return e + (ones & ((2ull << (kWinBits * n)) - 1));
}
// The digit of the window at bit pos, below bit i (the top window is short).
WW_HD u32 window_digit(u64 f, int pos, int i) { return (u32)(f >> pos) & ((1u << (i - pos)) - 1u); }

// A^2 / R mod n
WW_HD u64 lz_sqr1(u64 a, const LzMod &m) {
    u64 u;
    u32 neg;
    return lz_low(lz_square(a), m, u, neg);
}
// A 2^(d - 32) mod n for 0 <= d < 32 (lz_shift's low digit)
WW_HD u64 lz_shift1(u64 a, u32 d, const LzMod &m) {
    const u32 w = ((u32)a << d) * (u32)m.q;
    u32 neg;
    const u64 r = lz_sub(a >> (32 - d), (u64)w * (u32)(m.p >> 32) + (((u64)w * (u32)m.p) >> 32), neg);
    return lz_addp(r, neg, m);
}

#if defined(__CUDACC__)

// The base-2 strong probable-prime test (sprp2) for a whole warp: all 32
// lanes call it, and lanes with act false test the first active lane's number
// and return false.  The bits of n-1 above every lane's lowest set bit t touch
// neither the value at bit t nor the -1 check, so the powering takes them in
// windows of five, with the same number of squarings in every lane; from the
// warp's largest t down (some six squarings) it goes bit by bit, as sprp2
// does, and keeps the value at bit t and whether -1 appears below it.
__device__ __forceinline__ bool sprp2_warp(u64 n, bool act, u64 &q_out) {
    const u32 live = __ballot_sync(0xffffffffu, act);
    if (live == 0) {
        q_out = 0;
        return false;
    }
    const u64 src = __shfl_sync(0xffffffffu, n, __ffs((int)live) - 1);
    n = act ? n : src;
    const u64 q = inv64(n);
    q_out = q;
    const LzMod m = lz_mod(n, q);
    const u64 one = r_mod(n);
    const u64 mone = n - one;
    const u64 nm1 = n - 1;
    const int t = __ffsll((long long)nm1) - 1;  // >= 1: n is odd
    const int tw = (int)__reduce_max_sync(0xffffffffu, (unsigned)t);
    const int top = (int)__reduce_max_sync(0xffffffffu, (unsigned)(63 - __clzll((long long)nm1)));
    const int steps = top - tw > 5 ? top - tw - 5 : 0;
    const u64 f = power_windows(nm1 >> tw >> 1, steps);
    const u32 e0 = (u32)(f >> steps);
    u64 a = one, unused;
    if (e0) a = mod_est(one >> (64 - e0), one << e0, n, 1.0 / (double)n, unused);
    int i = steps, pos = (steps + kWinBits - 1) / kWinBits * kWinBits;
    while (i > 0) {
        pos -= kWinBits;
        const u32 d = window_digit(f, pos, i);
        for (; i > pos; --i) a = lz_sqr1(a, m);
        a = lz_shift1(a, d, m);
    }
    u64 ebits = nm1 << (63 - tw);  // bit tw at bit 63
    u64 at_t = 0;
    bool m1 = false;
    for (i = tw; i >= 1; --i) {
        a = lz_sqr1(a, m);
        const u64 d = add_mod(a, a, n);
        a = ((long long)ebits < 0) ? d : a;
        ebits <<= 1;
        at_t = (i == t) ? a : at_t;
        m1 |= (i < t) & (a == mone);
    }
    const bool ok = (at_t == one) | (at_t == mone) | m1;
    return act && ok;
}
#endif

// x1 < 2p made canonical
WW_HD D2 lz_canonical(D2 x, u64 p) {
    if (x.d1 >= p) x.d1 -= p;
    return x;
}

}  // namespace ww
