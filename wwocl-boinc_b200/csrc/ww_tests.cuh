// ww_tests.cuh -- the Wieferich and Wall-Sun-Sun tests of one prime, and the
// reference's hit classification.
//
// The ladders run on the two-digit arithmetic of ww_ladder.cuh.  Arith64
// (64-bit C products, ww_arith.cuh), Arith32 (explicit 32-bit PTX carry
// chains) and ArithWide (32x32+64 wide products, ww_chain.cuh) are the
// canonical forms that the operand-level checks compare; WW_ARITH also sets
// the PRP test's form.
#pragma once

#include "ww_arith.cuh"
#include "ww_chain.cuh"
#include "ww_ladder.cuh"

namespace ww {

struct Arith64 {
    u64 p, q;
    WW_HD Arith64(u64 p_, u64 q_) : p(p_), q(q_) {}
    WW_HD D2 mul(D2 x, D2 y) const { return m2_mul(x, y, p, q); }
    WW_HD D2 sqr(D2 x) const { return m2_sqr(x, p, q); }
    WW_HD D2 redc(D2 x) const { return m2_redc(x, p, q); }
};

struct Arith32 {
    P32 P;
    WW_HD Arith32(u64 p, u64 q) : P(make_p32(p, q)) {}
    WW_HD D2 mul(D2 x, D2 y) const { return m2_mul32(x, y, P); }
    WW_HD D2 sqr(D2 x) const { return m2_sqr32(x, P); }
    WW_HD D2 redc(D2 x) const { return m2_redc32(x, P); }
};

struct ArithWide {
    u64 p, q;
    WW_HD ArithWide(u64 p_, u64 q_) : p(p_), q(q_) {}
    WW_HD D2 mul(D2 x, D2 y) const { return m2_mul_w(x, y, p, q); }
    WW_HD D2 sqr(D2 x) const { return m2_sqr_w(x, p, q); }
    WW_HD D2 redc(D2 x) const { return m2_redc_w(x, p, q); }
};

// WW_ARITH_VERSION: 1 = 64-bit C products (default), 2 = PTX carry chains,
// 3 = wide 32x32+64 products.  All three give identical digits.
#if defined(WW_ARITH_VERSION) && WW_ARITH_VERSION == 2
typedef Arith32 WW_ARITH;
WW_HD bool prp_test(u64 n, u64 &q) { return sprp2_32(n, q); }
#elif defined(WW_ARITH_VERSION) && WW_ARITH_VERSION == 3
typedef ArithWide WW_ARITH;
WW_HD bool prp_test(u64 n, u64 &q) { return sprp2(n, q); }
#else
typedef Arith64 WW_ARITH;
WW_HD bool prp_test(u64 n, u64 &q) { return sprp2(n, q); }
#endif

#if defined(__CUDACC__)
// prp_test for a whole warp (all lanes call it; act false gives false)
__device__ __forceinline__ bool prp_test_warp(u64 n, bool act, u64 &q) {
#if defined(WW_ARITH_VERSION) && WW_ARITH_VERSION == 2
    return act && sprp2_32(n, q);
#else
    return sprp2_warp(n, act, q);
#endif
}
#endif

WW_HD int top_bit(u64 x) {
#if defined(__CUDA_ARCH__)
    return 63 - __clzll((long long)x);
#else
    return 63 - __builtin_clzll(x);
#endif
}

WW_HD D2 sel(bool c, D2 a, D2 b) {
    D2 r;
    r.d0 = c ? a.d0 : b.d0;
    r.d1 = c ? a.d1 : b.d1;
    return r;
}

// W_k = V_2k, the Lucas numbers of even index (P = 3, Q = 1), for 0 <= k <= 33,
// all below 2^46: the ladder's state after the top bits of its index.
#define WW_LUCAS_EVEN                                                                                       \
    2ull, 3ull, 7ull, 18ull, 47ull, 123ull, 322ull, 843ull, 2207ull, 5778ull, 15127ull, 39603ull,           \
        103682ull, 271443ull, 710647ull, 1860498ull, 4870847ull, 12752043ull, 33385282ull, 87403803ull,     \
        228826127ull, 599074578ull, 1568397607ull, 4106118243ull, 10749957122ull, 28143753123ull,           \
        73681302247ull, 192900153618ull, 505019158607ull, 1322157322203ull, 3461452808002ull,               \
        9062201101803ull, 23725150497407ull, 62113250390418ull
#if defined(__CUDACC__)
static __device__ const u64 g_lucas_even[34] = {WW_LUCAS_EVEN};
#endif
static const u64 h_lucas_even[34] = {WW_LUCAS_EVEN};

WW_HD u64 lucas_even(u32 k) {  // k <= 33
#if defined(__CUDA_ARCH__)
    return __ldg(&g_lucas_even[k]);
#else
    return h_lucas_even[k];
#endif
}

// The two exponents have the same length to within a bit: (p-1)/2 for the
// Wieferich powering of 2, and j = (p - (p|5))/2 for the Lucas ladder, since
// F_2j comes from W_j and W_j+1.  Both ladders take the same number of steps,
// and so do all lanes of a warp: the warp's longest j less five bits.  What
// lies above the steps' bits is at most 5 bits of the start (31, or 32 for a
// j of 2^k), fewer for a lane whose p is shorter.
WW_HD u64 lucas_index(u64 p) {
    const u32 pm5 = (u32)(p % 5);
    return ((pm5 == 2 || pm5 == 3) ? p + 1 : p - 1) >> 1;
}
// every lane of the warp calls it
WW_HD int ladder_steps(u64 j) {
    int top = j ? top_bit(j) : 0;
#if defined(__CUDA_ARCH__)
    top = (int)__reduce_max_sync(0xffffffffu, (unsigned)top);
#endif
    return top > 4 ? top - 4 : 0;
}

// L R mod p^2 as canonical digits for L <= 2^48 (a power of 2 of the Wieferich
// start; Lucas numbers are below 2^46), below 2^48 for p >= 2^62.  There the
// quotient of L 2^64 by p is below 2^50, as mod_est wants it, and it is the
// high digit as it stands: one reduction, where m2_small needs two and the
// products with the digits of R.
WW_HD D2 small_start(u64 L, D2 one, u64 p, double rp) {
    if (p >> 62) {
        D2 r;
        r.d0 = mod_est(L, 0, p, rp, r.d1);
        return r;
    }
    return m2_small(L, one, p, rp);
}

struct LadderConst {
    D2 m2h, m3;  // -2 R^2 (as lz_halve leaves it) and -3 R^2
};
WW_HD LadderConst ladder_const(D2 one, const LzMod &m, double rp) {
    // R 2^32, squared: R^2 2^64 / R = R^2
    const D2 r2 = lz_canonical(lz_sqr(small_start(1ull << 32, one, m.p, rp), m), m.p);
    const D2 zero = {0, 0};
    const D2 t2 = m2_dbl(r2, m.p);
    LadderConst c;
    const D2 m2 = m2_sub(zero, t2, m.p);
    c.m2h = lz_halve(m2, m.p);
    c.m3 = m2_sub(m2, r2, m.p);
    return c;
}

// One Lucas step on (e, o) = (W at the even, at the odd of the indices k,
// k+1): W_2k+1 = W_k W_k+1 - 3 is always the odd one, and the even one is
// W_2k = W_k^2 - 2 or W_2k+2, the square of e or of o by the bit and the
// parity of k.  Against two squarings and their difference (V_2k+1 =
// V_2k+2 - V_2k) the product costs a cross product more and saves the
// difference with its two corrections, whose operands would have to be
// canonical.
WW_HD void lucas_step(D2 &e, D2 &o, bool &kodd, bool bit, const LadderConst &c, const LzMod &m) {
    const D2 s = sel(bit == kodd, e, o);
    o = lz_mul_add(e, o, c.m3, m);
    e = lz_sqr_add(s, c.m2h, m);
    kodd = bit;
}

// F_n = (2 W_j+1 - 3 W_j) / 5 for n = 2j: 5 is a unit mod p^2 since p has no
// factor below 127.
WW_HD D2 lucas_finish(D2 e, D2 o, bool jodd, u64 p, u64 q) {
    const D2 a = lz_canonical(sel(jodd, o, e), p);  // W_j
    const D2 b = lz_canonical(sel(jodd, e, o), p);  // W_j+1
    const D2 d = m2_sub(b, a, p);
    return m2_div5(m2_redc(m2_sub(m2_dbl(d, p), a, p), p, q), p);
}

// For p < 2^32, p^2 fits a word: the same ladders on residues mod n = p^2 in
// one-word Montgomery form, a third of the multiplies.  A whole warp takes it
// or none of its lanes does (small_modulus); kept out of line, so that the
// kernels' main loops keep their registers.
WW_HD bool small_modulus(u64 p) {
#if defined(__CUDA_ARCH__)
    return __all_sync(0xffffffffu, (p >> 32) == 0);
#else
    return (p >> 32) == 0;
#endif
}

#if defined(__CUDACC__)
#define WW_HD_CALL static __host__ __device__ __noinline__
#else
#define WW_HD_CALL static inline
#endif

struct SmallMod {
    LzMod m;     // n = p^2
    u64 one;     // 2^64 mod n
    double rn;   // 1 / (double)n
};
WW_HD SmallMod small_mod(u64 p) {
    SmallMod s;
    const u64 n = p * p;
    s.m = lz_mod(n, inv64(n));
    s.one = r_mod(n);
    s.rn = 1.0 / (double)n;
    return s;
}
// L R mod n for 1 <= L <= 2^48
WW_HD u64 small_times_r(u64 L, const SmallMod &s) {
    u64 l, h, unused;
    mul_wide(L, s.one, l, h);
    return mod_est(h, l, s.m.p, s.rn, unused);
}
// (x R^-1 mod n) as digits by p
WW_HD D2 small_digits(u64 x, u64 p, const SmallMod &s) {
    D2 d;
    d.d0 = mod_est(0, redc(x, 0, s.m.p, s.m.q), p, 1.0 / (double)p, d.d1);
    return d;
}

WW_HD_CALL D2 wieferich_small(u64 p, int steps) {
    const SmallMod s = small_mod(p);
    const u64 f = power_windows(p >> 1, steps);
    u64 a = small_times_r(1ull << (f >> steps), s);
    int pos = (steps + kWinBits - 1) / kWinBits * kWinBits;
    int i = steps;
    while (i > 0) {
        pos -= kWinBits;
        const u32 d = window_digit(f, pos, i);
        for (; i > pos; --i) a = lz_sqr1(a, s.m);
        a = lz_shift1(a, d, s.m);
    }
    return small_digits(a, p, s);
}

WW_HD_CALL D2 wss_small(u64 p, u64 j, int steps) {
    const SmallMod s = small_mod(p);
    // R 2^32, squared: R^2; the constants -2 R^2 and -3 R^2
    const u64 r2 = lz_sqr1(small_times_r(1ull << 32, s), s.m);
    const u64 c2 = sub_mod(0, add_mod(r2, r2, s.m.p), s.m.p);
    const u64 c3 = sub_mod(c2, r2, s.m.p);
    const u32 k0 = (u32)(j >> steps);
    bool kodd = k0 & 1u;
    u64 e = small_times_r(lucas_even(k0 + (k0 & 1u)), s);
    u64 o = small_times_r(lucas_even(k0 | 1u), s);
    u64 jb = j << (63 - steps) << 1;
    for (int i = steps; i > 0; --i) {
        const bool bit = (long long)jb < 0;
        jb <<= 1;
        const u64 x = bit == kodd ? e : o;
        u64 u;
        u32 neg;
        o = lz_low(lz_mad(e, o, c3), s.m, u, neg);
        e = lz_low(lz_square_add(x, c2), s.m, u, neg);
        kodd = bit;
    }
    const u64 a = kodd ? o : e, b = kodd ? e : o;  // W_j, W_j+1
    const u64 d = sub_mod(b, a, s.m.p);
    return m2_div5(small_digits(sub_mod(add_mod(d, d, s.m.p), a, s.m.p), p, s), p);
}

// 2^((p-1)/2) mod p^2 as canonical digits (wieferich.cl:219-245).  The five
// squarings of a window are written out for the list kernels (1 658 M
// primes/s, as a loop 1 635) and a loop (kWriteOut false) in the tile engine,
// whose warps run sieve, PRP test and both ladders at the same time and were
// waiting for instructions (96 ranges: 42.2 ms written out, 40.3 as a loop).
template <bool kWriteOut = true>
WW_HD D2 wieferich_digits(u64 p, u64 q, D2 one) {
    const int steps = ladder_steps(lucas_index(p));
    if (small_modulus(p)) return wieferich_small(p, steps);
    const LzMod m = lz_mod(p, q);
    const double rp = 1.0 / (double)p;
    const u64 f = power_windows(p >> 1, steps);
    D2 w = small_start(1ull << (f >> steps), one, p, rp);
    int pos = (steps + kWinBits - 1) / kWinBits * kWinBits;  // the window's low bit, once it is taken
    int i = steps;
    while (i > 0) {
        pos -= kWinBits;
        const u32 d = window_digit(f, pos, i);
        if (kWriteOut && i - pos == kWinBits) {
            w = lz_sqr(w, m);
            w = lz_sqr(w, m);
            w = lz_sqr(w, m);
            w = lz_sqr(w, m);
            w = lz_sqr(w, m);
            i = pos;
        }
#if defined(__CUDA_ARCH__)
#pragma unroll 1
#endif
        for (; i > pos; --i) w = lz_sqr(w, m);
        w = lz_shift(w, d, m);
    }
    return m2_redc(lz_canonical(w, p), p, q);
}

// F_{p-(p|5)} mod p^2 as canonical digits (wallsunsun.cl:242-300).
WW_HD D2 wss_digits(u64 p, u64 q, D2 one) {
    const u64 j = lucas_index(p);
    const int steps = ladder_steps(j);
    if (small_modulus(p)) return wss_small(p, j, steps);
    const LzMod m = lz_mod(p, q);
    const double rp = 1.0 / (double)p;
    const LadderConst c = ladder_const(one, m, rp);
    const u32 k0 = (u32)(j >> steps);
    bool kodd = k0 & 1u;
    D2 e = small_start(lucas_even(k0 + (k0 & 1u)), one, p, rp);
    D2 o = small_start(lucas_even(k0 | 1u), one, p, rp);
    u64 jb = j << (63 - steps) << 1;  // the next bit at bit 63
    for (int i = steps; i > 0; --i) {
        lucas_step(e, o, kodd, (long long)jb < 0, c, m);
        jb <<= 1;
    }
    return lucas_finish(e, o, kodd, p, q);
}

// Both in one loop: the three products of a step are independent.  (2e9
// numbers from 1e9 on in the tile engine: 36.3 ms without the one-word path,
// 23.7 with it; 2e9 numbers above 2^63, which pay for its branch: 39.3 and
// 39.5.)
WW_HD void both_digits(u64 p, u64 q, D2 one, D2 &s_out, D2 &c_out) {
    const u64 j = lucas_index(p);
    const int steps = ladder_steps(j);
    if (small_modulus(p)) {
        s_out = wieferich_small(p, steps);
        c_out = wss_small(p, j, steps);
        return;
    }
    const LzMod m = lz_mod(p, q);
    const double rp = 1.0 / (double)p;
    const u64 f = power_windows(p >> 1, steps);
    const LadderConst c = ladder_const(one, m, rp);
    const u32 k0 = (u32)(j >> steps);
    bool kodd = k0 & 1u;
    D2 e = small_start(lucas_even(k0 + (k0 & 1u)), one, p, rp);
    D2 o = small_start(lucas_even(k0 | 1u), one, p, rp);
    D2 w = small_start(1ull << (f >> steps), one, p, rp);
    u64 jb = j << (63 - steps) << 1;
    int pos = (steps + kWinBits - 1) / kWinBits * kWinBits;
    int i = steps;
    while (i > 0) {
        pos -= kWinBits;
        const u32 d = window_digit(f, pos, i);
        for (; i > pos; --i) {
            lucas_step(e, o, kodd, (long long)jb < 0, c, m);
            w = lz_sqr(w, m);
            jb <<= 1;
        }
        w = lz_shift(w, d, m);
    }
    s_out = m2_redc(lz_canonical(w, p), p, q);
    c_out = lucas_finish(e, o, kodd, p, q);
}

// ------------------------------------------------------------ classification

constexpr u64 kThreshold = 1000;  // WW.h:8 SPECIAL_THRESHOLD

// wieferich.cl:248-293.  Returns true and fills rem/quot for a hit.
WW_HD bool wieferich_classify(u64 p, D2 s, int &rem, int &quot) {
    if (((s.d1 == 0) & (s.d0 == 1)) | ((s.d1 == p - 1) & (s.d0 == p - 1))) {
        rem = 1;
        quot = 0;
        return true;
    }
    if (s.d1 <= kThreshold) {
        if (s.d0 == 1) { rem = 1; quot = (int)s.d1; return true; }
        if (s.d0 == p - 1) { rem = -1; quot = (int)(s.d1 + 1); return true; }
        return false;
    }
    if (s.d1 >= p - kThreshold) {
        if (s.d0 == 1) { rem = 1; quot = (int)(s.d1 - p); return true; }
        if (s.d0 == p - 1) { rem = -1; quot = (int)(s.d1 + 1 - p); return true; }
    }
    return false;
}

// wallsunsun.cl:325-349.  result 1 = WSS prime, 2 = special instance.
WW_HD bool wss_classify(u64 p, D2 c, int &result, int &quot) {
    if (c.d1 == 0) { result = 1; quot = 0; return true; }
    if (c.d1 <= kThreshold) { result = 2; quot = (int)c.d1; return true; }
    if (c.d1 >= p - kThreshold) { result = 2; quot = (int)(c.d1 - p); return true; }
    return false;
}

}  // namespace ww
