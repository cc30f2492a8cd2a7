// ww_kernels.cuh -- kernels of the WWocl search path on sm_100a.
//
//   k_sieve_prp   getsegprimes (getsegprimes.cl:228-301): a CTA sieves one
//                 segment of 2*G::kOdd integers at a time (taken from a cursor,
//                 or by grid stride).  The odd numbers of the segment form a
//                 shared-memory bitmap; each thread ORs the composite patterns
//                 of 3..113 into its words (the reference's 27 constant tables,
//                 getsegprimes.cl:169-225, become per-prime bit offsets kept
//                 incrementally), the deep sieve marks the multiples of the
//                 primes up to 2^WW_DEEP_BITS that cannot be pseudoprimes
//                 (ww_deep.cuh), then each warp compacts the survivors with
//                 ballot/popc into a warp queue and runs the base-2 strong
//                 PRP test 32 candidates at a time, one atomic per warp for the
//                 output slots.
//   k_wieferich / k_wallsunsun   the two reference test kernels.
//   k_test_prps   both tests in one pass over the PRP list (warps pull work
//                 from a cursor, or stride).
//   k_digits      per-prime canonical digits (verification only).
#pragma once

#include "ww_device.cuh"

namespace ww {

// Threads per SM the sieve's launch bounds ask for: 1024 holds it to 64
// registers (2 CTAs of 512, or 4 of 256, per SM).  Uncapped it takes 128;
// at 512 or 768 (1 CTA of 512 per SM, 128 registers) the sieve measured
// 7.19 against 5.90 ms per 2^30 numbers on a B200 (with a doubling per bit
// in the PRP test; 4.87 ms with its windows).
#ifndef WW_SIEVE_MINB_THREADS
#define WW_SIEVE_MINB_THREADS 1024
#endif

// Sieve + SPRP over [lo, hi) in segments of shape G (SieveGeom).  b0 = lo & ~1;
// segment s holds the odd numbers b0 + 2(s*G::kOdd + j) + 1, j < G::kOdd.
// With a segment cursor (zeroed before the launch) the CTAs take segments
// one at a time from it; without one (a launch captured into a graph, or
// one that found every cursor of the library's pool busy) they stride over
// the segments.  marks (optional): the large deep primes' marks of the whole
// launch, bit j of word w = odd number b0 + 2(32 w + j) + 1 (ww_bucket.cu),
// ORed into each segment's bitmap.  plan: SievePlan.
template <class G>
__global__ void __launch_bounds__(G::kThreads, WW_SIEVE_MINB_THREADS / G::kThreads) k_sieve_prp(u64 lo, u64 hi, u64 nseg, PrpOut out,
                                                                              u64 *cursor, const DeepRow *deep,
                                                                              const u32 *__restrict__ marks,
                                                                              SievePlan plan) {
    extern __shared__ u32 sieve_smem[];
    int words, chunk_words;  // of a segment, and of the share a warp takes of it at a time
    if constexpr (G::kRuntime) {
        words = plan.words;
        chunk_words = min(32, words / G::kWarps);
    } else {
        words = G::kWords;
        chunk_words = 32;
    }
    const u64 odd = 32ull * (u64)words;  // odd numbers of a segment
    u32 *bitmap = sieve_smem;
    u32(*queue)[kQueueCap] = reinterpret_cast<u32(*)[kQueueCap]>(sieve_smem + words);
    __shared__ u32 s_chunk;
    __shared__ u64 s_seg;
    const u64 b0 = lo & ~1ull;
    const u64 span = hi - b0;
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;

    u64 seg = blockIdx.x;
    if (cursor) {
        if (threadIdx.x == 0) s_seg = atomicAdd((unsigned long long *)cursor, 1ull);
        __syncthreads();
        seg = s_seg;
    }
    while (seg < nseg) {
        const u64 seg_off = seg * 2 * odd;
        const u64 rem_span = span - seg_off;  // > 0
        const u64 nvalid = rem_span / 2 < odd ? rem_span / 2 : odd;

        // ---- pre-sieve 3..113 on this thread's contiguous words
        const int wpt = (words + G::kThreads - 1) / G::kThreads;
        const int w0 = threadIdx.x * wpt;
        const int w1 = G::kRuntime ? min(w0 + wpt, words) : w0 + wpt;
        if (!G::kRuntime || w0 < words) {
            const u64 n0 = b0 + seg_off + 64ull * (u64)w0 + 1;  // may wrap past 2^64 beyond hi
            const u32 *seg_marks = marks ? marks + seg * (u64)words : nullptr;
#define WW_J0(R) u32 j##R = first_hit<R>(n0);
            WW_FOR_SMALL_PRIMES(WW_J0)
#undef WW_J0
#pragma unroll 4
            for (int w = w0; w < w1; ++w) {
                u32 m = seg_marks ? seg_marks[w] : 0u;
#define WW_MASK(R) m |= prime_mask<R>(j##R); step_hit<R>(j##R);
                WW_FOR_SMALL_PRIMES(WW_MASK)
#undef WW_MASK
                // bits past the end of the range are not candidates
                const u64 first = (u64)w * 32;
                if (first + 32 > nvalid) {
                    const u64 keep = nvalid > first ? nvalid - first : 0;  // < 32
                    m |= ~((1u << keep) - 1u);
                }
                bitmap[w] = m;
            }
        }
        if (threadIdx.x == 0) s_chunk = 0;
        __syncthreads();

        // ---- deep sieve 113 < r < 2^WW_DEEP_BITS, sparing possible pseudoprimes
        const u64 nbase = b0 + seg_off + 1;
        deep_mark(nbase, (u32)nvalid, bitmap, threadIdx.x, G::kThreads, deep,
                  G::kRuntime ? plan.deep_n : kWideRows, G::kRuntime ? plan.warp_n : kDeepWarpPrimes);
        __syncthreads();

        // ---- warps take chunks of 32 words (or fewer) dynamically (so they reach the next
        // barrier together), compact the survivors with ballot/popc into a
        // warp queue and PRP-test them 32 at a time
        u32 *q = queue[warp];
        int qn = 0;
        for (;;) {
            u32 chunk = 0;
            if (lane == 0) chunk = atomicAdd(&s_chunk, 1u);
            chunk = __shfl_sync(0xffffffffu, chunk, 0);
            const bool more = (int)chunk * chunk_words < words;
            if (more) {
                const int w = chunk * chunk_words + lane;
                u32 cand = !G::kRuntime || lane < chunk_words ? ~bitmap[w] : 0u;
                const int cnt = __popc(cand);
                int incl = cnt;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int t = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += t;
                }
                const int total = __shfl_sync(0xffffffffu, incl, 31);
                int pos = qn + incl - cnt;
                while (cand) {
                    const int b = __ffs(cand) - 1;
                    q[pos++] = (u32)(w * 32 + b);
                    cand &= cand - 1;
                }
                qn += total;
                __syncwarp();
            }
            while (qn >= 32 || (!more && qn > 0)) {
                const int take = qn >= 32 ? 32 : qn;
                qn -= take;
                const bool act = lane < take;
                const u32 j = act ? q[qn + lane] : 0u;
                __syncwarp();
                sprp_emit(out, nbase + 2ull * j, act);
            }
            if (!more) break;
        }
        __syncthreads();  // bitmap reused by the next segment
        if (cursor) {
            if (threadIdx.x == 0) s_seg = atomicAdd((unsigned long long *)cursor, 1ull);
            __syncthreads();
            seg = s_seg;
        } else {
            seg += gridDim.x;
        }
    }
}

// ------------------------------------------------------------------ tests

__device__ __forceinline__ void count_update(u32 *primecount, u64 *totalprimecount) {
    // wieferich.cl:317-326: accumulate the launch's PRP count, keep the max
    const u32 pc = primecount[0];
    *totalprimecount += pc;
    if (pc > primecount[1]) primecount[1] = pc;
}

// Runs f(unit) on whole warps for every unit < n.  With a work cursor (zeroed
// before the launch) each warp pulls one unit at a time, so warps that run
// ahead take more of the work and all finish together; without one (a
// launch captured into a graph, or one that found every cursor of the
// library's pool busy) the grid strides.  Units that do not outnumber the
// grid's warps go one to a warp, neighbours to different SMs, without the
// cursor, whose atomics from every warp of the grid would take longer than a
// step of the ladders.
template <class F>
__device__ __forceinline__ void for_each_unit(u64 n, u64 *cursor, F &&f) {
    const int lane = threadIdx.x & 31;
    // a list has below 2^37 primes, so units fit 32 bits (64-bit ones in this
    // loop cost the test kernel 1 %)
    const u32 m = (u32)n;
    u32 unit = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
    if (m <= (gridDim.x * blockDim.x) >> 5) cursor = nullptr;
    for (;;) {
        if (cursor) {
            if (lane == 0) unit = (u32)atomicAdd((unsigned long long *)cursor, 1ull);
            unit = __shfl_sync(0xffffffffu, unit, 0);
        }
        if (unit >= m) break;
        f(unit);
        unit += (gridDim.x * blockDim.x) >> 5;
    }
}

// f(i, whether the lane is one of the list's) for 32 consecutive list indices
// a unit.  The ladders run on whole warps: lanes past the end repeat the last
// prime, whose size is its neighbours'.
template <class F>
__device__ __forceinline__ void for_each_prime(u64 n, u64 *cursor, F &&f) {
    for_each_unit((n + 31) / 32, cursor, [&](u32 unit) {
        const u64 i = 32ull * unit + (threadIdx.x & 31);
        f(min(i, n - 1), i < n);
    });
}

__global__ void __launch_bounds__(kTestThreads, WW_TEST_MINB) k_wieferich(u32 *primecount, const u64 *prime,
                                                             const u64 *inv, u64 *g_one, HitOut hits,
                                                             u64 *checksum, u64 *totalprimecount,
                                                             u64 capacity, u64 *cursor) {
    const u64 n = min((u64)primecount[0], capacity);
    u64 sum = 0;
    for_each_prime(n, cursor, [&](u64 i, bool act) {
        const u64 p = prime[i];
        const u64 q = inv ? inv[i] : inv64(p);
        const D2 one = m2_one(p);
        if (act && g_one) {
            g_one[2 * i] = one.d0;
            g_one[2 * i + 1] = one.d1;
        }
        const D2 s = wieferich_digits(p, q, one);
        if (act) {
            sum += s.d1 & 0xffffffffull;
            int rem, quot;
            if (wieferich_classify(p, s, rem, quot)) emit_hit(hits, p, 1093, rem, quot);
        }
    });
    sum = warp_sum(sum);
    if ((threadIdx.x & 31) == 0 && sum) atomicAdd(checksum, sum);
    if (blockIdx.x == 0 && threadIdx.x == 0) count_update(primecount, totalprimecount);
}

__global__ void __launch_bounds__(kTestThreads, WW_TEST_MINB) k_wallsunsun(const u32 *primecount, const u64 *prime,
                                                              const u64 *inv, const u64 *g_one,
                                                              HitOut hits, u64 *checksum, u64 capacity,
                                                              u64 *cursor) {
    const u64 n = min((u64)primecount[0], capacity);
    u64 sum = 0;
    for_each_prime(n, cursor, [&](u64 i, bool act) {
        const u64 p = prime[i];
        const u64 q = inv ? inv[i] : inv64(p);
        D2 one;
        if (g_one) {
            one.d0 = g_one[2 * i];
            one.d1 = g_one[2 * i + 1];
        } else {
            one = m2_one(p);
        }
        const D2 c = wss_digits(p, q, one);
        if (act) {
            sum += c.d1 & 0xffffffffull;
            int res, quot;
            if (wss_classify(p, c, res, quot)) emit_hit(hits, p, res, 0, quot);
        }
    });
    sum = warp_sum(sum);
    if ((threadIdx.x & 31) == 0 && sum) atomicAdd(checksum, sum);
}

// Both tests over the list in one launch.  A unit of work is one test of 32
// primes: the Wall-Sun-Sun units first, which take twice as long, then the
// Wieferich ones, so the last of a launch are short, and a list shorter than
// the grid's warps runs its two tests on different warps.  The two in one
// loop (both_digits, 78 registers) measured 1 509 against 1 543 M primes/s
// on 2^24 primes (with the products as __int128 multiplies; 1 660 M since).
__global__ void __launch_bounds__(kTestThreads, WW_TEST_MINB) k_test_prps(u32 *primecount, const u64 *prime,
                                                             const u64 *inv, HitOut hits, u64 *checksum,
                                                             u64 *totalprimecount, u64 capacity,
                                                             u64 *cursor) {
    const u64 n = min((u64)primecount[0], capacity);
    const u32 groups = (u32)((n + 31) / 32);
    u64 sum = 0;
    for_each_unit(2ull * groups, cursor, [&](u32 unit) {
        const bool wss = unit < groups;
        const u64 at = 32ull * (wss ? unit : unit - groups) + (threadIdx.x & 31);
        const bool act = at < n;
        const u64 i = min(at, n - 1);  // lanes past the end repeat the last prime
        const u64 p = prime[i];
        const u64 q = inv ? inv[i] : inv64(p);
        const D2 one = m2_one(p);
        int res = 1093, rem = 0, quot;
        u64 digit;
        bool hit;
        if (wss) {
            const D2 c = wss_digits(p, q, one);
            digit = c.d1;
            hit = wss_classify(p, c, res, quot);
        } else {
            const D2 s = wieferich_digits(p, q, one);
            digit = s.d1;
            hit = wieferich_classify(p, s, rem, quot);
        }
        if (act) {
            sum += digit & 0xffffffffull;
            if (hit) emit_hit(hits, p, res, rem, quot);
        }
    });
    sum = warp_sum(sum);
    if ((threadIdx.x & 31) == 0 && sum) atomicAdd(checksum, sum);
    if (blockIdx.x == 0 && threadIdx.x == 0) count_update(primecount, totalprimecount);
}

// Units as in k_test_prps.
__global__ void __launch_bounds__(kTestThreads, WW_TEST_MINB) k_digits(const u64 *primes, u64 n, u64 *out) {
    const u32 groups = (u32)((n + 31) / 32);
    for_each_unit(2ull * groups, nullptr, [&](u32 unit) {
        const bool wss = unit < groups;
        const u64 i = 32ull * (wss ? unit : unit - groups) + (threadIdx.x & 31);
        const u64 p = primes[min(i, n - 1)];
        const u64 q = inv64(p);
        const D2 one = m2_one(p);
        const D2 d = wss ? wss_digits(p, q, one) : wieferich_digits(p, q, one);
        if (i < n) {
            u64 *to = out + 4 * i + (wss ? 2 : 0);
            to[0] = d.d0;
            to[1] = d.d1;
        }
    });
}

// q = p^-1 mod 2^64 for a loaded list; sets the segment count.
__global__ void k_fill_inverse(const u64 *prime, u64 *inv, u64 n) {
    for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x)
        inv[i] = inv64(prime[i]);
}

}  // namespace ww
