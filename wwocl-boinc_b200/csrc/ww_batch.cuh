// ww_batch.cuh -- the tile engine of the batched search and of the request
// server: many ranges of uneven width in one persistent launch that pulls
// (range, segment) tiles from a device queue.
//
// One CTA takes one tile at a time (an atomic on the tile counter), sieves
// it in a shared-memory bitmap, and runs the whole path on it without a PRP
// list in global memory: warps take 32-word chunks of the bitmap from a
// shared counter (so the warps of a CTA finish a tile together), compact
// the survivors into a warp queue, run the base-2 strong PRP test 32 at a
// time, and push the PRPs into a second warp queue that feeds the
// Wieferich and Wall-Sun-Sun tests 32 (or 64 with two primes per thread) at
// a time.  That queue is kept from tile to tile, each PRP with its unit, and
// emptied at the end of the launch, so small tiles do not leave test batches
// half empty.  Checksums and PRP counts go to the unit with one atomic per
// batch (one per lane where a batch mixes units); the sums are order-free, so
// every unit's checksum is bit-identical to a run of that unit alone.
//
// A unit's tile is at most the configuration's segment and a power of two of
// words below it (UnitState::words): tiles small enough that the launch has
// several for every resident CTA, since 2^20-number tiles gave a batch of
// eight ranges of 1e5 to 1e6 numbers to eight CTAs.
#pragma once

#include "ww_device.cuh"

namespace ww {

// Device state of one range (a unit of a batch or a served request).
struct UnitState {
    u64 start, end;          // [start, end), start >= 127 unless empty
    u64 n_tiles;             // ceil((end - start) / tile)
    u64 checksum;            // sum of both checksum terms
    u64 prp_count;           // PRPs tested
    u64 *prp_out;            // optional PRP buffer of the range (nullptr: none)
    u64 prp_cap;
    u64 prp_written;         // PRPs found (may exceed prp_cap: overflow)
    u64 tiles_done;          // 64 bits: tiles of 2^18 numbers in a request of 2^50 pass 2^32
    u32 hits;
    u32 words;               // bitmap words of a tile of this unit
};

// A unit's finished tiles counted in full ones of `tile` numbers, whatever
// they were cut into.
WW_HD u32 full_tiles(const UnitState &u, u64 tile) {
    if (u.tiles_done < u.n_tiles) return (u32)(u.tiles_done * 64 * u.words / tile);
    const u64 w = u.end - u.start;
    return (u32)(w / tile + (w % tile ? 1 : 0));
}

// Tiles have kTileMinWords << k words, k < kTileSizes.
constexpr int kTileMinWords = 128;
constexpr int kTileSizes = 9;

// Serving: the tiles [next, end) of one unit that a launch hands out.
struct StepShare {
    u64 next, end;
    u32 unit, pad;
};

struct BatchArgs {
    UnitState *units;
    u32 n_units;
    // static tile table (batch): tile_first[k] = first tile of unit k, n_units + 1 entries
    const u64 *tile_first;
    u64 n_tiles;
    u64 *next_tile;          // queue head
    // serving: this launch's tiles, n_shares units in the order they go out
    // (earliest deadline first)
    StepShare *shares;
    u32 n_shares;
    u64 *hit_p;
    int *hit_result, *hit_rem, *hit_quot;
    u32 *hit_unit;
    u32 *hit_count;
    u32 hit_capacity;
    u32 *overflow;           // bit 1: hit list overflow, bit 0: a PRP buffer overflowed
    const DeepRow *deep;     // the deep-sieve table (deep_rows_device())
    int deep_n[kTileSizes];  // its rows used for tiles of kTileMinWords << k words
};

// A tile configuration: SEG_WORDS bitmap words, THREADS per CTA, PPT batches
// of 32 PRPs a warp collects before testing them, and JOINT = 1 for the
// Wieferich and WSS tests of a prime in one loop (the list kernel's form)
// instead of one after the other.
template <int SEG_WORDS, int THREADS, int PPT, int JOINT = 0>
struct BatchCfg {
    static constexpr int kWords = SEG_WORDS;
    static constexpr int kThreads = THREADS;
    static constexpr int kWarps = THREADS / 32;
    static constexpr int kPpt = PPT;
    static constexpr bool kJoint = JOINT != 0;
    // resident threads per SM the registers must allow: 1024 (64 registers,
    // 32 warps) with one or two batches of PRPs per warp -- left to the
    // compiler, the 512-thread tiles took 128 registers (16 warps per SM)
    // and ran 7 % slower; four or eight batches keep the compiler's choice
    // (110 registers at 256 threads, two CTAs per SM; 142 and 146 while the
    // batches were written out, then faster than 78 and 80 at three CTAs)
    static constexpr int kSmThreads = PPT >= 4 ? THREADS : 1024;
    static constexpr int kMinBlocks = kSmThreads / THREADS > 0 ? kSmThreads / THREADS : 1;
    static constexpr u64 kTileNumbers = 64ull * SEG_WORDS;  // integers per full tile
    static constexpr int kCandCap = 416;  // as kQueueCap: 31 carried + at most 378 per 32-word chunk
    static constexpr int kPrpCap = 32 * PPT + 32;
    static_assert(SEG_WORDS % THREADS == 0, "words per thread");
};

__device__ __forceinline__ void emit_batch_hit(const BatchArgs &a, u32 unit, u64 p, int result, int rem, int quot) {
    const u32 ix = atomicAdd(a.hit_count, 1u);
    if (ix < a.hit_capacity) {
        a.hit_p[ix] = p;
        a.hit_result[ix] = result;
        a.hit_rem[ix] = rem;
        a.hit_quot[ix] = quot;
        a.hit_unit[ix] = unit;
    } else {
        atomicOr(a.overflow, 2u);
    }
    atomicAdd(&a.units[unit].hits, 1u);
}

// Wieferich + WSS on the first n_valid of 32*PPT entries of the warp's PRP
// queue, each added to its own unit.
template <int PPT, bool JOINT>
__device__ __forceinline__ void test_batch(const u64 *qp, const u32 *qu, int n_valid, const BatchArgs &a) {
    const int lane = threadIdx.x & 31;
    // one copy of the ladders: written out PPT times, warps at different
    // places of them waited for instructions (96 ranges of 1e6 to 1e8 numbers
    // with 2, 4 and 8 primes per thread in 2^19-number tiles 49.3, 84.3 and
    // 126.6 ms, as a loop 41.3, 43.0 and 43.4; with one 41.1)
#pragma unroll 1
    for (int k = 0; k < PPT; ++k) {
        const int idx = k * 32 + lane;
        if (k * 32 >= n_valid) break;
        const bool act = idx < n_valid;
        const u64 p = qp[act ? idx : 0];  // idle lanes repeat the first
        const u32 unit = act ? qu[idx] : 0u;
        const u64 q = inv64(p);
        const D2 one = m2_one(p);
        // one after the other: fewer registers live at once, so the
        // 512-thread tiles fit 64 registers (two CTAs, 32 warps per SM);
        // the joint loop has three independent products per step
        D2 s, c;
        if (JOINT) {
            both_digits(p, q, one, s, c);
        } else {
            s = wieferich_digits<false>(p, q, one);
            c = wss_digits(p, q, one);
        }
        u64 sum = 0;
        if (act) {
            sum = (s.d1 & 0xffffffffull) + (c.d1 & 0xffffffffull);
            int rem, quot_w, res, quot_s;
            const bool hw = wieferich_classify(p, s, rem, quot_w);
            const bool hs = wss_classify(p, c, res, quot_s);
            if (hw) emit_batch_hit(a, unit, p, 1093, rem, quot_w);  // as the wieferich kernel would
            if (hs) emit_batch_hit(a, unit, p, res, 0, quot_s);     // as the wallsunsun kernel would
        }
        // one atomic a batch when its PRPs are of one unit
        const u32 live = __ballot_sync(0xffffffffu, act);
        const u32 unit0 = __shfl_sync(0xffffffffu, unit, __ffs((int)live) - 1);
        if (__all_sync(0xffffffffu, !act || unit == unit0)) {
            sum = warp_sum(sum);
            if (lane == 0) {
                atomicAdd((unsigned long long *)&a.units[unit0].checksum, (unsigned long long)sum);
                atomicAdd((unsigned long long *)&a.units[unit0].prp_count, (unsigned long long)__popc(live));
            }
        } else if (act) {
            atomicAdd((unsigned long long *)&a.units[unit].checksum, (unsigned long long)sum);
            atomicAdd((unsigned long long *)&a.units[unit].prp_count, 1ull);
        }
    }
}

// Bitmap words of a unit's tiles: the largest power of two, up to the
// configuration's segment, that cuts `numbers` (what is left of the launch
// from this unit on) into kTileRounds tiles for each of `slots` resident CTAs.
#ifndef WW_TILE_ROUNDS
#define WW_TILE_ROUNDS 2
#endif
constexpr double kTileRounds = WW_TILE_ROUNDS;
inline u32 tile_words(double numbers, int slots, u32 seg_words) {
    u32 w = seg_words;
    while (w > (u32)kTileMinWords && 64.0 * w * kTileRounds * slots > numbers) w /= 2;
    return w;
}

template <class Cfg>
constexpr size_t batch_smem_bytes() {
    return (size_t)Cfg::kWarps * Cfg::kPrpCap * 12 + (size_t)Cfg::kWords * 4 +
           (size_t)Cfg::kWarps * Cfg::kCandCap * 4;
}

// Hand out the next tile.  Batch: the global queue head over the static
// tile table.  Serving: the first of the launch's shares with tiles left,
// through that share's own cursor.  The host cuts the shares to the step's
// size, so a step hands out exactly those tiles, whichever CTAs come first;
// the loop is bounded by the number of shares, so an exhausted step ends the
// kernel instead of spinning.
template <bool SERVE>
__device__ __forceinline__ bool next_tile(const BatchArgs &a, u32 &unit, u64 &tile) {
    if constexpr (!SERVE) {
        const u64 t = atomicAdd((unsigned long long *)a.next_tile, 1ull);
        if (t >= a.n_tiles) return false;
        u32 lo = 0, hi = a.n_units;  // last k with tile_first[k] <= t
        while (hi - lo > 1) {
            const u32 mid = (lo + hi) >> 1;
            if (a.tile_first[mid] <= t) lo = mid; else hi = mid;
        }
        unit = lo;
        tile = t - a.tile_first[lo];
        return true;
    } else {
        for (u32 i = 0; i < a.n_shares; ++i) {
            StepShare &sh = a.shares[i];
            // the cursor is read past L1 (other CTAs move it); a stale value
            // only costs an atomic that finds the share exhausted
            if (*(volatile u64 *)&sh.next >= sh.end) continue;
            const u64 t = atomicAdd((unsigned long long *)&sh.next, 1ull);
            if (t < sh.end) {
                unit = sh.unit;
                tile = t;
                return true;
            }
        }
        return false;
    }
}

template <class Cfg, bool SERVE>
__global__ void __launch_bounds__(Cfg::kThreads, Cfg::kMinBlocks) k_tiles(BatchArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr size_t kPrps = (size_t)Cfg::kWarps * Cfg::kPrpCap;
    u64(*prpq)[Cfg::kPrpCap] = reinterpret_cast<u64(*)[Cfg::kPrpCap]>(smem);
    u32 *bitmap = reinterpret_cast<u32 *>(smem + kPrps * 8);
    u32(*candq)[Cfg::kCandCap] = reinterpret_cast<u32(*)[Cfg::kCandCap]>(smem + kPrps * 8 + Cfg::kWords * 4);
    u32(*unitq)[Cfg::kPrpCap] = reinterpret_cast<u32(*)[Cfg::kPrpCap]>(
        smem + kPrps * 8 + Cfg::kWords * 4 + (size_t)Cfg::kWarps * Cfg::kCandCap * 4);
    __shared__ u64 s_lo, s_hi;
    __shared__ u32 s_unit, s_chunk, s_ok, s_words;
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    u32 *cq = candq[warp];
    u64 *pq = prpq[warp];
    u32 *uq = unitq[warp];
    int pn = 0;  // PRPs in the warp's queue, kept from tile to tile

    for (;;) {
        if (threadIdx.x == 0) {
            u32 k = 0;
            u64 t = 0;
            s_chunk = 0;
            s_ok = next_tile<SERVE>(a, k, t) ? 1u : 0u;
            if (s_ok) {
                const UnitState &u = a.units[k];
                const u64 numbers = 64ull * (u64)u.words;
                const u64 tlo = u.start + t * numbers;
                const u64 room = u.end - tlo;
                s_unit = k;
                s_words = u.words;
                s_lo = tlo;
                s_hi = room > numbers ? tlo + numbers : u.end;
            }
        }
        __syncthreads();
        if (!s_ok) break;
        const u64 lo = s_lo, hi = s_hi;
        const u32 unit = s_unit;
        const int words = (int)s_words;
        const int chunk_words = min(32, words / Cfg::kWarps);  // a warp's share at a time

        // ---- pre-sieve 3..113 over [lo, hi): bit j of the tile is b0 + 2j + 1
        const u64 b0 = lo & ~1ull;
        const u64 span = hi - b0;
        const u64 odd = 32ull * (u64)words;
        const u64 nvalid = span / 2 < odd ? span / 2 : odd;
        const int wpt = (words + Cfg::kThreads - 1) / Cfg::kThreads;
        const int w0 = threadIdx.x * wpt;
        if (w0 < words) {
            const int w1 = min(w0 + wpt, words);
            const u64 n0 = b0 + 64ull * (u64)w0 + 1;
#define WW_J0(R) u32 j##R = first_hit<R>(n0);
            WW_FOR_SMALL_PRIMES(WW_J0)
#undef WW_J0
#pragma unroll 2
            for (int w = w0; w < w1; ++w) {
                u32 m = 0;
#define WW_MASK(R) m |= prime_mask<R>(j##R); step_hit<R>(j##R);
                WW_FOR_SMALL_PRIMES(WW_MASK)
#undef WW_MASK
                const u64 first = (u64)w * 32;
                if (first + 32 > nvalid) {
                    const u64 keep = nvalid > first ? nvalid - first : 0;
                    m |= ~((1u << keep) - 1u);
                }
                bitmap[w] = m;
            }
        }
        __syncthreads();

        // ---- deep sieve 113 < r < 2^WW_DEEP_BITS, sparing possible pseudoprimes
        const u64 nbase = b0 + 1;
        deep_mark(nbase, (u32)nvalid, bitmap, threadIdx.x, Cfg::kThreads, a.deep,
                  a.deep_n[__ffs(words) - __ffs(kTileMinWords)], min(words / 8, kDeepWarpPrimes));
        __syncthreads();

        // ---- chunks of 32 words (or fewer), taken dynamically by the warps
        int cn = 0;
        // one PRP test per lane; passing numbers go to the warp's PRP queue,
        // which feeds the Wieferich + WSS batches
        auto sprp_step = [&](u32 j, bool act) {
            const u64 n = nbase + 2ull * j;
            u64 q = 0;
            const bool pass = prp_test_warp(n, act, q);
            const u32 ballot = __ballot_sync(0xffffffffu, pass);
            const u32 rank = __popc(ballot & ((1u << lane) - 1u));
            if (pass) {
                pq[pn + rank] = n;
                uq[pn + rank] = unit;
            }
            if (a.units[unit].prp_out && ballot) {  // the range's PRP buffer (serving)
                u64 base = 0;
                if (lane == 0)
                    base = atomicAdd((unsigned long long *)&a.units[unit].prp_written,
                                     (unsigned long long)__popc(ballot));
                base = __shfl_sync(0xffffffffu, base, 0);
                if (pass) {
                    if (base + rank < a.units[unit].prp_cap) a.units[unit].prp_out[base + rank] = n;
                    else atomicOr(a.overflow, 1u);
                }
            }
            pn += __popc(ballot);
            __syncwarp();
            while (pn >= 32 * Cfg::kPpt) {
                pn -= 32 * Cfg::kPpt;
                test_batch<Cfg::kPpt, Cfg::kJoint>(pq + pn, uq + pn, 32 * Cfg::kPpt, a);
                __syncwarp();
            }
        };
        for (;;) {
            u32 chunk = 0;
            if (lane == 0) chunk = atomicAdd(&s_chunk, 1u);
            chunk = __shfl_sync(0xffffffffu, chunk, 0);
            const bool more = (int)chunk * chunk_words < words;
            if (more) {
                const int w = chunk * chunk_words + lane;
                u32 cand = lane < chunk_words ? ~bitmap[w] : 0u;
                const int c = __popc(cand);
                int incl = c;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int t = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += t;
                }
                const int total = __shfl_sync(0xffffffffu, incl, 31);
                int pos = cn + incl - c;
                while (cand) {
                    const int b = __ffs(cand) - 1;
                    cq[pos++] = (u32)(w * 32 + b);
                    cand &= cand - 1;
                }
                cn += total;
                __syncwarp();
            }
            // SPRP 32 candidates at a time; the last partial batch once the bitmap is done
            while (cn >= 32 || (!more && cn > 0)) {
                const int take = cn >= 32 ? 32 : cn;
                cn -= take;
                const bool act = lane < take;
                const u32 j = act ? cq[cn + lane] : 0u;
                __syncwarp();
                sprp_step(j, act);
            }
            if (!more) break;
        }
        __syncthreads();
        // some of the tile's PRPs may still wait in the warps' queues: the
        // count is read only after the launch, which empties them
        if (threadIdx.x == 0) {
            __threadfence();
            atomicAdd((unsigned long long *)&a.units[unit].tiles_done, 1ull);
        }
    }
    if (pn > 0) test_batch<Cfg::kPpt, Cfg::kJoint>(pq, uq, pn, a);
}

}  // namespace ww
