// CTA-level building blocks shared by the kernels: warp and CTA scans, the k-ary search used
// for partitioning, and the bounded look-back of the single-pass scans.
#pragma once

#include "common.cuh"

namespace nb200 {

constexpr unsigned FULL_MASK = 0xffffffffu;

// ---- warp scans -----------------------------------------------------------------------

__device__ __forceinline__ int warp_incl_sum(int v) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int n = __shfl_up_sync(FULL_MASK, v, o);
        if (lane_id() >= o) v += n;
    }
    return v;
}

__device__ __forceinline__ unsigned warp_incl_max(unsigned v) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        unsigned n = __shfl_up_sync(FULL_MASK, v, o);
        if (lane_id() >= o) v = max(v, n);
    }
    return v;
}

// Exclusive sum over a CTA of NT threads; `total` receives their sum. `tmp` is >= 33
// ints of shared memory; the function syncs before reusing it, so calls may follow one another.
template <int NT>
__device__ __forceinline__ int block_excl_sum(int v, int *tmp, int &total) {
    constexpr int NW = NT / 32;
    int incl = warp_incl_sum(v);
    __syncthreads();
    if (lane_id() == 31) tmp[warp_id()] = incl;
    __syncthreads();
    if (warp_id() == 0) {
        int w = lane_id() < NW ? tmp[lane_id()] : 0;
        int wi = warp_incl_sum(w);
        if (lane_id() < NW) tmp[lane_id()] = wi - w;
        if (lane_id() == NW - 1) tmp[32] = wi;
    }
    __syncthreads();
    total = tmp[32];
    return tmp[warp_id()] + incl - v;
}

// Two exclusive sums at once (va, vb) over a CTA of NT threads; `ta` / `tb` receive the totals.
// `tmp` is >= 66 ints of shared memory.
template <int NT>
__device__ __forceinline__ void block_excl_sum2(int va, int vb, int *tmp, int &ea, int &eb, int &ta, int &tb) {
    constexpr int NW = NT / 32;
    const int ia = warp_incl_sum(va), ib = warp_incl_sum(vb);
    __syncthreads();
    if (lane_id() == 31) {
        tmp[warp_id()] = ia;
        tmp[33 + warp_id()] = ib;
    }
    __syncthreads();
    if (warp_id() == 0) {
        const int wa = lane_id() < NW ? tmp[lane_id()] : 0, wb = lane_id() < NW ? tmp[33 + lane_id()] : 0;
        const int sa = warp_incl_sum(wa), sb = warp_incl_sum(wb);
        if (lane_id() < NW) {
            tmp[lane_id()] = sa - wa;
            tmp[33 + lane_id()] = sb - wb;
        }
        if (lane_id() == NW - 1) {
            tmp[32] = sa;
            tmp[65] = sb;
        }
    }
    __syncthreads();
    ta = tmp[32];
    tb = tmp[65];
    ea = tmp[warp_id()] + ia - va;
    eb = tmp[33 + warp_id()] + ib - vb;
}

// ---- k-ary search -----------------------------------------------------------------------

// Number of leading true values of a monotone pred over [lo, hi), returned as lo + count; G
// neighbouring lanes search together, each group of a warp on its own range. All 32 lanes call this
// together; a group that is done idles until the warp's last one is.
template <int G, typename Pred>
__device__ __forceinline__ uint32_t group_count_true(uint32_t lo, uint32_t hi, Pred pred) {
    const int in_group = lane_id() & (G - 1), shift = lane_id() & ~(G - 1);
    while (__any_sync(FULL_MASK, lo < hi)) {
        const uint32_t step = lo < hi ? (hi - lo + G - 1) / G : 0u;
        const uint32_t p = lo + (in_group + 1) * step - 1;
        const bool ok = step > 0 && p < hi && pred(p);
        const unsigned votes = __ballot_sync(FULL_MASK, ok);
        const int c = __popc(G == 32 ? votes : (votes >> shift) & ((1u << (G & 31)) - 1u));
        if (step > 0) {
            lo += c * step;
            hi = min(hi, lo + step - 1);
        }
    }
    return lo;
}

// ---- bounded decoupled look-back ----------------------------------------------------------

// Chained scan across CTAs in one pass: every tile publishes its own count ("aggregate") as
// soon as it knows it, then walks back over its predecessors' words, 32 at a time, adding
// aggregates until it meets a tile that already knows its inclusive prefix. A word carries a
// 2-bit state and a 62-bit value and is written with one 8-byte store, so no fence is needed
// between the two. A tile waits only on tiles with lower numbers, so tiles must be numbered in
// an order in which their CTAs start: the CTA index (the hardware hands CTAs out in index
// order, the numbering the kernels here use) or an atomic ticket taken at CTA start.
//
// Every wait is bounded: after LOOKBACK_POLL_LIMIT polls the walk gives up, records the tile in `status` and
// returns -1; the caller then skips its writes. A give-up is never lost, however late it comes: the waiter puts
// LB_FAILED in the place of the word it misses (unless that word has come after all), a word is first published only
// in the place of zero, and so no tile behind the missing word gets a base, the last one among them, which is the
// one that publishes the total.
constexpr uint64_t LB_AGGREGATE = 1ull << 62;
constexpr uint64_t LB_PREFIX = 2ull << 62;
constexpr uint64_t LB_FAILED = 3ull << 62;
constexpr uint64_t LB_VALUE_MASK = (1ull << 62) - 1;
constexpr int LOOKBACK_POLL_LIMIT = 1 << 22;
constexpr int ERR_LOOKBACK_TIMEOUT = 1;

__device__ __forceinline__ uint64_t ld_relaxed_gpu(const volatile uint64_t *p) {
    uint64_t v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void st_relaxed_gpu(volatile uint64_t *p, uint64_t v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

__device__ __forceinline__ int ld_relaxed_gpu_i32(const int *p) {
    int v;
    asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Writes `v` into a word that is still zero; returns what the word held.
__device__ __forceinline__ uint64_t set_if_zero(volatile uint64_t *word, uint64_t v) {
    return atomicCAS(reinterpret_cast<unsigned long long *>(const_cast<uint64_t *>(word)), 0ull, (unsigned long long)v);
}

// Sum of the counts of tiles [0, t), read off the tile words of the predecessors, 32 at a time
// from the nearest one backwards; publishes nothing. A round is complete once every word up to
// the nearest tile that already knows its prefix is published (the words beyond it are not
// needed). Returns -1 (and records the tile in `status`) if a bounded wait gives up, here or on the way. Called by
// all 32 lanes of one warp, t > 0.
__device__ __forceinline__ int64_t lookback_predecessors(volatile uint64_t *state, int t, DeviceStatus *status) {
    int64_t exclusive = 0;
    for (int pos = t - 1;; pos -= 32) {  // lane l looks at tile pos - l
        const int idx = pos - lane_id();
        uint64_t s;
        unsigned prefixes, need;
        for (int polls = 0;; ++polls) {
            s = idx >= 0 ? ld_relaxed_gpu(state + idx) : LB_PREFIX;  // before tile 0: an empty prefix
            prefixes = __ballot_sync(FULL_MASK, (s >> 62) == 2);
            const unsigned published = __ballot_sync(FULL_MASK, (s >> 62) != 0);
            need = prefixes ? FULL_MASK >> (32 - __ffs(prefixes)) : FULL_MASK;
            if ((published & need) == need) break;
            if (polls >= LOOKBACK_POLL_LIMIT) {
                if (s == 0 && ((need >> lane_id()) & 1u)) {
                    s = set_if_zero(state + idx, LB_FAILED);
                    if (s == 0) s = LB_FAILED;
                }
                prefixes = __ballot_sync(FULL_MASK, (s >> 62) == 2);
                need = prefixes ? FULL_MASK >> (32 - __ffs(prefixes)) : FULL_MASK;
                break;
            }
            __nanosleep(32);
        }
        if (__ballot_sync(FULL_MASK, s >= LB_FAILED) & need) {
            if (lane_id() == 0 && atomicCAS(&status->error, 0, ERR_LOOKBACK_TIMEOUT) == 0) status->detail = t;
            return -1;
        }
        long long v = (need >> lane_id()) & 1u ? (long long)(s & LB_VALUE_MASK) : 0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL_MASK, v, o);
        exclusive += v;
        if (prefixes) return exclusive;
    }
}

// Publishes the tile's count, walks back, publishes the inclusive prefix. Returns the sum of the
// counts of tiles [0, t), or -1 after a give-up. Called by all 32 lanes of one warp.
__device__ __forceinline__ int64_t lookback_exclusive(volatile uint64_t *state, int t, int64_t aggregate,
                                                      DeviceStatus *status) {
    uint64_t before = 0;  // not zero: some tile has given up on this one
    if (lane_id() == 0) before = set_if_zero(state + t, (t == 0 ? LB_PREFIX : LB_AGGREGATE) | (uint64_t)aggregate);
    if (t == 0) return 0;
    const int64_t exclusive = lookback_predecessors(state, t, status);
    if (exclusive < 0) __threadfence();  // the error word goes out before the word that tells the successors
    if (lane_id() == 0 && before == 0) st_relaxed_gpu(state + t, exclusive < 0 ? LB_FAILED : LB_PREFIX | (uint64_t)(exclusive + aggregate));
    return exclusive;
}

}  // namespace nb200
