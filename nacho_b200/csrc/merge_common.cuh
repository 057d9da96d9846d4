// Definitions shared by the merge kernels (CSR element-wise, COO3 / CSF3 tensor add): the set
// operation and launch-mode enums, the control block of single-pass launches, and the small
// scan kernel that sits between the two passes of the count -> scan -> fill route.
#pragma once

#include "block_utils.cuh"
#include "common.cuh"

namespace nb200 {

enum SetOp { OP_UNION = 0, OP_INTERSECT = 1 };

// What one launch of the tile kernel does.
//   MODE_COUNT  count the tile's result entries (first pass of the two-pass scheme)
//   MODE_FILL   write the result; the tile's output base comes from the scanned counts
//   MODE_FUSED  single pass: count, obtain the output base (below), write
//   MODE_REDUCE no result tensor: the products of the entries both operands hold are summed
//               (inner product); the tile's partial sum is added to a double in the control block
enum Mode { MODE_COUNT = 0, MODE_FILL = 1, MODE_FUSED = 2, MODE_REDUCE = 3 };

// Device-side control block of a fused launch.
struct FusedCtl {
    int hollow;           // offsets mode: a result entry stands for empty ranges only
    DeviceStatus status;  // bounded-wait failures
    long long total;      // result entries, written by whoever has all counts: the last of few tiles, else CTA 0 (MODE_REDUCE: the bits of a double, the running sum)
};

// ------------------------------------------------------------------- output bases ----
//
// The output base of a tile is the number of results of all earlier tiles, some 600 of which may still be
// at work. One warp -- CTA 0 of the launch, the first to be dispatched -- reads the counts in order and
// hands every tile its base in a word that only this tile polls. Letting tiles read
// their predecessors' words instead loses to the polling itself: hundreds of tiles reading the lines that
// hundreds of others are about to write. Measured at 64 M entries per operand, whole kernel: walking the
// counts back 32 at a time 609 us, per-group sums that every tile reads in one round 519 us, this 470 us.
// Up to DIRECT_TILES tiles, when everything is resident and little is polled, a tile adds up the counts
// before it itself, one hop less.
//
// Whoever publishes the length (CTA 0, or the last tile) has read every count, and reads the status behind a fence
// after that. A tile that gives up writes the status, and behind a fence looks at the word it misses once more: it is
// still missing only if the publisher's look at the status is yet to come. So a length goes out as good only if
// every tile has, or will find, its base.
constexpr int DIRECT_TILES = 128;

// Words of one launch, zero at the start: a count and a base per tile.
struct TileWords {
    uint64_t *count, *base;
    __host__ __device__ static constexpr size_t needed(size_t num_tiles) { return 2 * num_tiles; }
    __host__ __device__ static TileWords at(uint64_t *p, int num_tiles) { return TileWords{p, p + num_tiles}; }
};

__device__ __forceinline__ void publish_count(const TileWords &words, const int t, const int count) {
    st_relaxed_gpu(words.count + t, LB_AGGREGATE | (uint64_t)count);
}

// Runs in one warp. Publishes the base of every tile; returns the number of results, or -1 after
// `poll_limit` rounds without a new count (the tiles that wait are told, and the error word is set). The
// next round's load is on its way while a round is summed up: a round takes one trip to L2 and no more.
__device__ __forceinline__ int64_t scan_tile_counts(const TileWords &words, const int num_tiles, DeviceStatus *status, const int poll_limit) {
    const int lane = lane_id();
    int64_t run = 0;
    int idle = 0;
    uint64_t w = lane < num_tiles ? ld_relaxed_gpu(words.count + lane) : 0;
    for (int pos = 0;;) {
        const unsigned missing = __ballot_sync(FULL_MASK, (w >> 62) == 0);
        const int n = missing ? __ffs(missing) - 1 : 32;
        const int next = pos + n;
        const uint64_t w_next = next + lane < num_tiles ? ld_relaxed_gpu(words.count + next + lane) : 0;
        if (n > 0) {
            const int v = lane < n ? (int)(w & LB_VALUE_MASK) : 0;
            const int incl = warp_incl_sum(v);
            if (lane < n) st_relaxed_gpu(words.base + pos + lane, LB_PREFIX | (uint64_t)(run + incl - v));
            run += __shfl_sync(FULL_MASK, incl, 31);
            idle = 0;
            if (next >= num_tiles) {
                __syncwarp();  // the bases of all lanes lie before the fence of the one that publishes the length
                return run;
            }
        } else if (++idle > poll_limit) {
            if (lane == 0 && atomicCAS(&status->error, 0, ERR_LOOKBACK_TIMEOUT) == 0) status->detail = pos;
            __threadfence();
            for (int i = pos + lane; i < num_tiles; i += 32) st_relaxed_gpu(words.base + i, LB_FAILED);
            return -1;
        }
        pos = next;
        w = w_next;
    }
}

// Output base of tile t, or -1 after a give-up. Called by all 32 lanes of one warp.
__device__ __forceinline__ int64_t tile_base(const TileWords &words, const int t, const int num_tiles, DeviceStatus *status, const int poll_limit) {
    if (t == 0) return 0;
    auto record = [&]() {
        if (lane_id() == 0 && atomicCAS(&status->error, 0, ERR_LOOKBACK_TIMEOUT) == 0) status->detail = t;
        __syncwarp();
        __threadfence();
    };
    uint64_t w = LB_AGGREGATE;  // lanes past the last predecessor add nothing
    if (num_tiles <= DIRECT_TILES) {
        int sum = 0;
        for (int first = 0; first < t; first += 32) {
            const int at = first + lane_id();
            w = LB_AGGREGATE;
            for (int polls = 0;; ++polls) {
                if (at < t) w = ld_relaxed_gpu(words.count + at);
                if (__all_sync(FULL_MASK, (w >> 62) != 0)) break;
                if (polls >= poll_limit) {
                    record();
                    if (at < t) w = ld_relaxed_gpu(words.count + at);
                    if (__all_sync(FULL_MASK, (w >> 62) != 0)) break;
                    return -1;
                }
            }
            sum += (int)(w & LB_VALUE_MASK);
        }
        __syncwarp();  // every lane's look at the counts lies before the fence of the one that publishes the length
        return __reduce_add_sync(FULL_MASK, sum);
    }
    for (int polls = 0;; ++polls) {
        if (lane_id() == 0) w = ld_relaxed_gpu(words.base + t);
        w = __shfl_sync(FULL_MASK, w, 0);
        if (w >> 62) break;
        if (polls >= poll_limit) {
            record();
            if (lane_id() == 0) w = ld_relaxed_gpu(words.base + t);
            w = __shfl_sync(FULL_MASK, w, 0);
            break;
        }
        __nanosleep(64);
    }
    return (w >> 62) == 2 ? (int64_t)(w & LB_VALUE_MASK) : -1;
}

// Exclusive prefix of the per-tile counts, in place, by one CTA; the grand total goes to
// *total_out (64-bit so that the host can detect int32 overflow).
static __global__ void __launch_bounds__(1024) k_scan_tiles(int32_t *counts, int32_t n, int64_t *total_out) {
    __shared__ long long warp_sums[33];
    __shared__ long long carry_s;
    if (threadIdx.x == 0) carry_s = 0;
    __syncthreads();
    for (int base = 0; base < n; base += 1024) {
        const int i = base + threadIdx.x;
        const long long v = i < n ? counts[i] : 0;
        long long incl = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            long long nb = __shfl_up_sync(FULL_MASK, incl, o);
            if (lane_id() >= o) incl += nb;
        }
        if (lane_id() == 31) warp_sums[warp_id()] = incl;
        __syncthreads();
        if (warp_id() == 0) {
            long long w = warp_sums[lane_id()];
            long long wi = w;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                long long nb = __shfl_up_sync(FULL_MASK, wi, o);
                if (lane_id() >= o) wi += nb;
            }
            warp_sums[lane_id()] = wi - w;
            if (lane_id() == 31) warp_sums[32] = wi;
        }
        __syncthreads();
        const long long carry = carry_s;
        const long long excl = carry + warp_sums[warp_id()] + incl - v;
        if (i < n) counts[i] = (int32_t)min(excl, (long long)INT32_MAX);
        __syncthreads();
        if (threadIdx.x == 0) carry_s = carry + warp_sums[32];
        __syncthreads();
    }
    if (threadIdx.x == 0) *total_out = carry_s;
}

// Device-wide exclusive prefix of n int32 counts, in place, in one pass: 2048 counts per CTA,
// CTA totals chained by bounded look-back. `state` holds one zeroed 8-byte word per CTA and
// `ctl` is zeroed; the grand total lands in ctl->total. A give-up of a bounded wait is
// recorded in ctl->status and leaves the tail of the array unscanned.
constexpr int SCAN_NT = 256, SCAN_VT = 8;

static __global__ void __launch_bounds__(SCAN_NT) k_scan_lookback(int32_t *data, int32_t n, uint64_t *state_raw, FusedCtl *ctl) {
    __shared__ int scan_tmp[40];
    __shared__ long long s_base;
    volatile uint64_t *state = state_raw;
    const int tid = threadIdx.x;
    const int t = blockIdx.x;  // CTAs are dispatched in index order; waits on earlier tiles are bounded
    const int64_t p0 = ((int64_t)t * SCAN_NT + tid) * SCAN_VT;
    int v[SCAN_VT];
    int mine = 0;
#pragma unroll
    for (int q = 0; q < SCAN_VT; ++q) {
        v[q] = p0 + q < n ? data[p0 + q] : 0;
        mine += v[q];
    }
    int total;
    int run = block_excl_sum<SCAN_NT>(mine, scan_tmp, total);
    if (warp_id() == 0) {
        const int64_t b = lookback_exclusive(state, t, total, &ctl->status);
        if (lane_id() == 0) s_base = b;
    }
    __syncthreads();
    const long long base = s_base;
    if (base < 0) return;
    long long acc = base + run;
#pragma unroll
    for (int q = 0; q < SCAN_VT; ++q) {
        if (p0 + q < n) data[p0 + q] = (int32_t)min(acc, (long long)INT32_MAX);
        acc += v[q];
    }
    if (t == (int)gridDim.x - 1 && tid == SCAN_NT - 1) ctl->total = acc;
}

// The same scan out of place, for counts that turn into offsets: out[i] = sum of data[0 .. i), i = 0 .. n, and
// the total as a result word.
static __global__ void __launch_bounds__(SCAN_NT) k_scan_offsets(const int32_t *__restrict__ data, int32_t n, int32_t *__restrict__ out,
                                                                uint64_t *state, FusedCtl *ctl, unsigned long long *word) {
    __shared__ int scan_tmp[40];
    __shared__ long long s_base;
    const int tid = threadIdx.x, t = blockIdx.x;  // CTAs are dispatched in index order; waits on earlier tiles are bounded
    const int64_t p0 = ((int64_t)t * SCAN_NT + tid) * SCAN_VT;
    int v[SCAN_VT], mine = 0;
#pragma unroll
    for (int q = 0; q < SCAN_VT; ++q) {
        v[q] = p0 + q < n ? ld_nc(data + p0 + q) : 0;
        mine += v[q];
    }
    int total;
    const int run = block_excl_sum<SCAN_NT>(mine, scan_tmp, total);
    if (warp_id() == 0) {
        const int64_t b = lookback_exclusive(state, t, total, &ctl->status);
        if (lane_id() == 0) s_base = b;
    }
    __syncthreads();
    const bool last = t == (int)gridDim.x - 1;
    if (last && tid == 0) {
        if (s_base >= 0) ctl->total = s_base + total;
        publish_result_word(word, s_base < 0 || ld_relaxed_gpu_i32(&ctl->status.error) != 0 ? NB200_E_TIMEOUT : NB200_OK, s_base < 0 ? 0 : s_base + total);
    }
    if (s_base < 0) return;
    long long acc = s_base + run;
#pragma unroll
    for (int q = 0; q < SCAN_VT; ++q) {
        if (p0 + q <= n) out[p0 + q] = (int32_t)min(acc, (long long)INT32_MAX);
        acc += v[q];
    }
}

}  // namespace nb200
