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
    long long total;      // result entries, written by the last tile (MODE_REDUCE: the bits of a double, the running sum)
};

// ------------------------------------------------------------------- output bases ----
//
// The output base of a tile is the number of results of all earlier tiles, some 600 of which may still be at work. Every tile
// has a word: first its own count, then, once the tile has its base, the count of all results up to its end. A tile reads the
// words in front of its own, 32 in a trip to L2, back to the nearest one that holds such a sum: while 40 tiles end
// in a microsecond that is one to five trips away, and the words that are looked at first are those that come last. What this replaced,
// one CTA that read the counts in order and handed every tile its base, was two trips one after the other for every tile and handed out no more
// than 32 bases in one: 2.0 of the 13 us of a tile between the last count in front of it and its base (67 M entries per operand), 3.0 of
// the 13.4 us of a merge of 521 tiles, which all count at once. 410 -> 397 us a call of the former, 23.8 -> 22.3 of the latter, 16 M
// entries intersected 114 -> 110, 100 M coordinates per operand 1086 -> 1040. Several windows in flight (64, 96, 128 words: 397, 404, 406 us) cost more in
// registers than they save in trips.
//
// A word is {tag, 28 bits; state, 2 bits; value, 34 bits} and is only ever raised (atomicMax), so a word of an earlier call,
// whose tag is lower, counts as unpublished and needs no clearing. Tiles are numbered by CTA index, in which order CTAs start,
// so a tile waits only on CTAs that started before it.
//
// Every wait is bounded. Who gives up on a word puts "failed" in its place, by compare and swap with what it held: a count that comes
// later does not undo it, and one that came in between is used after all. A tile without a base marks its own word the same
// way, and so does one whose columns did not land. No tile behind a failed word gets a base, the last one among
// them, which reports the call's length: a length goes out only if every tile has, or will find, its base.

// Words of one launch, one per tile, with its tag (shifted into place; not zero). Words of lower tags may lie there.
struct TileWords {
    uint64_t *word;
    uint64_t tag;
    static constexpr int TAG_SHIFT = 36;
    __host__ __device__ static constexpr size_t needed(size_t num_tiles) { return num_tiles; }
    // Words that are zero, or of lower tags, at the start.
    __host__ __device__ static TileWords at(uint64_t *p, uint32_t tag = 1) { return TileWords{p, (uint64_t)tag << TAG_SHIFT}; }
};
constexpr uint64_t TW_COUNT = 1ull << 34, TW_SUM = 2ull << 34, TW_FAILED = 3ull << 34;

__device__ __forceinline__ void raise_word(const TileWords &words, const int t, const uint64_t state_and_value) {
    atomicMax(reinterpret_cast<unsigned long long *>(words.word + t), (unsigned long long)(words.tag | state_and_value));
}

// A tile's count, by one thread, as soon as it is known.
__device__ __forceinline__ void publish_count(const TileWords &words, const int t, const int count) {
    raise_word(words, t, (t == 0 ? TW_SUM : TW_COUNT) | (uint64_t)count);
}
// The tile has no count, and nobody behind it a base.
__device__ __forceinline__ void publish_failure(const TileWords &words, const int t) { raise_word(words, t, TW_FAILED); }

// Output base of tile t, which has published `count`, or -1 after a give-up, here or in front of it. Called by all 32 lanes of one warp.
__device__ __forceinline__ int64_t tile_base(const TileWords &words, const int t, const int count, DeviceStatus *status, const int poll_limit) {
    if (t == 0) return 0;
    const int lane = lane_id();
    const uint32_t tag = (uint32_t)(words.tag >> 32);  // the upper word with no state in it
    uint32_t sum = 0;                                  // two operands of up to 2^31 - 1 entries
    bool failed = false;
    int polls = 0;
    for (int at = t - 1 - lane;;) {  // lane l looks at tile t - 1 - l, then 32 further back each time
        uint64_t w = at >= 0 ? ld_relaxed_gpu(words.word + at) : words.tag | TW_SUM;  // before tile 0: an empty sum
        uint32_t state = ((uint32_t)(w >> 32) ^ tag) >> 2;  // 1 to 3; anything else: unpublished
        unsigned sums = __ballot_sync(FULL_MASK, state == 2u);
        unsigned need = sums ? sums ^ (sums - 1u) : FULL_MASK;  // up to the nearest sum
        const unsigned missing = __ballot_sync(FULL_MASK, state - 1u >= 3u) & need;
        if (missing) {
            if (++polls <= poll_limit) continue;
            if ((missing >> lane) & 1u) {  // gives up on what is missing, unless it has come after all
                const uint64_t now = atomicCAS(reinterpret_cast<unsigned long long *>(words.word + at), (unsigned long long)w, (unsigned long long)(words.tag | TW_FAILED));
                w = now == w ? words.tag | TW_FAILED : now;
                state = ((uint32_t)(w >> 32) ^ tag) >> 2;
            }
            sums = __ballot_sync(FULL_MASK, state == 2u);
            need = sums ? sums ^ (sums - 1u) : FULL_MASK;
        }
        failed = (__ballot_sync(FULL_MASK, state == 3u) & need) != 0u;
        if ((need >> lane) & 1u) sum += (uint32_t)w;
        if (sums || failed) break;
        at -= 32;
    }
    const int64_t base = failed ? -1 : (int64_t)__reduce_add_sync(FULL_MASK, sum);
    if (lane == 0) {
        if (failed) {
            if (atomicCAS(&status->error, 0, ERR_LOOKBACK_TIMEOUT) == 0) status->detail = t;
            publish_failure(words, t);
        } else {
            raise_word(words, t, TW_SUM | (uint64_t)(base + count));
        }
    }
    return base;
}

// ------------------------------------------------------------------------- tile cuts ----
//
// A merge whose call waits for its length is one launch, where it does not have too many tiles: they find their cuts themselves, with words of their own
// (acquire_tagged) in which nothing needs to be cleared but the control block of a later merge. The first tiles, those that are at work at once from
// the start (four CTAs on each of 148 SMs), search for both of their cuts before anything else. For all others a few CTAs in front of
// the tiles make the cuts, in order and faster than tiles end, and leave them in tagged words. A launch in front of the merge makes all cuts
// before the first tile begins; the other routes keep it (asynchronous calls, whose launches may be captured and run again; counts before a
// fill; a call profiled with 1, which is to tell the searches from the merge). us a call, with that launch and without: sums of 10900 entries per operand
// 15.6 and 14.9, 0.5 M 19.1 and 17.7, 3.3 M 44.2 and 40.4, 4.5 M in short rows 66.5 and 57.9; intersection of 16 M 88.5 and 83.5; three operands of 9 M 183 and
// 176; trees of 100 K 45.8 and 41.8. Coordinate lists have such CTAs nowhere: their probes, of up to six loads far apart, cannot keep up
// with the tiles (100 M entries per operand 1024 us with the launch, 1341 so), so they stay with RESIDENT tiles (inner product of 300 K entries 20.9 and 18.3).
constexpr int RESIDENT = 592;  // tiles at work at once
constexpr int CUTTERS = 32;    // CTAs that make cuts, where there are more tiles than that
struct OwnWords {
    FusedCtl *ctl = nullptr, *clear = nullptr;  // of this merge; of a later one
    TileWords words{nullptr, 0};
    uint64_t *cut = nullptr;  // four words a cut
    int cutters = 0;          // leading CTAs that make the cuts from first_cut() on
    __host__ __device__ int first_cut() const { return RESIDENT - CUTTERS; }
};
// `wanted` is withdrawn where the device has no room for the words: the call then has the launch for its cuts, whose scratch it holds anyway
// (and which asynchronous calls on the stream, that may be captured, find there).
inline int take_own_words(cudaStream_t stream, int num_tiles, bool *wanted, OwnWords *out) {
    static_assert(sizeof(FusedCtl) <= 8 * sizeof(uint64_t), "a control block takes a piece");
    if (!*wanted) return NB200_OK;
    const bool many = num_tiles > RESIDENT;
    Tagged block;
    const int st = acquire_tagged(stream, many ? 5 * (size_t)num_tiles + 4 : RESIDENT, &block);
    if (st == NB200_E_NOMEM) *wanted = false;
    if (st != NB200_OK) return *wanted ? st : NB200_OK;
    out->ctl = reinterpret_cast<FusedCtl *>(block.mine);
    out->clear = reinterpret_cast<FusedCtl *>(block.later);
    out->words = TileWords::at(block.words, block.tag);
    out->cut = block.words + num_tiles;
    out->cutters = many ? CUTTERS : 0;
    return NB200_OK;
}

// One thread. A word carries its tag and its part of the cut together, and what a tile reads with them lies behind its own wait_for_previous:
// nothing needs an order among these writes or beside others.
__device__ __forceinline__ void store_cut(const OwnWords &own, const int t, const int4 cut) {
    uint64_t *w = own.cut + 4 * (size_t)t;
    st_relaxed_gpu(w, own.words.tag | (uint32_t)cut.x);
    st_relaxed_gpu(w + 1, own.words.tag | (uint32_t)cut.y);
    st_relaxed_gpu(w + 2, own.words.tag | (uint32_t)cut.z);
}
// All lanes of a warp; every lane gets the cut. False after a give-up.
__device__ __forceinline__ bool await_cut(const OwnWords &own, const int t, const int poll_limit, int4 *cut) {
    const uint64_t *w = own.cut + 4 * (size_t)t + min(lane_id(), 2);
    uint64_t v = 0;
    for (int polls = 0;; ++polls) {
        v = ld_relaxed_gpu(w);
        if (__all_sync(FULL_MASK, (v ^ own.words.tag) >> TileWords::TAG_SHIFT == 0)) break;
        if (polls >= poll_limit) return false;
    }
    *cut = make_int4(__shfl_sync(FULL_MASK, (int)v, 0), __shfl_sync(FULL_MASK, (int)v, 1), __shfl_sync(FULL_MASK, (int)v, 2), 0);
    return true;
}
// One thread, without waiting: whether the cut is there.
__device__ __forceinline__ bool peek_cut(const OwnWords &own, const int t, int4 *cut) {
    const uint64_t *w = own.cut + 4 * (size_t)t;
    const uint64_t x = ld_relaxed_gpu(w), y = ld_relaxed_gpu(w + 1), z = ld_relaxed_gpu(w + 2);
    *cut = make_int4((int)x, (int)y, (int)z, 0);
    return (((x ^ own.words.tag) | (y ^ own.words.tag) | (z ^ own.words.tag)) >> TileWords::TAG_SHIFT) == 0;
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
