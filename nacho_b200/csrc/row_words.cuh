// The rows of a CSR matrix as bitmap words: for every 32 neighbouring columns of which a row stores any, one item
// {number of the word, bits of its columns}. The rows of a graph are clustered, so a product that only asks which columns
// there are (the symbolic pass of SpGEMM) walks half as many items as entries
// (R-MAT graphs of 50000 to 65536 vertices: 2.0 entries per item, weighted by how often a row is selected), and no two
// items of a row lie in one word.
#pragma once

#include "merge_common.cuh"

namespace nb200 {

// Items of row r: items[rp[r]] .. items[rp[r + 1] - 1], in the order of their columns.
struct RowWords {
    uint2 *items = nullptr;
    int32_t *rp = nullptr;
};

constexpr int WORDS_NT = 256, WORDS_TILE = WORDS_NT * 8;  // entries of a CTA: eight groups of 32 per warp

// Scratch of the three kernels below for a matrix of `nnz` entries.
struct RowWordsScratch {
    RowWords out;
    uint32_t *starts;   // bit p: entry p is the first of its row
    uint64_t *state;    // look-back words
    uint2 *groups;      // per 32 entries: items before them, and which of them begin an item
    static int tiles(int64_t nnz) { return (int)((nnz + WORDS_TILE) / WORDS_TILE); }  // position nnz has a group too
    template <typename C>
    static RowWordsScratch carve(C &c, int64_t rows, int64_t nnz, size_t *clear_from, size_t *clear_bytes) {
        RowWordsScratch s;
        *clear_from = c.used();
        s.starts = c.template take<uint32_t>((size_t)tiles(nnz) * (WORDS_TILE / 32) + 1);
        s.state = c.template take<uint64_t>((size_t)tiles(nnz) + 1);
        *clear_bytes = c.used() - *clear_from;
        s.out.items = c.template take<uint2>((size_t)nnz);
        s.out.rp = c.template take<int32_t>((size_t)rows + 1);
        s.groups = c.template take<uint2>((size_t)tiles(nnz) * (WORDS_TILE / 32));
        return s;
    }
};

static __global__ void __launch_bounds__(256) k_words_starts(const int32_t *rp, int32_t rows, uint32_t *starts) {
    wait_for_previous();
    trigger_dependents();
    const int64_t r = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (r >= rows) return;
    const int32_t base = ld_late(rp), lo = ld_late(rp + r) - base, hi = ld_late(rp + r + 1) - base;
    if (lo < hi) atomicOr(starts + (lo >> 5), 1u << (lo & 31));
}

// Entry p begins an item where its row begins or its word differs from that of entry p - 1. Lane = entry; the bits of an
// item are collected by a segmented scan within 32 entries, and what runs over into the next 32 is added there. The
// number of items before a CTA comes from the bounded look-back.
static __global__ void __launch_bounds__(WORDS_NT) k_words_build(const int32_t *rp, const int32_t *col, int32_t nnz, const uint32_t *starts, uint2 *groups,
                                                                uint2 *items, uint64_t *state, FusedCtl *ctl) {
    constexpr int G = WORDS_TILE / WORDS_NT;
    __shared__ int s_warp[WORDS_NT / 32];
    __shared__ long long s_base;
    wait_for_previous();
    trigger_dependents();
    const int t = blockIdx.x, lane = lane_id(), wid = warp_id();  // CTAs are dispatched in index order; waits on earlier tiles are bounded
    const int64_t p0 = (int64_t)t * WORDS_TILE + wid * 32 * G;
    col += ld_late(rp);
    int32_t c[G + 1];
    uint32_t start[G + 1];
#pragma unroll
    for (int g = 0; g <= G; ++g) {
        const int64_t p = p0 + 32 * g + lane;
        c[g] = p < nnz ? ld_late(col + p) : -1;
        start[g] = ld_late(starts + (p0 >> 5) + g);
    }
    int32_t last = p0 > 0 && p0 <= nnz ? ld_late(col + p0 - 1) : -1;  // the column in front of the group
    uint32_t heads[G + 1], bits[G + 1];
    int mine = 0;
#pragma unroll
    for (int g = 0; g <= G; ++g) {
        const bool there = p0 + 32 * g + lane < nnz;
        int32_t before = __shfl_up_sync(FULL_MASK, c[g], 1);
        if (lane == 0) before = last;
        last = __shfl_sync(FULL_MASK, c[g], 31);
        heads[g] = __ballot_sync(FULL_MASK, there && (((start[g] >> lane) & 1u) || (c[g] >> 5) != (before >> 5)));
        const uint32_t later = lane < 31 ? heads[g] >> (lane + 1) : 0u;
        const int end = later ? lane + __ffs((int)later) : 32;  // first lane of the next item
        uint32_t v = there ? 1u << (c[g] & 31) : 0u;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t w = __shfl_down_sync(FULL_MASK, v, d);
            if (lane + d < end) v |= w;
        }
        bits[g] = v;
        if (g < G) mine += __popc(heads[g]);
    }
    if (lane == 0) s_warp[wid] = mine;
    __syncthreads();
    int before = 0, total = 0;
#pragma unroll
    for (int w = 0; w < WORDS_NT / 32; ++w) {
        before += w < wid ? s_warp[w] : 0;
        total += s_warp[w];
    }
    if (wid == 0) {
        const int64_t b = lookback_exclusive(state, t, total, &ctl->status);
        if (lane == 0) s_base = b;
    }
    __syncthreads();
    if (s_base < 0) return;  // a bounded wait gave up: k_words_rp leaves every row empty, and the call reports it
    uint32_t run = (uint32_t)s_base + (uint32_t)before;
#pragma unroll
    for (int g = 0; g < G; ++g) {
        const uint32_t over = __shfl_sync(FULL_MASK, bits[g + 1], 0);  // what lies before the first head of the next group
        const bool is_last = heads[g] >> lane == 1u;
        const uint32_t v = bits[g] | (is_last && !(heads[g + 1] & 1u) ? over : 0u);
        if ((heads[g] >> lane) & 1u) items[run + __popc(heads[g] & ((1u << lane) - 1u))] = make_uint2((uint32_t)c[g] >> 5, v);
        if (lane == 0) groups[(p0 >> 5) + g] = make_uint2(run, heads[g]);
        run += __popc(heads[g]);
    }
}

static __global__ void __launch_bounds__(256) k_words_rp(const int32_t *rp, int32_t rows, const uint2 *groups, const FusedCtl *ctl, int32_t *item_rp) {
    trigger_dependents();  // k_words_build has begun, so everything in front of these kernels is complete
    wait_for_previous();
    const int64_t r = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (r > rows) return;
    const int32_t p = ld_late(rp + r) - ld_late(rp);
    const uint2 g = ld_late(groups + (p >> 5));
    item_rp[r] = ctl->status.error != 0 ? 0 : (int32_t)(g.x + __popc(g.y & ((1u << (p & 31)) - 1u)));
}

// Queues the three kernels; what carve() calls clear must be zero. A give-up of the look-back goes to ctl->status.
inline cudaError_t build_row_words(const int32_t *rp, const int32_t *col, int32_t rows, int32_t nnz, const RowWordsScratch &s, FusedCtl *ctl, cudaStream_t stream) {
    cudaError_t e;
    {
        LaunchScope scope("row_words_starts", stream);
        e = launch_overlapped(k_words_starts, dim3((unsigned)(((int64_t)rows + 255) / 256)), dim3(256), 0, stream, rp, rows, s.starts);
    }
    if (e == cudaSuccess) {
        LaunchScope scope("row_words_build", stream);
        e = launch_overlapped(k_words_build, dim3(RowWordsScratch::tiles(nnz)), dim3(WORDS_NT), 0, stream, rp, col, nnz, s.starts, s.groups, s.out.items, s.state, ctl);
    }
    if (e == cudaSuccess) {
        LaunchScope scope("row_words_rp", stream);
        e = launch_overlapped(k_words_rp, dim3((unsigned)(((int64_t)rows + 1 + 255) / 256)), dim3(256), 0, stream, rp, rows, s.groups, ctl, s.out.rp);
    }
    return e;
}

}  // namespace nb200
