// Masked SpGEMM ("sssmm"): Z_ik = sum_j a_ij * b_jk * c_ik on the positions the mask C stores and
// at least one product reaches. The reference declares it as one fused kernel
// (compiler.cpp:150-153: Sum_j a_ij * b_jk * c_ik) and runs it through the same expand / sort /
// compress machinery as its SpGEMM (src/backend/stitch_and_generate_gpu.cpp:14-139), on the products
// that survive the three-way intersection.
//
// Here the mask drives the accumulation, so nothing outside it is ever formed, sorted or written:
//   k_sssmm_classify    how many products does a row have, and how wide (first to last column) and
//                       how long is its mask row? The row goes on one of six lists.
//   k_sssmm_bitmap      rows with many products, one CTA per row taken from a ticket: the mask row
//                       becomes a bitmap over its column span in shared memory plus, per 64-bit
//                       word, the count of set bits before it. A product tests one bit; a hit finds
//                       its position in the mask row as rank + popcount and adds
//                       (a_ij * b_jk) * c_ik -- the reference's expression, left to right -- to a
//                       shared-memory accumulator (rows whose mask row is too long for that, or
//                       whose span needs the whole shared memory, accumulate in global memory).
//                       Three list classes, by the shared memory a row needs.
//   k_sssmm_look_up     rows with a mask row of some dozens of positions, one warp per row: the other way round,
//                       the mask's columns are searched in the rows of B, sums in registers.
//   k_sssmm_search_*    rows with few products (one warp per row) and rows whose span exceeds the
//                       largest bitmap (one CTA per row): binary search of the product's column in
//                       the mask row, float atomics on the global accumulators.
//   k_sssmm_scan        exclusive scan of the "reached" flags (the result position of every mask position)
//                       and, in the same pass, the reached positions written there.
//   k_sssmm_compact     reached positions move to their result slot (column, value); the result's
//                       row offsets are the scanned flags at the mask's row starts.
// The sums are float32 atomics in arrival order, as the reference's compress is for every row.
#include <algorithm>

#include "block_utils.cuh"
#include "merge_common.cuh"

namespace nb200 {

namespace {

constexpr int LIGHT_P = 256;    // rows with fewer products than this are searched by one warp
constexpr int SEARCH_NT = 128;  // threads of a searching CTA
// lists: bitmap classes 0..2, wide rows (searched by a CTA), light rows (searched by a warp), rows whose mask
// positions are looked up in B
constexpr int LIST_WIDE = 3, LIST_LIGHT = 4, LIST_MASK = 5;
constexpr int MASK_UNIT = 8;    // entries of A's row that one warp looks the mask row up for: its searches are a chain of loads
                                // (R-MAT 15021 vertices: 83 us with 8, 89 with 16, 134 with 64)
constexpr int WARP_ENTRIES = 8; // entries of A's row one warp of a unit takes

// Work classes. A unit of work is a run of `unit` consecutive entries of one row of A (a row with
// more entries becomes several units, so a hub row spreads over the SMs), worked by one CTA of
// `nt` threads. The bitmap classes keep `words` 64-bit bitmap words and `entries` accumulators of
// the mask row in shared memory: bytes = 12 * words + 5 * entries (bitmap, ranks; sums, flags).
struct WorkClass {
    int words, entries, nt;
    __host__ __device__ constexpr int unit() const { return WARP_ENTRIES * (nt / 32); }
    constexpr size_t smem() const { return size_t(12) * words + size_t(5) * entries + 16; }
};
constexpr WorkClass CLASS[4] = {
    {1024, 2048, 256},    //  65536 columns of span, 22.5 KB: eight CTAs per SM
    {4096, 8192, 1024},   // 262144 columns, 88 KB: two CTAs per SM
    {16384, 0, 1024},     // 2^20 columns, 192 KB, sums in global memory: one CTA per SM
    {0, 0, SEARCH_NT},    // wider still: no bitmap, binary search
};

// Entries of A's row in a unit of a list (LIST_LIGHT has whole rows).
__device__ __forceinline__ int unit_of(int list) {
    return list == LIST_MASK ? MASK_UNIT : list == 0 ? CLASS[0].unit() : list == LIST_WIDE ? CLASS[LIST_WIDE].unit() : CLASS[1].unit();
}

struct CsrView {
    const int32_t *rp, *col;
    const float *val;
};

struct SssmmCtl {
    int count[8];   // units (light list: rows) on each list
    int ticket[8];  // next list position to hand out
};

// Rows of one CTA of the classification. A warp has the dependent loads of eight rows (A's columns, then B's offsets)
// in flight together, rows of more than LONG_ROW entries are left to the whole CTA, and a list's length is
// advanced once per CTA: with a warp per row, one row after the other, the chains of loads and 50021 atomics on
// six words took 39 us on a graph of 50021 vertices. A CTA's rows lie far apart: the hubs of a graph are often
// neighbours.
constexpr int ROWS_PER_WARP = 8, ROWS_PER_CTA = 8 * ROWS_PER_WARP, LONG_ROW = 128;

__global__ void __launch_bounds__(256) k_sssmm_classify(CsrView A, CsrView B, CsrView C, int32_t rows, int64_t list_cap,
                                                       int2 *__restrict__ units, int32_t *__restrict__ light,
                                                       SssmmCtl *__restrict__ ctl) {
    __shared__ int s_lo[ROWS_PER_CTA], s_hi[ROWS_PER_CTA], s_list[ROWS_PER_CTA], s_units[ROWS_PER_CTA], s_at[ROWS_PER_CTA];
    __shared__ float s_products[ROWS_PER_CTA];
    __shared__ int s_long[ROWS_PER_CTA], s_n_long, s_count[LIST_MASK + 1];
    trigger_dependents();
    const int tid = threadIdx.x, lane = lane_id(), first = warp_id() * ROWS_PER_WARP;
    auto row_of = [&](int r) -> int64_t { return (int64_t)r * gridDim.x + blockIdx.x; };  // neighbouring rows in different CTAs
    if (tid <= LIST_MASK) s_count[tid] = 0;
    if (tid == 0) s_n_long = 0;
    __syncthreads();
    {
        int32_t lo = 0, hi = 0;  // lane r: A's entries of the warp's row r; none where the mask has none
        if (lane < ROWS_PER_WARP && row_of(first + lane) < rows) {
            const int64_t i = row_of(first + lane);
            lo = ld_nc(A.rp + i);
            hi = ld_nc(C.rp + i) == ld_nc(C.rp + i + 1) ? lo : ld_nc(A.rp + i + 1);
        }
        const bool is_long = hi - lo > LONG_ROW;
        if (lane < ROWS_PER_WARP) {
            s_lo[first + lane] = lo;
            s_hi[first + lane] = hi;
            s_products[first + lane] = 0.f;
            if (is_long) s_long[atomicAdd(&s_n_long, 1)] = first + lane;
        }
        const int len = is_long ? 0 : hi - lo;
        const int most = __reduce_max_sync(FULL_MASK, (unsigned)len);
        float mine[ROWS_PER_WARP] = {};  // rounding does not matter: the counts only choose a list
        for (int p = lane; p - lane < most; p += 32) {
            int32_t j[ROWS_PER_WARP];
#pragma unroll
            for (int r = 0; r < ROWS_PER_WARP; ++r) {
                const int n = __shfl_sync(FULL_MASK, len, r), from = __shfl_sync(FULL_MASK, lo, r);
                j[r] = p < n ? ld_nc(A.col + from + p) : -1;
            }
#pragma unroll
            for (int r = 0; r < ROWS_PER_WARP; ++r)
                if (j[r] >= 0) mine[r] += (float)(ld_nc(B.rp + j[r] + 1) - ld_nc(B.rp + j[r]));
        }
#pragma unroll
        for (int r = 0; r < ROWS_PER_WARP; ++r) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) mine[r] += __shfl_xor_sync(FULL_MASK, mine[r], o);
            if (lane == r && !is_long) s_products[first + r] = mine[r];
        }
    }
    __syncthreads();
    for (int l = 0; l < s_n_long; ++l) {
        const int row = s_long[l];
        float mine = 0.f;
#pragma unroll 4
        for (int32_t p = s_lo[row] + tid; p < s_hi[row]; p += 256) {
            const int32_t j = ld_nc(A.col + p);
            mine += (float)(ld_nc(B.rp + j + 1) - ld_nc(B.rp + j));
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mine += __shfl_xor_sync(FULL_MASK, mine, o);
        if (lane == 0) atomicAdd(s_products + row, mine);
    }
    __syncthreads();
    if (tid < ROWS_PER_CTA) {
        const float products = s_products[tid];
        const int32_t a_lo = s_lo[tid], a_hi = s_hi[tid];
        int list = -1, n_units = 0, at = 0;
        if (products > 0.f && products < (float)LIGHT_P) {
            list = LIST_LIGHT;
            n_units = 1;
        } else if (products > 0.f) {
            const int64_t i = row_of(tid);
            const int32_t c_lo = ld_nc(C.rp + i), c_hi = ld_nc(C.rp + i + 1);
            const int32_t words = (ld_nc(C.col + c_hi - 1) >> 6) - (ld_nc(C.col + c_lo) >> 6) + 1, entries = c_hi - c_lo;
            // Warp instructions of the two ways, roughly: looking the mask row up in every selected row of B costs
            // 150 per entry and 32 mask positions; walking the products costs 4000 for the bitmap of the mask row,
            // 200 per entry and 0.7 per product. R-MAT rows of a few dozen entries are an order of magnitude cheaper
            // to look up, hub rows are not. (50021 vertices, 800003 edges: 506 us with 150, 534 with 300, 693 without
            // the look-up.)
            const float entries_a = (float)(a_hi - a_lo);
            const bool by_mask = 150.f * entries_a * (float)((entries + 31) / 32) <= 4000.f + 200.f * entries_a + 0.7f * products;
            list = LIST_WIDE;
            if (by_mask) list = LIST_MASK;
            else if (words <= CLASS[0].words && entries <= CLASS[0].entries) list = 0;
            else if (words <= CLASS[1].words && entries <= CLASS[1].entries) list = 1;
            else if (words <= CLASS[2].words) list = 2;
            n_units = (a_hi - a_lo + unit_of(list) - 1) / unit_of(list);
        }
        if (list >= 0) at = atomicAdd(&s_count[list], n_units);
        s_list[tid] = list;
        s_units[tid] = n_units;
        s_at[tid] = at;
    }
    __syncthreads();
    if (tid <= LIST_MASK && s_count[tid] > 0) s_count[tid] = atomicAdd(&ctl->count[tid], s_count[tid]);  // from here on: where the CTA's units begin
    __syncthreads();
#pragma unroll
    for (int r = first; r < first + ROWS_PER_WARP; ++r) {
        const int list = s_list[r], n_units = s_units[r];
        if (list < 0) continue;
        const int64_t at = s_count[list] + s_at[r];
        if (list == LIST_LIGHT) {
            if (lane == 0) light[at] = (int32_t)row_of(r);
            continue;
        }
        const int unit = unit_of(list);
        int2 *to = units + (list == LIST_MASK ? 4 : list) * list_cap + at;
        for (int u = lane; u < n_units; u += 32) to[u] = make_int2((int)row_of(r), s_lo[r] + u * unit);
    }
}

// One product column k of the mask row [c_lo, c_hi) by binary search; on a hit the product goes to
// the global sums.
__device__ __forceinline__ void search_product(const CsrView &B, const CsrView &C, int32_t q, int32_t k, float av, int32_t c_lo,
                                               int32_t c_hi, int32_t c0, float *__restrict__ acc, int32_t *__restrict__ hit) {
    int32_t lo = c_lo, hi = c_hi;  // first position of the mask's row with column >= k
    while (lo < hi) {
        const int32_t mid = lo + ((hi - lo) >> 1);
        if (ld_nc(C.col + mid) < k) lo = mid + 1; else hi = mid;
    }
    if (lo < c_hi && ld_nc(C.col + lo) == k) {
        atomicAdd(acc + (lo - c0), (av * ld_nc(B.val + q)) * ld_nc(C.val + lo));
        hit[lo - c0] = 1;
    }
}

__global__ void __launch_bounds__(256) k_sssmm_search_warp(CsrView A, CsrView B, CsrView C, const int32_t *__restrict__ list,
                                                          SssmmCtl *__restrict__ ctl, float *__restrict__ acc,
                                                          int32_t *__restrict__ hit) {
    trigger_dependents();
    const int lane = lane_id();
    const int32_t c0 = ld_nc(C.rp);  // the mask may be a row block of a larger matrix: positions count from its first entry
    const int count = ctl->count[LIST_LIGHT];
    for (;;) {
        int t = 0;
        if (lane == 0) t = atomicAdd(&ctl->ticket[LIST_LIGHT], 1);
        t = __shfl_sync(0xffffffffu, t, 0);
        if (t >= count) {
            finish_after_previous();
            return;
        }
        const int64_t i = ld_nc(list + t);
        const int32_t c_lo = ld_nc(C.rp + i), c_hi = ld_nc(C.rp + i + 1);
        for (int32_t p = ld_nc(A.rp + i), a_hi = ld_nc(A.rp + i + 1); p < a_hi; ++p) {
            const int32_t j = ld_nc(A.col + p);
            const float av = ld_nc(A.val + p);
            for (int32_t q = ld_nc(B.rp + j) + lane, b_hi = ld_nc(B.rp + j + 1); q < b_hi; q += 32)
                search_product(B, C, q, ld_nc(B.col + q), av, c_lo, c_hi, c0, acc, hit);
        }
    }
}

// The mask positions of one row, tile by tile of 32 NR, looked up in the rows of B that the entries
// [p_begin, p_end) of A's row select, NE entries at a time: a lane keeps the sums of its NR positions in
// registers and searches NE * NR rows side by side, so that the dependent loads of one search hide the others'.
// The number of steps depends on the row of B alone, so the warp stays together. Terms are added in the order of
// A's entries.
template <int NE, int NR>
__device__ __forceinline__ void look_up_tile(const CsrView &A, const CsrView &B, int32_t p_begin, int32_t p_end, const int32_t (&k)[4],
                                             const float (&cv)[4], float (&sum)[4], unsigned &found) {
    const int lane = lane_id();
    for (int32_t p0 = p_begin; p0 < p_end; p0 += 32) {
        int32_t my_lo = 0, my_len = 0;
        float my_a = 0.f;
        if (p0 + lane < p_end) {
            const int32_t j = ld_nc(A.col + p0 + lane);
            my_lo = ld_nc(B.rp + j);
            my_len = ld_nc(B.rp + j + 1) - my_lo;
            my_a = ld_nc(A.val + p0 + lane);
        }
        const int n_here = min(32, p_end - p0);
        for (int e0 = 0; e0 < n_here; e0 += NE) {
            int32_t at[NE][NR];
            int n[NE], len[NE], longest = 0;
#pragma unroll
            for (int e = 0; e < NE; ++e) {
                const int32_t lo = __shfl_sync(FULL_MASK, my_lo, (e0 + e) & 31);
                const int32_t l = __shfl_sync(FULL_MASK, my_len, (e0 + e) & 31);
                len[e] = n[e] = e0 + e < n_here ? l : 0;
                longest = max(longest, n[e]);
#pragma unroll
                for (int r = 0; r < NR; ++r) at[e][r] = lo;
            }
            for (; longest > 1; longest -= longest >> 1) {  // the last position of the row whose column is <= k, or its first
#pragma unroll
                for (int e = 0; e < NE; ++e) {
                    if (n[e] > 1) {  // uniform
                        const int half = n[e] >> 1;
#pragma unroll
                        for (int r = 0; r < NR; ++r) at[e][r] += ld_nc(B.col + at[e][r] + half) <= k[r] ? half : 0;
                        n[e] -= half;
                    }
                }
            }
#pragma unroll
            for (int e = 0; e < NE; ++e) {
                const float a = __shfl_sync(FULL_MASK, my_a, (e0 + e) & 31);
                if (len[e] > 0) {  // uniform
#pragma unroll
                    for (int r = 0; r < NR; ++r) {
                        if (ld_nc(B.col + at[e][r]) == k[r]) {
                            sum[r] += (a * ld_nc(B.val + at[e][r])) * cv[r];
                            found |= 1u << r;
                        }
                    }
                }
            }
        }
    }
}

__global__ void __launch_bounds__(256) k_sssmm_look_up(CsrView A, CsrView B, CsrView C, const int2 *__restrict__ units,
                                                      SssmmCtl *__restrict__ ctl, float *__restrict__ acc, int32_t *__restrict__ hit) {
    trigger_dependents();
    const int lane = lane_id();
    const int32_t c0 = ld_nc(C.rp);
    const int count = ctl->count[LIST_MASK];
    for (;;) {
        int t = 0;
        if (lane == 0) t = atomicAdd(&ctl->ticket[LIST_MASK], 1);
        t = __shfl_sync(FULL_MASK, t, 0);
        if (t >= count) break;
        const int2 unit = units[t];
        const int64_t i = unit.x;
        const int32_t c_lo = ld_nc(C.rp + i), c_hi = ld_nc(C.rp + i + 1), a_lo = ld_nc(A.rp + i), a_hi = ld_nc(A.rp + i + 1);
        const int32_t p_end = min(unit.y + MASK_UNIT, a_hi);
        const bool alone = a_hi - a_lo <= MASK_UNIT;  // no other unit adds to this row's sums
        for (int32_t m0 = c_lo; m0 < c_hi; m0 += 128) {
            int32_t k[4];
            float cv[4], sum[4] = {0.f, 0.f, 0.f, 0.f};
            unsigned found = 0;
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int32_t m = m0 + 32 * r + lane;
                k[r] = m < c_hi ? ld_nc(C.col + m) : -1;
                cv[r] = m < c_hi ? ld_nc(C.val + m) : 0.f;
            }
            const int left = c_hi - m0;
            if (left <= 32) look_up_tile<8, 1>(A, B, unit.y, p_end, k, cv, sum, found);
            else if (left <= 64) look_up_tile<4, 2>(A, B, unit.y, p_end, k, cv, sum, found);
            else look_up_tile<2, 4>(A, B, unit.y, p_end, k, cv, sum, found);
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                if (!((found >> r) & 1u)) continue;
                const int32_t at = m0 + 32 * r + lane - c0;
                if (alone) acc[at] = sum[r]; else atomicAdd(acc + at, sum[r]);
                hit[at] = 1;
            }
        }
    }
    finish_after_previous();
}

// Shared memory of unit_products: for every entry of the unit, the bounds of its row of B, its
// value, and the number of chunks in front of it.
template <int NT>
struct UnitRows {
    static constexpr int E = WARP_ENTRIES * (NT / 32);
    int32_t lo[E], hi[E], first[E];
    float av[E];
    int tmp[34];
};

// The products of the entries [p_begin, p_end) of A's row, spread evenly over the warps of the CTA: the rows of B the entries
// select are cut into chunks, the chunks are numbered through (an exclusive sum over the entries) and every warp takes a
// contiguous share of them. For 32 chunks at a time every lane finds the entry of one of them by binary search in the
// shared-memory sums; then the chunks go by, what their lane knows broadcast. The CTA must be in step on entry. `reaches(k)` says
// whether the mask may hold column k; `hit(q, a)` receives the position in B and A's value of those products that
// pass. The two are apart because few pass (one in sixteen on R-MAT graphs) and a lane that does makes its whole warp walk the
// long way: the tests of a chunk are done first, then every lane works off its own hits, so the long way is walked as often
// as the luckiest lane has hits (under 3 times per 8 products) and not once per product.
template <int NT, typename Reaches, typename Hit>
__device__ __forceinline__ void unit_products(const CsrView &A, const CsrView &B, int32_t p_begin, int32_t p_end, UnitRows<NT> &rows, Reaches reaches, Hit hit) {
    constexpr int NW = NT / 32;
    constexpr int PER_LANE = 8, CHUNK = 32 * PER_LANE;  // products of a chunk per lane: that many loads in flight
    const int tid = threadIdx.x, lane = lane_id(), n_e = p_end - p_begin;
    int chunks = 0;
    if (tid < n_e) {
        const int32_t j = ld_nc(A.col + p_begin + tid);
        const int32_t lo = ld_nc(B.rp + j), hi = ld_nc(B.rp + j + 1);
        rows.av[tid] = ld_nc(A.val + p_begin + tid);
        rows.lo[tid] = lo;
        rows.hi[tid] = hi;
        chunks = (hi - lo + CHUNK - 1) / CHUNK;
    }
    int total;
    const int before = block_excl_sum<NT>(chunks, rows.tmp, total);
    if (tid < n_e) rows.first[tid] = before;
    __syncthreads();

    const int share = (total + NW - 1) / NW, end = min((warp_id() + 1) * share, total);
    for (int c0 = warp_id() * share; c0 < end; c0 += 32) {
        const int mine = min(c0 + lane, end - 1);
        int e = 0, above = n_e;  // the last entry whose first chunk is at or before this lane's
        while (above - e > 1) {
            const int mid = (e + above) >> 1;
            if (rows.first[mid] <= mine) e = mid; else above = mid;
        }
        const int32_t my_q = rows.lo[e] + (mine - rows.first[e]) * CHUNK, my_hi = rows.hi[e];
        const float my_a = rows.av[e];
        const int here = min(32, end - c0);
        for (int u = 0; u < here; ++u) {
            const int32_t q = __shfl_sync(FULL_MASK, my_q, u) + lane, n = __shfl_sync(FULL_MASK, my_hi, u) - q;
            const float a = __shfl_sync(FULL_MASK, my_a, u);
            int32_t k[PER_LANE];
#pragma unroll
            for (int t = 0; t < PER_LANE; ++t) k[t] = 32 * t < n ? ld_nc(B.col + q + 32 * t) : -1;
            unsigned hits = 0;
#pragma unroll
            for (int t = 0; t < PER_LANE; ++t)
                if (k[t] >= 0 && reaches(k[t])) hits |= 1u << t;
            for (; hits; hits &= hits - 1u) hit(q + 32 * (__ffs((int)hits) - 1), a);
        }
    }
}

__global__ void __launch_bounds__(SEARCH_NT) k_sssmm_search_cta(CsrView A, CsrView B, CsrView C, const int2 *__restrict__ units,
                                                               SssmmCtl *__restrict__ ctl, float *__restrict__ acc,
                                                               int32_t *__restrict__ hit) {
    trigger_dependents();
    __shared__ UnitRows<SEARCH_NT> s_rows;
    const int32_t c0 = ld_nc(C.rp);
    const int count = ctl->count[LIST_WIDE];
    for (int t = blockIdx.x; t < count; t += gridDim.x) {
        const int2 unit = units[t];
        const int64_t i = unit.x;
        const int32_t c_lo = ld_nc(C.rp + i), c_hi = ld_nc(C.rp + i + 1);
        unit_products<SEARCH_NT>(A, B, unit.y, min(unit.y + CLASS[LIST_WIDE].unit(), ld_nc(A.rp + i + 1)), s_rows, [](int32_t) { return true; },
                                 [&](int32_t q, float av) { search_product(B, C, q, ld_nc(B.col + q), av, c_lo, c_hi, c0, acc, hit); });
        __syncthreads();
    }
    finish_after_previous();
}

// What covers the latency of a product's loads is the number of warps, so a thread is held to 32 registers, eight and two CTAs
// per SM instead of six and one: a graph of 50021 vertices squared on its own positions 484 -> 412 us a call, of 24405 204 -> 190, of
// 131072 2270 -> 1555. (The rows of B as bitmap words, 32 columns to a test, need 48 and 64 registers, three kernels in front and 12
// bytes of scratch per entry of B, and were behind at every size: 450, 204 and 1806 us.)
template <int NT, bool SHARED_ACC>
__global__ void __launch_bounds__(NT, 2048 / NT) k_sssmm_bitmap(CsrView A, CsrView B, CsrView C, const int2 *units,
                                                    SssmmCtl *ctl, int which, int words_cap, int entries_cap,
                                                    float *__restrict__ acc, int32_t *__restrict__ hit) {
    extern __shared__ uint64_t sm_words[];
    uint64_t *bm = sm_words;                                         // bit (k - 64 * w0) set: the mask row stores column k
    uint32_t *bm32 = reinterpret_cast<uint32_t *>(bm);               // the same bits, for 32-bit shared-memory atomics
    uint32_t *rank = reinterpret_cast<uint32_t *>(bm + words_cap);   // set bits in front of each 64-bit word
    float *acc_s = reinterpret_cast<float *>(rank + words_cap);
    unsigned char *flag_s = reinterpret_cast<unsigned char *>(acc_s + entries_cap);
    __shared__ int2 s_unit;
    __shared__ UnitRows<NT> s_rows;
    // The list kernels run side by side. Only the first (which == 2) waits for the lists, and lets the next
    // one start after that; each of the others lets its successor start at once.
    if (which == 2) wait_for_previous();
    trigger_dependents();
    const int tid = threadIdx.x;
    const int32_t c0 = ld_nc(C.rp);
    const int count = ctl->count[which];
    for (;;) {
        if (tid == 0) {
            const int t = atomicAdd(&ctl->ticket[which], 1);
            s_unit = t < count ? units[t] : make_int2(-1, 0);
        }
        __syncthreads();
        const int2 unit = s_unit;
        const int64_t i = unit.x;
        if (i < 0) {
            finish_after_previous();
            return;
        }
        const int32_t c_lo = ld_nc(C.rp + i), c_hi = ld_nc(C.rp + i + 1);
        const int32_t w0 = ld_nc(C.col + c_lo) >> 6;
        const int32_t words = (ld_nc(C.col + c_hi - 1) >> 6) - w0 + 1, entries = c_hi - c_lo;
        for (int w = tid; w < words; w += NT) bm[w] = 0;
        if (SHARED_ACC)
            for (int p = tid; p < entries; p += NT) {
                acc_s[p] = 0.0f;
                flag_s[p] = 0;
            }
        __syncthreads();
        for (int32_t p = c_lo + tid; p < c_hi; p += NT) {
            const int32_t k = ld_nc(C.col + p) - (w0 << 6);
            atomicOr(bm32 + (k >> 5), 1u << (k & 31));
        }
        __syncthreads();
        {   // ranks: every thread counts a run of consecutive words, the CTA scans the runs
            const int per = (words + NT - 1) / NT;
            const int w_lo = min(tid * per, words), w_hi = min(w_lo + per, words);
            int mine = 0, total;
            for (int w = w_lo; w < w_hi; ++w) mine += __popcll(bm[w]);
            int before = block_excl_sum<NT>(mine, s_rows.tmp, total);
            for (int w = w_lo; w < w_hi; ++w) {
                rank[w] = (uint32_t)before;
                before += __popcll(bm[w]);
            }
        }
        __syncthreads();
        const int32_t col0 = w0 << 6;
        const uint32_t span = (uint32_t)words << 6;
        unit_products<NT>(A, B, unit.y, min(unit.y + WARP_ENTRIES * (NT / 32), ld_nc(A.rp + i + 1)), s_rows, [&](int32_t k) {
            const uint32_t bit = (uint32_t)(k - col0);
            return bit < span && ((bm32[bit >> 5] >> (bit & 31)) & 1u) != 0u;  // most products end here
        }, [&](int32_t q, float av) {
            const uint32_t bit = (uint32_t)(ld_nc(B.col + q) - col0);  // the column again, from cache: an index into registers would cost more
            const uint32_t w = bit >> 6, sh = bit & 63;
            const int32_t pos = (int32_t)rank[w] + __popcll(bm[w] & ((1ull << sh) - 1));
            const float v = (av * ld_nc(B.val + q)) * ld_nc(C.val + c_lo + pos);
            if (SHARED_ACC) {
                atomicAdd(acc_s + pos, v);
                flag_s[pos] = 1;
            } else {
                atomicAdd(acc + (c_lo - c0 + pos), v);
                hit[c_lo - c0 + pos] = 1;
            }
        });
        __syncthreads();
        if (SHARED_ACC) {  // other units of the same row add to the same sums
            for (int p = tid; p < entries; p += NT)
                if (flag_s[p]) {
                    atomicAdd(acc + (c_lo - c0 + p), acc_s[p]);
                    hit[c_lo - c0 + p] = 1;
                }
            __syncthreads();
        }
    }
}

// Exclusive scan of the flags over nnz + 1 entries, in place (the last flag is 0, so pos[nnz] is the total, which
// also goes to `word`), and, where the caller's arrays hold every mask position (`z_col` set), the reached
// positions written to their places in the same pass.
__global__ void __launch_bounds__(SCAN_NT) k_sssmm_scan(int32_t *pos, const float *acc, const int32_t *__restrict__ c_rp,
                                                       const int32_t *__restrict__ c_col, int32_t nnz, uint64_t *state, FusedCtl *ctl,
                                                       int32_t *z_col, float *z_val, unsigned long long *word) {
    __shared__ int scan_tmp[40];
    __shared__ long long s_base;
    trigger_dependents();
    wait_for_previous();
    const int tid = threadIdx.x, t = blockIdx.x;  // CTAs are dispatched in index order; waits on earlier tiles are bounded
    const int64_t n = (int64_t)nnz + 1, p0 = ((int64_t)t * SCAN_NT + tid) * SCAN_VT;
    int v[SCAN_VT], mine = 0;
#pragma unroll
    for (int q = 0; q < SCAN_VT; ++q) {
        v[q] = p0 + q < n ? pos[p0 + q] : 0;
        mine += v[q];
    }
    int total;
    const int run = block_excl_sum<SCAN_NT>(mine, scan_tmp, total);
    if (warp_id() == 0) {
        const int64_t b = lookback_exclusive(state, t, total, &ctl->status);
        if (lane_id() == 0) s_base = b;
    }
    __syncthreads();
    if (t == (int)gridDim.x - 1 && tid == 0)
        publish_result_word(word, s_base < 0 || ld_relaxed_gpu_i32(&ctl->status.error) != 0 ? NB200_E_TIMEOUT : NB200_OK, s_base < 0 ? 0 : s_base + total);
    if (s_base < 0) return;
    int32_t at = (int32_t)s_base + run;  // at most nnz
    const int32_t *mask_col = c_col + ld_nc(c_rp);
    float sum[SCAN_VT];  // fetched together: a plain load stays behind the stores in front of it
#pragma unroll
    for (int q = 0; q < SCAN_VT; ++q) sum[q] = v[q] && z_col ? ld_late(acc + p0 + q) : 0.f;
#pragma unroll
    for (int q = 0; q < SCAN_VT; ++q) {
        if (p0 + q >= n) break;
        pos[p0 + q] = at;
        if (v[q]) {
            if (z_col) {
                z_col[at] = ld_nc(mask_col + p0 + q);
                z_val[at] = sum[q];
            }
            ++at;
        }
    }
}

__global__ void __launch_bounds__(256) k_sssmm_row_offsets(const int32_t *pos, const int32_t *__restrict__ c_rp,
                                                          int32_t rows, int32_t *z_rp) {
    wait_for_previous();
    const int64_t r = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (r > rows) return;
    z_rp[r] = ld_late(pos + (ld_nc(c_rp + r) - ld_nc(c_rp)));
}

// Writes the reached positions after the scan, for callers with less room than the mask has entries.
__global__ void __launch_bounds__(256) k_sssmm_compact(const int32_t *__restrict__ pos, const float *__restrict__ acc,
                                                      const int32_t *__restrict__ c_rp, const int32_t *__restrict__ c_col, int32_t nnz,
                                                      int32_t *__restrict__ z_col, float *__restrict__ z_val) {
    const int64_t p = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (p >= nnz) return;
    const int32_t at = ld_nc(pos + p);
    if (ld_nc(pos + p + 1) > at) {
        z_col[at] = ld_nc(c_col + ld_nc(c_rp) + p);
        z_val[at] = ld_nc(acc + p);
    }
}

int check(const nb200_csr *m) {
    if (!m || m->rows < 0 || m->cols < 0 || m->nnz < 0 || !m->row_ptr) return NB200_E_BADARG;
    if (m->nnz > 0 && (!m->col || !m->val)) return NB200_E_BADARG;
    return NB200_OK;
}

int sssmm_run(const nb200_csr *a, const nb200_csr *b, const nb200_csr *c, nb200_csr *z, int64_t capacity, void *stream_v) {
    int st;
    if ((st = check(a)) || (st = check(b)) || (st = check(c))) return st;
    if (!z || !z->row_ptr || capacity < 0 || a->cols != b->rows || c->rows != a->rows || c->cols != b->cols) return NB200_E_BADARG;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
    const int32_t rows = a->rows, nnz = c->nnz;
    z->rows = rows;
    z->cols = b->cols;
    z->nnz = 0;
    if (nnz == 0 || a->nnz == 0 || b->nnz == 0) {
        NB200_CUDA(cudaMemsetAsync(z->row_ptr, 0, sizeof(int32_t) * ((size_t)rows + 1), stream));
        return NB200_OK;
    }
    // per device, so set on every call: cheap next to the launches that follow
    NB200_CUDA(cudaFuncSetAttribute(k_sssmm_bitmap<1024, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CLASS[1].smem()));
    NB200_CUDA(cudaFuncSetAttribute(k_sssmm_bitmap<1024, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CLASS[2].smem()));
    int device = 0, sms = 148;
    NB200_CUDA(cudaGetDevice(&device));
    NB200_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));

    const int scan_ctas = (int)(((int64_t)nnz + 1 + SCAN_NT * SCAN_VT - 1) / (SCAN_NT * SCAN_VT));
    const int64_t list_cap = (int64_t)rows + a->nnz / CLASS[LIST_WIDE].unit() + 1;  // the smallest unit of those classes bounds every list
    const int64_t mask_cap = (int64_t)rows + a->nnz / MASK_UNIT + 1;
    Carver sizes;
    sizes.take<float>((size_t)nnz);
    sizes.take<int32_t>((size_t)nnz + 1);
    sizes.take<uint64_t>((size_t)scan_ctas + 8);
    sizes.take<SssmmCtl>(1);
    sizes.take<int2>((size_t)4 * list_cap + mask_cap);
    sizes.take<int32_t>((size_t)rows);
    Workspace *ws = nullptr;
    if ((st = acquire_workspace(stream, sizes.used(), &ws, 1))) return st;
    Carver carve(ws->dev);
    float *acc = carve.take<float>((size_t)nnz);
    int32_t *hit = carve.take<int32_t>((size_t)nnz + 1);
    uint64_t *scan_block = carve.take<uint64_t>((size_t)scan_ctas + 8);
    SssmmCtl *sctl = carve.take<SssmmCtl>(1);
    int2 *units = carve.take<int2>((size_t)4 * list_cap + mask_cap);
    int32_t *light = carve.take<int32_t>((size_t)rows);
    FusedCtl *ctl = reinterpret_cast<FusedCtl *>(scan_block);
    // sums, flags and control blocks lie next to one another: one fill clears them all
    NB200_CUDA(cudaMemsetAsync(acc, 0, (size_t)(reinterpret_cast<unsigned char *>(units) - reinterpret_cast<unsigned char *>(acc)), stream));
    unsigned long long *word = result_word(ws, 0);
    const CsrView A{a->row_ptr, a->col, a->val}, B{b->row_ptr, b->col, b->val}, C{c->row_ptr, c->col, c->val};
    const int row_warps_grid = (int)std::min<int64_t>(((int64_t)rows + 7) / 8, (int64_t)sms * 8);
    const int most = (int)std::min<int64_t>(list_cap, 1 << 30);
    {
        LaunchScope scope("sssmm_classify", stream);
        k_sssmm_classify<<<(int)(((int64_t)rows + ROWS_PER_CTA - 1) / ROWS_PER_CTA), 256, 0, stream>>>(A, B, C, rows, list_cap, units, light, sctl);
    }
    // Every list is worked by resident CTAs that take units from a ticket; a list's length stays on
    // the device, so an empty list costs one launch of CTAs that leave at once.
    {
        LaunchScope scope("sssmm_bitmap_wide", stream);
        NB200_CUDA(launch_overlapped(k_sssmm_bitmap<1024, false>, dim3(std::min(sms, most)), dim3(1024), CLASS[2].smem(), stream, A, B, C,
                                     units + 2 * list_cap, sctl, 2, CLASS[2].words, 0, acc, hit));
    }
    {
        LaunchScope scope("sssmm_bitmap_medium", stream);
        NB200_CUDA(launch_overlapped(k_sssmm_bitmap<1024, true>, dim3(std::min(2 * sms, most)), dim3(1024), CLASS[1].smem(), stream, A, B, C,
                                     units + list_cap, sctl, 1, CLASS[1].words, CLASS[1].entries, acc, hit));
    }
    {
        LaunchScope scope("sssmm_bitmap_narrow", stream);
        NB200_CUDA(launch_overlapped(k_sssmm_bitmap<256, true>, dim3(std::min(8 * sms, most)), dim3(256), CLASS[0].smem(), stream, A, B, C, units, sctl, 0,
                                     CLASS[0].words, CLASS[0].entries, acc, hit));
    }
    {
        LaunchScope scope("sssmm_look_up", stream);
        NB200_CUDA(launch_overlapped(k_sssmm_look_up, dim3(row_warps_grid), dim3(256), 0, stream, A, B, C, units + (size_t)4 * list_cap, sctl, acc, hit));
    }
    {
        LaunchScope scope("sssmm_search_wide", stream);
        NB200_CUDA(launch_overlapped(k_sssmm_search_cta, dim3(std::min(16 * sms, most)), dim3(SEARCH_NT), 0, stream, A, B, C,
                                     units + (size_t)LIST_WIDE * list_cap, sctl, acc, hit));
    }
    {
        LaunchScope scope("sssmm_search_light", stream);
        NB200_CUDA(launch_overlapped(k_sssmm_search_warp, dim3(row_warps_grid), dim3(256), 0, stream, A, B, C, light, sctl, acc, hit));
    }
    const bool room = capacity >= nnz && z->col && z->val;  // then every reached position has its place already
    {
        LaunchScope scope("sssmm_scan", stream);
        NB200_CUDA(launch_overlapped(k_sssmm_scan, dim3(scan_ctas), dim3(SCAN_NT), 0, stream, hit, acc, c->row_ptr, c->col, nnz, scan_block + 4, ctl,
                                     room ? z->col : nullptr, z->val, word));
    }
    {
        LaunchScope scope("sssmm_row_offsets", stream);
        NB200_CUDA(launch_overlapped(k_sssmm_row_offsets, dim3((int)(((int64_t)rows + 1 + 255) / 256)), dim3(256), 0, stream, hit, c->row_ptr, rows, z->row_ptr));
    }
    int64_t length;
    int device_status;
    if ((st = wait_result_word(word, stream, &length, &device_status))) return st;
    if (device_status != 0) return note_timeout(ERR_LOOKBACK_TIMEOUT, 0, "sssmm scan");
    z->nnz = (int32_t)length;
    if (room) return NB200_OK;
    if (length > capacity) return NB200_E_CAPACITY;
    if (length > 0) {
        if (!z->col || !z->val) return NB200_E_BADARG;
        LaunchScope scope("sssmm_compact", stream);
        k_sssmm_compact<<<(int)(((int64_t)nnz + 255) / 256), 256, 0, stream>>>(hit, acc, c->row_ptr, c->col, nnz, z->col, z->val);
        NB200_CUDA(cudaGetLastError());
    }
    return NB200_OK;
}

}  // namespace

}  // namespace nb200

using namespace nb200;

extern "C" {

int nb200_sssmm_f32_into(const nb200_csr *a, const nb200_csr *b, const nb200_csr *c, nb200_csr *z, int64_t capacity, void *stream) {
    return sssmm_run(a, b, c, z, capacity, stream);
}

}  // extern "C"
