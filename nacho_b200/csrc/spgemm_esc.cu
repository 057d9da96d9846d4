// SpGEMM C = A * B by expand - sort - compress, row by row.
//
// What the reference does (GPU only, compiler.cpp:145-148): expand every product
// a.values[p] * b.values[q] with key k = b.cols[q] in (i, j ascending, k ascending) order
// (src/backend/compute.cpp:526-611), sort each row's products by k with a global segmented sort
// (src/backend/stitch_and_generate_gpu.cpp:79-94), flag run heads, scan, and sum runs with
// warp shuffles plus atomics (:96-124, :257-363). All its counters are int32 and it
// materialises every product in HBM.
//
// Here rows are binned by their product count P_i (64-bit counters throughout) and no product
// ever reaches HBM:
//   small   P_i <= 32      one warp per row: products in registers, bitonic sort by shuffles
//   medium  P_i <= 256     one CTA per row: products in shared memory, bitonic sort there
//   ranked  P_i <= 65535   one CTA per row: a bitmap of the produced columns in shared memory is
//   heavy   P_i  > 65535   turned into the rank of every column within the result row, then every
//                          product is added straight into its position of the row, in shared memory
//                          where the row's result fits there. Heavy rows start in order of weight.
// Matrices wider than the bitmap (262144 columns) are walked in column windows of that width.
// Two passes: symbolic (unique columns per row -> row offsets by a scan) and numeric (fill).
// Small and medium rows sum equal-column products in expansion order (ascending j), a fixed
// order; ranked and heavy rows sum with float32 atomics, like the reference does for every row.
#include <algorithm>
#include <climits>
#include <cstring>
#include <mutex>
#include <type_traits>

#include "merge_common.cuh"
#include "row_words.cuh"

namespace nb200 {

namespace {

constexpr int SMALL_P = 32;
#ifndef ESC_MEDIUM_P
#define ESC_MEDIUM_P 256
#endif
constexpr int MEDIUM_P = ESC_MEDIUM_P;
constexpr int MED_NT = 128;
constexpr unsigned long long RANKED_P = 65535;   // rows above are heavy: larger symbolic CTAs, first in every list
constexpr unsigned long long GIANT_P = 1ull << 18;

struct CsrView {
    const int32_t *rp;
    const int32_t *col;
    const float *val;
};

enum { BIN_SMALL, BIN_MEDIUM, BIN_RANKED, BIN_GIANT, BIN_HEAVY, BINS };  // heavy rows with more / at most GIANT_P products

// Device-side counters of one call.
struct EscCtl {
    unsigned long long products;
    int n_rows[BINS];
    int max_entries;       // longest row of A
    int arrived;           // CTAs of the binning kernel that are done
};

// Result words of the binning kernel, in this order.
enum { W_PRODUCTS, W_SMALL, W_MEDIUM, W_RANKED, W_GIANT, W_HEAVY, W_ENTRIES, W_NNZ, W_COUNT };

// The last CTA of the binning kernel to get here tells the host the counters. `prefix` may be null.
__device__ __forceinline__ void publish_counters(EscCtl *ctl, const FusedCtl *prefix, unsigned long long *words) {
    __syncthreads();
    if (threadIdx.x != 0) return;
    __threadfence();
    if (atomicAdd(&ctl->arrived, 1) != (int)gridDim.x - 1) return;
    __threadfence();
    const volatile EscCtl *c = ctl;
    publish_result_word(words + W_SMALL, 0, c->n_rows[BIN_SMALL]);
    publish_result_word(words + W_MEDIUM, 0, c->n_rows[BIN_MEDIUM]);
    publish_result_word(words + W_RANKED, 0, c->n_rows[BIN_RANKED]);
    publish_result_word(words + W_GIANT, 0, c->n_rows[BIN_GIANT]);
    publish_result_word(words + W_HEAVY, 0, c->n_rows[BIN_HEAVY]);
    publish_result_word(words + W_ENTRIES, 0, c->max_entries);
    publish_result_word(words + W_PRODUCTS, prefix && prefix->status.error != 0 ? NB200_E_TIMEOUT : NB200_OK, (long long)c->products);
}

// heavy_rows holds the giant rows from its front and the other heavy rows from its back, so
// that the heaviest rows are handed out first.
struct RowLists {
    int32_t *small_rows, *medium_rows, *ranked_rows, *heavy_rows;
};

// P[p] = products of the first p stored entries of A (p = 0 .. nnz(A), counted from A's first row
// offset, which need not be 0): B's row lengths summed
// in one pass, 2048 entries per CTA, CTA totals chained by bounded look-back.
__global__ void __launch_bounds__(256) k_esc_product_prefix(CsrView A, CsrView B, int32_t nnz_a, unsigned long long *__restrict__ P,
                                                             uint64_t *state_raw, FusedCtl *ctl) {
    trigger_dependents();
    constexpr int VT = 8;
    __shared__ unsigned long long warp_sums[9];
    __shared__ long long s_base;
    volatile uint64_t *state = state_raw;
    const int tid = threadIdx.x, t = blockIdx.x;  // CTAs are dispatched in index order; waits on earlier tiles are bounded
    const int64_t p0 = ((int64_t)t * 256 + tid) * VT;
    const int32_t *a_col = A.col + ld_nc(A.rp);
    unsigned len[VT];
    unsigned long long mine = 0;
#pragma unroll
    for (int q = 0; q < VT; ++q) {
        len[q] = 0;
        if (p0 + q < nnz_a) {
            const int32_t j = ld_nc(a_col + p0 + q);
            len[q] = (unsigned)(ld_nc(B.rp + j + 1) - ld_nc(B.rp + j));
        }
        mine += len[q];
    }
    unsigned long long incl = mine;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const unsigned long long up = __shfl_up_sync(FULL_MASK, incl, d);
        if (lane_id() >= d) incl += up;
    }
    if (lane_id() == 31) warp_sums[warp_id()] = incl;
    __syncthreads();
    if (tid == 0) {
        unsigned long long run = 0;
        for (int w = 0; w < 8; ++w) {
            const unsigned long long c = warp_sums[w];
            warp_sums[w] = run;
            run += c;
        }
        warp_sums[8] = run;
    }
    __syncthreads();
    if (warp_id() == 0) {
        const int64_t b = lookback_exclusive(state, t, (int64_t)warp_sums[8], &ctl->status);
        if (lane_id() == 0) s_base = b;
    }
    __syncthreads();
    if (s_base < 0) return;
    unsigned long long run = (unsigned long long)s_base + warp_sums[warp_id()] + incl - mine;
#pragma unroll
    for (int q = 0; q < VT; ++q) {
        if (p0 + q <= nnz_a) P[p0 + q] = run;
        run += len[q];
    }
}

// Puts row i (p products) of every thread of the CTA on its list, and adds the products up. A CTA advances each list
// once: every warp's atomics on the same few words held the kernel up (262144 rows of a mesh 22.2 -> 14.6 us).
__device__ __forceinline__ void bin_rows(const int i, const unsigned long long p, const int32_t rows, int32_t *row_count, const RowLists &lists, EscCtl *ctl) {
    __shared__ unsigned long long s_products;
    __shared__ int s_count[BINS];
    if (threadIdx.x < BINS) s_count[threadIdx.x] = 0;
    if (threadIdx.x == 0) s_products = 0;
    __syncthreads();
    const int bin = p == 0 ? -1 : p <= SMALL_P ? BIN_SMALL : p <= MEDIUM_P ? BIN_MEDIUM : p <= RANKED_P ? BIN_RANKED : p > GIANT_P ? BIN_GIANT : BIN_HEAVY;
    int at = 0;
#pragma unroll
    for (int b = 0; b < BINS; ++b) {  // the rows of a list stay in order within a warp
        const unsigned same = __ballot_sync(FULL_MASK, bin == b);
        if (same == 0u) continue;
        int first = 0;
        if (lane_id() == 0) first = atomicAdd(&s_count[b], __popc(same));
        first = __shfl_sync(FULL_MASK, first, 0);
        if (bin == b) at = first + __popc(same & ((1u << lane_id()) - 1u));
    }
    unsigned long long sum = p;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(FULL_MASK, sum, o);
    if (lane_id() == 0 && sum) atomicAdd(&s_products, sum);
    __syncthreads();
    if (threadIdx.x < BINS && s_count[threadIdx.x] > 0) s_count[threadIdx.x] = atomicAdd(&ctl->n_rows[threadIdx.x], s_count[threadIdx.x]);  // from here on: where the CTA's rows begin
    if (threadIdx.x == BINS && s_products) atomicAdd(&ctl->products, s_products);
    __syncthreads();
    if (bin >= 0) {
        at += s_count[bin];
        if (bin == BIN_SMALL) lists.small_rows[at] = i;
        else if (bin == BIN_MEDIUM) lists.medium_rows[at] = i;
        else if (bin == BIN_RANKED) lists.ranked_rows[at] = i;
        else lists.heavy_rows[bin == BIN_GIANT ? at : rows - 1 - at] = i;
    } else if (i < rows && row_count) {
        row_count[i] = 0;
    }
}

// Expand phase 1 (src/backend/compute.cpp:541-611): per-row product counts, and the bins.
// Rows without products get their count (0) written here. The counts come from the prefix P of
// B's row lengths over A's entries (k_esc_product_prefix): a hub row costs one subtraction.
__global__ void __launch_bounds__(256) k_esc_rowwork(CsrView A, const unsigned long long *P, int32_t rows,
                                                     int32_t *__restrict__ row_count, RowLists lists, EscCtl *ctl,
                                                     const FusedCtl *prefix, unsigned long long *words) {
    wait_for_previous();
    const int i = blockIdx.x * 256 + threadIdx.x;  // one lane per row: its products are a difference of the prefix
    unsigned long long p = 0;
    if (i < rows) {
        const int32_t base = ld_nc(A.rp);
        p = ld_late(P + (ld_nc(A.rp + i + 1) - base)) - ld_late(P + (ld_nc(A.rp + i) - base));  // (A lay ready before the prefix pass began)
    }
    bin_rows(i, p, rows, row_count, lists, ctl);
    publish_counters(ctl, prefix, words);
}

// The same with the product counts taken row by row: one lane per row walks its entries (the warp
// shares the work of its longer rows). For matrices of short rows, where a prefix pass over A's
// entries costs more than it saves.
__global__ void __launch_bounds__(256) k_esc_rowwork_walk(CsrView A, CsrView B, int32_t rows, int32_t *__restrict__ row_count,
                                                     RowLists lists, EscCtl *ctl, unsigned long long *words) {
    const int i = blockIdx.x * 256 + threadIdx.x;  // one lane per row; the warp shares the work of its longer rows
    int32_t lo = 0, hi = 0;
    if (i < rows) {
        lo = ld_nc(A.rp + i);
        hi = ld_nc(A.rp + i + 1);
    }
    unsigned long long p = 0;
    const bool together = hi - lo > 32;
    if (!together) {
        for (int32_t e = lo; e < hi; e += 4) {  // four entries' loads in flight
            int32_t j[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) j[q] = e + q < hi ? ld_nc(A.col + e + q) : -1;
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (j[q] >= 0) p += (unsigned long long)(ld_nc(B.rp + j[q] + 1) - ld_nc(B.rp + j[q]));
        }
    }
    for (unsigned todo = __ballot_sync(FULL_MASK, together); todo; todo &= todo - 1) {
        const int r = __ffs(todo) - 1;
        const int32_t l = __shfl_sync(FULL_MASK, lo, r), h = __shfl_sync(FULL_MASK, hi, r);
        unsigned long long q = 0;
        for (int32_t e = l + lane_id(); e < h; e += 128) {  // a hub row is a chain of these: four entries' loads in flight
            int32_t j[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) j[u] = e + 32 * u < h ? ld_nc(A.col + e + 32 * u) : -1;
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (j[u] >= 0) q += (unsigned long long)(ld_nc(B.rp + j[u] + 1) - ld_nc(B.rp + j[u]));
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) q += __shfl_xor_sync(FULL_MASK, q, o);
        if (lane_id() == r) p = q;
    }
    __shared__ int s_longest;
    if (threadIdx.x == 0) s_longest = 0;
    bin_rows(i, p, rows, row_count, lists, ctl);
    const int longest = __reduce_max_sync(FULL_MASK, hi - lo);
    if (lane_id() == 0) atomicMax(&s_longest, longest);
    __syncthreads();
    if (threadIdx.x == 0 && s_longest > 0) atomicMax(&ctl->max_entries, s_longest);
    publish_counters(ctl, nullptr, words);
}

// ------------------------------------------------------------------------- small rows ----

// Compare-exchange step of a 32-wide bitonic sort held one key per lane.
__device__ __forceinline__ uint64_t warp_bitonic_sort(uint64_t key) {
#pragma unroll
    for (int k = 2; k <= 32; k <<= 1) {
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            const uint64_t other = __shfl_xor_sync(FULL_MASK, key, j);
            const bool up = (lane_id() & k) == 0;        // ascending block?
            const bool lower = (lane_id() & j) == 0;     // lower lane of the pair?
            const bool take_min = up == lower;
            key = take_min ? min(key, other) : max(key, other);
        }
    }
    return key;
}

__device__ __forceinline__ uint32_t warp_bitonic_sort32(uint32_t key) {
#pragma unroll
    for (int k = 2; k <= 32; k <<= 1) {
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            const uint32_t other = __shfl_xor_sync(FULL_MASK, key, j);
            const bool take_min = ((lane_id() & k) == 0) == ((lane_id() & j) == 0);
            key = take_min ? min(key, other) : max(key, other);
        }
    }
    return key;
}

#ifndef ESC_SMALL_ROWS
#define ESC_SMALL_ROWS 4
#endif

// Rows with at most 32 products, ESC_SMALL_ROWS of them per warp. Lane l holds product l of a row's
// expansion order; the sort key is (column << 32 | l), so equal columns stay in expansion order.
// NARROW: B has fewer than 2^27 columns, so (column << 5 | lane) fits 32 bits and the sort
// moves half as much through the shuffles.
//
// A row's work is a chain of five dependent loads (row number, A's offsets, A's columns, B's
// offsets, B's columns) and little else, so a warp walks the chain for its rows side by side: the
// loads of one link are issued for all of them before any is used.
template <bool NUMERIC, bool NARROW>
__global__ void __launch_bounds__(256) k_esc_small(CsrView A, CsrView B, const int32_t *__restrict__ row_list, int n_rows,
                                                   int32_t *__restrict__ row_count, const int32_t *__restrict__ c_rp,
                                                   int32_t *__restrict__ c_col, float *__restrict__ c_val) {
    trigger_dependents();
    constexpr int R = ESC_SMALL_ROWS;
    const int w = ((blockIdx.x * 256 + threadIdx.x) >> 5) * R;
    if (w >= n_rows) return;
    const int lane = lane_id();
    int32_t i[R], lo[R], hi[R], out[R];
    uint32_t my_col[R];
    float my_val[R];
    bool have[R];
#pragma unroll
    for (int r = 0; r < R; ++r) i[r] = w + r < n_rows ? ld_nc(row_list + w + r) : -1;
    bool one_round = true;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        lo[r] = hi[r] = out[r] = 0;
        if (i[r] >= 0) {
            lo[r] = ld_nc(A.rp + i[r]);
            hi[r] = ld_nc(A.rp + i[r] + 1);
            if (NUMERIC) out[r] = ld_nc(c_rp + i[r]);
        }
        one_round &= hi[r] - lo[r] <= 32;
        my_col[r] = 0;
        my_val[r] = 0.f;
        have[r] = false;
    }
    // Expansion, 32 entries of a row at a time (one round unless the row holds entries whose rows of B
    // are empty): lane l reads entry l and its row of B; the products of the round take the lanes
    // [base, base + total) in expansion order, each finding its entry among the round's non-empty
    // ones from the mask of slice starts.
    auto place = [&](int r, int base, int32_t b_lo, int len, float a) -> int {
        const int incl = warp_incl_sum(len);
        const int start = base + incl - len;                       // first lane of this entry's products
        const unsigned nonempty = __ballot_sync(FULL_MASK, len > 0);
        const unsigned starts = __reduce_or_sync(FULL_MASK, len > 0 ? 1u << start : 0u);  // the row has at most 32 products
        const int total = __shfl_sync(FULL_MASK, incl, 31);
        // the entry of lane `lane`'s product: the n-th non-empty one, n = slice starts at or before the lane
        const int nth = __popc(starts & (0xffffffffu >> (31 - lane)));
        const int owner = nth > 0 ? (int)__fns(nonempty, 0, nth) : 0;
        const int32_t o_lo = __shfl_sync(FULL_MASK, b_lo, owner);
        const int o_start = __shfl_sync(FULL_MASK, start, owner);
        const float o_a = __shfl_sync(FULL_MASK, a, owner);
        if (lane >= base && lane < base + total) {
            my_col[r] = (uint32_t)ld_nc(B.col + o_lo + (lane - o_start));
            if (NUMERIC) my_val[r] = o_a * ld_nc(B.val + o_lo + (lane - o_start));
            have[r] = true;
        }
        return total;
    };
    if (one_round) {  // uniform: every link of the chain for all rows at once
        int32_t j[R], b_lo[R], len[R];
        float a[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            j[r] = lo[r] + lane < hi[r] ? ld_nc(A.col + lo[r] + lane) : -1;
            a[r] = NUMERIC && j[r] >= 0 ? ld_nc(A.val + lo[r] + lane) : 0.f;
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
            b_lo[r] = len[r] = 0;
            if (j[r] >= 0) {
                b_lo[r] = ld_nc(B.rp + j[r]);
                len[r] = ld_nc(B.rp + j[r] + 1) - b_lo[r];
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) place(r, 0, b_lo[r], len[r], a[r]);
    } else {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            int base = 0;
            for (int32_t chunk = lo[r]; chunk < hi[r]; chunk += 32) {  // uniform across the warp
                int32_t b_lo = 0, len = 0;
                float a = 0.f;
                if (chunk + lane < hi[r]) {
                    const int32_t j = ld_nc(A.col + chunk + lane);
                    b_lo = ld_nc(B.rp + j);
                    len = ld_nc(B.rp + j + 1) - b_lo;
                    if (NUMERIC) a = ld_nc(A.val + chunk + lane);
                }
                base += place(r, base, b_lo, len, a);
            }
        }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
        if (i[r] < 0) continue;  // uniform
        if (!NUMERIC) {
            // distinct columns: a lane counts if it is the first of the lanes that hold its column
            const unsigned peers = __match_any_sync(FULL_MASK, have[r] ? my_col[r] : 0x80000000u | (uint32_t)lane);
            const unsigned firsts = __ballot_sync(FULL_MASK, have[r] && lane == __ffs(peers) - 1);
            if (lane == 0) row_count[i[r]] = __popc(firsts);
            continue;
        }
        uint32_t col;
        int src;
        bool valid;
        if (NARROW) {
            uint32_t key = have[r] ? ((my_col[r] << 5) | (uint32_t)lane) : ~0u;
            key = warp_bitonic_sort32(key);
            col = key >> 5;
            src = (int)(key & 31u);
            valid = key != ~0u;
        } else {
            uint64_t key = have[r] ? (((uint64_t)my_col[r] << 32) | (uint32_t)lane) : ~0ull;
            key = warp_bitonic_sort(key);
            col = (uint32_t)(key >> 32);
            src = (int)(key & 31u);
            valid = key != ~0ull;
        }
        const uint32_t prev_col = __shfl_up_sync(FULL_MASK, col, 1);
        const bool head = valid && (lane == 0 || prev_col != col);
        const unsigned heads = __ballot_sync(FULL_MASK, head);
        float v = __shfl_sync(FULL_MASK, my_val[r], src);  // value of the product now at this lane
        float acc = v;
        // longest run of equal columns in this row (distance from a head to the next head or to
        // the end of the valid lanes): the summation loop needs no more steps than that
        const unsigned later = lane < 31 ? (heads >> (lane + 1)) : 0u;
        const int n_valid = __popc(__ballot_sync(FULL_MASK, valid));
        const int my_run = head ? (later ? __ffs(later) : n_valid - lane) : 0;
        const int longest = __reduce_max_sync(FULL_MASK, my_run);
        for (int t = 1; t < longest; ++t) {  // head lanes add their run in sorted (= expansion) order
            const float nv = __shfl_down_sync(FULL_MASK, v, t);
            if (t < my_run) acc += nv;
        }
        if (head) {
            const int pos = out[r] + __popc(heads & ((1u << lane) - 1u));
            c_col[pos] = (int32_t)col;
            c_val[pos] = acc;
        }
    }
    finish_after_previous();
}

// ------------------------------------------------------------------------ medium rows ----

// One CTA per row with at most MEDIUM_P products: expand into shared memory in expansion
// order, bitonic sort on (column << 32 | expansion index), then each run head sums its run.
template <bool NUMERIC>
__global__ void __launch_bounds__(MED_NT) k_esc_medium(CsrView A, CsrView B, const int32_t *__restrict__ row_list,
                                                       int32_t *__restrict__ row_count, const int32_t *__restrict__ c_rp,
                                                       int32_t *__restrict__ c_col, float *__restrict__ c_val) {
    __shared__ uint64_t keys[MEDIUM_P];
    __shared__ float vals[NUMERIC ? MEDIUM_P : 1];
    __shared__ int seg_off[MED_NT], seg_start[MED_NT];
    __shared__ float seg_a[NUMERIC ? MED_NT : 1];
    __shared__ int scan_tmp[72];
    trigger_dependents();
    const int tid = threadIdx.x;
    const int32_t i = ld_nc(row_list + blockIdx.x);
    const int32_t lo = ld_nc(A.rp + i), hi = ld_nc(A.rp + i + 1);

    int p_total = 0, rows_of_b = 0;
    for (int32_t chunk = lo; chunk < hi; chunk += MED_NT) {  // expand phase 2, MED_NT entries of A at a time
        const int32_t e = chunk + tid;
        int32_t b_lo = 0, len = 0;
        float a = 0.f;
        if (e < hi) {
            const int32_t j = ld_nc(A.col + e);
            b_lo = ld_nc(B.rp + j);
            len = ld_nc(B.rp + j + 1) - b_lo;
            if (NUMERIC) a = ld_nc(A.val + e);
        }
        int k, off, n, chunk_total;
        block_excl_sum2<MED_NT>(len > 0 ? 1 : 0, len, scan_tmp, k, off, n, chunk_total);
        if (len > 0) {
            seg_off[k] = off;
            seg_start[k] = b_lo;
            if (NUMERIC) seg_a[k] = a;
        }
        __syncthreads();
        for (int p = tid; p < chunk_total; p += MED_NT) {  // thread = product: a long row of B is not one thread's work
            int seg = 0, above = n;
            while (above - seg > 1) {
                const int mid = (seg + above) >> 1;
                if (seg_off[mid] <= p) seg = mid; else above = mid;
            }
            const int32_t q = seg_start[seg] + (p - seg_off[seg]);
            const int idx = p_total + p;
            keys[idx] = ((uint64_t)(uint32_t)ld_nc(B.col + q) << 32) | (uint32_t)idx;
            if (NUMERIC) vals[idx] = seg_a[seg] * ld_nc(B.val + q);
        }
        p_total += chunk_total;
        rows_of_b += n;
        __syncthreads();
    }
    int n2 = 2;
    while (n2 < p_total) n2 <<= 1;
    for (int p = p_total + tid; p < n2; p += MED_NT) keys[p] = ~0ull;
    __syncthreads();

    for (int k = rows_of_b > 1 ? 2 : n2 + 1; k <= n2; k <<= 1) {  // sort (one row of B is in order)
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int p = tid; p < (n2 >> 1); p += MED_NT) {
                const int i1 = 2 * j * (p / j) + (p % j), i2 = i1 + j;
                const bool up = (i1 & k) == 0;
                const uint64_t x = keys[i1], y = keys[i2];
                if ((x > y) == up) {
                    keys[i1] = y;
                    keys[i2] = x;
                }
            }
            __syncthreads();
        }
    }

    // compress: thread t looks after sorted positions [t * per, (t + 1) * per)
    const int per = (n2 + MED_NT - 1) / MED_NT;
    const int p_lo = min(tid * per, p_total), p_hi = min(p_lo + per, p_total);
    int heads = 0;
    for (int p = p_lo; p < p_hi; ++p) heads += p == 0 || (uint32_t)(keys[p] >> 32) != (uint32_t)(keys[p - 1] >> 32);
    int unique;
    int rank = block_excl_sum<MED_NT>(heads, scan_tmp, unique);
    if (!NUMERIC && tid == 0) row_count[i] = unique;
    const int32_t out = NUMERIC ? ld_nc(c_rp + i) : 0;
    for (int p = p_lo; NUMERIC && p < p_hi; ++p) {
        const uint32_t col = (uint32_t)(keys[p] >> 32);
        if (p == 0 || col != (uint32_t)(keys[p - 1] >> 32)) {
            float acc = vals[(uint32_t)keys[p]];
            for (int q = p + 1; q < p_total && (uint32_t)(keys[q] >> 32) == col; ++q) acc += vals[(uint32_t)keys[q]];
            c_col[out + rank] = (int32_t)col;
            c_val[out + rank] = acc;
            ++rank;
        }
    }
    finish_after_previous();
}

// ----------------------------------------------------------------- product walk ----

// A warp takes FLIGHT times 32 products at a time, in pieces that lie in one row of B each: of LONG products where there
// are rows enough to keep the chip busy, because the broadcasts and addresses of a piece cost as much as 32 of its products
// (pieces of 32 took 33 instructions per 32 products in the symbolic pass of 32768 vertices' heavy rows, of 128 take 23);
// of SHORT products where there are few rows and the latency of each counts: the rows of B are then often shorter than LONG,
// and the loads of four of them are in flight together (whole calls on graphs of 2700 / 9000 vertices with SHORT pieces 98 / 229 us;
// with LONG ones such graphs took a seventh more).
constexpr int FLIGHT = 4, SHORT = 32, LONG = 32 * FLIGHT;

// The rows of B that a chunk of A's row selects, as segments: segment k covers the pieces [first[k], first[k + 1]) of
// the flat sequence of pieces, and its products are the entries start[k] .. start[k] + len[k] - 1 of B, each multiplied by
// a[k]. Only non-empty segments.
template <int NT>
struct Segments {
    int first[NT], start[NT], len[NT];
    float a[NT];
    int n, pieces;
};

// Lists the segments of the CTA's threads ({start, len, a} of the thread's entry of A; len 0: none). All NT threads; ends
// with a barrier. `tmp`: 72 ints.
template <int NT, int PIECE>
__device__ __forceinline__ void list_segments(Segments<NT> &seg, int *tmp, int32_t start, int len, float a) {
    int k, off, n, pieces;
    block_excl_sum2<NT>(len > 0 ? 1 : 0, (len + PIECE - 1) / PIECE, tmp, k, off, n, pieces);
    if (len > 0) {
        seg.first[k] = off;
        seg.start[k] = start;
        seg.len[k] = len;
        seg.a[k] = a;
    }
    if (threadIdx.x == 0) {
        seg.n = n;
        seg.pieces = pieces;
    }
    __syncthreads();
}

// Walks all products of the segments: f(what load(position in B) gives, a). Every warp takes one contiguous share of the
// pieces. For 32 pieces at a time every lane finds the segment of one of them by binary search; then the pieces go by one
// after the other, what their lane knows broadcast, lane = product, so that the loads from B coalesce and nothing diverges.
template <int NT, int PIECE, bool VALUES, typename Load, typename F>
__device__ __forceinline__ void walk_segments(const Segments<NT> &seg, Load load, F f) {
    constexpr int NW = NT / 32, TOGETHER = LONG / PIECE, EACH = PIECE / 32;  // pieces in flight, loads per lane of each
    const int lane = lane_id(), n_seg = seg.n, share = (seg.pieces + NW - 1) / NW;
    const int end = min((warp_id() + 1) * share, seg.pieces);
    for (int c = warp_id() * share; c < end; c += 32) {
        const int mine = min(c + lane, end - 1);
        int k = 0, above = n_seg;  // the last segment that begins at or before this lane's piece
        while (above - k > 1) {
            const int mid = (k + above) >> 1;
            if (seg.first[mid] <= mine) k = mid; else above = mid;
        }
        const int at = (mine - seg.first[k]) * PIECE;
        const int my_q = seg.start[k] + at, my_n = c + lane < end ? seg.len[k] - at : 0;
        const float my_a = VALUES ? seg.a[k] : 0.f;
        const int here = min(32, end - c);
        for (int u = 0; u < here; u += TOGETHER) {  // (u + t stays below 32; pieces past the share have n = 0)
            decltype(load(0)) x[FLIGHT];
            float a[TOGETHER];
            unsigned live = 0;
#pragma unroll
            for (int t = 0; t < TOGETHER; ++t) {
                const int q = __shfl_sync(FULL_MASK, my_q, u + t) + lane, n = __shfl_sync(FULL_MASK, my_n, u + t) - lane;
                a[t] = VALUES ? __shfl_sync(FULL_MASK, my_a, u + t) : 0.f;
#pragma unroll
                for (int j = 0; j < EACH; ++j)
                    if (32 * j < n) {
                        x[t * EACH + j] = load(q + 32 * j);
                        live |= 1u << (t * EACH + j);
                    }
            }
#pragma unroll
            for (int j = 0; j < FLIGHT; ++j)
                if ((live >> j) & 1u) f(x[j], a[j / EACH]);
        }
    }
}

// ------------------------------------------------------------- ranked and heavy rows ----
//
// Rows of more than MEDIUM_P products. The symbolic pass (k_esc_mark) sets a bit per produced column in a shared-memory
// bitmap and counts; its bitmaps are kept for the numeric pass (k_esc_rank), which turns them into the rank of every
// word's columns within the result row, writes the row's columns, walks the products and adds each one into its position.
// Matrices wider than one bitmap are walked in column windows.

constexpr int RK_WORDS = 8192;                     // bitmap words of one column window in shared memory
constexpr int RK_WINDOW_COLS = RK_WORDS * 32;      // 262144 columns per window
constexpr size_t RK_PTR_BUDGET = size_t(1) << 30;  // bytes of the window pointer table; beyond it windows are searched on the fly
constexpr int RK_NT = 256, HEAVY_NT = 512;         // threads of a symbolic CTA for rows up to / above RANKED_P products ...
// ... and up to RANKED_P where there are many, in windows of up to 131072 columns. A wider window's table takes 64 KB: rows of few results
// then share an SM better without sums beside it. (Products per row, result columns: 6000, 200000 907 us with the numeric pass by classes
// and the small symbolic CTAs, 685 without; 400, 400000 22.5 against 18.3 ms; 441 of a band, 200000 6.88 against 5.40; R-MAT graph of
// 262144 vertices with 16 / 4 edges each 18.4 against 17.0 and 3.64 against 3.16. Up to 131072 columns the classes win: 131072
// vertices 6.29 ms before them, 5.43.)
constexpr int MANY_NT = 128, MANY_ROWS = 8192, MANY_WORDS = 4096;

// Where the word w of a window lies in shared memory. The low bits of a graph's column numbers are far from uniform (in an
// R-MAT graph each is 0 three times in four, so a quarter of all words would lie in one bank; random look-ups with that skew
// take 8 cycles per warp instead of 3); folding the bits above into them spreads the banks. One to one on any power
// of two of words. FOLD false: in order, for the kernels of few rows, which wait for loads and not for banks.
template <bool FOLD>
__device__ __forceinline__ uint32_t spread(uint32_t w) { return FOLD ? w ^ (w >> 4) ^ (w >> 8) : w; }

// First index in [lo, hi) whose column is >= key (hi if none).
__device__ __forceinline__ int32_t first_col_at_least(const int32_t *__restrict__ col, int32_t lo, int32_t hi, int64_t key) {
    while (lo < hi) {
        const int32_t mid = lo + ((hi - lo) >> 1);
        if (ld_nc(col + mid) < key)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

// Window pointer table of B, built only for matrices wider than one window:
// ptr[j * (n_win + 1) + w] = first position of row j whose column is >= w * RK_WINDOW_COLS
// (w = 0 .. n_win), so that window w of row j is [ptr[w], ptr[w + 1]).
__global__ void __launch_bounds__(256) k_esc_window_ptr(CsrView B, int32_t b_rows, int n_win, int32_t *__restrict__ ptr) {
    const int64_t t = (int64_t)blockIdx.x * 256 + threadIdx.x;
    const int per = n_win + 1;
    if (t >= (int64_t)b_rows * per) return;
    const int32_t j = (int32_t)(t / per);
    const int w = (int)(t - (int64_t)j * per);
    const int32_t lo = ld_nc(B.rp + j), hi = ld_nc(B.rp + j + 1);
    ptr[t] = w == 0 ? lo : w == n_win ? hi : first_col_at_least(B.col, lo, hi, (int64_t)w * RK_WINDOW_COLS);
}

// Column windows of B: their number, and the window pointer table (null: one window, or a table beyond its budget).
struct Windows {
    int n;
    const int32_t *ptr;
    // The entries of row j whose columns lie in window w.
    __device__ __forceinline__ void range(const CsrView &B, int32_t j, int w, int32_t &start, int32_t &len) const {
        if (n == 1) {
            start = ld_nc(B.rp + j);
            len = ld_nc(B.rp + j + 1) - start;
        } else if (ptr) {
            const int64_t at = (int64_t)j * (n + 1) + w;
            start = ld_nc(ptr + at);
            len = ld_nc(ptr + at + 1) - start;
        } else {
            const int32_t b_lo = ld_nc(B.rp + j), b_hi = ld_nc(B.rp + j + 1), c_first = w * RK_WINDOW_COLS;
            start = w == 0 ? b_lo : first_col_at_least(B.col, b_lo, b_hi, c_first);
            len = (w == n - 1 ? b_hi : first_col_at_least(B.col, start, b_hi, (int64_t)c_first + RK_WINDOW_COLS)) - start;
        }
    }
};

// The entries of A's row and the walks over what they select, NT entries at a time (a thread keeps its entry where one
// chunk is all).
template <int NT, int PIECE, bool VALUES>
struct RowWalk {
    int32_t lo, hi, my_j = -1;
    float my_a = 0.f;
    __device__ __forceinline__ RowWalk(const CsrView &A, int32_t i) : lo(ld_nc(A.rp + i)), hi(ld_nc(A.rp + i + 1)) {
        if (one_chunk()) fetch(A, lo);
    }
    __device__ __forceinline__ bool one_chunk() const { return hi - lo <= NT; }
    __device__ __forceinline__ void fetch(const CsrView &A, int32_t chunk) {
        my_j = -1;
        if (chunk + (int)threadIdx.x >= hi) return;
        my_j = ld_nc(A.col + chunk + threadIdx.x);
        if (VALUES) my_a = ld_nc(A.val + chunk + threadIdx.x);
    }
    // range(j, start, len) gives the segment of an entry. `build` false: the segments of a single chunk are there already.
    // Returns whether there was any segment; ends with a barrier.
    template <typename Range, typename Load, typename F>
    __device__ __forceinline__ bool run(const CsrView &A, Segments<NT> &seg, int *tmp, bool build, Range range, Load load, F f) {
        bool any = false;
        for (int32_t chunk = lo; chunk < hi; chunk += NT) {
            if (build) {
                if (!one_chunk()) fetch(A, chunk);
                int32_t start = 0, len = 0;
                if (my_j >= 0) range(my_j, start, len);
                list_segments<NT, PIECE>(seg, tmp, start, len, my_a);
            }
            any |= seg.n > 0;
            walk_segments<NT, PIECE, VALUES>(seg, load, f);
            __syncthreads();  // the segment arrays are rewritten by the next chunk
        }
        return any;
    }
};

// Symbolic pass, one CTA per row: a bit per produced column, window by window, and their number. WORDS: the rows of B are
// walked as bitmap words (row_words.cuh), one window only. `row_list` is read from the front for the first n_front CTAs and from the back (list_len - 1
// downwards) for the others. `words`: bitmap words in use, a power of two of at least 128. `cache` (one window only), when
// given, receives the bitmaps, `words` per CTA, word w at place w.
//
// Bound by instructions and shared-memory wavefronts together; a pass over entries instead of words sets twice the bits.
template <int NT, int PIECE, bool WORDS>
__global__ void __launch_bounds__(NT, 1536 / NT) k_esc_mark(CsrView A, CsrView B, RowWords B_words, Windows windows, const int32_t *__restrict__ row_list,
                                                 int32_t list_len, int n_front, int words, uint4 *cache, int32_t *__restrict__ row_count) {
    extern __shared__ __align__(16) unsigned char rk_smem[];
    uint32_t *bitmap = reinterpret_cast<uint32_t *>(rk_smem);
    __shared__ Segments<NT> seg;
    __shared__ int scan_tmp[72];
    __shared__ int s_count;
    trigger_dependents();
    const int tid = threadIdx.x, r = blockIdx.x;
    const int32_t i = ld_nc(row_list + (r < n_front ? r : list_len - 1 - (r - n_front)));
    RowWalk<NT, PIECE, false> row(A, i);
    if (tid == 0) s_count = 0;
    int count = 0;
    for (int w = 0; w < windows.n; ++w) {
        const int32_t c_first = w * RK_WINDOW_COLS;  // below 2^31: it is a column of B
        for (int c = tid; c < words / 4; c += NT) reinterpret_cast<uint4 *>(bitmap)[c] = make_uint4(0u, 0u, 0u, 0u);
        __syncthreads();
        bool any;
        if (WORDS) {
            any = row.run(A, seg, scan_tmp, true, [&](int32_t j, int32_t &start, int32_t &len) {
                start = ld_nc(B_words.rp + j);
                len = ld_nc(B_words.rp + j + 1) - start;
            }, [&](int q) { return __ldg(B_words.items + q); }, [&](uint2 item, float) { atomicOr(bitmap + spread<PIECE == LONG>(item.x), item.y); });
        } else {
            any = row.run(A, seg, scan_tmp, true, [&](int32_t j, int32_t &start, int32_t &len) { windows.range(B, j, w, start, len); },
                          [&](int q) { return ld_nc(B.col + q); }, [&](int32_t col, float) {
                              const uint32_t cw = (uint32_t)(col - c_first);
                              atomicOr(bitmap + spread<PIECE == LONG>(cw >> 5), 1u << (cw & 31u));
                          });
        }
        if (!any) continue;  // uniform
        for (int q = tid; q < words / 4; q += NT) {
            uint4 v;
            v.x = bitmap[spread<PIECE == LONG>(4 * q)], v.y = bitmap[spread<PIECE == LONG>(4 * q + 1)], v.z = bitmap[spread<PIECE == LONG>(4 * q + 2)], v.w = bitmap[spread<PIECE == LONG>(4 * q + 3)];
            count += __popc(v.x) + __popc(v.y) + __popc(v.z) + __popc(v.w);
            if (cache) __stcs(cache + (size_t)r * (words / 4) + q, v);
        }
        __syncthreads();  // the next window clears the bitmap
    }
    count = __reduce_add_sync(FULL_MASK, count);
    if (lane_id() == 0 && count) atomicAdd(&s_count, count);
    __syncthreads();
    if (tid == 0) row_count[i] = s_count;
    finish_after_previous();
}

// The rows of the heavy and the ranked list, numbered through: heavy rows first (giant ones from the front of their list,
// the others from its back). The number is also the place of a row's bitmap.
struct ListedRows {
    const int32_t *heavy_rows, *ranked_rows;
    int32_t rows;  // length of the heavy list
    int n_giant, n_heavy, n;
    __device__ __forceinline__ int32_t row(int t) const {
        return t < n_giant ? ld_nc(heavy_rows + t) : t < n_heavy ? ld_nc(heavy_rows + rows - 1 - (t - n_giant)) : ld_nc(ranked_rows + (t - n_heavy));
    }
};

// The numeric pass takes its rows by the length of their results: a row's sums, four bytes per entry, should lie in shared
// memory (float32 atomics there run at 960 G per second, reductions in L2 at 182), and the shorter the rows the more CTAs
// share an SM. A class holds the rows whose results fit what its CTAs have beside the table of words; what does not fit the
// last one keeps the rest of its sums in L2.
struct RankClass {
    int nt, per_sm;       // threads of a CTA, CTAs of an SM
    size_t smem;          // dynamic shared memory of a CTA
    bool columns_walked;  // the walk of the products notes their columns, in shared memory too (below)
    int piece;
};
constexpr int CLASSES = 5, FEW = 5, FEW_HEAVY = 6;  // the last two: few rows, or windows too wide, for the rows to be sorted by class
constexpr RankClass RANK_CLASS[] = {{128, 8, 25 * 1024, true, LONG},  {256, 4, 50 * 1024, true, LONG},    {320, 3, 68 * 1024, true, LONG},   {512, 2, 104 * 1024, true, LONG},
                                    {1024, 1, 208 * 1024, false, LONG}, {256, 5, 0, false, SHORT}, {1024, 1, 208 * 1024, false, SHORT}};
constexpr int NARROW_WORDS = 2048;  // windows of up to 65536 columns: the table has 16 columns and their rank in 32 bits
// Sums of a CTA of class `cls` beside a table of `words` bitmap words.
constexpr int rank_slots(int cls, int words) {
    const bool narrow = words <= NARROW_WORDS;
    const size_t table = (size_t)words * 8, slot = !RANK_CLASS[cls].columns_walked ? 4 : narrow ? 6 : 8;
    return RANK_CLASS[cls].smem < table + 1024 ? 0 : (int)((RANK_CLASS[cls].smem - table) / slot) & ~1;
}

struct ClassSlots {
    int slots[CLASSES];
};
struct ClassCtl {
    int count[CLASSES], ticket[CLASSES];
};

// Puts the listed rows on the list of their class (`stride` apart): {row, place of its bitmap}, the heaviest first as far as
// the order of the CTAs goes.
__global__ void __launch_bounds__(256) k_esc_classes(ListedRows listed, const int32_t *__restrict__ c_rp, const ClassSlots most, int2 *__restrict__ out,
                                                     int64_t stride, ClassCtl *ctl) {
    __shared__ int s_count[CLASSES];
    if (threadIdx.x < CLASSES) s_count[threadIdx.x] = 0;
    __syncthreads();
    const int t = blockIdx.x * 256 + threadIdx.x;
    int cls = -1, at = 0;
    int32_t row = 0;
    if (t < listed.n) {
        row = listed.row(t);
        const int32_t length = ld_nc(c_rp + row + 1) - ld_nc(c_rp + row);
        cls = 0;
#pragma unroll
        for (int k = 0; k < CLASSES - 1; ++k) cls += length > most.slots[k] ? 1 : 0;  // slots grow with the class
        at = atomicAdd(&s_count[cls], 1);
    }
    __syncthreads();
    if (threadIdx.x < CLASSES && s_count[threadIdx.x] > 0) s_count[threadIdx.x] = atomicAdd(&ctl->count[threadIdx.x], s_count[threadIdx.x]);
    __syncthreads();
    if (cls >= 0) out[cls * stride + s_count[cls] + at] = make_int2(row, t);
}

// Column and value of every entry of B side by side: a product of the numeric pass is one 8-byte load.
__global__ void __launch_bounds__(256) k_esc_pairs(const int32_t *__restrict__ rp, const int32_t *__restrict__ col, const float *__restrict__ val, int32_t nnz,
                                                   uint2 *__restrict__ pairs) {
    const int64_t p = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (p >= nnz) return;
    const int64_t at = (int64_t)ld_nc(rp) + p;
    pairs[p] = make_uint2((uint32_t)ld_nc(col + at), __float_as_uint(ld_nc(val + at)));
}

// The columns of a window and their ranks, by bitmap words, in one of three forms:
//   HALVES  16 columns in the lower half of a 32-bit word, the number of columns before them in the upper one (a look-up is one 4-byte
//           load: 3 cycles of the shared-memory pipe for random words against 5 for 8 bytes); windows of up to 65536 columns
//   PAIRS   32 columns and their rank in 64 bits
//   SPLIT   the words, and behind them 16 bits of rank for each: 6 bytes where the others take 8, so that four CTAs instead of three
//           have room for the widest window on an SM, and half as much to empty; rows of at most 65535 products
enum Table { HALVES, PAIRS, SPLIT };
template <Table KIND, bool FOLD>
struct RankTable {
    static_assert(KIND != SPLIT || !FOLD, "the words of a split table lie in order");
    unsigned char *at;
    int words;
    static __host__ __device__ constexpr size_t bytes(int words) { return (size_t)words * (KIND == SPLIT ? 6 : 8); }
    __device__ __forceinline__ uint32_t &half(uint32_t h) const { return reinterpret_cast<uint32_t *>(at)[FOLD ? h ^ (h >> 5) ^ (h >> 10) : h]; }
    __device__ __forceinline__ uint2 &full(uint32_t w) const { return reinterpret_cast<uint2 *>(at)[spread<FOLD>(w)]; }
    __device__ __forceinline__ uint16_t *ranks() const { return reinterpret_cast<uint16_t *>(at + 4 * (size_t)words); }
    // Empties what mark() writes into.
    template <int NT>
    __device__ __forceinline__ void clear() const {
        for (int c = threadIdx.x; c < words / (KIND == SPLIT ? 4 : 2); c += NT) reinterpret_cast<uint4 *>(at)[c] = make_uint4(0u, 0u, 0u, 0u);
    }
    __device__ __forceinline__ void mark(uint32_t cw) const {  // column cw of the window
        if (KIND == HALVES) atomicOr(&half(cw >> 4), 1u << (cw & 15u));
        else if (KIND == PAIRS) atomicOr(&full(cw >> 5).x, 1u << (cw & 31u));
        else atomicOr(reinterpret_cast<uint32_t *>(at) + (cw >> 5), 1u << (cw & 31u));
    }
    // Word w of a marked table, and the same with `rank` columns before it.
    __device__ __forceinline__ uint32_t marked(uint32_t w) const { return KIND == HALVES ? half(2 * w) | half(2 * w + 1) << 16 : full(w).x; }
    __device__ __forceinline__ void put(uint32_t w, uint32_t bits, uint32_t rank) const {
        if (KIND == HALVES) {
            half(2 * w) = (bits & 0xffffu) | rank << 16;
            half(2 * w + 1) = bits >> 16 | (rank + __popc(bits & 0xffffu)) << 16;
        } else {
            full(w) = make_uint2(bits, rank);
        }
    }
    // The words 4 q to 4 q + 3 of a table in order, 16 bytes at a time: the lanes of a warp take neighbouring ones.
    __device__ __forceinline__ uint4 marked4(uint32_t q) const {
        const uint4 *from = reinterpret_cast<const uint4 *>(at);
        if (KIND == SPLIT) return from[q];
        const uint4 lo = from[2 * q], hi = from[2 * q + 1];
        return KIND == HALVES ? make_uint4(lo.x | lo.y << 16, lo.z | lo.w << 16, hi.x | hi.y << 16, hi.z | hi.w << 16) : make_uint4(lo.x, lo.z, hi.x, hi.z);
    }
    __device__ __forceinline__ void put4(uint32_t q, uint4 v, uint32_t rank) const {
        const uint32_t r1 = rank + __popc(v.x), r2 = r1 + __popc(v.y), r3 = r2 + __popc(v.z);
        uint4 *to = reinterpret_cast<uint4 *>(at);
        if (KIND == SPLIT) {
            to[q] = v;
            reinterpret_cast<uint2 *>(ranks())[q] = make_uint2(rank | r1 << 16, r2 | r3 << 16);
        } else if (KIND == HALVES) {
            auto lower = [](uint32_t bits, uint32_t r) { return (bits & 0xffffu) | r << 16; };
            auto upper = [](uint32_t bits, uint32_t r) { return bits >> 16 | (r + __popc(bits & 0xffffu)) << 16; };
            to[2 * q] = make_uint4(lower(v.x, rank), upper(v.x, rank), lower(v.y, r1), upper(v.y, r1));
            to[2 * q + 1] = make_uint4(lower(v.z, r2), upper(v.z, r2), lower(v.w, r3), upper(v.w, r3));
        } else {
            to[2 * q] = make_uint4(v.x, rank, v.y, r1);
            to[2 * q + 1] = make_uint4(v.z, r2, v.w, r3);
        }
    }
    // columns up to and with cw, which is one of them: its position plus one
    __device__ __forceinline__ uint32_t find(uint32_t cw) const {
        if (KIND == HALVES) {
            const uint32_t e = half(cw >> 4);
            return (e >> 16) + __popc(e << (31u - (cw & 15u)));
        }
        if (KIND == SPLIT) return (uint32_t)ranks()[cw >> 5] + __popc(reinterpret_cast<const uint32_t *>(at)[cw >> 5] << (~cw & 31u));
        const uint2 e = full(cw >> 5);
        return e.y + __popc(e.x << (~cw & 31u));
    }
};

// Numeric pass, one CTA per row: CTAs take the rows of a class from a ticket; where rows are not sorted by class, CTA t takes
// the listed row first + t. Per window the row's bitmap, from the symbolic pass's store or from a walk of its own, becomes the table
// of ranks; the products are walked and each one added into its position: a look-up, a popcount and an atomic. Positions beyond
// `acc_slots` (last class; all of them where there are few rows, which the latency of shared-memory atomics would hold up) take a float32
// reduction in L2 on the row's own output range, which this CTA zeroed first. The columns are noted by the products themselves
// (WALKED) or written out of the bitmap into the place of the sums before the walk; both ways they are stored coalesced. (Out of the
// bitmap every lane loops over the bits of its words, and a warp over those of its densest: rows of up to 6144 entries spent a
// third of their instructions there. The longest rows, 7 products per entry, still do it.)
//
// `pairs`: B's entries as {column, value}, or null. What bounds it is the shared-memory pipe beside latency: per 32 products 3
// cycles for the pairs, 3 for the look-up, 3 for noting the column, 10 for the atomic, of 28 to 34 that it takes at 32 to
// 40 warps per SM. R-MAT graph of 65536 vertices times its transpose (403 M products): both passes of these rows 2.2 ms with entries
// instead of words in the symbolic one, 5120 sums in shared memory and the others in L2, columns out of the bitmap; 1.5 ms now.
template <int CLS, Table KIND, bool BY_PAIR>
__global__ void __launch_bounds__(RANK_CLASS[CLS].nt, RANK_CLASS[CLS].per_sm)
    k_esc_rank(CsrView A, CsrView B, const uint2 *pairs, Windows windows, ListedRows listed, int first, int last, const int2 *list, ClassCtl *ctl, int words,
               int acc_slots, const uint4 *cache, const int32_t *__restrict__ c_rp, int32_t *__restrict__ c_col, float *__restrict__ c_val) {
    constexpr RankClass K = RANK_CLASS[CLS];
    constexpr int NT = K.nt;
    constexpr bool WALKED = K.columns_walked, BY_CLASS = CLS < CLASSES, IN_L2 = K.smem == 0;
    using Col = typename std::conditional<KIND == HALVES, uint16_t, uint32_t>::type;
    extern __shared__ __align__(16) unsigned char rk_smem[];
    const RankTable<KIND, K.piece == LONG> table{rk_smem, words};
    float *acc = reinterpret_cast<float *>(rk_smem + table.bytes(words));
    int32_t *stage = reinterpret_cast<int32_t *>(acc);
    Col *noted = reinterpret_cast<Col *>(acc + acc_slots);  // WALKED
    __shared__ Segments<NT> seg;
    __shared__ int scan_tmp[72];
    __shared__ int s_next;
    trigger_dependents();
    const int tid = threadIdx.x, count = BY_CLASS ? ctl->count[BY_CLASS ? CLS : 0] : last;
    const int quads = words / 4;
    const int32_t b_base = BY_PAIR ? ld_nc(B.rp) : 0;
    auto load = [&](int q) -> uint2 {
        return BY_PAIR ? __ldg(pairs + (q - b_base)) : make_uint2((uint32_t)ld_nc(B.col + q), __float_as_uint(ld_nc(B.val + q)));
    };
    if (BY_CLASS) {
        if (tid == 0) s_next = atomicAdd(&ctl->ticket[BY_CLASS ? CLS : 0], 1);
        __syncthreads();
    }
    for (;;) {
        const int r = BY_CLASS ? s_next : first + (int)blockIdx.x;
        if (r >= count) break;  // uniform
        int next = count;
        if (BY_CLASS && tid == 0) next = atomicAdd(&ctl->ticket[BY_CLASS ? CLS : 0], 1);
        const int2 at = BY_CLASS ? list[r] : make_int2(listed.row(r), r);
        const int32_t i = at.x;
        RowWalk<NT, K.piece, true> row(A, i);
        int64_t out = ld_nc(c_rp + i);  // next free position of the row
        for (int w = 0; w < windows.n; ++w) {
            const int32_t c_first = w * RK_WINDOW_COLS;  // below 2^31: it is a column of B
            auto range = [&](int32_t j, int32_t &start, int32_t &len) { windows.range(B, j, w, start, len); };
            const uint4 *from = cache ? cache + (size_t)at.y * quads : nullptr;
            auto write_columns = [&](int c, uint32_t bits, int &rank, int cnt) {  // of word c
                const int32_t col0 = c_first + c * 32 - 1;
                if (!IN_L2 && cnt <= acc_slots) {
                    for (; bits; bits &= bits - 1u) stage[rank++] = col0 + __ffs((int)bits);
                } else {
                    for (; bits; bits &= bits - 1u) c_col[out + rank++] = col0 + __ffs((int)bits);
                }
            };
            if (!cache) {
                table.template clear<NT>();
                __syncthreads();
                const bool any = row.run(A, seg, scan_tmp, true, range, [&](int q) { return ld_nc(B.col + q); },
                                         [&](int32_t col, float) { table.mark((uint32_t)(col - c_first)); });
                if (!any) continue;  // uniform
            }
            int cnt;
            if constexpr (BY_CLASS) {  // neighbouring words fall to one thread; the fold keeps them off one another's banks
                const int per = quads >= NT ? 4 * ((quads + NT - 1) / NT) : (words + NT - 1) / NT;
                const int w_lo = min(tid * per, words), w_hi = min(w_lo + per, words);
                auto each_word = [&](auto f) {  // f(word, bits) for the thread's words
                    if (!cache) {
                        for (int c = w_lo; c < w_hi; ++c) f(c, table.marked(c));
                    } else if (quads >= NT) {
                        for (int c = w_lo; c < w_hi; c += 4) {
                            const uint4 v = __ldg(from + c / 4);
                            f(c, v.x), f(c + 1, v.y), f(c + 2, v.z), f(c + 3, v.w);
                        }
                    } else {
                        for (int c = w_lo; c < w_hi; ++c) f(c, __ldg(reinterpret_cast<const uint32_t *>(from) + c));
                    }
                };
                int mine = 0;
                each_word([&](int, uint32_t bits) { mine += __popc(bits); });
                int rank = block_excl_sum<NT>(mine, scan_tmp, cnt);
                each_word([&](int c, uint32_t bits) {
                    table.put(c, bits, rank);
                    if (WALKED) rank += __popc(bits);
                    else write_columns(c, bits, rank, cnt);
                });
            } else {
                // A warp looks after a run of neighbouring words, four to a lane and step: the loads of a step are one piece of memory,
                // and its stores meet a bank twice at most. (With a run of words to a thread, as above, those of the widest window lay
                // 32 to a bank: 2000 rows of 20000 products in 2 M columns 1968 us a call, 1017 like this, 782 with six bytes to a word.)
                const int share = (quads + NT - 1) / NT * 32;
                const int q_lo = min(warp_id() * share, quads) + lane_id(), q_hi = min((warp_id() + 1) * share, quads);
                auto fetch = [&](int q) { return q >= q_hi ? make_uint4(0u, 0u, 0u, 0u) : cache ? __ldg(from + q) : table.marked4(q); };
                auto columns = [](uint4 v) { return __popc(v.x) + __popc(v.y) + __popc(v.z) + __popc(v.w); };
                const uint4 held = fetch(q_lo);  // the first step's words are not fetched again
                int mine = columns(held);
                for (int q = q_lo + 32; q < q_hi; q += 32) mine += columns(fetch(q));
                int run = __shfl_sync(FULL_MASK, block_excl_sum<NT>(mine, scan_tmp, cnt), 0);  // columns before the step's
                for (int q = q_lo; q - lane_id() < q_hi; q += 32) {
                    const uint4 v = q == q_lo ? held : fetch(q);
                    const int here = columns(v), incl = warp_incl_sum(here);
                    int rank = run + incl - here;
                    run += __shfl_sync(FULL_MASK, incl, 31);
                    if (q >= q_hi) continue;
                    table.put4(q, v, rank);
                    write_columns(4 * q, v.x, rank, cnt), write_columns(4 * q + 1, v.y, rank, cnt);
                    write_columns(4 * q + 2, v.z, rank, cnt), write_columns(4 * q + 3, v.w, rank, cnt);
                }
            }
            const bool fits = !IN_L2 && cnt <= acc_slots;
            if (!WALKED && !IN_L2) __syncthreads();
            float *row_val = c_val + out;  // the window's part of the row; its length fits 32 bits
            const int in_acc = IN_L2 ? 0 : min(cnt, acc_slots);
            for (int k = tid; k < in_acc; k += NT) {
                if (!WALKED && fits) c_col[out + k] = stage[k];
                acc[k] = 0.f;
            }
            if (!WALKED) for (int k = (IN_L2 ? 0 : acc_slots) + tid; k < cnt; k += NT) row_val[k] = 0.f;  // positions beyond the shared sums
            __syncthreads();  // table complete, sums zeroed (the reductions below come from this CTA only)
            row.run(A, seg, scan_tmp, cache || !row.one_chunk(), range, load, [&](uint2 product, float a) {
                const uint32_t cw = product.x - (uint32_t)c_first, to = table.find(cw) - 1;
                const float v = a * __uint_as_float(product.y);
                if (WALKED) noted[to] = (Col)cw;
                if (WALKED || (!IN_L2 && to < (uint32_t)acc_slots)) atomicAdd(acc + to, v);
                else atomicAdd(row_val + to, v);  // reduction in L2
            });
            // the pass ends with a barrier: every sum is in place
            for (int k = tid; k < in_acc; k += NT) {
                if (WALKED) c_col[out + k] = c_first + (int32_t)noted[k];
                row_val[k] = acc[k];
            }
            out += cnt;
        }
        if (!BY_CLASS) break;
        if (tid == 0) s_next = next;
        __syncthreads();  // also: this row's sums are stored before the next row's take their place
    }
    finish_after_previous();
}

// ------------------------------------------------------------- matrices of short rows ----

constexpr int SHORT_NT = 128, SHORT_ENTRIES = 8;

// The whole product in one pass, for matrices whose rows of A hold at most K <= 8 entries and reach at
// most SMALL_P products (meshes, bands). One THREAD merges one row: the K rows of B are sorted lists whose
// heads it keeps in registers, with the entry behind each (the steps are bound by the latency of these loads, at the
// 24 warps per SM that the staging leaves); a step takes the smallest head and adds up the lists that hold it, in the
// order of A's entries (ascending j, the same sum as the other kernels form). A row is staged in shared memory
// at the offset of its product count, the CTA's result count goes through the cross-tile scan of the merge
// kernels, and the rows are copied out eight lanes to a row. 512 x 512 5-point mesh squared: a warp per row with
// a 32-wide bitonic sort, counting first, took 240 instructions a row and 156 us in two kernels; without the entry
// behind each head this one took 49 us, with it 44.
template <int K>
__global__ void __launch_bounds__(SHORT_NT) k_esc_short(CsrView A, CsrView B, int32_t rows, TileWords words, FusedCtl *ctl, int num_tiles,
                                                       int32_t *__restrict__ c_rp, int32_t *__restrict__ c_col, float *__restrict__ c_val,
                                                       unsigned long long *word) {
    constexpr uint32_t END = 0xffffffffu;
    __shared__ uint32_t s_col[SHORT_NT * SMALL_P];
    __shared__ float s_val[SHORT_NT * SMALL_P];
    __shared__ int scan_tmp[40];
    __shared__ long long s_base;
    const int t = blockIdx.x, tid = threadIdx.x, lane = lane_id();
    const int64_t i = (int64_t)t * SHORT_NT + tid;
    const int32_t lo = i < rows ? ld_nc(A.rp + i) : 0, hi = i < rows ? ld_nc(A.rp + i + 1) : 0;
    uint32_t pos[K], end[K];  // one past the last entry of 2^31 - 1 is still a position
    uint32_t head[K], next[K];
    float a[K], head_val[K], next_val[K];
    int products = 0;
#pragma unroll
    for (int e = 0; e < K; ++e) {
        const int32_t j = lo + e < hi ? ld_nc(A.col + lo + e) : -1;
        a[e] = j >= 0 ? ld_nc(A.val + lo + e) : 0.f;
        pos[e] = j >= 0 ? ld_nc(B.rp + j) : 0;
        end[e] = j >= 0 ? ld_nc(B.rp + j + 1) : 0;
        products += end[e] - pos[e];
    }
#pragma unroll
    for (int e = 0; e < K; ++e) {
        auto fetch = [&](uint32_t q, uint32_t &col, float &val) {
            col = q < end[e] ? (uint32_t)ld_nc(B.col + q) : END;
            val = q < end[e] ? ld_nc(B.val + q) : 0.f;
        };
        fetch(pos[e], head[e], head_val[e]);
        fetch(++pos[e], next[e], next_val[e]);  // from here on pos is that of `next`
    }
    int tile_products;
    const int staged = block_excl_sum<SHORT_NT>(products, scan_tmp, tile_products);
    int count = 0;
    for (;;) {
        uint32_t m = head[0];
#pragma unroll
        for (int e = 1; e < K; ++e) m = min(m, head[e]);
        if (m == END) break;
        float acc = 0.f;
        bool first = true;
#pragma unroll
        for (int e = 0; e < K; ++e) {
            if (head[e] == m) {
                const float v = a[e] * head_val[e];
                acc = first ? v : acc + v;
                first = false;
                head[e] = next[e];
                head_val[e] = next_val[e];
                if (++pos[e] < end[e]) {
                    next[e] = (uint32_t)ld_nc(B.col + pos[e]);
                    next_val[e] = ld_nc(B.val + pos[e]);
                } else {
                    next[e] = END;
                }
            }
        }
        s_col[staged + count] = m;
        s_val[staged + count] = acc;
        ++count;
    }
    int total;
    const int rank = block_excl_sum<SHORT_NT>(count, scan_tmp, total);
    if (tid == 0) publish_count(words, t, total);
    if (warp_id() == 0) {
        const int64_t b = tile_base(words, t, total, &ctl->status, LOOKBACK_POLL_LIMIT);
        if (lane == 0) {
            s_base = b;
            if (t == num_tiles - 1) publish_result_word(word, b < 0 ? NB200_E_TIMEOUT : NB200_OK, b < 0 ? 0 : b + total);
        }
    }
    __syncthreads();
    const long long base = s_base;
    if (base < 0) return;  // a bounded wait gave up; the host reports it
    if (i < rows) c_rp[i] = (int32_t)(base + rank);
    if (t == num_tiles - 1 && tid == 0) c_rp[rows] = (int32_t)(base + total);
#pragma unroll
    for (int s = 0; s < 8; ++s) {
        const int r = 4 * s + (lane >> 3);
        const int n = __shfl_sync(FULL_MASK, count, r), from = __shfl_sync(FULL_MASK, staged, r), to = __shfl_sync(FULL_MASK, rank, r);
        for (int q = lane & 7; q < n; q += 8) {
            c_col[base + to + q] = (int32_t)s_col[from + q];
            c_val[base + to + q] = s_val[from + q];
        }
    }
}

// ------------------------------------------------------------------------ host driver ----

// Bitmap words of a row for B's column count (one window's worth at most): a power of two.
int ranked_words(int32_t b_cols) {
    const int64_t need = (std::min<int64_t>(b_cols, RK_WINDOW_COLS) + 31) / 32;
    int words = 128;
    while (words < need) words *= 2;
    return words;
}

int check_operand(const nb200_csr *m) {
    if (!m || m->rows < 0 || m->cols < 0 || m->nnz < 0 || !m->row_ptr) return NB200_E_BADARG;
    if (m->nnz > 0 && (!m->col || !m->val)) return NB200_E_BADARG;
    return NB200_OK;
}

struct EscPlan {
    Workspace *ws;
    RowLists lists;
    int32_t *row_count;    // rows entries (symbolic pass)
    uint64_t *scan_block;  // FusedCtl + one word per scan CTA
    int scan_ctas;
    EscCtl *ctl;
    int n_win;             // column windows of RK_WINDOW_COLS
    int32_t *win_ptr;      // window pointer table (null: one window, or beyond its budget)
    int words;             // bitmap words of a row in a window
    uint4 *cache;          // bitmaps carried from the symbolic to the numeric pass, heavy rows first (or null)
    int2 *class_rows;      // rows of every class, as many apart as there are rows above MEDIUM_P products (null: not sorted by class)
    ClassCtl *classes;
    RowWords b_words;      // rows of B as bitmap words for the symbolic pass (or null)
    Workspace *cache_ws;   // pool block of the bitmaps (null without them)
    EscCtl host;           // counters reported by the binning kernel
    uint64_t *short_block; // FusedCtl + tile words of the short-row kernel
    int short_tiles;
    unsigned long long *result;  // result words
};

bool many_rows(int64_t listed, int words) { return listed >= MANY_ROWS && words <= MANY_WORDS; }

// Another form of B is made for products that read every entry of it this often, and of which there are this many: its words take
// four short launches (some 25 us with nothing beside them, and 11 per million entries), its pairs one of 9. A graph of 24405 vertices, 49 M
// products: the whole call 468 -> 357 us with both and the classes; of 9000 vertices, 7 M products, it would take 20 us more. How
// much the words save depends on how the columns lie together, which is not known before they are made: the entries of a band,
// read 41 times each, 2514 -> 2175 us a call; scattered ones, read 23 to 30 times, cost 4 to 5 % (9000 rows of 6000 products, 130000
// columns: 493 us with, 470 without).
constexpr unsigned long long PAIRS_REUSE = 16, WORDS_REUSE = 32, FORMS_FROM = 32 << 20;
constexpr int WORDS_SLOT = 4, PAIRS_SLOT = 5;  // their pool blocks
constexpr size_t BITMAP_CACHE_BUDGET = size_t(8) << 30;  // bytes of bitmaps carried between the passes of one call

// Bins the rows (kernel + one read-back) and carves the scratch of a symbolic pass, a numeric
// pass, or one after the other. `counts`: rows without products get their count written
// (needed by the symbolic pass).
int esc_prepare(const nb200_csr *a, const nb200_csr *b, bool counts, bool carry_bitmaps, cudaStream_t stream, EscPlan *plan) {
    const int32_t rows = a->rows;
    const int64_t n_win = std::max<int64_t>(1, ((int64_t)b->cols + RK_WINDOW_COLS - 1) / RK_WINDOW_COLS);
    const size_t ptr_entries = n_win > 1 ? (size_t)b->rows * (size_t)(n_win + 1) : 0;
    const bool with_table = ptr_entries > 0 && ptr_entries * 4 <= RK_PTR_BUDGET;
    const int scan_ctas = (int)(((int64_t)rows + 1 + SCAN_NT * SCAN_VT - 1) / (SCAN_NT * SCAN_VT));
    Carver sizes;
    for (int q = 0; q < 4; ++q) sizes.take<int32_t>((size_t)rows);
    sizes.take<int32_t>((size_t)rows + 1);
    sizes.take<ClassCtl>(1);
    if (with_table) sizes.take<int32_t>(ptr_entries);
    const int prefix_ctas = (int)(((int64_t)a->nnz + 1 + 2047) / 2048);
    const int short_tiles = (int)(((int64_t)rows + SHORT_NT - 1) / SHORT_NT);
    sizes.take<unsigned long long>((size_t)a->nnz + 1);
    const size_t clear_from = sizes.used();
    sizes.take<uint64_t>((size_t)scan_ctas + 8);
    sizes.take<EscCtl>(1);
    sizes.take<uint64_t>((size_t)prefix_ctas + 8);
    sizes.take<uint64_t>(TileWords::needed(short_tiles) + 4);
    int st;
    if ((st = acquire_workspace(stream, sizes.used(), &plan->ws))) return st;
    Carver carve(plan->ws->dev);
    plan->lists.small_rows = carve.take<int32_t>((size_t)rows);
    plan->lists.medium_rows = carve.take<int32_t>((size_t)rows);
    plan->lists.ranked_rows = carve.take<int32_t>((size_t)rows);
    plan->lists.heavy_rows = carve.take<int32_t>((size_t)rows);
    plan->row_count = carve.take<int32_t>((size_t)rows + 1);
    plan->classes = carve.take<ClassCtl>(1);
    plan->n_win = (int)n_win;
    plan->words = ranked_words(b->cols);
    plan->win_ptr = with_table ? carve.take<int32_t>(ptr_entries) : nullptr;
    unsigned long long *prefix = carve.take<unsigned long long>((size_t)a->nnz + 1);
    plan->scan_block = carve.take<uint64_t>((size_t)scan_ctas + 8);
    plan->scan_ctas = scan_ctas;
    plan->ctl = carve.take<EscCtl>(1);
    uint64_t *prefix_block = carve.take<uint64_t>((size_t)prefix_ctas + 8);
    plan->short_block = carve.take<uint64_t>(TileWords::needed(short_tiles) + 4);
    plan->short_tiles = short_tiles;
    plan->result = result_word(plan->ws, 0);
    for (int k = 1; k < W_COUNT; ++k) result_word(plan->ws, k);

    // every control block and tile word of the call lies in one piece: one fill clears them all
    NB200_CUDA(cudaMemsetAsync(static_cast<unsigned char *>(plan->ws->dev) + clear_from, 0, carve.used() - clear_from, stream));
    plan->host = EscCtl{};
    const CsrView A{a->row_ptr, a->col, a->val}, B{b->row_ptr, b->col, b->val};
    const bool short_rows = (int64_t)a->nnz <= 8 * (int64_t)rows;  // then a lane walks its row faster than a prefix pass pays
    if (rows > 0 && short_rows) {
        LaunchScope scope("esc_rowwork", stream);
        k_esc_rowwork_walk<<<(rows + 255) / 256, 256, 0, stream>>>(A, B, rows, counts ? plan->row_count : nullptr, plan->lists, plan->ctl, plan->result);
        NB200_CUDA(cudaGetLastError());
    } else if (rows > 0) {
        {
            LaunchScope scope("esc_product_prefix", stream);
            k_esc_product_prefix<<<prefix_ctas, 256, 0, stream>>>(A, B, a->nnz, prefix, prefix_block + 4, reinterpret_cast<FusedCtl *>(prefix_block));
        }
        LaunchScope scope("esc_rowwork", stream);
        NB200_CUDA(launch_overlapped(k_esc_rowwork, dim3((rows + 255) / 256), dim3(256), 0, stream, A, prefix, rows, counts ? plan->row_count : nullptr,
                                     plan->lists, plan->ctl, reinterpret_cast<const FusedCtl *>(prefix_block), plan->result));
    }
    if (rows > 0) {
        int64_t v[W_NNZ];
        int device_status = 0, failed = 0;
        for (int k = 0; k < W_NNZ; ++k) {
            if ((st = wait_result_word(plan->result + k, stream, &v[k], &device_status))) return st;
            failed |= device_status;
        }
        // a prefix whose look-back gave up leaves rows with wrong product counts: nothing may be built on them
        if (failed) return note_timeout(ERR_LOOKBACK_TIMEOUT, 0, "spgemm product prefix");
        plan->host.products = (unsigned long long)v[W_PRODUCTS];
        plan->host.n_rows[BIN_SMALL] = (int)v[W_SMALL], plan->host.n_rows[BIN_MEDIUM] = (int)v[W_MEDIUM], plan->host.n_rows[BIN_RANKED] = (int)v[W_RANKED];
        plan->host.n_rows[BIN_GIANT] = (int)v[W_GIANT], plan->host.n_rows[BIN_HEAVY] = (int)v[W_HEAVY];
        plan->host.max_entries = short_rows ? (int)v[W_ENTRIES] : INT_MAX;
    }
    if (with_table && plan->host.n_rows[BIN_RANKED] + plan->host.n_rows[BIN_GIANT] + plan->host.n_rows[BIN_HEAVY] > 0) {
        LaunchScope scope("esc_window_ptr", stream);
        k_esc_window_ptr<<<(unsigned)((ptr_entries + 255) / 256), 256, 0, stream>>>(B, b->rows, plan->n_win, plan->win_ptr);
        NB200_CUDA(cudaGetLastError());
    }
    plan->cache = nullptr;
    plan->cache_ws = nullptr;
    plan->b_words = RowWords{};
    plan->class_rows = nullptr;
    const int64_t listed = (int64_t)plan->host.n_rows[BIN_RANKED] + plan->host.n_rows[BIN_GIANT] + plan->host.n_rows[BIN_HEAVY];
    if (listed > 0) {
        // a second pool block: its size is only known now, and the first must not move
        const size_t bitmap_bytes = (size_t)listed * plan->words * 4;
        const bool many = many_rows(listed, plan->words), carry = carry_bitmaps && plan->n_win == 1 && bitmap_bytes <= BITMAP_CACHE_BUDGET;
        auto carve_rows = [&](Carver &c) {
            if (many) plan->class_rows = c.take<int2>((size_t)CLASSES * listed);
            if (carry) plan->cache = c.take<uint4>(bitmap_bytes / 16);
        };
        Carver row_sizes;
        carve_rows(row_sizes);
        Workspace *row_ws = nullptr;
        const int row_st = many || carry ? acquire_workspace(stream, row_sizes.used(), &row_ws, 3) : NB200_E_NOMEM;
        if (row_st == NB200_OK) {
            Carver row_carve(row_ws->dev);
            carve_rows(row_carve);
            plan->cache_ws = row_ws;
        } else if (row_st != NB200_E_NOMEM) {
            return row_st;
        }  // without room the numeric pass walks the products twice, as it does on its own, and takes all rows in one launch
    }
    if (listed > 0 && counts && plan->n_win == 1 && plan->host.products >= FORMS_FROM && plan->host.products >= WORDS_REUSE * (unsigned long long)b->nnz) {
        size_t clear_from, clear_bytes;
        Carver word_sizes;
        RowWordsScratch::carve(word_sizes, b->rows, b->nnz, &clear_from, &clear_bytes);
        Workspace *word_ws = nullptr;
        const int word_st = acquire_workspace(stream, word_sizes.used(), &word_ws, WORDS_SLOT);
        if (word_st == NB200_OK) {  // without room the entries are walked
            Carver word_carve(word_ws->dev);
            const RowWordsScratch scratch = RowWordsScratch::carve(word_carve, b->rows, b->nnz, &clear_from, &clear_bytes);
            NB200_CUDA(cudaMemsetAsync(static_cast<unsigned char *>(word_ws->dev) + clear_from, 0, clear_bytes, stream));
            // a give-up is reported by the scan that ends the symbolic pass
            NB200_CUDA(build_row_words(b->row_ptr, b->col, b->rows, b->nnz, scratch, reinterpret_cast<FusedCtl *>(plan->scan_block), stream));
            plan->b_words = scratch.out;
        } else if (word_st != NB200_E_NOMEM) {
            return word_st;
        }
    }
    return NB200_OK;
}

// The bins of a pass touch different rows, so each kernel after the first starts beside the one before it
// (a few hub rows on as many CTAs would otherwise leave the rest of the chip idle: 16 of them took 150 us of
// 780 on a graph of 24405 vertices).
template <typename... P, typename... V>
int launch_bin(bool beside, void (*kernel)(P...), int grid, int block, size_t smem, cudaStream_t stream, V... args) {
    if (beside) {
        NB200_CUDA(launch_overlapped(kernel, dim3(grid), dim3(block), smem, stream, args...));
    } else {
        kernel<<<grid, block, smem, stream>>>(args...);
        NB200_CUDA(cudaGetLastError());
    }
    return NB200_OK;
}

template <int NT, int PIECE>
int launch_mark(const CsrView &A, const CsrView &B, const EscPlan &plan, const int32_t *list, int32_t list_len, int n_front, int n_rows, int first,
                cudaStream_t stream, bool beside) {
    uint4 *cache = plan.cache ? plan.cache + (size_t)first * (plan.words / 4) : nullptr;  // `first`: place of the first of these rows
    auto kernel = plan.b_words.items ? k_esc_mark<NT, PIECE, true> : k_esc_mark<NT, PIECE, false>;
    return launch_bin(beside, kernel, n_rows, NT, (size_t)plan.words * 4, stream, A, B, plan.b_words, Windows{plan.n_win, plan.win_ptr}, list, list_len, n_front,
                      plan.words, cache, plan.row_count);
}

int launch_sorted(bool numeric, const CsrView &A, const CsrView &B, const EscPlan &plan, int32_t b_cols, const nb200_csr *c, cudaStream_t stream, bool beside) {
    int32_t *count = numeric ? nullptr : plan.row_count, *c_col = numeric ? c->col : nullptr;
    const int32_t *c_rp = numeric ? c->row_ptr : nullptr;
    float *c_val = numeric ? c->val : nullptr;
    int st;
    if (plan.host.n_rows[BIN_MEDIUM] > 0) {
        LaunchScope scope(numeric ? "esc_medium_numeric" : "esc_medium_symbolic", stream);
        if ((st = launch_bin(beside, numeric ? k_esc_medium<true> : k_esc_medium<false>, plan.host.n_rows[BIN_MEDIUM], MED_NT, 0, stream, A, B,
                             plan.lists.medium_rows, count, c_rp, c_col, c_val)))
            return st;
        beside = true;
    }
    if (plan.host.n_rows[BIN_SMALL] > 0) {
        LaunchScope scope(numeric ? "esc_small_numeric" : "esc_small_symbolic", stream);
        const int rows = plan.host.n_rows[BIN_SMALL], warps = (rows + ESC_SMALL_ROWS - 1) / ESC_SMALL_ROWS;
        const bool narrow = b_cols < (1 << 27);
        auto kernel = numeric ? (narrow ? k_esc_small<true, true> : k_esc_small<true, false>) : (narrow ? k_esc_small<false, true> : k_esc_small<false, false>);
        if ((st = launch_bin(beside, kernel, (warps + 7) / 8, 256, 0, stream, A, B, plan.lists.small_rows, rows, count, c_rp, c_col, c_val))) return st;
    }
    return NB200_OK;
}

int run_symbolic(const nb200_csr *a, const nb200_csr *b, const EscPlan &plan, cudaStream_t stream) {
    const CsrView A{a->row_ptr, a->col, a->val}, B{b->row_ptr, b->col, b->val};
    int st;
    const int n_heavy = plan.host.n_rows[BIN_GIANT] + plan.host.n_rows[BIN_HEAVY], n_ranked = plan.host.n_rows[BIN_RANKED];
    const bool many = many_rows(n_heavy + n_ranked, plan.words);
    if (n_heavy > 0) {  // first: the heaviest rows take longest
        LaunchScope scope("esc_heavy_symbolic", stream);
        auto launch = many ? launch_mark<HEAVY_NT, LONG> : launch_mark<HEAVY_NT, SHORT>;
        if ((st = launch(A, B, plan, plan.lists.heavy_rows, a->rows, plan.host.n_rows[BIN_GIANT], n_heavy, 0, stream, false))) return st;
    }
    if (n_ranked > 0) {
        LaunchScope scope("esc_ranked_symbolic", stream);
        auto launch = many ? launch_mark<MANY_NT, LONG> : launch_mark<RK_NT, SHORT>;
        if ((st = launch(A, B, plan, plan.lists.ranked_rows, a->rows, n_ranked, n_ranked, n_heavy, stream, n_heavy > 0))) return st;
    }
    return launch_sorted(false, A, B, plan, b->cols, nullptr, stream, n_heavy + n_ranked > 0);
}

ListedRows listed_rows(const EscPlan &plan, int32_t rows) {
    const int n_heavy = plan.host.n_rows[BIN_GIANT] + plan.host.n_rows[BIN_HEAVY];
    return ListedRows{plan.lists.heavy_rows, plan.lists.ranked_rows, rows, plan.host.n_rows[BIN_GIANT], n_heavy, n_heavy + plan.host.n_rows[BIN_RANKED]};
}

// What the numeric pass needs besides the result's row offsets: the rows of every class (`classes`; few rows go straight
// to one launch), and B's entries side by side where enough products read them. Made anew for every numeric pass (the
// values may be others than at the symbolic one).
struct NumericPlan {
    bool classes = false;
    const uint2 *pairs = nullptr;
};

int prepare_numeric(const nb200_csr *a, const nb200_csr *b, const EscPlan &plan, const int32_t *c_rp, NumericPlan *numeric, cudaStream_t stream) {
    *numeric = NumericPlan{};
    const ListedRows listed = listed_rows(plan, a->rows);
    if (listed.n == 0) return NB200_OK;
    numeric->classes = plan.class_rows != nullptr;
    if (numeric->classes) {
        NB200_CUDA(cudaMemsetAsync(plan.classes, 0, sizeof(ClassCtl), stream));
        LaunchScope scope("esc_classes", stream);
        ClassSlots most;
        for (int k = 0; k < CLASSES; ++k) most.slots[k] = rank_slots(k, plan.words);
        k_esc_classes<<<(listed.n + 255) / 256, 256, 0, stream>>>(listed, c_rp, most, plan.class_rows, listed.n, plan.classes);
        NB200_CUDA(cudaGetLastError());
    }
    if (!numeric->classes || plan.host.products < FORMS_FROM || plan.host.products < PAIRS_REUSE * (unsigned long long)b->nnz) return NB200_OK;
    Workspace *ws = nullptr;
    const int st = acquire_workspace(stream, (size_t)b->nnz * sizeof(uint2), &ws, PAIRS_SLOT);
    if (st != NB200_OK) return st == NB200_E_NOMEM ? NB200_OK : st;  // without room columns and values are loaded apart
    LaunchScope scope("esc_pairs", stream);
    uint2 *pairs = static_cast<uint2 *>(ws->dev);
    k_esc_pairs<<<(unsigned)(((int64_t)b->nnz + 255) / 256), 256, 0, stream>>>(b->row_ptr, b->col, b->val, b->nnz, pairs);
    NB200_CUDA(cudaGetLastError());
    numeric->pairs = pairs;
    return NB200_OK;
}

// An SM's split between L1 and shared memory stays while CTAs are on it, and the kernel of the sorted rows, which starts beside that of
// a few ranked rows, wants 100 KB for a full SM: a split that suits a short table alone (512 columns, 32 KB) shuts it out. (Graphs of
// 500 / 2000 / 2700 vertices with 16 / 4 / 4 edges each: calls of 67 / 74 / 75 us, with room for both 57 / 65 / 64. All of the SM for
// shared memory is no better, and 1 % behind where the tables are long.)
constexpr size_t FEW_STATIC = 6 * 1024, BESIDE_SMEM = 100 * 1024, SM_SMEM = 228 * 1024;
int shared_percent(size_t wanted) { return (int)std::min<size_t>(100, (100 * std::max(wanted, BESIDE_SMEM) + SM_SMEM - 1) / SM_SMEM); }

template <int CLS>
int launch_rank(const nb200_csr *a, const nb200_csr *b, const EscPlan &plan, const NumericPlan &numeric, int first, int last, const nb200_csr *c, cudaStream_t stream,
                bool beside) {
    static const char *const names[] = {"esc_rank_0", "esc_rank_1", "esc_rank_2", "esc_rank_3", "esc_rank_4", "esc_rank_few", "esc_rank_few_heavy"};
    constexpr RankClass K = RANK_CLASS[CLS];
    // A table that leaves no room for sums: no row is of this class, and where rows are not sorted all their sums are in L2.
    const int slots = rank_slots(CLS, plan.words);
    if (CLS < CLASSES && slots == 0) return NB200_OK;
    const bool halves = plan.words <= NARROW_WORDS;
    constexpr Table WIDE = CLS == FEW ? SPLIT : PAIRS;
    const size_t smem = std::max(K.smem, halves ? RankTable<HALVES, false>::bytes(plan.words) : RankTable<WIDE, false>::bytes(plan.words));
    int device = 0, ctas = last - first;
    if (CLS < CLASSES) {
        NB200_CUDA(cudaGetDevice(&device));
        NB200_CUDA(cudaDeviceGetAttribute(&ctas, cudaDevAttrMultiProcessorCount, device));
        ctas *= K.per_sm;
    }
    LaunchScope scope(names[CLS], stream);
    auto kernel = halves ? k_esc_rank<CLS, HALVES, false> : k_esc_rank<CLS, WIDE, false>;
    if constexpr (CLS < CLASSES)
        if (numeric.pairs) kernel = halves ? k_esc_rank<CLS, HALVES, true> : k_esc_rank<CLS, WIDE, true>;
    // the most that any call asks for: several threads may be here with different sizes
    NB200_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)std::max(K.smem, (size_t)RK_WORDS * 8)));
    if (CLS >= CLASSES)
        NB200_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, shared_percent(K.per_sm * (smem + FEW_STATIC))));
    return launch_bin(beside, kernel, ctas, K.nt, smem, stream, CsrView{a->row_ptr, a->col, a->val},
                      CsrView{b->row_ptr, b->col, b->val}, numeric.pairs, Windows{plan.n_win, plan.win_ptr}, listed_rows(plan, a->rows), first, last,
                      CLS < CLASSES ? plan.class_rows + (size_t)CLS * last : nullptr, plan.classes, plan.words, slots, plan.cache, c->row_ptr, c->col, c->val);
}

// The heaviest rows first: they take longest.
int launch_ranks(const nb200_csr *a, const nb200_csr *b, const EscPlan &plan, const NumericPlan &numeric, const nb200_csr *c, cudaStream_t stream) {
    const ListedRows listed = listed_rows(plan, a->rows);
    int st;
    if (numeric.classes) {
        if ((st = launch_rank<4>(a, b, plan, numeric, 0, listed.n, c, stream, false))) return st;
        if ((st = launch_rank<3>(a, b, plan, numeric, 0, listed.n, c, stream, true))) return st;
        if ((st = launch_rank<2>(a, b, plan, numeric, 0, listed.n, c, stream, true))) return st;
        if ((st = launch_rank<1>(a, b, plan, numeric, 0, listed.n, c, stream, true))) return st;
        return launch_rank<0>(a, b, plan, numeric, 0, listed.n, c, stream, true);
    }
    const int n_heavy = listed.n_heavy;
    if (n_heavy > 0 && (st = launch_rank<FEW_HEAVY>(a, b, plan, numeric, 0, n_heavy, c, stream, false))) return st;
    return listed.n > n_heavy ? launch_rank<FEW>(a, b, plan, numeric, n_heavy, listed.n, c, stream, n_heavy > 0) : NB200_OK;
}

// The numeric pass after prepare_numeric.
int run_numeric(const nb200_csr *a, const nb200_csr *b, const EscPlan &plan, const NumericPlan &numeric, const nb200_csr *c, cudaStream_t stream) {
    const CsrView A{a->row_ptr, a->col, a->val}, B{b->row_ptr, b->col, b->val};
    const bool any = listed_rows(plan, a->rows).n > 0;
    int st;
    if (any && (st = launch_ranks(a, b, plan, numeric, c, stream))) return st;
    return launch_sorted(true, A, B, plan, b->cols, c, stream, any);
}

// The plan of the latest symbolic pass, kept for the numeric pass that normally follows it on the
// same operands: the bins, the window pointer table and the bitmaps are then not computed again.
// It is used only if the operand arrays, sizes, device and stream are the same, the result's row
// offsets are the array that symbolic pass filled (with the length it reported), and neither pool
// block was handed out to anyone in between (their generations are unchanged). The patterns of A
// and B must not have been rewritten in place between the two passes; their values may change.
struct SavedPlan {
    bool valid = false;
    EscPlan plan{};
    const void *a_rp = nullptr, *a_col = nullptr, *b_rp = nullptr, *b_col = nullptr, *c_rp = nullptr;
    int32_t a_rows = 0, a_nnz = 0, b_rows = 0, b_cols = 0, b_nnz = 0, c_nnz = 0;
    cudaStream_t stream = nullptr;
    int device = -1;
    uint64_t gen_main = 0, gen_cache = 0, epoch = 0;
};
std::mutex g_saved_mutex;
SavedPlan g_saved;

void save_plan(const nb200_csr *a, const nb200_csr *b, const nb200_csr *c, const EscPlan &plan, cudaStream_t stream) {
    std::lock_guard<std::mutex> g(g_saved_mutex);
    g_saved.valid = cudaGetDevice(&g_saved.device) == cudaSuccess;
    g_saved.plan = plan;
    g_saved.a_rp = a->row_ptr, g_saved.a_col = a->col, g_saved.b_rp = b->row_ptr, g_saved.b_col = b->col;
    g_saved.c_rp = c->row_ptr, g_saved.c_nnz = c->nnz;
    g_saved.a_rows = a->rows, g_saved.a_nnz = a->nnz, g_saved.b_rows = b->rows, g_saved.b_cols = b->cols, g_saved.b_nnz = b->nnz;
    g_saved.stream = stream;
    g_saved.epoch = workspace_epoch();
    g_saved.gen_main = plan.ws->generation;
    g_saved.gen_cache = plan.cache_ws ? plan.cache_ws->generation : 0;
}

bool take_saved_plan(const nb200_csr *a, const nb200_csr *b, const nb200_csr *c, cudaStream_t stream, EscPlan *out) {
    std::lock_guard<std::mutex> g(g_saved_mutex);
    int dev = -1;
    if (!g_saved.valid || g_saved.epoch != workspace_epoch()) return false;  // the pool blocks may be gone
    if (cudaGetDevice(&dev) != cudaSuccess || dev != g_saved.device || stream != g_saved.stream) return false;
    if (a->row_ptr != g_saved.a_rp || a->col != g_saved.a_col || b->row_ptr != g_saved.b_rp || b->col != g_saved.b_col) return false;
    if (c->row_ptr != g_saved.c_rp || c->nnz != g_saved.c_nnz) return false;  // row offsets obtained elsewhere: recompute
    if (a->rows != g_saved.a_rows || a->nnz != g_saved.a_nnz || b->rows != g_saved.b_rows || b->cols != g_saved.b_cols ||
        b->nnz != g_saved.b_nnz)
        return false;
    if (g_saved.plan.ws->generation != g_saved.gen_main) return false;
    if (g_saved.plan.cache_ws && g_saved.plan.cache_ws->generation != g_saved.gen_cache) return false;
    *out = g_saved.plan;
    return true;
}

// What every form of the call checks first. *done is set where the product has no rows.
int spgemm_begin(const nb200_csr *a, const nb200_csr *b, nb200_csr *c, cudaStream_t stream, bool *done) {
    int st;
    if ((st = check_operand(a)) || (st = check_operand(b))) return st;
    if (!c || !c->row_ptr || a->cols != b->rows) return NB200_E_BADARG;
    c->rows = a->rows;
    c->cols = b->cols;
    c->nnz = 0;
    *done = a->rows == 0;
    if (*done) NB200_CUDA(cudaMemsetAsync(c->row_ptr, 0, sizeof(int32_t), stream));
    return NB200_OK;
}

// The symbolic pass on rows that `plan` has just binned (its control blocks serve one call).
// `numeric` set: the numeric pass follows, and what it needs is queued before the host waits.
int symbolic_on(const EscPlan &plan, const nb200_csr *a, const nb200_csr *b, nb200_csr *c, NumericPlan *numeric, cudaStream_t stream) {
    int st;
    if ((st = run_symbolic(a, b, plan, stream))) return st;
    {
        LaunchScope scope("esc_scan_offsets", stream);
        k_scan_offsets<<<plan.scan_ctas, SCAN_NT, 0, stream>>>(plan.row_count, a->rows, c->row_ptr, plan.scan_block + 4,
                                                              reinterpret_cast<FusedCtl *>(plan.scan_block), plan.result + W_NNZ);
        NB200_CUDA(cudaGetLastError());
    }
    if (numeric && (st = prepare_numeric(a, b, plan, c->row_ptr, numeric, stream))) return st;
    int64_t nnz;
    int device_status;
    if ((st = wait_result_word(plan.result + W_NNZ, stream, &nnz, &device_status))) return st;
    if (device_status != 0) return note_timeout(ERR_LOOKBACK_TIMEOUT, 0, "spgemm row scan");
    if (nnz > INT32_MAX) return NB200_E_OVERFLOW;
    c->nnz = (int32_t)nnz;
    return NB200_OK;
}

int spgemm_symbolic(const nb200_csr *a, const nb200_csr *b, nb200_csr *c, int64_t *products, void *stream_v) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
    bool done;
    int st;
    if (products) *products = 0;
    if ((st = spgemm_begin(a, b, c, stream, &done)) || done) return st;
    EscPlan plan{};
    if ((st = esc_prepare(a, b, true, true, stream, &plan))) return st;
    if (products) *products = (int64_t)plan.host.products;
    if ((st = symbolic_on(plan, a, b, c, nullptr, stream))) return st;
    save_plan(a, b, c, plan, stream);
    return NB200_OK;
}

int spgemm_numeric(const nb200_csr *a, const nb200_csr *b, nb200_csr *c, void *stream_v) {
    int st;
    if ((st = check_operand(a)) || (st = check_operand(b))) return st;
    if (!c || !c->row_ptr || a->cols != b->rows || c->nnz < 0) return NB200_E_BADARG;
    if (c->nnz > 0 && (!c->col || !c->val)) return NB200_E_BADARG;
    if (a->rows == 0 || c->nnz == 0) return NB200_OK;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
    EscPlan plan{};
    if (!take_saved_plan(a, b, c, stream, &plan) && (st = esc_prepare(a, b, false, false, stream, &plan))) return st;
    NumericPlan numeric;
    if ((st = prepare_numeric(a, b, plan, c->row_ptr, &numeric, stream))) return st;
    return run_numeric(a, b, plan, numeric, c, stream);
}

// Whether the one-pass kernel can do the product. It wants room for as many entries as there are products, an upper bound of nnz(C).
bool is_short(const EscPlan &plan) {
    return plan.host.n_rows[BIN_MEDIUM] + plan.host.n_rows[BIN_RANKED] + plan.host.n_rows[BIN_GIANT] + plan.host.n_rows[BIN_HEAVY] == 0 && plan.host.max_entries <= SHORT_ENTRIES &&
           plan.host.products > 0 && plan.host.products <= INT32_MAX;
}

int short_on(const EscPlan &plan, const nb200_csr *a, const nb200_csr *b, nb200_csr *c, cudaStream_t stream) {
    const CsrView A{a->row_ptr, a->col, a->val}, B{b->row_ptr, b->col, b->val};
    FusedCtl *ctl = reinterpret_cast<FusedCtl *>(plan.short_block);
    const TileWords words = TileWords::at(plan.short_block + 4);
    auto kernel = plan.host.max_entries <= 4 ? k_esc_short<4> : plan.host.max_entries <= 6 ? k_esc_short<6> : k_esc_short<8>;
    {
        LaunchScope scope("esc_short", stream);
        kernel<<<plan.short_tiles, SHORT_NT, 0, stream>>>(
            A, B, a->rows, words, ctl, plan.short_tiles, c->row_ptr, c->col, c->val, plan.result + W_NNZ);
        NB200_CUDA(cudaGetLastError());
    }
    int st;
    int64_t nnz;
    int device_status;
    if ((st = wait_result_word(plan.result + W_NNZ, stream, &nnz, &device_status))) return st;
    if (device_status != 0) return note_timeout(ERR_LOOKBACK_TIMEOUT, 0, "spgemm of short rows");
    c->nnz = (int32_t)nnz;
    return NB200_OK;
}

int spgemm_bound(const nb200_csr *a, const nb200_csr *b, int64_t *capacity, void *stream_v) {
    int st;
    if ((st = check_operand(a)) || (st = check_operand(b))) return st;
    if (!capacity || a->cols != b->rows) return NB200_E_BADARG;
    *capacity = 0;
    if (a->rows == 0) return NB200_OK;
    EscPlan plan{};
    if ((st = esc_prepare(a, b, false, false, static_cast<cudaStream_t>(stream_v), &plan))) return st;
    if (is_short(plan)) *capacity = (int64_t)plan.host.products;
    return NB200_OK;
}

int spgemm_into(const nb200_csr *a, const nb200_csr *b, nb200_csr *c, int64_t capacity, void *stream_v) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
    bool done;
    int st;
    if (!c || capacity < 0 || (capacity > 0 && (!c->col || !c->val))) return NB200_E_BADARG;
    if ((st = spgemm_begin(a, b, c, stream, &done)) || done) return st;
    EscPlan plan{};
    if ((st = esc_prepare(a, b, true, true, stream, &plan))) return st;
    if (is_short(plan) && capacity >= (int64_t)plan.host.products) return short_on(plan, a, b, c, stream);
    NumericPlan numeric;
    if ((st = symbolic_on(plan, a, b, c, &numeric, stream))) return st;
    if (c->nnz > capacity) return NB200_E_CAPACITY;
    return c->nnz > 0 ? run_numeric(a, b, plan, numeric, c, stream) : NB200_OK;
}

// The whole product into arrays that the caller hands out once their length is known: no plan outlives the call.
int spgemm_with(const nb200_csr *a, const nb200_csr *b, nb200_csr *c, nb200_take_fn take, void *ctx, bool one_pass, void *stream_v) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
    bool done;
    int st;
    if (!c || !take) return NB200_E_BADARG;
    c->col = nullptr;
    c->val = nullptr;
    if ((st = spgemm_begin(a, b, c, stream, &done)) || done) return st;
    EscPlan plan{};
    if ((st = esc_prepare(a, b, true, true, stream, &plan))) return st;
    if (one_pass && is_short(plan)) {
        const int64_t products = (int64_t)plan.host.products;
        st = take(ctx, products, &c->col, &c->val);
        if (st == NB200_OK) {
            if ((st = short_on(plan, a, b, c, stream))) return st;
            // A result holds at most twice its length, as a union's does: one that has shrunk further (32 products
            // can meet in 4 entries) moves to arrays of its own, where there is room for them.
            int32_t *col = nullptr;
            float *val = nullptr;
            if (2 * (int64_t)c->nnz >= products || take(ctx, c->nnz, &col, &val) != NB200_OK) return NB200_OK;
            NB200_CUDA(cudaMemcpyAsync(col, c->col, sizeof(int32_t) * (size_t)c->nnz, cudaMemcpyDeviceToDevice, stream));
            NB200_CUDA(cudaMemcpyAsync(val, c->val, sizeof(float) * (size_t)c->nnz, cudaMemcpyDeviceToDevice, stream));
            c->col = col;
            c->val = val;
            return NB200_OK;
        }
        if (st != NB200_E_NOMEM) return st;  // no room for an entry per product: count first
    }
    NumericPlan numeric;
    if ((st = symbolic_on(plan, a, b, c, &numeric, stream)) || c->nnz == 0) return st;
    st = take(ctx, c->nnz, &c->col, &c->val);
    if (st == NB200_E_NOMEM && (plan.b_words.items || numeric.pairs)) {  // the other forms of B are not worth a call's end
        const bool words = drop_workspace(stream, WORDS_SLOT), pairs = drop_workspace(stream, PAIRS_SLOT);
        numeric.pairs = nullptr;
        if (words || pairs) st = take(ctx, c->nnz, &c->col, &c->val);
    }
    if (st != NB200_OK) return st;
    return run_numeric(a, b, plan, numeric, c, stream);
}

}  // namespace

}  // namespace nb200

using namespace nb200;

extern "C" {

int nb200_spgemm_f32_bound(const nb200_csr *a, const nb200_csr *b, int64_t *capacity, void *stream) {
    return spgemm_bound(a, b, capacity, stream);
}

int nb200_spgemm_f32_into(const nb200_csr *a, const nb200_csr *b, nb200_csr *c, int64_t capacity, void *stream) {
    return spgemm_into(a, b, c, capacity, stream);
}

int nb200_spgemm_f32_with(const nb200_csr *a, const nb200_csr *b, nb200_csr *c, nb200_take_fn take, void *ctx, void *stream) {
    return spgemm_with(a, b, c, take, ctx, true, stream);
}

int nb200_spgemm_f32_symbolic(const nb200_csr *a, const nb200_csr *b, nb200_csr *c, int64_t *products, void *stream) {
    return spgemm_symbolic(a, b, c, products, stream);
}

int nb200_spgemm_f32_numeric(const nb200_csr *a, const nb200_csr *b, nb200_csr *c, void *stream) {
    return spgemm_numeric(a, b, c, stream);
}

int nb200_spgemm_f32(const nb200_csr *a, const nb200_csr *b, nb200_csr *c, int32_t, int32_t, void *stream_v) {
    if (!a || !c) return NB200_E_BADARG;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
    c->row_ptr = nullptr;
    c->col = nullptr;
    c->val = nullptr;
    NB200_CUDA(cudaMallocAsync(reinterpret_cast<void **>(&c->row_ptr), sizeof(int32_t) * ((size_t)std::max(a->rows, 0) + 1), stream));
    auto take = [](void *ctx, int64_t entries, int32_t **col, float **val) -> int {
        cudaStream_t on = static_cast<cudaStream_t>(ctx);
        NB200_CUDA(cudaMallocAsync(reinterpret_cast<void **>(col), sizeof(int32_t) * (size_t)entries, on));
        NB200_CUDA(cudaMallocAsync(reinterpret_cast<void **>(val), sizeof(float) * (size_t)entries, on));
        return NB200_OK;
    };
    const int st = spgemm_with(a, b, c, take, stream_v, false, stream_v);  // arrays of nnz(C) entries, so the rows are counted first
    if (st != NB200_OK) {
        if (c->row_ptr) cudaFreeAsync(c->row_ptr, stream);
        if (c->col) cudaFreeAsync(c->col, stream);
        if (c->val) cudaFreeAsync(c->val, stream);
        c->row_ptr = c->col = nullptr;
        c->val = nullptr;
    }
    return st;
}

}  // extern "C"
