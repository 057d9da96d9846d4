// CSF3 tensor add: Z = A + B for tensors stored as three compressed levels (i list, j fibres
// under each i, k fibres under each (i, j)). The reference emits a three-level nested union
// (src/backend/compute.cpp:619-1392 with the runtime-exclusion partition of
// src/backend/partition.cpp:286-328, 586-811): merge the i lists, under equal i merge the j
// fibres, under equal (i, j) merge k, otherwise copy the subtree. The result is the unique
// canonical tree of the union of the coordinate sets, so it is produced here from flat merges, by
// one of two routes (levels_pay chooses; NACHO_B200_CSF_TWO_LEVEL=0 / 1 forces one).
// Route over expanded coordinates (an operand that stores empty slices or fibres, capacities below the worst
// case):
//   1. k_csf_expand    every stored entry gets its (i, j) written out next to its k: one warp
//                      per 32 (i, j) fibres finds their i by binary search and fills their ranges;
//   2. coo3_add_run    the sorted-union merge of the two coordinate lists (coo3_merge.cu); k and
//                      the values go straight into the result's k_idx / val arrays;
//   3. k_csf_compress  one pass over the merged (i, j) columns: head flags for new i and new
//                      (i, j), a packed two-counter scan across tiles by bounded look-back, and
//                      the scatter of i_idx / j_ptr / j_idx / k_ptr.
// Level-by-level route (described above csf_add_levels): one merge per
// level, each of which tells the next where the ranges of A and B begin, so that no per-entry (i, j) is
// ever written.
#include <algorithm>
#include <cstdlib>
#include <cstring>

#include "csr_common.cuh"

namespace nb200 {

int coo3_add_run(const nb200_coo3 *a, const nb200_coo3 *b, nb200_coo3 *z, bool alloc, int64_t capacity, void *stream_v,
                 void *scratch, Workspace *ws);
int coo3_inner_run(const nb200_coo3 *a, const nb200_coo3 *b, float *z, void *stream_v, void *scratch, Workspace *ws);
size_t coo3_add_scratch_bytes(int64_t total_entries);
int64_t coo3_add_tiles(int64_t total_entries);

namespace {

constexpr int NT = 256;

// One warp per 32 consecutive (i, j) fibres. Each lane looks up its fibre's i (the last
// fibre-list start <= q, by binary search) and j; the warp then walks the entries of its 32
// fibres together, 32 entries at a time, each lane taking the (i, j) of its entry's fibre from
// the lane that holds it, so that the writes are coalesced however short the fibres are.
__global__ void __launch_bounds__(NT) k_csf_expand(int32_t n_i, int32_t n_j, const int32_t *__restrict__ i_idx,
                                                   const int32_t *__restrict__ j_ptr, const int32_t *__restrict__ j_idx,
                                                   const int32_t *__restrict__ k_ptr, int32_t *__restrict__ out_i,
                                                   int32_t *__restrict__ out_j) {
    const int w = (blockIdx.x * NT + threadIdx.x) >> 5;
    const int q0 = w * 32;
    if (q0 >= n_j) return;
    const int lane = lane_id();
    const int q = q0 + lane;
    int32_t start = INT32_MAX, i = 0, j = 0;
    if (q < n_j) {
        int lo = 0, hi = n_i - 1;  // largest r with j_ptr[r] <= q
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (ld_nc(j_ptr + mid) <= q) lo = mid; else hi = mid - 1;
        }
        i = ld_nc(i_idx + lo);
        j = ld_nc(j_idx + q);
        start = ld_nc(k_ptr + q);
    }
    const int32_t p_begin = __shfl_sync(FULL_MASK, start, 0);
    const int32_t p_end = ld_nc(k_ptr + min(q0 + 32, n_j));
    // Within a block of 32 entries the fibre starts form a bit mask, and an entry's fibre is the
    // number of fibres started at or before it. An empty fibre shares its start with its
    // successor; a block that sees one falls back to a search over the 32 starts by shuffles.
    for (int32_t base = p_begin; base < p_end; base += 32) {
        const int32_t rel = start - base;  // INT32_MAX - base for lanes past the last fibre: never in range
        const bool in_block = rel >= 0 && rel < 32;
        const int started = __popc(__ballot_sync(FULL_MASK, rel < 0));  // fibres that start before the block
        const unsigned starts = __reduce_or_sync(FULL_MASK, in_block ? 1u << rel : 0u);
        const int32_t p = base + lane;
        int f = started + __popc(starts & (0xffffffffu >> (31 - lane))) - 1;
        if (__popc(__ballot_sync(FULL_MASK, in_block)) != __popc(starts)) {  // uniform: an empty fibre in the block
            int lo = 0, hi = 31;  // largest lane whose fibre starts at or before p
#pragma unroll
            for (int step = 0; step < 5; ++step) {
                const int mid = (lo + hi + 1) >> 1;
                const int32_t sm = __shfl_sync(FULL_MASK, start, mid);
                if (sm <= p) lo = mid; else hi = mid - 1;
            }
            f = lo;
        }
        const int32_t vi = __shfl_sync(FULL_MASK, i, f), vj = __shfl_sync(FULL_MASK, j, f);
        if (p < p_end) {
            out_i[p] = vi;
            out_j[p] = vj;
        }
    }
}

struct CompressCtl {
    DeviceStatus status;
    int n_i, n_j;
};

constexpr int CVT = 32;  // entries per thread in the compress pass (one bit each in the head masks)
constexpr int CCH = 8;   // entries per load step: two 16-byte loads per coordinate array

// Loads entries [p, p + CCH) of `z` (-1 beyond the end). p is a multiple of CCH, so the fast
// path is two aligned 16-byte loads.
__device__ __forceinline__ void load_chunk(const int32_t *__restrict__ z, int64_t p, int32_t nnz, int32_t (&out)[CCH]) {
    if (p + CCH <= nnz) {
        const int4 lo = __ldg(reinterpret_cast<const int4 *>(z + p)), hi = __ldg(reinterpret_cast<const int4 *>(z + p) + 1);
        out[0] = lo.x, out[1] = lo.y, out[2] = lo.z, out[3] = lo.w, out[4] = hi.x, out[5] = hi.y, out[6] = hi.z, out[7] = hi.w;
    } else {
#pragma unroll
        for (int q = 0; q < CCH; ++q) out[q] = p + q < nnz ? ld_nc(z + p + q) : -1;
    }
}

// Head flags + packed scan + scatter. A tile's count is (new i's << 31 | new (i, j)'s).
__global__ void __launch_bounds__(NT) k_csf_compress(int32_t nnz, const int32_t *__restrict__ zi,
                                                     const int32_t *__restrict__ zj, int32_t cap_i, int32_t cap_j,
                                                     int32_t *__restrict__ i_idx, int32_t *__restrict__ j_ptr,
                                                     int32_t *__restrict__ j_idx, int32_t *__restrict__ k_ptr,
                                                     uint64_t *tile_state_raw, CompressCtl *ctl) {
    __shared__ int scan_tmp[72];
    __shared__ long long s_base;
    volatile uint64_t *tile_state = tile_state_raw;
    const int tid = threadIdx.x;
    const int t = blockIdx.x;  // CTAs are dispatched in index order; waits on earlier tiles are bounded
    const int64_t p0 = ((int64_t)t * NT + tid) * CVT;
    unsigned head_i = 0, head_ij = 0;
    {
        int32_t prev_i = p0 > 0 && p0 - 1 < nnz ? ld_nc(zi + p0 - 1) : -1;
        int32_t prev_j = p0 > 0 && p0 - 1 < nnz ? ld_nc(zj + p0 - 1) : -1;
#pragma unroll
        for (int c = 0; c < CVT / CCH; ++c) {
            int32_t ci[CCH], cj[CCH];
            load_chunk(zi, p0 + c * CCH, nnz, ci);
            load_chunk(zj, p0 + c * CCH, nnz, cj);
#pragma unroll
            for (int q = 0; q < CCH; ++q) {
                const bool live = p0 + c * CCH + q < nnz;
                const bool ni = live && ci[q] != prev_i;
                const bool nij = live && (ni || cj[q] != prev_j);
                head_i |= (unsigned)ni << (c * CCH + q);
                head_ij |= (unsigned)nij << (c * CCH + q);
                prev_i = ci[q];
                prev_j = cj[q];
            }
        }
    }
    int tot_i, tot_ij;
    int rank_i = block_excl_sum<NT>(__popc(head_i), scan_tmp, tot_i);
    int rank_ij = block_excl_sum<NT>(__popc(head_ij), scan_tmp, tot_ij);
    if (warp_id() == 0) {
        const int64_t packed = ((int64_t)tot_i << 31) | (int64_t)tot_ij;
        const int64_t b = lookback_exclusive(tile_state, t, packed, &ctl->status);
        if (lane_id() == 0) s_base = b;
    }
    __syncthreads();
    const long long base = s_base;
    if (base < 0) return;
    int r = (int)(base >> 31) + rank_i;
    int f = (int)(base & 0x7fffffff) + rank_ij;
#pragma unroll
    for (int c = 0; c < CVT / CCH; ++c) {
        if (((head_ij >> (c * CCH)) & 0xffu) == 0) continue;  // no fibre starts in this chunk
        int32_t ci[CCH], cj[CCH];
        load_chunk(zi, p0 + c * CCH, nnz, ci);  // second read, from cache
        load_chunk(zj, p0 + c * CCH, nnz, cj);
#pragma unroll
        for (int q = 0; q < CCH; ++q) {
            const int bit = c * CCH + q;
            if ((head_ij >> bit) & 1u) {
                if (f < cap_j) {
                    j_idx[f] = cj[q];
                    k_ptr[f] = (int32_t)(p0 + bit);
                }
                if ((head_i >> bit) & 1u) {
                    if (r < cap_i) {
                        i_idx[r] = ci[q];
                        j_ptr[r] = f;
                    }
                    ++r;
                }
                ++f;
            }
        }
    }
    if (t == (int)gridDim.x - 1 && tid == NT - 1) {  // last thread of the last tile holds the totals
        ctl->n_i = r;
        ctl->n_j = f;
        if (f <= cap_j) k_ptr[f] = nnz;
        if (r <= cap_i) j_ptr[r] = f;
    }
}

// The route over expanded coordinates: steps 1-3 of the file comment. `z`'s arrays exist and hold
// cap_i / cap_j / cap_k entries (cap_k >= n_k(A) + n_k(B)); nothing is freed here on failure.
int csf_add_expanded(const nb200_csf3 *a, const nb200_csf3 *b, nb200_csf3 *z, int64_t cap_i, int64_t cap_j, cudaStream_t stream) {
    const int64_t total = (int64_t)a->n_k + b->n_k;
    cudaError_t e;
    int st;
    // one pool block: expanded (i, j) of A, of B and of the merged list, the merge's own scratch
    // and the compress pass's control block and tile words
    const int64_t compress_tiles = (total + NT * CVT - 1) / (NT * CVT);
    Carver sizes;
    sizes.take<int32_t>((size_t)a->n_k);
    sizes.take<int32_t>((size_t)a->n_k);
    sizes.take<int32_t>((size_t)b->n_k);
    sizes.take<int32_t>((size_t)b->n_k);
    sizes.take<int32_t>((size_t)total);
    sizes.take<int32_t>((size_t)total);
    sizes.take<uint64_t>((size_t)compress_tiles + 8);
    const size_t own = sizes.used();
    Workspace *ws = nullptr;
    if ((st = acquire_workspace(stream, own + coo3_add_scratch_bytes(total) + 256, &ws))) return (st);
    Carver carve(ws->dev);
    int32_t *ai = carve.take<int32_t>((size_t)a->n_k), *aj = carve.take<int32_t>((size_t)a->n_k);
    int32_t *bi = carve.take<int32_t>((size_t)b->n_k), *bj = carve.take<int32_t>((size_t)b->n_k);
    int32_t *zi = carve.take<int32_t>((size_t)total), *zj = carve.take<int32_t>((size_t)total);
    uint64_t *compress_block = carve.take<uint64_t>((size_t)compress_tiles + 8);
    void *merge_scratch = static_cast<unsigned char *>(ws->dev) + own;

    if (a->n_j > 0) {
        LaunchScope scope("csf_expand", stream);
        k_csf_expand<<<(int)(((int64_t)a->n_j + 31) / 32 * 32 + NT - 1) / NT, NT, 0, stream>>>(a->n_i, a->n_j, a->i_idx, a->j_ptr, a->j_idx, a->k_ptr, ai, aj);
    }
    if (b->n_j > 0) {
        LaunchScope scope("csf_expand", stream);
        k_csf_expand<<<(int)(((int64_t)b->n_j + 31) / 32 * 32 + NT - 1) / NT, NT, 0, stream>>>(b->n_i, b->n_j, b->i_idx, b->j_ptr, b->j_idx, b->k_ptr, bi, bj);
    }
    e = cudaGetLastError();
    if (e != cudaSuccess) return (note_cuda_error(e, "k_csf_expand"));

    nb200_coo3 ca{{a->dims[0], a->dims[1], a->dims[2]}, a->n_k, ai, aj, a->k_idx, a->val};
    nb200_coo3 cb{{b->dims[0], b->dims[1], b->dims[2]}, b->n_k, bi, bj, b->k_idx, b->val};
    nb200_coo3 cz{{0, 0, 0}, 0, zi, zj, z->k_idx, z->val};
    CompressCtl *ctl = reinterpret_cast<CompressCtl *>(compress_block);
    static_assert(sizeof(CompressCtl) <= 4 * sizeof(uint64_t), "control block must fit its slot");
    uint64_t *tile_state = compress_block + 4;

    if ((st = coo3_add_run(&ca, &cb, &cz, false, total, stream, merge_scratch, ws))) return (st);
    const int32_t nnz = cz.nnz;
    z->n_k = nnz;
    const int tiles = (int)(((int64_t)nnz + NT * CVT - 1) / (NT * CVT));
    e = cudaMemsetAsync(compress_block, 0, sizeof(uint64_t) * ((size_t)tiles + 4), stream);
    if (e != cudaSuccess) return (note_cuda_error(e, "cudaMemsetAsync"));
    {
        LaunchScope scope("csf_compress", stream);
        k_csf_compress<<<tiles, NT, 0, stream>>>(nnz, zi, zj, (int32_t)std::min<int64_t>(cap_i, INT32_MAX),
                                                 (int32_t)std::min<int64_t>(cap_j, INT32_MAX), z->i_idx, z->j_ptr, z->j_idx,
                                                 z->k_ptr, tile_state, ctl);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) return (note_cuda_error(e, "k_csf_compress"));
    e = cudaMemcpyAsync(ws->host, ctl, sizeof(CompressCtl), cudaMemcpyDeviceToHost, stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    if (e != cudaSuccess) return (note_cuda_error(e, "read result lengths"));
    CompressCtl h;
    std::memcpy(&h, ws->host, sizeof(h));
    if (h.status.error != 0) return note_timeout(h.status.error, h.status.detail, "csf3 level compress");
    z->n_i = h.n_i;
    z->n_j = h.n_j;
    if (h.n_i > cap_i || h.n_j > cap_j) return (NB200_E_CAPACITY);
    return NB200_OK;
}

// -------------------------------------------------------------- the level-by-level route ----
//
// Expanding (i, j) for every entry moves more bytes than the tensor has. The same union comes from one merge
// per level, none of which waits for the host:
//   1. the slice lists of A and B, as matrices of one row whose columns are the slice numbers, in the
//      offsets mode of the CSR tile kernel: Z's i_idx, and over Z's slices a row-offset array into the
//      fibres of A (of B) in which a slice the operand lacks is an empty row;
//   2. with those, the fibre lists are CSR matrices with one row per slice of Z: the offsets mode again
//      gives Z's j_ptr and j_idx and, over Z's fibres, offsets into the entries of A and of B;
//   3. with those, A's and B's (k_idx, val) arrays are CSR matrices with one row per fibre of Z, and the
//      CSR union writes Z's k_ptr, k_idx and val.
// Steps 2 and 3 read their row count from device memory.

// Measured against the expanded route: 25 M entries per operand in fibres of 7, 262 us against 625; 5 M in
// fibres of 4, 96 against 205; 5000 in fibres of 1, 39 against 63. So it is taken wherever it applies.
bool levels_pay(const nb200_csf3 *a, const nb200_csf3 *b) {
    if (a->n_j == 0 || b->n_j == 0) return false;
    if (const char *e = std::getenv("NACHO_B200_CSF_TWO_LEVEL")) return e[0] != '0';  // read per call: tests take both routes
    return true;
}

// Up to this many entries per fibre of the operands, the tile for short rows takes the entries. Whole call, that tile against the large one, with 1, 2, 4,
// 12, 30 and 62 entries per fibre: 3 M entries per operand 94, 80, 70, 62, 60, 60 us and 111, 92, 72, 65, 60, 61; 8 M 174, 146, 124, 109, 105, 103 and 204, 160, 119, 104, 99, 98;
// 25 M 440, 370, 292, 239, 220, 217 and 532, 409, 280, 228, 206, 203. The line was drawn when tiles gathered their values; since they copy them, the tile for
// short rows earns its place up to some three entries per fibre, and beyond those among the smaller trees alone.
constexpr int64_t SHORT_FIBRE = 64;

// `done` tells whether the result is in place; it is not where an operand stores empty slices or fibres, which
// the canonical tree does not have (the caller then takes the other route).
int csf_add_levels(const nb200_csf3 *a, const nb200_csf3 *b, nb200_csf3 *z, cudaStream_t stream, bool *done,
                   const LaunchKnobs &first_knobs = LaunchKnobs()) {
    *done = false;
    const int64_t bound_i = (int64_t)a->n_i + b->n_i, bound_j = (int64_t)a->n_j + b->n_j, total = (int64_t)a->n_k + b->n_k;
    if (bound_j > INT32_MAX - 1) return NB200_E_OVERFLOW;
    Carver sizes;
    sizes.take<int32_t>((size_t)bound_i + 1);
    sizes.take<int32_t>((size_t)bound_i + 1);
    sizes.take<int32_t>((size_t)bound_j + 1);
    sizes.take<int32_t>((size_t)bound_j + 1);
    const size_t own = sizes.used(), list_bytes = csr2_scratch_bytes(bound_i), fibre_bytes = csr2_scratch_bytes(bound_j);
    Workspace *ws = nullptr;
    int st;
    if ((st = acquire_workspace(stream, own + list_bytes + fibre_bytes + csr2_scratch_bytes(total), &ws, 3))) return st;
    Carver carve(ws->dev);
    int32_t *ja = carve.take<int32_t>((size_t)bound_i + 1), *jb = carve.take<int32_t>((size_t)bound_i + 1);
    int32_t *ka = carve.take<int32_t>((size_t)bound_j + 1), *kb = carve.take<int32_t>((size_t)bound_j + 1);
    unsigned char *scratch_i = static_cast<unsigned char *>(ws->dev) + own, *scratch_j = scratch_i + list_bytes, *scratch_k = scratch_j + fibre_bytes;
    unsigned long long *word[3] = {result_word(ws, 0), result_word(ws, 1), result_word(ws, 2)};
    FusedCtl *ctl[3] = {};

    const LevelOffsets slices{a->j_ptr, b->j_ptr, ja, jb}, fibres{a->k_ptr, b->k_ptr, ka, kb};
    if ((st = csr2_enqueue(OP_UNION, CsrIn{nullptr, a->i_idx, nullptr, a->n_i}, CsrIn{nullptr, b->i_idx, nullptr, b->n_i}, RowCount{1}, a->dims[0],
                           CsrOut{nullptr, z->i_idx, nullptr, nullptr, word[0]}, &slices, scratch_i, stream, &ctl[0], first_knobs)))
        return st;
    if ((st = csr2_enqueue(OP_UNION, CsrIn{ja, a->j_idx, nullptr, a->n_j}, CsrIn{jb, b->j_idx, nullptr, b->n_j}, RowCount{(int32_t)std::min<int64_t>(bound_i, a->dims[0]), &ctl[0]->total}, a->dims[1],
                           CsrOut{z->j_ptr, z->j_idx, nullptr, nullptr, word[1], ctl[0]}, &fibres, scratch_j, stream, &ctl[1])))
        return st;
    if ((st = csr2_enqueue(OP_UNION, CsrIn{ka, a->k_idx, a->val, a->n_k}, CsrIn{kb, b->k_idx, b->val, b->n_k}, RowCount{(int32_t)std::min<int64_t>(bound_j, (int64_t)a->dims[0] * a->dims[1]), &ctl[1]->total, total < SHORT_FIBRE * bound_j}, a->dims[2],
                           CsrOut{z->k_ptr, z->k_idx, z->val, nullptr, word[2], ctl[1]}, nullptr, scratch_k, stream, &ctl[2])))
        return st;
    int64_t length[3];
    for (int q = 0; q < 3; ++q) {
        int device_status;
        if ((st = wait_result_word(word[q], stream, &length[q], &device_status))) return st;
        if (device_status != 0) {
            NB200_CUDA(cudaMemcpyAsync(ws->host, ctl[q], sizeof(FusedCtl), cudaMemcpyDeviceToHost, stream));
            NB200_CUDA(cudaStreamSynchronize(stream));
            FusedCtl h;
            std::memcpy(&h, ws->host, sizeof(h));
            return note_timeout(h.status.error, h.status.detail, "csf3 levels");
        }
    }
    if (length[2] & RW_HOLLOW) return NB200_OK;
    z->n_i = (int32_t)(length[0] & (RW_HOLLOW - 1));
    z->n_j = (int32_t)(length[1] & (RW_HOLLOW - 1));
    z->n_k = (int32_t)length[2];
    *done = true;
    return NB200_OK;
}

int check_csf3(const nb200_csf3 *t) {
    if (!t || t->n_i < 0 || t->n_j < 0 || t->n_k < 0) return NB200_E_BADARG;
    if (t->n_k > 0 && (!t->i_idx || !t->j_ptr || !t->j_idx || !t->k_ptr || !t->k_idx || !t->val)) return NB200_E_BADARG;
    return NB200_OK;
}

int csf_add_run(const nb200_csf3 *a, const nb200_csf3 *b, nb200_csf3 *z, bool alloc, int64_t cap_i, int64_t cap_j,
                int64_t cap_k, void *stream_v) {
    int st;
    if ((st = check_csf3(a)) || (st = check_csf3(b))) return st;
    if (!z || a->dims[0] != b->dims[0] || a->dims[1] != b->dims[1] || a->dims[2] != b->dims[2]) return NB200_E_BADARG;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
    const int64_t total = (int64_t)a->n_k + b->n_k;
    if (total > INT32_MAX) return NB200_E_OVERFLOW;
    if (total > 0 && (a->dims[0] < 0 || a->dims[1] < 0 || a->dims[2] < 0)) return NB200_E_BADARG;
    const int64_t bound_i = (int64_t)a->n_i + b->n_i, bound_j = (int64_t)a->n_j + b->n_j;
    for (int d = 0; d < 3; ++d) z->dims[d] = a->dims[d];
    z->n_i = z->n_j = z->n_k = 0;
    cudaError_t e;
    if (alloc) {
        z->i_idx = z->j_ptr = z->j_idx = z->k_ptr = z->k_idx = nullptr;
        z->val = nullptr;
        cap_i = bound_i;
        cap_j = bound_j;
        cap_k = total;
        struct { void **p; size_t n; } arrays[6] = {
            {reinterpret_cast<void **>(&z->i_idx), (size_t)bound_i}, {reinterpret_cast<void **>(&z->j_ptr), (size_t)bound_i + 1},
            {reinterpret_cast<void **>(&z->j_idx), (size_t)bound_j}, {reinterpret_cast<void **>(&z->k_ptr), (size_t)bound_j + 1},
            {reinterpret_cast<void **>(&z->k_idx), (size_t)total},   {reinterpret_cast<void **>(&z->val), (size_t)total}};
        for (auto &arr : arrays) {
            if (arr.n == 0) continue;
            e = cudaMallocAsync(arr.p, 4 * arr.n, stream);
            if (e != cudaSuccess) {
                for (auto &other : arrays) {
                    if (*other.p) cudaFreeAsync(*other.p, stream);
                    *other.p = nullptr;
                }
                return note_cuda_error(e, "cudaMallocAsync");
            }
        }
    } else {
        if (cap_i < 0 || cap_j < 0 || cap_k < 0 || !z->j_ptr || !z->k_ptr) return NB200_E_BADARG;
        if (cap_k < total) return NB200_E_CAPACITY;  // the merge needs room for every operand entry
        if (total > 0 && (!z->i_idx || !z->j_idx || !z->k_idx || !z->val)) return NB200_E_BADARG;
    }
    auto fail = [&](int code) {
        if (alloc) {
            void **ps[6] = {reinterpret_cast<void **>(&z->i_idx), reinterpret_cast<void **>(&z->j_ptr),
                            reinterpret_cast<void **>(&z->j_idx), reinterpret_cast<void **>(&z->k_ptr),
                            reinterpret_cast<void **>(&z->k_idx), reinterpret_cast<void **>(&z->val)};
            for (auto p : ps) {
                if (*p) cudaFreeAsync(*p, stream);
                *p = nullptr;
            }
        }
        return code;
    };
    if (total == 0) {  // empty result: the two offset arrays hold their single leading zero
        e = cudaMemsetAsync(z->j_ptr, 0, sizeof(int32_t), stream);
        if (e == cudaSuccess) e = cudaMemsetAsync(z->k_ptr, 0, sizeof(int32_t), stream);
        if (e != cudaSuccess) return fail(note_cuda_error(e, "cudaMemsetAsync"));
        return NB200_OK;
    }

    // (the levels are written in one pass each: room for the worst case, or the other route)
    bool done = false;
    st = NB200_OK;
    if (levels_pay(a, b) && cap_i >= bound_i && cap_j >= bound_j) st = csf_add_levels(a, b, z, stream, &done);
    if (st == NB200_OK && !done) st = csf_add_expanded(a, b, z, cap_i, cap_j, stream);
    return st == NB200_OK ? NB200_OK : fail(st);
}

// Inner product of two CSF3 tensors (compiler.cpp:141): every entry gets its (i, j) written out
// next to its k (k_csf_expand), then the coordinate lists go through the inner-product mode of the
// COO3 tile kernel.
int csf_inner_run(const nb200_csf3 *a, const nb200_csf3 *b, float *z, void *stream_v) {
    int st;
    if ((st = check_csf3(a)) || (st = check_csf3(b))) return st;
    if (!z || a->dims[0] != b->dims[0] || a->dims[1] != b->dims[1] || a->dims[2] != b->dims[2]) return NB200_E_BADARG;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
    if (a->n_k == 0 || b->n_k == 0) {
        NB200_CUDA(cudaMemsetAsync(z, 0, sizeof(float), stream));
        return NB200_OK;
    }
    const int64_t total = (int64_t)a->n_k + b->n_k;
    if (total > INT32_MAX) return NB200_E_OVERFLOW;
    Carver sizes;
    sizes.take<int32_t>((size_t)a->n_k);
    sizes.take<int32_t>((size_t)a->n_k);
    sizes.take<int32_t>((size_t)b->n_k);
    sizes.take<int32_t>((size_t)b->n_k);
    const size_t own = sizes.used();
    Workspace *ws = nullptr;
    if ((st = acquire_workspace(stream, own + coo3_add_scratch_bytes(total) + 256, &ws))) return st;
    Carver carve(ws->dev);
    int32_t *ai = carve.take<int32_t>((size_t)a->n_k), *aj = carve.take<int32_t>((size_t)a->n_k);
    int32_t *bi = carve.take<int32_t>((size_t)b->n_k), *bj = carve.take<int32_t>((size_t)b->n_k);
    void *merge_scratch = static_cast<unsigned char *>(ws->dev) + own;
    {
        LaunchScope scope("csf_expand", stream);
        k_csf_expand<<<(int)(((int64_t)a->n_j + 31) / 32 * 32 + NT - 1) / NT, NT, 0, stream>>>(a->n_i, a->n_j, a->i_idx, a->j_ptr, a->j_idx, a->k_ptr, ai, aj);
    }
    {
        LaunchScope scope("csf_expand", stream);
        k_csf_expand<<<(int)(((int64_t)b->n_j + 31) / 32 * 32 + NT - 1) / NT, NT, 0, stream>>>(b->n_i, b->n_j, b->i_idx, b->j_ptr, b->j_idx, b->k_ptr, bi, bj);
    }
    NB200_CUDA(cudaGetLastError());
    nb200_coo3 ca{{a->dims[0], a->dims[1], a->dims[2]}, a->n_k, ai, aj, a->k_idx, a->val};
    nb200_coo3 cb{{b->dims[0], b->dims[1], b->dims[2]}, b->n_k, bi, bj, b->k_idx, b->val};
    return coo3_inner_run(&ca, &cb, z, stream_v, merge_scratch, ws);
}

}  // namespace

}  // namespace nb200

using namespace nb200;

extern "C" {

int nb200_csf_add_f32(const nb200_csf3 *a, const nb200_csf3 *b, nb200_csf3 *z, int32_t, int32_t, void *stream) {
    return csf_add_run(a, b, z, true, 0, 0, 0, stream);
}

int nb200_csf_add_f32_into(const nb200_csf3 *a, const nb200_csf3 *b, nb200_csf3 *z, int64_t cap_i, int64_t cap_j,
                           int64_t cap_k, void *stream) {
    return csf_add_run(a, b, z, false, cap_i, cap_j, cap_k, stream);
}

int nb200_inner_prod_f32(const nb200_csf3 *a, const nb200_csf3 *b, float *z, void *stream) {
    return csf_inner_run(a, b, z, stream);
}

int nb200_selftest_levels_timeout(const nb200_csf3 *a, const nb200_csf3 *b, nb200_csf3 *z, int64_t cap_i, int64_t cap_j, int64_t cap_k,
                                  int32_t polls, void *stream) {
    int st;
    if ((st = check_csf3(a)) || (st = check_csf3(b))) return st;
    if ((int64_t)a->n_i + b->n_i < SELFTEST_ENTRIES) return NB200_E_BADARG;
    if (polls < 1 || !z || cap_i < (int64_t)a->n_i + b->n_i || cap_j < (int64_t)a->n_j + b->n_j || cap_k < (int64_t)a->n_k + b->n_k) return NB200_E_BADARG;
    LaunchKnobs knobs;
    knobs.first_tile = 1;
    knobs.poll_limit = polls;
    bool done;
    return csf_add_levels(a, b, z, static_cast<cudaStream_t>(stream), &done, knobs);
}

}  // extern "C"
