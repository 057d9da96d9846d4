// The 2-D formats beside CSR: coordinate lists (COO) and doubly compressed rows (DCSR), and the
// element-wise kernels the reference declares over them (compiler.cpp:118-126):
//   coo_add, coo_mul        COO  (+|.*) COO  -> COO
//   coo_csr_add             CSR  +      COO  -> CSR
//   dcsr_add, dcsr_mul      DCSR (+|.*) DCSR -> DCSR
// Both formats hold their columns and values in CSR order, so each kernel here runs the CSR merge kernels of
// csr_merge.cu on the caller's own column / value arrays; what differs is the row level.
//   COO   the missing row offsets are built (one small pass over the rows) and the row index of every
//         result entry is written out (one warp per 32 rows).
//   DCSR  the two row lists are merged first, as matrices of one row whose columns are the row numbers
//         (offsets mode of the tile kernel): that yields the union of the stored rows and, over it, a row
//         offset array for each operand in which a row it lacks is empty. With those the entries are a
//         CSR merge whose rows are the stored ones only, however many the matrix has; its row count is
//         read from device memory, so nothing waits in between. The sum keeps the rows that hold a result
//         entry: all of the union, unless an operand stores empty rows. The product keeps the rows that
//         BOTH operands store -- also those whose columns do not meet, which the reference keeps as an
//         empty fibre (its intersection works level by level: src/backend/compute.cpp:619-1392 run on the
//         i level first, then on j inside the matched rows). Rows are dropped by a scan and a scatter.
#include <algorithm>
#include <cstring>

#include "csr_common.cuh"

namespace nb200 {

namespace {

constexpr int NT = 256;

// rp[r] = ptr[q(r)] where q(r) is the number of ids below r (ids sorted ascending, n of them);
// ptr == nullptr stands for ptr[q] = q. Thread q writes the rows in (ids[q - 1], ids[q]]; the rows
// after the last id get ptr[n]. With repeated ids (a coordinate list) a thread whose id equals its
// predecessor's has no row to write.
__global__ void __launch_bounds__(NT) k_row_offsets(const int32_t *__restrict__ ids, const int32_t *__restrict__ ptr, int32_t n,
                                                   int32_t rows, int32_t *__restrict__ rp) {
    const int64_t q = (int64_t)blockIdx.x * NT + threadIdx.x;
    if (q > n) return;
    const int64_t first = q == 0 ? 0 : (int64_t)ld_nc(ids + q - 1) + 1;
    const int64_t last = q == n ? rows : ld_nc(ids + q);
    const int32_t v = ptr ? ld_nc(ptr + q) : (int32_t)q;
    for (int64_t r = first; r <= last && r <= rows; ++r) rp[r] = v;
}

// out[p] = the row of entry p, for every entry of a CSR structure: one warp per 32 consecutive
// rows walks their entries 32 at a time; an entry's row is the last of the 32 whose start is at
// or before it (found with five shuffles), so the writes are coalesced however short the rows are.
__global__ void __launch_bounds__(NT) k_expand_rows(const int32_t *__restrict__ rp, int32_t rows, int32_t *__restrict__ out) {
    const int w = (blockIdx.x * NT + threadIdx.x) >> 5;
    const int64_t r0 = (int64_t)w * 32;
    if (r0 >= rows) return;
    const int lane = lane_id();
    const int32_t start = r0 + lane < rows ? ld_nc(rp + r0 + lane) : INT32_MAX;
    const int32_t p_begin = __shfl_sync(FULL_MASK, start, 0);
    const int32_t p_end = ld_nc(rp + min(r0 + 32, (int64_t)rows));
    for (int32_t base = p_begin; base < p_end; base += 32) {
        const int32_t p = base + lane;
        int lo = 0, hi = 31;  // largest lane whose row starts at or before p
#pragma unroll
        for (int step = 0; step < 5; ++step) {
            const int mid = (lo + hi + 1) >> 1;
            const int32_t sm = __shfl_sync(FULL_MASK, start, mid);
            if (sm <= p) lo = mid; else hi = mid - 1;
        }
        if (p < p_end) out[p] = (int32_t)(r0 + lo);
    }
}

// keep[u] = 1 for the rows of a CSR structure that hold an entry.
__global__ void __launch_bounds__(NT) k_rows_nonempty(const int32_t *__restrict__ rp, int32_t rows, int32_t *__restrict__ keep) {
    const int64_t u = (int64_t)blockIdx.x * NT + threadIdx.x;
    if (u < rows) keep[u] = ld_nc(rp + u + 1) > ld_nc(rp + u);
}

// After the exclusive scan of keep[]: row u, if kept, is result row pos[u]. The flag is recomputed
// (pos[u + 1] > pos[u], with the total after the last row). The result length goes to `word`.
__global__ void __launch_bounds__(NT) k_rows_scatter(const int32_t *__restrict__ pos, const FusedCtl *__restrict__ ctl, const int32_t *__restrict__ ids,
                                                    const int32_t *__restrict__ rp, int32_t rows, int32_t *__restrict__ i_idx,
                                                    int32_t *__restrict__ j_ptr, unsigned long long *word) {
    const int64_t u = (int64_t)blockIdx.x * NT + threadIdx.x;
    if (u > rows) return;
    const int32_t n = (int32_t)ctl->total;
    if (u == rows) {
        j_ptr[n] = ld_nc(rp + rows);
        publish_result_word(word, ctl->status.error != 0 ? NB200_E_TIMEOUT : NB200_OK, n);
        return;
    }
    const int32_t at = ld_nc(pos + u);
    const int32_t next = u + 1 < rows ? ld_nc(pos + u + 1) : n;
    if (next > at) {
        i_idx[at] = ld_nc(ids + u);
        j_ptr[at] = ld_nc(rp + u);
    }
}

int check_coo(const nb200_coo *m) {
    if (!m || m->rows < 0 || m->cols < 0 || m->nnz < 0) return NB200_E_BADARG;
    if (m->nnz > 0 && (!m->i || !m->j || !m->val)) return NB200_E_BADARG;
    return NB200_OK;
}

int check_dcsr(const nb200_dcsr *m) {
    if (!m || m->rows < 0 || m->cols < 0 || m->n_i < 0 || m->nnz < 0 || m->n_i > m->rows) return NB200_E_BADARG;
    if (!m->j_ptr || (m->n_i > 0 && !m->i_idx) || (m->nnz > 0 && (!m->j_idx || !m->val))) return NB200_E_BADARG;
    return NB200_OK;
}

cudaError_t launch_row_offsets(const int32_t *ids, const int32_t *ptr, int32_t n, int32_t rows, int32_t *rp, cudaStream_t stream) {
    LaunchScope scope("row_offsets", stream);
    k_row_offsets<<<(int)(((int64_t)n + 1 + NT - 1) / NT), NT, 0, stream>>>(ids, ptr, n, rows, rp);
    return cudaGetLastError();
}

typedef int (*csr_into_fn)(const nb200_csr *, const nb200_csr *, nb200_csr *, int64_t, void *);

// Scratch of a call on coordinate lists: row offsets of A, B and the result. Pool slot 1: the CSR kernels
// underneath use slot 0.
struct Scratch2d {
    int32_t *rpa, *rpb, *rpz;
};

int take_scratch(int32_t rows, cudaStream_t stream, Scratch2d *s) {
    Carver sizes;
    for (int q = 0; q < 3; ++q) sizes.take<int32_t>((size_t)rows + 2);
    Workspace *ws = nullptr;
    int st;
    if ((st = acquire_workspace(stream, sizes.used(), &ws, 1))) return st;
    Carver carve(ws->dev);
    s->rpa = carve.take<int32_t>((size_t)rows + 2);
    s->rpb = carve.take<int32_t>((size_t)rows + 2);
    s->rpz = carve.take<int32_t>((size_t)rows + 2);
    return NB200_OK;
}

int coo2_run(csr_into_fn op, bool is_union, const nb200_coo *a, const nb200_coo *b, nb200_coo *z, int64_t capacity, void *stream_v) {
    int st;
    if ((st = check_coo(a)) || (st = check_coo(b))) return st;
    if (!z || a->rows != b->rows || a->cols != b->cols || capacity < 0) return NB200_E_BADARG;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
    z->rows = a->rows;
    z->cols = a->cols;
    z->nnz = 0;
    const int64_t total = (int64_t)a->nnz + b->nnz;
    if (total == 0 || (!is_union && (a->nnz == 0 || b->nnz == 0))) return NB200_OK;
    if (capacity > 0 && (!z->i || !z->j || !z->val)) return NB200_E_BADARG;
    Scratch2d s;
    if ((st = take_scratch(a->rows, stream, &s))) return st;
    cudaError_t e = launch_row_offsets(a->i, nullptr, a->nnz, a->rows, s.rpa, stream);
    if (e == cudaSuccess) e = launch_row_offsets(b->i, nullptr, b->nnz, b->rows, s.rpb, stream);
    if (e != cudaSuccess) return note_cuda_error(e, "k_row_offsets");
    const nb200_csr ca{a->rows, a->cols, a->nnz, s.rpa, a->j, a->val}, cb{b->rows, b->cols, b->nnz, s.rpb, b->j, b->val};
    nb200_csr cz{a->rows, a->cols, 0, s.rpz, z->j, z->val};
    st = op(&ca, &cb, &cz, capacity, stream_v);
    z->nnz = cz.nnz;
    if (st != NB200_OK) return st;
    if (cz.nnz > 0) {
        LaunchScope scope("expand_rows", stream);
        const int64_t warps = ((int64_t)a->rows + 31) / 32;
        k_expand_rows<<<(int)((warps * 32 + NT - 1) / NT), NT, 0, stream>>>(s.rpz, a->rows, z->i);
        e = cudaGetLastError();
        if (e != cudaSuccess) return note_cuda_error(e, "k_expand_rows");
    }
    return NB200_OK;
}

// Numbers the kept ones of `n` rows (flags in `keep`, overwritten) and writes the compressed row level of the
// result; *count receives its length. `block` holds the scan's control block and tile words.
int compress_rows(int32_t *keep, int32_t n, const int32_t *ids, const int32_t *rp, uint64_t *block, nb200_dcsr *z, unsigned long long *word,
                  cudaStream_t stream) {
    const int ctas = (int)(((int64_t)n + SCAN_NT * SCAN_VT - 1) / (SCAN_NT * SCAN_VT));
    FusedCtl *ctl = reinterpret_cast<FusedCtl *>(block);
    NB200_CUDA(cudaMemsetAsync(block, 0, sizeof(uint64_t) * ((size_t)ctas + 4), stream));
    {
        LaunchScope scope("scan_lookback", stream);
        k_scan_lookback<<<ctas, SCAN_NT, 0, stream>>>(keep, n, block + 4, ctl);
    }
    {
        LaunchScope scope("dcsr_scatter", stream);
        k_rows_scatter<<<(int)(((int64_t)n + 1 + NT - 1) / NT), NT, 0, stream>>>(keep, ctl, ids, rp, n, z->i_idx, z->j_ptr, word);
    }
    NB200_CUDA(cudaGetLastError());
    int64_t kept;
    int st, device_status;
    if ((st = wait_result_word(word, stream, &kept, &device_status))) return st;
    if (device_status != 0) return note_timeout(ERR_LOOKBACK_TIMEOUT, 0, "dcsr row compress");
    z->n_i = (int32_t)kept;
    return NB200_OK;
}

int dcsr2_run(csr_into_fn op, bool is_union, const nb200_dcsr *a, const nb200_dcsr *b, nb200_dcsr *z, int64_t cap_i, int64_t capacity,
              void *stream_v) {
    int st;
    if ((st = check_dcsr(a)) || (st = check_dcsr(b))) return st;
    if (!z || a->rows != b->rows || a->cols != b->cols || capacity < 0 || cap_i < 0 || !z->j_ptr) return NB200_E_BADARG;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
    z->rows = a->rows;
    z->cols = a->cols;
    z->n_i = z->nnz = 0;
    const int64_t stored = (int64_t)a->n_i + b->n_i;  // most rows of the union
    const int64_t bound_i = is_union ? std::min<int64_t>(stored, a->rows) : std::min(a->n_i, b->n_i);
    if (cap_i < bound_i) return NB200_E_CAPACITY;  // the row level is written in one pass: room for the worst case
    if (bound_i > 0 && !z->i_idx) return NB200_E_BADARG;
    const int64_t total = (int64_t)a->nnz + b->nnz;
    if (bound_i == 0 || total == 0) {  // no row survives: one leading zero in the offsets
        NB200_CUDA(cudaMemsetAsync(z->j_ptr, 0, sizeof(int32_t), stream));
        return NB200_OK;
    }
    if (capacity > 0 && (!z->j_idx || !z->val)) return NB200_E_BADARG;
    if (stored > INT32_MAX - 1) return NB200_E_OVERFLOW;

    // pool slot 1: the union's rows, the offsets of both operands over it, flags, the result's offsets over it
    const size_t scan_words = (size_t)stored / (SCAN_NT * SCAN_VT) + 8;
    Carver sizes;
    for (int q = 0; q < 5; ++q) sizes.take<int32_t>((size_t)stored + 2);
    sizes.take<uint64_t>(scan_words);
    const size_t own = sizes.used();
    const size_t list_bytes = csr2_scratch_bytes(stored), entry_bytes = csr2_scratch_bytes(total);
    Workspace *ws = nullptr;
    if ((st = acquire_workspace(stream, own + list_bytes + entry_bytes, &ws, 1))) return st;
    Carver carve(ws->dev);
    int32_t *off_a = carve.take<int32_t>((size_t)stored + 2), *off_b = carve.take<int32_t>((size_t)stored + 2);
    int32_t *keep = carve.take<int32_t>((size_t)stored + 2), *ids = carve.take<int32_t>((size_t)stored + 2);
    int32_t *rpz = carve.take<int32_t>((size_t)stored + 2);
    uint64_t *scan_block = carve.take<uint64_t>(scan_words);
    unsigned char *list_scratch = static_cast<unsigned char *>(ws->dev) + own, *entry_scratch = list_scratch + list_bytes;
    unsigned long long *rows_word = result_word(ws, 0), *length_word = result_word(ws, 1), *kept_word = result_word(ws, 2);

    // ---- the stored rows of both operands, and where their entries begin
    const LevelOffsets levels{a->j_ptr, b->j_ptr, off_a, off_b, is_union ? nullptr : keep};
    FusedCtl *rows_ctl = nullptr, *ctl = nullptr;
    int32_t *union_rows = is_union ? z->i_idx : ids;
    if ((st = csr2_enqueue(OP_UNION, CsrIn{nullptr, a->i_idx, nullptr, a->n_i}, CsrIn{nullptr, b->i_idx, nullptr, b->n_i}, RowCount{1}, a->rows,
                           CsrOut{nullptr, union_rows, nullptr, nullptr, rows_word}, &levels, list_scratch, stream, &rows_ctl)))
        return st;

    // ---- the entries, on the rows of the union
    int64_t length, n_rows;
    int rows_status, device_status = 0;
    int32_t *result_rp = is_union ? z->j_ptr : rpz;
    const CsrIn A{off_a, a->j_idx, a->val, a->nnz}, B{off_b, b->j_idx, b->val, b->nnz};
    const bool one_pass = capacity >= (is_union ? total : std::min<int64_t>(a->nnz, b->nnz));
    bool hollow = false;
    if (one_pass) {
        if ((st = csr2_enqueue(is_union ? OP_UNION : OP_INTERSECT, A, B, RowCount{(int32_t)std::min<int64_t>(stored, a->rows), &rows_ctl->total}, a->cols,
                               CsrOut{result_rp, z->j_idx, z->val, nullptr, length_word, rows_ctl}, nullptr, entry_scratch, stream, &ctl)))
            return st;
    }
    if ((st = wait_result_word(rows_word, stream, &n_rows, &rows_status))) return st;
    n_rows &= RW_HOLLOW - 1;
    if (one_pass) {
        if ((st = wait_result_word(length_word, stream, &length, &device_status))) return st;
        hollow = (length & RW_HOLLOW) != 0;
        length &= RW_HOLLOW - 1;
        if (length > INT32_MAX) return NB200_E_OVERFLOW;
        z->nnz = (int32_t)length;
    }
    if (rows_status != 0 || device_status != 0) {
        NB200_CUDA(cudaMemcpyAsync(ws->host, rows_status != 0 ? rows_ctl : ctl, sizeof(FusedCtl), cudaMemcpyDeviceToHost, stream));
        NB200_CUDA(cudaStreamSynchronize(stream));
        FusedCtl h;
        std::memcpy(&h, ws->host, sizeof(h));
        return note_timeout(h.status.error, h.status.detail, "dcsr merge");
    }
    if (!one_pass) {  // less room than the worst case: count first
        const nb200_csr ca{(int32_t)n_rows, a->cols, a->nnz, off_a, a->j_idx, a->val}, cb{(int32_t)n_rows, b->cols, b->nnz, off_b, b->j_idx, b->val};
        nb200_csr cz{(int32_t)n_rows, a->cols, 0, result_rp, z->j_idx, z->val};
        st = op(&ca, &cb, &cz, capacity, stream_v);
        z->nnz = cz.nnz;
        if (st != NB200_OK) return st;
        hollow = true;  // (not reported on this route: check below)
    }

    // ---- the rows the result stores
    if (!is_union) return compress_rows(keep, (int32_t)n_rows, ids, rpz, scan_block, z, kept_word, stream);
    z->n_i = (int32_t)n_rows;
    if (!hollow) return NB200_OK;
    NB200_CUDA(cudaMemcpyAsync(ids, z->i_idx, sizeof(int32_t) * (size_t)n_rows, cudaMemcpyDeviceToDevice, stream));
    NB200_CUDA(cudaMemcpyAsync(rpz, z->j_ptr, sizeof(int32_t) * ((size_t)n_rows + 1), cudaMemcpyDeviceToDevice, stream));
    {
        LaunchScope scope("dcsr_keep", stream);
        k_rows_nonempty<<<(int)((n_rows + NT - 1) / NT), NT, 0, stream>>>(rpz, (int32_t)n_rows, keep);
    }
    NB200_CUDA(cudaGetLastError());
    return compress_rows(keep, (int32_t)n_rows, ids, rpz, scan_block, z, kept_word, stream);
}

}  // namespace

}  // namespace nb200

using namespace nb200;

extern "C" {

int nb200_coo_add_f32_into(const nb200_coo *a, const nb200_coo *b, nb200_coo *z, int64_t capacity, void *stream) {
    return coo2_run(nb200_csr_add_f32_into, true, a, b, z, capacity, stream);
}

int nb200_coo_mul_f32_into(const nb200_coo *a, const nb200_coo *b, nb200_coo *z, int64_t capacity, void *stream) {
    return coo2_run(nb200_csr_mul_f32_into, false, a, b, z, capacity, stream);
}

int nb200_coo_csr_add_f32_into(const nb200_csr *a, const nb200_coo *b, nb200_csr *z, int64_t capacity, void *stream_v) {
    int st;
    if ((st = check_coo(b))) return st;
    if (!a || a->rows != b->rows || a->cols != b->cols) return NB200_E_BADARG;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
    Scratch2d s;
    if ((st = take_scratch(b->rows, stream, &s))) return st;
    cudaError_t e = launch_row_offsets(b->i, nullptr, b->nnz, b->rows, s.rpb, stream);
    if (e != cudaSuccess) return note_cuda_error(e, "k_row_offsets");
    const nb200_csr cb{b->rows, b->cols, b->nnz, s.rpb, b->j, b->val};
    return nb200_csr_add_f32_into(a, &cb, z, capacity, stream_v);
}

int nb200_dcsr_add_f32_into(const nb200_dcsr *a, const nb200_dcsr *b, nb200_dcsr *z, int64_t cap_i, int64_t capacity, void *stream) {
    return dcsr2_run(nb200_csr_add_f32_into, true, a, b, z, cap_i, capacity, stream);
}

int nb200_dcsr_mul_f32_into(const nb200_dcsr *a, const nb200_dcsr *b, nb200_dcsr *z, int64_t cap_i, int64_t capacity, void *stream) {
    return dcsr2_run(nb200_csr_mul_f32_into, false, a, b, z, cap_i, capacity, stream);
}

}  // extern "C"
