// Types and small helpers shared by the CSR element-wise kernels (csr_merge.cu) and by the formats that run on
// them (formats2d.cu, csf3_add.cu).
#pragma once

#include <stdint.h>

#include "block_utils.cuh"
#include "common.cuh"
#include "merge_common.cuh"
#include "tma.cuh"

namespace nb200 {

constexpr int CSR_NT = 256;  // threads of a CSR tile CTA

struct CsrIn {
    const int32_t *rp;  // null: a single row that holds all entries
    const int32_t *col;
    const float *val;
    int32_t nnz;                         // stored entries, or the most there can be where
    const long long *nnz_dev = nullptr;  // an earlier launch on the stream leaves their number in device memory
    __device__ __forceinline__ int32_t entries() const { return nnz_dev ? (int32_t)*nnz_dev : nnz; }
};

struct CsrOut {
    int32_t *rp;
    int32_t *col;
    float *val;
    // Asynchronous calls only: three device words {result entries, status, rows} the kernels fill
    // themselves. The partition kernel writes rows and a status of 0, the last tile the length, and
    // any tile whose bounded wait gives up (or a length beyond int32) raises the status.
    long long *result = nullptr;
    // Calls that wait for their length: the result word in pinned host memory that the last tile writes.
    unsigned long long *host = nullptr;
    // ... and the control block of the earlier merge that this one builds on: the word reports its status and hollow flag
    // too, and where it gave up nothing that it should have left is read.
    const FusedCtl *earlier = nullptr;
};

// What a merge of positions carries instead of values (offsets mode of the tile kernel): the operands'
// entries stand for ranges of a lower level, entry p of A for [a[p], a[p + 1]). For every result entry u,
// off_a[u] is the start of A's range where A holds the entry, else the start of its next one (the end of
// the last range behind the last entry), so that off_a is a row-offset array over the result entries in
// which an entry that A lacks is an empty row; off_b likewise. keep[u], when asked for, says that both hold
// u with a range that is not empty. *hollow is raised if a result entry stands for no range but empty ones.
struct LevelOffsets {
    const int32_t *a = nullptr, *b = nullptr;
    int32_t *off_a = nullptr, *off_b = nullptr, *keep = nullptr;
};

__device__ __forceinline__ int32_t row_offset(const CsrIn &m, int64_t r) { return m.rp ? ld_late(m.rp + r) : r > 0 ? m.entries() : 0; }

constexpr int MBAR_POLL_LIMIT = 1 << 24;
constexpr int ERR_COPY_TIMEOUT = 2;

// Number of 4-byte elements from `p` up to the next 16-byte boundary (0..3).
__device__ __forceinline__ int head_elems(const void *p) {
    return (int)(((16u - (unsigned)(reinterpret_cast<uintptr_t>(p) & 15u)) & 15u) >> 2);
}

inline int col_bits(int32_t cols) {
    int b = 1;
    while (b < 32 && (int64_t(1) << b) < (int64_t)cols) ++b;
    return b;
}

inline int check_csr(const nb200_csr *m, bool need_arrays) {
    if (!m || m->rows < 0 || m->cols < 0 || m->nnz < 0) return NB200_E_BADARG;
    if (need_arrays && (!m->row_ptr || (m->nnz > 0 && (!m->col || !m->val)))) return NB200_E_BADARG;
    return NB200_OK;
}

// A row count that a call knows (`dev` null) or that an earlier launch on the stream leaves in device memory.
struct RowCount {
    int32_t value = 0;  // beside `dev`: the most there can be (0: unknown; chooses the tile, nothing else)
    const long long *dev = nullptr;
    bool short_rows = false;  // rows of a few dozen entries or less (chooses the tile, nothing else)
    __device__ __forceinline__ int32_t get() const { return dev ? (int32_t)*dev : value; }
};

constexpr long long RW_HOLLOW = 1ll << 48;  // beside the length in a result word: the hollow flag of this or an earlier launch

// Test knobs of a launch: the first tile to run (a self-test of the bounded waits leaves tile 0
// out, so that every other tile waits for a count that never comes) and the number of polls after
// which a tile gives up on a cut or on its output base.
struct LaunchKnobs {
    int first_tile = 0;
    int poll_limit = LOOKBACK_POLL_LIMIT;
};
constexpr int64_t SELFTEST_ENTRIES = 24000;  // three tiles, of whatever size: enough for one to be left out

// One single-pass merge as part of a longer call: the partition and the tile kernel are queued and nothing
// is waited for. `scratch` holds csr2_scratch_bytes(entries) bytes; the control block (length, status) that
// *ctl then points to lies in it, or in a block of the stream's that the next three merges there leave alone. With `levels` the offsets mode runs (values are not read).
size_t csr2_scratch_bytes(int64_t entries);
int csr2_enqueue(SetOp op, const CsrIn &A, const CsrIn &B, const RowCount &rows, int32_t cols, const CsrOut &Z, const LevelOffsets *levels,
                 void *scratch, cudaStream_t stream, FusedCtl **ctl, const LaunchKnobs &knobs = LaunchKnobs());

}  // namespace nb200
