// CSR + CSR element-wise kernels: sorted union (add) and intersection (multiply) of two CSR
// operands, as flat merge-path over the (row, column) order.
//
// The merged sequence of all stored entries of A and B, ordered by (row, column) with A first
// on ties, is cut into tiles of a few thousand entries. A partition kernel finds every cut with
// k-ary searches (rows on the summed row offsets, then the merge-path diagonal inside the row).
// One CTA then owns one tile: the copy engine stages the tile's columns in shared memory (the values are
// prefetched into L2 meanwhile), every row that begins in the tile adds one to the upper bits of its first column (so a
// key of the next entry is "row of the entry before it + this word"), every thread finds where its
// share of the merged sequence begins with two searches in shared memory, and merges the columns of its entries
// one result after the other, noting where each comes from. The tile's count goes out; the columns of the results are taken into
// registers by those notes, in order, and for a sum the values then take the place of the columns in shared memory; both are written
// back coalesced. Row offsets of the result are produced by
// the same pass: a tile owns the offsets of the rows that begin inside it.
//
// Reference behaviour restated (not its code): partition src/backend/partition.cpp:813-993
// (equal columns never split, :964-983), count src/backend/compute.cpp:152-271, fill
// :273-411, value expressions :426-440, empty-result path
// src/backend/stitch_and_generate.cpp:168-220.
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <type_traits>

#include "csr_common.cuh"

namespace nb200 {

namespace {

constexpr int NT = CSR_NT;

// Tile cuts: for cut t, {the row it falls in, the absolute positions in A and B, unused}. Without them the tiles find their cuts themselves, every
// `step` merged entries, with words of their own (no step: a single tile, whose two cuts need no search).
struct Cuts {
    int4 *at = nullptr;
    int32_t step = 0;
    OwnWords own;
};

// One tile: rows i0 (where it begins) .. i1 (where the next one begins), its entries in A and B.
struct TileRange {
    int32_t i0, i1, a0, b0;
    int na, nb;
};

// Result words of an asynchronous call (CsrOut::result), written from inside the tile kernel.
__device__ __forceinline__ void publish_length(long long *result, long long total) {
    if (!result) return;
    result[0] = total;
    if (total > INT32_MAX) atomicMax(result + 1, (long long)NB200_E_OVERFLOW);
}
__device__ __forceinline__ void publish_timeout(long long *result) {
    if (result) atomicMax(result + 1, (long long)NB200_E_TIMEOUT);
}

// Whether an earlier launch on the stream, whose results a kernel builds on, ended without them.
__device__ __forceinline__ bool gave_up(const FusedCtl *earlier) { return earlier && earlier->status.error != 0; }

// The last tile has its base: the result length (negative after a give-up of any tile) goes to the control block and to whoever waits for it.
__device__ __forceinline__ void finish_total(FusedCtl *ctl, const CsrOut &Z, long long total) {
    int status = total < 0 ? NB200_E_TIMEOUT : NB200_OK;
    if (total >= 0) {
        ctl->total = total;
        publish_length(Z.result, total);
    } else {
        publish_timeout(Z.result);
    }
    long long value = total < 0 ? 0 : total;
    if (Z.earlier) {  // complete since before this launch; handed on, so that the last launch of a chain reports all of it
        if (gave_up(Z.earlier)) {
            status = NB200_E_TIMEOUT;
            ctl->status = Z.earlier->status;
        }
        if (Z.earlier->hollow) {
            ctl->hollow = 1;
            value |= RW_HOLLOW;
        }
    }
    publish_result_word(Z.host, status, value);
}

// ------------------------------------------------------------------------- partition ----

// Cut t, at merged position min(t * tile_step, total), by G neighbouring lanes; all lanes of a warp call this together.
template <int G>
__device__ __forceinline__ int4 find_cut(const CsrIn &A, const CsrIn &B, const int32_t rows, const int32_t tile_step, const int t, const int num_tiles,
                                         const bool failed) {
    const uint32_t total = (uint32_t)A.entries() + (uint32_t)B.entries();  // may be less than the tiles cover
    const int32_t a_base = row_offset(A, 0), b_base = row_offset(B, 0);
    const uint32_t d = (uint32_t)min((int64_t)t * tile_step, (int64_t)total);
    const bool inner = t > 0 && t < num_tiles && d < total && !failed;
    // Row holding merged position d: the largest i with work(i) <= d, where work(i) is the number of
    // entries of A and B in rows before i; work(0) = 0, so it is the number of rows i >= 1 that satisfy it.
    const int32_t row = (int32_t)group_count_true<G>(1, inner ? (uint32_t)rows : 1u, [&](uint32_t i) {
        return (uint32_t)(row_offset(A, i) - a_base) + (uint32_t)(row_offset(B, i) - b_base) <= d;
    }) - 1;
    const int32_t a_lo = row_offset(A, row), a_hi = row_offset(A, row + 1);
    const int32_t b_lo = row_offset(B, row), b_hi = row_offset(B, row + 1);
    const int64_t dd = (int64_t)d - ((int64_t)(a_lo - a_base) + (int64_t)(b_lo - b_base));
    const int64_t len_a = a_hi - a_lo, len_b = b_hi - b_lo;
    // Merge-path diagonal dd inside the row: x entries of A and dd - x of B come first.
    const uint32_t x_lo = (uint32_t)max((int64_t)0, dd - len_b), x_hi = (uint32_t)min(dd, len_a);
    const uint32_t x = group_count_true<G>(x_lo, inner ? x_hi : x_lo, [&](uint32_t m) {
        return ld_late(A.col + a_lo + m) <= ld_late(B.col + b_lo + (dd - 1 - m));
    });
    int64_t y = dd - x;
    if (failed) return make_int4(0, 0, 0, 0);
    if (!inner) return t == 0 ? make_int4(0, a_base, b_base, 0) : make_int4(rows, a_base + A.entries(), b_base + B.entries(), 0);
    // Keep a column present in both operands on one side of the cut.
    if (x > 0 && y < len_b && ld_late(A.col + a_lo + x - 1) == ld_late(B.col + b_lo + y)) ++y;
    return make_int4(row, a_lo + (int32_t)x, b_lo + (int32_t)y, 0);
}

// The same by a warp, for a tile of its own accord.
__device__ __forceinline__ int4 tile_cut(const CsrIn &A, const CsrIn &B, const RowCount &row_count, const int32_t tile_step, const int t, const int num_tiles,
                                      const FusedCtl *earlier) {
    return find_cut<32>(A, B, row_count.get(), tile_step, t, num_tiles, gave_up(earlier));
}

// A CTA in front of the tiles: eight lanes per cut, NT / 8 cuts a round.
__device__ __forceinline__ void make_cuts(const CsrIn &A, const CsrIn &B, const RowCount &row_count, const Cuts &cuts, const int num_tiles, const FusedCtl *earlier) {
    constexpr int G = 8;
    const int32_t rows = row_count.get();
    const bool failed = gave_up(earlier);
    for (int first = cuts.own.first_cut() + blockIdx.x * (NT / G); first <= num_tiles; first += CUTTERS * (NT / G)) {
        const int t = first + threadIdx.x / G;
        const int4 cut = find_cut<G>(A, B, rows, cuts.step, min(t, num_tiles), num_tiles, failed);
        if ((threadIdx.x & (G - 1)) == 0 && t <= num_tiles) store_cut(cuts.own, t, cut);
    }
}

// G lanes per cut.
template <int G>
__global__ void __launch_bounds__(NT) k_csr2_partition(CsrIn A, CsrIn B, RowCount row_count,
                                                       int32_t tile_step, int32_t num_tiles, int4 *cuts, long long *result,
                                                       uint64_t *zero_block, int zero_words, const FusedCtl *earlier) {
    wait_for_previous();   // the scratch that is cleared below may still be in use
    trigger_dependents();  // the tile kernel may take its places; it waits for the cuts
    const int64_t gid = (int64_t)blockIdx.x * NT + threadIdx.x;
    const int32_t rows = row_count.get();
    // The merge in front of this one gave up: its offsets and columns are whatever the scratch held. No offset is
    // followed, and every tile is empty; the tile kernel hands the status on.
    const bool failed = gave_up(earlier);
    if (result && gid == 0) {  // the tile kernel that follows fills in the rest
        result[1] = NB200_OK;
        result[2] = rows;
    }
    // the control block and the tile words of the kernel that follows start from zero (the grid has at
    // least G >= 8 threads per tile word, so one word per thread covers them)
    if (gid < zero_words) zero_block[gid] = 0;
    const int t = (int)min(gid / G, (int64_t)num_tiles);  // spare groups repeat the last cut
    const int4 cut = find_cut<G>(A, B, rows, tile_step, t, num_tiles, failed);
    if ((threadIdx.x & (G - 1)) == 0 && gid / G <= num_tiles) cuts[t] = cut;
}

// ------------------------------------------------------------------------ tile kernel ----


// Large tile where the caller says that rows are short (the fibres of a tree): a tile of 31 with more rows than fit takes
// longer than the others and holds up their output bases, and the twin mask by entries (below) pays. Trees of 25 M entries per operand, whole call, with 1, 2, 4, 12
// entries per fibre 440, 370, 292, 239 us with 21, 447, 373, 305, 250 with 17, 533, 358, 283, 232 with 23 and 532, 409, 280, 228 with 31; 8 M with 1 and 2 174 and 146 with
// 21, 204 and 160 with 31.
constexpr int V_FIBRES = 21, V_MOST = 31;  // V_MOST: the large tile otherwise

// Shared-memory plan of the tile body. The column words of both operands lie in one array: A's entry e at
// word oa + e, B's at word ob + e, where oa and ob are chosen so that a global address on a 16-byte
// boundary lands on a 16-byte boundary in shared memory too (what a bulk copy needs). Behind them, one
// 16-bit word per result entry says where it comes from (offsets mode: two, for both operands).
template <int VT, bool LEVELS>
struct TilePlan {
    static constexpr int CAP = NT * VT;         // most merged entries of one tile
    static constexpr int SLOTS = CAP + 16;      // + alignment words of both operands and their sentinels
    // Row starts kept in shared memory; tiles with more rows search the offsets in global memory. The most of which four CTAs
    // fit an SM; the small tile and that for fibres have room for a row per entry.
    static constexpr int ROWS = VT > 21 ? 1856 : VT > 15 ? CAP : 4096;
    static constexpr size_t ROWS_AT = (LEVELS ? 8 : 6) * (size_t)SLOTS;
    static constexpr size_t BYTES = ROWS_AT + 4 * (size_t)(ROWS + 2);
    static_assert(VT <= 31, "a thread's twins are kept in the lower 31 bits of a word");
    static_assert(4 * SLOTS < 32768, "byte offsets of entries are kept in 15 bits");
};
constexpr uint32_t ROW_FAR = 0xffffu;

// A tile, other than the large one, asks for the row offsets of one that starts a few microseconds later, so that they wait in L2:
// they are read by plain loads, a few dependent rounds of them. (Trees of 50 M entries per operand in fibres of 1, 6 and 30 entries 827, 498, 400 us without, 807, 495, 396
// so; of 8 M no difference. The columns ahead as well cost the largest sums 1 to 4 %, whether 64, 148, 296 or 592 tiles ahead, when tiles gathered their values.) Not for a tile that starts with the
// first ones, and at most as many offsets as a tile keeps: beyond those lie runs of empty rows, which could fill the L2.
constexpr int TILES_AHEAD = 148;
// Tiles up to which a call that waits for its length is one launch. Two operands of 24, 32, 40 and 50 M entries (6050, 8070, 10090 and 12610 tiles) take
// 171.4, 217.4, 262.1 and 319.4 us with a launch for the cuts in front, 168.8, 216.3, 263.9 and 323.6 without: the places of the CTAs that make
// the cuts are worth more than the time before the first tile then.
constexpr int OWN_CUTS_UP_TO = 8192;

// Fixed shared memory of a tile (one block for both key widths).
struct TileShared {
    uint64_t mbar;
    long long base;                 // output base of the tile
    int4 cut[2];                    // where it begins and ends, if it finds that out itself
    int lost;                       // a cut did not come in time
    int trow[NT], wrow[NT / 32];    // the last row that starts at or before a thread's / between two warps' diagonals;
                                    // once every thread has its row, trow holds the threads' first results instead
    unsigned twin[NT];
    int wtotal[NT / 32];            // survivors of each warp
};

// The last of rows from + 1 .. nr (relative to the tile) that starts at or before an entry, by bisection of the row offsets. A call,
// because a merge with 64-bit keys has it twice in each of its steps, up to 62 times in a kernel: with the loop in every place such a
// kernel waited for its instructions more than for anything else (9.8 of 18 stalled warps for each that issues, a third of the slots
// used; beside the larger second half of a tile a sum of 33 M entries in columns beyond 2^30 went from 524 to 747 us a call; so 400).
__device__ __noinline__ int far_row(const int32_t *rp, const int32_t entry, const int from, const int nr) {
    int r = from + 1, top = nr;
    while (r < top) {
        const int mid = (r + top + 1) >> 1;
        if (ld_late(rp + mid) <= entry) r = mid; else top = mid - 1;
    }
    return r;
}

// The tile body. Keys order entries by (row in tile, column):
//   narrow  32 bits, (row << cbits) | column. A staged word is a column; the first entry of a row also
//           carries, above the column bits, how many rows begin there, so that the key after key k of the
//           same operand is (k & row bits) + next word. That is all the row handling there is: no key array
//           is ever written.
//   WIDE    64 bits, row and column, for tiles that span too many rows for that (rows of an entry or two,
//           long runs of empty rows): the row of an entry that begins one comes from its row mark.
// A row mark is 16 bits per staged word, in the place of the source indices that come later: the last row
// that begins at the entry (ROW_FAR: beyond 16 bits, looked up in the row offsets).
//
// What bounds this kernel is instruction issue and, for a tile, latency: phases that barriers separate, with a wait for its columns in front (2.97 of
// its 13 us; the wait for the counts of all earlier tiles is 0.15). So
//   - the merge is sequential and moves columns only: one compare and at most two loads per result entry
//     (a key-building pass, a register merge network and a per-entry value gather took four times the
//     instructions), and it leaves a 16-bit source index per result entry;
//   - the tile's count goes out right after it; a sum's results take their columns into registers, which frees the words for a
//     second copy, of the values, while the count travels. One wait covers both, and no thread fetches a value from L2 with an
//     address of its own: gathering values in four batches behind the base took 17 instructions and 2 trips to L2 more per eight results
//     (67 M entries 446 -> 410 us a call, 16 M in rows of 16 172 -> 138, three operands of 9 M 239 -> 194, a tree of 25 M 359 -> 323);
//   - an intersection keeps the gather: its results are few, and most values would be copied for nothing. What follows from a twin is done in a
//     loop over a thread's twins, not as a test per step (16 M entries, half of them shared: 122 -> 114 us);
//   - a tile needs 6 bytes of shared memory per entry instead of 16: 55 KB with 31 entries per thread, so four CTAs share an SM.
template <int VT, int OP, int MODE, bool LEVELS, bool OWN, bool WIDE>
__device__ __forceinline__ void csr2_tile(const CsrIn &A, const CsrIn &B, const TileRange &tile, const int cbits, const int t,
                                          const int num_tiles, int32_t *tile_count, const TileWords &words, FusedCtl *ctl,
                                          const CsrOut &Z, const LevelOffsets &L, unsigned char *smem_raw, TileShared &sh,
                                          const int poll_limit) {
    using P = TilePlan<VT, LEVELS>;
    using Key = typename std::conditional<WIDE, uint64_t, uint32_t>::type;
    constexpr int W = NT / 32;
    constexpr Key END = WIDE ? (Key)~0ull : (Key)0x80000000u;  // after every key (narrow: keys are below 2^31), also with row bits added
    constexpr bool WRITES = MODE != MODE_COUNT;
    // Rows of an entry or two: a mask by entries instead of steps spares every row offset a search of it (trees of 25 M entries per
    // operand with 1 and 2 in a fibre: 461 -> 440, 378 -> 370 us). With fewer rows the mask costs more than the searches (12 in a fibre 235 -> 239).
    constexpr bool MANY_ROWS = VT == V_FIBRES;
    uint32_t *s_rows = reinterpret_cast<uint32_t *>(smem_raw + P::ROWS_AT);  // start of row r in the tile: A's in the lower half, B's in the upper
    int *s_trow = sh.trow, *s_wrow = sh.wrow, *s_rank = sh.trow, *s_wtotal = sh.wtotal;
    unsigned *s_twin = sh.twin;
    long long &s_base = sh.base;
    uint64_t *mbar = &sh.mbar;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int na = tile.na, nb = tile.nb, n = na + nb;
    const int nr = tile.i1 - tile.i0;  // rows 1 .. nr (relative) begin in this tile
    const bool rows_fit = nr <= P::ROWS;
    const uint32_t cmask = WIDE ? 0xffffffffu : (1u << cbits) - 1u;
    uint32_t *keys = reinterpret_cast<uint32_t *>(smem_raw);
    using Src = typename std::conditional<LEVELS, uint32_t, uint16_t>::type;
    Src *src_of = reinterpret_cast<Src *>(smem_raw + 4 * P::SLOTS);
    uint16_t *row_mark = reinterpret_cast<uint16_t *>(smem_raw + 4 * P::SLOTS);
    auto word_at = [&](uint32_t byte) -> uint32_t & { return *reinterpret_cast<uint32_t *>(smem_raw + byte); };

    const int32_t *ga_col = A.col + tile.a0, *gb_col = B.col + tile.b0;
    const float *ga_val = A.val + tile.a0, *gb_val = B.val + tile.b0;
    const int ha = head_elems(ga_col), hb = head_elems(gb_col);
    const int oa = (4 - ha) & 3;
    const int ob = ((oa + na + 1 + 3) & ~3) + ((4 - hb) & 3);  // A's sentinel lies before it

    // ---- stage the columns. One thread hands the 16-byte-aligned interior of each array to the copy
    // engine (and asks for the values' lines in L2); a few others load the ragged ends (at most 3 entries
    // each side).
    const int head_a = min(na, ha), head_b = min(nb, hb);
    const int nva = (na - head_a) >> 2, nvb = (nb - head_b) >> 2;  // 16-byte vectors in the interior
    if (tid == 0) {
        mbar_arrive_expect_tx(mbar, 16u * (uint32_t)(nva + nvb));
        if (nva) bulk_load(keys + oa + head_a, ga_col + head_a, 16u * nva, mbar);
        if (nvb) bulk_load(keys + ob + head_b, gb_col + head_b, 16u * nvb, mbar);
        if (WRITES && OP == OP_UNION && !LEVELS) {
            prefetch_l2(ga_val, na);
            prefetch_l2(gb_val, nb);
        }
        if (!rows_fit) {  // read three times
            if (A.rp) prefetch_l2(A.rp + tile.i0 + 1, nr);
            if (B.rp) prefetch_l2(B.rp + tile.i0 + 1, nr);
        }
    }
    if (tid >= 32 && tid < 32 + 12) {  // ragged ends: 3 head + 3 tail slots for A, then for B
        const int k = tid - 32;
        const bool is_b = k >= 6;
        const int e = is_b ? k - 6 : k;
        const int count = is_b ? nb : na, head = is_b ? head_b : head_a, nv = is_b ? nvb : nva;
        const int idx = e < 3 ? e : head + 4 * nv + (e - 3);
        if (e < 3 ? e < head : idx < count) keys[(is_b ? ob : oa) + idx] = (uint32_t)ld_late((is_b ? gb_col : ga_col) + idx);
    }
    if (tid == 64) keys[oa + na] = (uint32_t)END;
    if (tid == 65) keys[ob + nb] = (uint32_t)END;
    s_trow[tid] = 0;
    if (WIDE) for (int i = tid; i < P::SLOTS / 2; i += NT) reinterpret_cast<uint32_t *>(row_mark)[i] = 0u;
    if (tid < W) s_wrow[tid] = 0;

    // ---- row starts (relative to the tile), while the copies fly. Row 0 is the one the tile begins in. A few rows fall to
    // the last warps, which have nothing to stage: plain loads do not pass the staging.
    auto global_start = [&](int r) -> uint32_t {
        return (uint32_t)(row_offset(A, (int64_t)tile.i0 + r) - tile.a0) | (uint32_t)(row_offset(B, (int64_t)tile.i0 + r) - tile.b0) << 16;
    };
    constexpr int RB = 4;  // rows a thread fetches together
    if (nr <= NT) {
        if (NT - tid <= nr) s_rows[NT - tid] = global_start(NT - tid);
    } else if (rows_fit) {
        for (int r0 = 1; r0 <= nr; r0 += RB * NT) {
            uint32_t w[RB];
#pragma unroll
            for (int u = 0; u < RB; ++u) {
                const int r = r0 + u * NT + tid;
                w[u] = r <= nr ? global_start(r) : 0u;
            }
#pragma unroll
            for (int u = 0; u < RB; ++u) {
                const int r = r0 + u * NT + tid;
                if (r <= nr) s_rows[r] = w[u];
            }
        }
    }
    if (rows_fit && tid == 0) {
        s_rows[0] = 0u;
        s_rows[nr + 1] = (uint32_t)na | (uint32_t)nb << 16;
    }
    auto row_start = [&](int r) -> uint32_t {  // packed like s_rows, r in [0, nr + 1]
        if (rows_fit) return s_rows[r];
        return r == 0 ? 0u : r > nr ? (uint32_t)na | (uint32_t)nb << 16 : global_start(r);
    };
    const bool landed = wid > 0 || mbar_wait_bounded(mbar, 0, MBAR_POLL_LIMIT);  // one warp polls; the others' issue slots are worth more
    if (!__syncthreads_and(landed)) {  // the copies did not land in time: report, touch nothing
        if (tid == 0) {
            if (atomicCAS(&ctl->status.error, 0, ERR_COPY_TIMEOUT) == 0) ctl->status.detail = t;
            publish_timeout(Z.result);
            if (MODE == MODE_FUSED) {
                publish_failure(words, t);
                if (t == num_tiles - 1) publish_result_word(Z.host, NB200_E_TIMEOUT, 0);
            }
            mbar_wait_bounded(mbar, 0, MBAR_POLL_LIMIT);        // second bounded wait for copies in flight
        }
        return;
    }

    // ---- every row that begins in the tile adds one above the column bits of its first entry (several
    // where empty rows share a start), and the last row that starts at or before a thread's diagonal is
    // noted for that thread, and for its warp
    auto begin_row = [&](const int r, const uint32_t w, const uint32_t w_next) {
        const int sa = (int)(w & 0xffffu), sb = (int)(w >> 16);
        if (!WIDE) {
            if (sa < na) atomicAdd(keys + oa + sa, 1u << cbits);
            if (sb < nb) atomicAdd(keys + ob + sb, 1u << cbits);
        }
        const uint16_t mark = (uint16_t)min((uint32_t)r, ROW_FAR);
        if (sa < (int)(w_next & 0xffffu)) row_mark[oa + sa] = mark;  // row r holds entries of A: nothing else marks that word
        if (sb < (int)(w_next >> 16)) row_mark[ob + sb] = mark;
        const int q = (sa + sb + VT - 1) / VT;  // the first thread whose diagonal is not before this row
        const int q_next = r < nr ? ((int)(w_next & 0xffffu) + (int)(w_next >> 16) + VT - 1) / VT : NT + 32;
        if (q < NT && q_next != q) {
            s_trow[q] = r;
            if ((q_next >> 5) != (q >> 5)) s_wrow[q >> 5] = r;
        }
    };
    if (rows_fit) {
        for (int r = 1 + tid; r <= nr; r += NT) begin_row(r, s_rows[r], s_rows[r + 1]);
    } else {
        for (int r0 = 1; r0 <= nr; r0 += RB * NT) {
            uint32_t w[RB], w_next[RB];
#pragma unroll
            for (int u = 0; u < RB; ++u) {
                const int r = r0 + u * NT + tid;
                w[u] = r <= nr ? global_start(r) : 0u;
                w_next[u] = r <= nr ? row_start(r + 1) : 0u;
            }
#pragma unroll
            for (int u = 0; u < RB; ++u)
                if (r0 + u * NT + tid <= nr) begin_row(r0 + u * NT + tid, w[u], w_next[u]);
        }
    }
    __syncthreads();

    // ---- where this thread's share begins: the row of merged position tid * VT, then the merge-path
    // diagonal inside that row (ties take A first; a column both operands hold stays on one side)
    const int diag = min(tid * VT, n);
    int x, y, shifted = 0, row;
    Key ka = END, kb = END;
    int row_a = 0, row_b = 0;  // WIDE: row of each head
    // row of the entry at staged word `at`, position `pos` of its operand, that begins one after row `from`
    auto marked_row = [&](const int at, const int pos, const int from, const int shift) -> int {
        const uint32_t mark = row_mark[at];
        if (mark != ROW_FAR) return (int)mark;
        return shift ? far_row(B.rp + tile.i0, tile.b0 + pos, from, nr) : far_row(A.rp + tile.i0, tile.a0 + pos, from, nr);
    };
    {
        row = (int)warp_incl_max((unsigned)s_trow[tid]);
        row = max(row, (int)__reduce_max_sync(FULL_MASK, lane < wid ? (unsigned)s_wrow[lane & (W - 1)] : 0u));
        const uint32_t w0 = row_start(row), w1 = row_start(row + 1);
        const int a_lo = (int)(w0 & 0xffffu), b_lo = (int)(w0 >> 16), a_hi = (int)(w1 & 0xffffu), b_hi = (int)(w1 >> 16);
        const int dd = diag - a_lo - b_lo;
        int lo = max(0, dd - (b_hi - b_lo)), up = min(dd, a_hi - a_lo);
        const uint32_t *ca = keys + oa + a_lo, *cb = keys + ob + b_lo + dd - 1;
        while (lo < up) {
            const int mid = (lo + up) >> 1;
            if ((ca[mid] & cmask) <= (cb[-mid] & cmask)) lo = mid + 1; else up = mid;
        }
        x = a_lo + lo;
        y = b_lo + dd - lo;
        if (lo > 0 && y < b_hi && ((keys[oa + x - 1] ^ keys[ob + y]) & cmask) == 0u) {
            ++y;
            shifted = 1;
        }
        // keys of the two heads. A head beyond this row begins a later row of its operand.
        auto head_key = [&](const int at, const int pos, const int end, const int count, const int shift, int &head_row) -> Key {
            head_row = row;
            if (pos >= count) return END;
            if (pos >= end) head_row = marked_row(at, pos, row, shift);
            return WIDE ? (Key)((uint64_t)(uint32_t)head_row << 32 | keys[at]) : (Key)((uint32_t)head_row << cbits | (keys[at] & cmask));
        };
        if (diag < n) {
            ka = head_key(oa + x, x, a_hi, na, 0, row_a);
            kb = head_key(ob + y, y, b_hi, nb, 16, row_b);
        }
    }

    // ---- merge, one result entry per step: take the smaller head, or both where they are equal. Offsets are
    // in bytes from the start of the column words. src[i]: the entry step i took (A's where both), with
    // the top bit set where it took both; in the offsets mode both heads, bit 0 of each half set where it was taken.
    const uint32_t pa0 = 4u * (uint32_t)(oa + x), pb0 = 4u * (uint32_t)(ob + y);
    uint32_t src[VT];
    unsigned twin = 0;  // bit i: step i took an entry of each operand
    int steps;
    {
        // Every thread takes VT steps, whatever its share: what runs over the end (into the next thread's share, or past
        // a sentinel into other words of the tile's shared memory) is cut off afterwards, which is cheaper than a test
        // per step. The word behind each head is loaded a step ahead, so that a step waits for no load of its own.
        uint32_t pa = pa0, pb = pb0;
        uint32_t next_a = word_at(pa + 4), next_b = word_at(pb + 4);
#pragma unroll
        for (int i = 0; i < VT; ++i) {
            const bool ta = ka <= kb, tb = kb <= ka;
            const uint32_t row_bits = (uint32_t)min(ka, kb) & ~cmask;
            if (LEVELS) {
                src[i] = (pa | (ta ? 1u : 0u)) | (pb | (tb ? 1u : 0u)) << 16;
            } else {
                src[i] = ta ? pa : pb;
            }
            if (ta && tb) twin |= 1u << i;
            if (ta) {
                pa += 4;
                if (!WIDE) {
                    ka = (Key)(row_bits + next_a);
                    next_a = word_at(pa + 4);
                } else {
                    const int at = (int)(pa >> 2), pos = at - oa;
                    if (pos < na && row_mark[at]) row_a = marked_row(at, pos, row_a, 0);
                    ka = pos < na ? (Key)(((uint64_t)(uint32_t)row_a << 32) | word_at(pa)) : END;
                }
            }
            if (tb) {
                pb += 4;
                if (!WIDE) {
                    kb = (Key)(row_bits + next_b);
                    next_b = word_at(pb + 4);
                } else {
                    const int at = (int)(pb >> 2), pos = at - ob;
                    if (pos < nb && row_mark[at]) row_b = marked_row(at, pos, row_b, 16);
                    kb = pos < nb ? (Key)(((uint64_t)(uint32_t)row_b << 32) | word_at(pb)) : END;
                }
            }
        }
        // step i is the thread's where the entries taken before it, i + (twins before it), are fewer than its share
        const int share = min(tid * VT + VT, n) - diag - shifted;
        steps = share;
        if (__any_sync(FULL_MASK, twin != 0u)) {
            int lo = 0, hi = share;
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (mid + __popc(twin & ((1u << mid) - 1u)) >= share) hi = mid; else lo = mid + 1;
            }
            steps = lo;
        }
        twin &= (1u << steps) - 1u;
    }

    // ---- rank the survivors inside the tile
    const int mine = OP == OP_UNION ? steps : __popc(twin);
    const int incl = warp_incl_sum(mine);
    if (lane == 31) s_wtotal[wid] = incl;
    if (!MANY_ROWS) s_twin[tid] = twin | (unsigned)shifted << 31;  // bit i: step i took an entry of each operand
    __syncthreads();  // also retires the merge of every thread: words of consumed twins may change from here on
    int total = 0, wbase = 0;
#pragma unroll
    for (int w = 0; w < W; ++w) {
        const int c = s_wtotal[w];
        wbase += w < wid ? c : 0;
        total += c;
    }
    const int rank = wbase + incl - mine;
    if (MODE == MODE_COUNT) {
        if (tid == 0) tile_count[t] = total;
        return;
    }
    if (MODE == MODE_FUSED && tid == 0) publish_count(words, t, total);
    s_rank[tid] = rank;
    // The last tile has the result length as soon as it has its base: the host learns it here, and prepares what
    // comes next while the results are still on their way (a call on 200 x 180: 2.6 us earlier).
    const bool last = MODE == MODE_FUSED && t == num_tiles - 1;
    auto ask_base = [&]() {
        const int64_t b = tile_base(words, t, total, &ctl->status, poll_limit);
        if (lane == 0) {
            s_base = b;
            if (b < 0) publish_timeout(Z.result);
            if (last) finish_total(ctl, Z, b < 0 || (OWN && sh.lost) ? -1 : b + total);
        }
    };
    if (last && wid == 0) ask_base();

    // ---- compact: source of every result entry, in order
    if (MANY_ROWS) {
        // The row offsets ask how many of a thread's first m entries are a twin's second: bit e for its entry e
        unsigned second = 0;
        for (unsigned left = twin << 1; left; left = (left & (left - 1u)) << 1) second |= left & (0u - left);
        s_twin[tid] = (second & 0x7fffffffu) | (unsigned)shifted << 31;
    }
    {
        Src *to = src_of + rank;
#pragma unroll
        for (int i = 0; i < VT; ++i) {
            if (OP == OP_UNION) {
                if (i < steps) to[i] = (Src)src[i];
            } else if ((twin >> i) & 1u) {
                *to++ = (Src)src[i];
            }
        }
    }
    // Byte offset of the B word of the k-th of this thread's twins, taken by step i, whose A word is `at`: step i began at
    // pa0 + pb0 + 4 (i + twins before it).
    const uint32_t begun = pa0 + pb0;
    auto partner = [&](const int i, const int k, const uint32_t at) { return begun + 4u * (uint32_t)(i + k) - at; };

    if (LEVELS) {
        __syncthreads();
        if (MODE == MODE_FUSED && !last && wid == 0) ask_base();
        __syncthreads();
        const long long base = MODE == MODE_FILL ? (long long)tile_count[t] : s_base;
        if (base < 0) return;  // a bounded wait gave up; the host reports it
        // ---- offsets mode: the column and the two range starts of every result entry
        constexpr int LB = 4;  // result entries a thread fetches together
        const int32_t *from_a = L.a + (tile.a0 - oa), *from_b = L.b + (tile.b0 - ob);
        for (int o0 = tid; o0 < total; o0 += LB * NT) {
            int32_t at_a[LB], at_b[LB], end_a[LB], end_b[LB], col[LB];
#pragma unroll
            for (int u = 0; u < LB; ++u) {
                const uint32_t s = src_of[min(o0 + u * NT, total - 1)], pa = s & 0xfffcu, pb = (s >> 16) & 0xfffcu;
                const int32_t *la = from_a + (pa >> 2), *lb = from_b + (pb >> 2);
                at_a[u] = ld_late(la), end_a[u] = ld_late(la + (s & 1u));
                at_b[u] = ld_late(lb), end_b[u] = ld_late(lb + ((s >> 16) & 1u));
                col[u] = (int32_t)(word_at(s & 1u ? pa : pb) & cmask);
            }
#pragma unroll
            for (int u = 0; u < LB; ++u) {
                if (o0 + u * NT >= total) break;
                const long long o = base + o0 + u * NT;
                const bool full_a = end_a[u] > at_a[u], full_b = end_b[u] > at_b[u];
                Z.col[o] = col[u];
                L.off_a[o] = at_a[u];
                L.off_b[o] = at_b[u];
                if (L.keep) L.keep[o] = full_a && full_b;
                if (!full_a && !full_b) ctl->hollow = 1;
            }
        }
        if (t == num_tiles - 1 && tid == 0) {
            L.off_a[base + total] = ld_late(L.a + tile.a0 + na);
            L.off_b[base + total] = ld_late(L.b + tile.b0 + nb);
        }
        if (!Z.rp) return;
    }
    const char *va = reinterpret_cast<const char *>(ga_val) - 4 * (int64_t)oa, *vb = reinterpret_cast<const char *>(gb_val) - 4 * (int64_t)ob;
    auto live = [&](const int q) { return q < VT && q * NT + tid < total; };
    if (!LEVELS && OP == OP_UNION) {
        __syncthreads();
        // ---- the columns of the results, q * NT + tid, into registers: then the words are free for the values. A fill knows its place and
        // writes them at once: beside all of a large tile's columns it had 80 bytes of registers spilled (67 M entries, given room for the
        // result alone, 338 -> 316 us a call; 317 with values gathered from L2).
        constexpr bool AT_ONCE = MODE == MODE_FILL;
        uint32_t col[AT_ONCE ? 1 : VT];
        if (AT_ONCE) {
            int32_t *gz_col = Z.col + tile_count[t] + tid;
#pragma unroll
            for (int q = 0; q < VT; ++q)
                if (live(q)) gz_col[q * NT] = (int32_t)(word_at(src_of[q * NT + tid]) & cmask);
        } else {
#pragma unroll
            for (int q = 0; q < VT; ++q) col[q] = live(q) ? word_at(src_of[q * NT + tid]) & cmask : 0u;
        }
        __syncthreads();
        // ---- bring the values to the places of their columns, and ask for the output base meanwhile
        const bool same_a = head_elems(ga_val) == ha, same_b = head_elems(gb_val) == hb;
        if (tid == 0) {
            fence_async_shared();  // the words were read and written by the threads so far
            mbar_arrive_expect_tx(mbar, 16u * (uint32_t)((same_a ? nva : 0) + (same_b ? nvb : 0)));
            if (same_a && nva) bulk_load(keys + oa + head_a, ga_val + head_a, 16u * nva, mbar);
            if (same_b && nvb) bulk_load(keys + ob + head_b, gb_val + head_b, 16u * nvb, mbar);
        }
        if (tid >= 32 && tid < 32 + 12) {  // ragged ends, as for the columns
            const int k = tid - 32;
            const bool is_b = k >= 6;
            const int e = is_b ? k - 6 : k;
            const int count = is_b ? nb : na, head = is_b ? head_b : head_a, nv = is_b ? nvb : nva;
            const int idx = e < 3 ? e : head + 4 * nv + (e - 3);
            if (e < 3 ? e < head : idx < count) keys[(is_b ? ob : oa) + idx] = __float_as_uint(ld_late((is_b ? gb_val : ga_val) + idx));
        }
        if (!same_a) for (int e = tid; e < na; e += NT) keys[oa + e] = __float_as_uint(ld_late(ga_val + e));
        if (!same_b) for (int e = tid; e < nb; e += NT) keys[ob + e] = __float_as_uint(ld_late(gb_val + e));
        if (MODE == MODE_FUSED && !last && wid == 0) ask_base();
        const bool values = wid != 1 || mbar_wait_bounded(mbar, 1, MBAR_POLL_LIMIT);
        const bool all_values = __syncthreads_and(values);
        const long long base = MODE == MODE_FILL ? (long long)tile_count[t] : s_base;
        if (base >= 0) {
            int32_t *gz_col = Z.col + base + tid;
            float *gz_val = Z.val + base + tid;
            if (!AT_ONCE) {
#pragma unroll
                for (int q = 0; q < VT; ++q)
                    if (live(q)) gz_col[q * NT] = (int32_t)col[q];
            }
            if (all_values) {
                if (total < n) {  // there are twins: the value of the A entry becomes the sum
                    const Src *of = src_of + rank;
                    int k = 0;
                    for (unsigned left = twin; left; left &= left - 1u, ++k) {
                        const int i = __ffs(left) - 1;
                        const uint32_t at = of[i];
                        word_at(at) = __float_as_uint(__uint_as_float(word_at(at)) + __uint_as_float(word_at(partner(i, k, at))));
                    }
                    __syncthreads();
                }
#pragma unroll
                for (int q = 0; q < VT; ++q)
                    if (live(q)) gz_val[q * NT] = __uint_as_float(word_at(src_of[q * NT + tid]));
            } else {  // the copies did not land in time: every thread fetches the values of its own share
                int k = 0;
                for (int i = 0; i < steps; ++i) {
                    const uint32_t at = src_of[rank + i];
                    float v = ld_late(reinterpret_cast<const float *>((at >= 4u * (uint32_t)ob ? vb : va) + at));
                    if ((twin >> i) & 1u) v = v + ld_late(reinterpret_cast<const float *>(vb + partner(i, k++, at)));
                    Z.val[base + rank + i] = v;
                }
            }
        }
        if (!all_values) mbar_wait_bounded(mbar, 1, MBAR_POLL_LIMIT);  // second bounded wait for copies in flight
        if (base < 0) return;  // a bounded wait gave up; the host reports it
    }
    long long base;
    if (!LEVELS && OP == OP_INTERSECT) {
        // ---- a result's A word points to its B word
        {
            const Src *of = src_of + rank;
            int k = 0;
            for (unsigned left = twin; left; left &= left - 1u, ++k) {
                const uint32_t at = of[k];
                word_at(at) = partner(__ffs(left) - 1, k, at);
            }
        }
        __syncthreads();
        // ---- fetch columns and values, results q * NT + tid; the first batch before the output base is asked for
        constexpr int GATHER = 8;
        uint32_t col[GATHER];
        float val[GATHER];
        auto gather = [&](const int q0) {
            uint32_t s[GATHER];
#pragma unroll
            for (int g = 0; g < GATHER; ++g) s[g] = live(q0 + g) ? (uint32_t)src_of[(q0 + g) * NT + tid] : 0u;
#pragma unroll
            for (int g = 0; g < GATHER; ++g) {
                val[g] = 0.0f;
                if (live(q0 + g)) {
                    const uint32_t other = word_at(s[g]);
                    col[g] = word_at(other) & cmask;
                    val[g] = ld_late(reinterpret_cast<const float *>(va + s[g])) * ld_late(reinterpret_cast<const float *>(vb + other));
                }
            }
        };
        gather(0);
        if (MODE == MODE_FUSED && !last && wid == 0) ask_base();
        __syncthreads();
        base = MODE == MODE_FILL ? (long long)tile_count[t] : s_base;
        if (base < 0) return;  // a bounded wait gave up; the host reports it
        int32_t *gz_col = Z.col + base + tid;
        float *gz_val = Z.val + base + tid;
#pragma unroll
        for (int q0 = 0; q0 < VT; q0 += GATHER) {
            if (q0 > 0) {
                if (q0 * NT >= total) break;
                gather(q0);
            }
#pragma unroll
            for (int g = 0; g < GATHER; ++g) {
                if (live(q0 + g)) {
                    gz_col[(q0 + g) * NT] = (int32_t)col[g];
                    gz_val[(q0 + g) * NT] = val[g];
                }
            }
        }
    }
    base = MODE == MODE_FILL ? (long long)tile_count[t] : s_base;

    // ---- row offsets. Result row r starts after every result entry of rows < r; inside this tile those
    // are the survivors among the first d = (A entries before row r) + (B entries before row r) merged
    // entries: all of them up to the thread that holds position d, then, in that thread, a step per entry
    // except that a twin step covers two. The tile owns rows i0+1 .. i1 (the next tile's first row).
    auto end_row = [&](const int r, const uint32_t w) {
        const int d = (int)((w & 0xffffu) + (w >> 16));
        const int owner = d / VT;
        int before = total;
        if (owner < NT) {
            const unsigned info = s_twin[owner];
            const int m = d - owner * VT - (int)(info >> 31);  // merged entries of that thread before the row, fewer than VT
            int twins;
            if (MANY_ROWS) {
                twins = __popc(info & ((1u << m) - 1u));  // no row begins between a twin's two
            } else {  // the steps that take m entries: s + (twins among the first s) grows with s
                int lo = m >> 1, hi = m;
                if ((info << 1) == 0u) lo = m;
                while (lo < hi) {
                    const int mid = (lo + hi) >> 1;
                    if (mid + __popc(info & ((1u << mid) - 1u)) >= m) hi = mid; else lo = mid + 1;
                }
                twins = m - lo;
            }
            before = s_rank[owner] + (OP == OP_UNION ? m - twins : twins);
        }
        Z.rp[tile.i0 + (int64_t)r] = (int32_t)(base + before);
    };
    if (rows_fit) {
        for (int r = 1 + tid; r <= nr; r += NT) end_row(r, s_rows[r]);
    } else {
        for (int r0 = 1; r0 <= nr; r0 += RB * NT) {
            uint32_t w[RB];
#pragma unroll
            for (int u = 0; u < RB; ++u) w[u] = r0 + u * NT + tid <= nr ? global_start(r0 + u * NT + tid) : 0u;
#pragma unroll
            for (int u = 0; u < RB; ++u)
                if (r0 + u * NT + tid <= nr) end_row(r0 + u * NT + tid, w[u]);
        }
    }
    if (t == 0 && tid == 0) Z.rp[0] = 0;
}

template <int VT, int OP, int MODE, bool LEVELS, bool OWN>
__device__ __noinline__ void csr2_tile_wide(const CsrIn &A, const CsrIn &B, const TileRange tile, const int cbits, const int t,
                                            const int num_tiles, int32_t *tile_count, const TileWords &words, FusedCtl *ctl,
                                            const CsrOut &Z, const LevelOffsets &L, unsigned char *smem_raw, TileShared &sh,
                                          const int poll_limit) {
    csr2_tile<VT, OP, MODE, LEVELS, OWN, true>(A, B, tile, cbits, t, num_tiles, tile_count, words, ctl, Z, L, smem_raw, sh, poll_limit);
}

// OWN: without a launch in front of it. (A kernel of its own: with both in one the merges that have such a launch are 1.4 % slower, 67 M entries
// per operand 394 -> 400 us.)
template <int V, int OP, int MODE, bool LEVELS, bool OWN>
__global__ void __launch_bounds__(NT, 4) k_csr2_tile(const __grid_constant__ CsrIn A, const __grid_constant__ CsrIn B,
                                                                    const RowCount row_count, const Cuts cuts, int cbits,
                                                                    int32_t *tile_count, const __grid_constant__ TileWords words, FusedCtl *ctl,
                                                                    const __grid_constant__ CsrOut Z, const __grid_constant__ LevelOffsets L, int num_tiles,
                                                                    int first_tile, int poll_limit) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ TileShared sh;
    if (threadIdx.x == 0) {
        mbar_init(&sh.mbar, 1);
        mbar_fence_init();
        if (OWN) sh.lost = 0;
    }
    __syncthreads();
    trigger_dependents();  // whatever follows on the stream that was launched for it may take its places, and waits
    wait_for_previous();   // the cuts (no wait where no partition kernel ran)
    // Tiles are numbered by CTA index: CTAs are dispatched in increasing index order, so a tile
    // only ever waits on CTAs that were dispatched before it (and every such wait is bounded).
    // first_tile is 0 except in the self-tests that leave tile 0 out; poll_limit is smaller in all self-tests.
    const int t = OWN ? (int)blockIdx.x - cuts.own.cutters + first_tile : (int)blockIdx.x + first_tile;
    TileRange tile;
    if (OWN) {
        if (blockIdx.x == 0 && threadIdx.x == 0) *cuts.own.clear = FusedCtl{};
        if (t < first_tile) {  // one of the CTAs in front of the tiles
            make_cuts(A, B, row_count, cuts, num_tiles, Z.earlier);
            return;
        }
        const int w = threadIdx.x >> 5;
        const bool given = cuts.own.cutters && t >= cuts.own.first_cut();
        if (w < 2) {
            int4 cut = make_int4(0, 0, 0, 0);
            const bool ok = !given || await_cut(cuts.own, t + w, poll_limit, &cut);
            if (!given) cut = tile_cut(A, B, row_count, cuts.step, t + w, num_tiles, Z.earlier);
            if (lane_id() == 0) {
                sh.cut[w] = cut;
                if (!ok) {  // reported, and the tile is empty
                    sh.lost = 1;
                    if (atomicCAS(&ctl->status.error, 0, ERR_LOOKBACK_TIMEOUT) == 0) ctl->status.detail = t;
                    publish_failure(words, t);
                }
            }
        }
        __syncthreads();
        const int4 c0 = sh.cut[0], c1 = sh.lost ? c0 : sh.cut[1];
        tile = TileRange{c0.x, c1.x, c0.y, c0.z, c1.y - c0.y, c1.z - c0.z};
        if (V != V_MOST && given && threadIdx.x == 96 && t + TILES_AHEAD < num_tiles) {
            int4 from, to;
            if (peek_cut(cuts.own, t + TILES_AHEAD, &from) && peek_cut(cuts.own, t + TILES_AHEAD + 1, &to)) {
                const int32_t n = min(to.x - from.x, TilePlan<V, LEVELS>::ROWS) + 1;
                if (A.rp) prefetch_l2(A.rp + from.x, n);
                if (B.rp) prefetch_l2(B.rp + from.x, n);
            }
        }
    } else if (cuts.at) {
        const int4 c0 = cuts.at[t], c1 = cuts.at[t + 1];
        tile = TileRange{c0.x, c1.x, c0.y, c0.z, c1.y - c0.y, c1.z - c0.z};
        if (V != V_MOST && threadIdx.x == 96 && t + TILES_AHEAD >= RESIDENT && t + TILES_AHEAD < num_tiles) {
            const int32_t r0 = cuts.at[t + TILES_AHEAD].x, n = min(cuts.at[t + TILES_AHEAD + 1].x - r0, TilePlan<V, LEVELS>::ROWS) + 1;
            if (A.rp) prefetch_l2(A.rp + r0, n);
            if (B.rp) prefetch_l2(B.rp + r0, n);
        }
    } else {
        const int32_t rows = row_count.get();
        tile = TileRange{0, rows, row_offset(A, 0), row_offset(B, 0), A.entries(), B.entries()};
        if (gave_up(Z.earlier)) tile = TileRange{0, 0, 0, 0, 0, 0};
        if (threadIdx.x == 0) {  // what the partition kernel does otherwise
            *ctl = FusedCtl{};
            if (Z.result) Z.result[1] = NB200_OK, Z.result[2] = rows;
        }
        __syncthreads();
    }
    // 32-bit keys hold (row in tile << cbits | column) when that fits; tiles that span too many rows for
    // that (long runs of empty rows) use 64-bit keys.
    const uint64_t nr = (uint64_t)(tile.i1 - tile.i0) + 1;
    const bool narrow = cbits < 31 && (nr << cbits) <= 0x80000000ull;
    if (narrow) {
        csr2_tile<V, OP, MODE, LEVELS, OWN, false>(A, B, tile, cbits, t, num_tiles, tile_count, words, ctl, Z, L, smem_raw, sh, poll_limit);
    } else {
        csr2_tile_wide<V, OP, MODE, LEVELS, OWN>(A, B, tile, cbits, t, num_tiles, tile_count, words, ctl, Z, L, smem_raw, sh, poll_limit);
    }
}

// ------------------------------------------------------------------------ host driver ----

constexpr int tile_step(int v) { return NT * v - 1; }  // merged entries between two tile cuts (a twin may add one)

// Merged entries per worker thread. Large tiles amortise what a tile costs whatever its size (searches, barriers, the wait for the
// earlier counts): 64 M entries per operand take 397 us with 31, 403 with 29, 407 with 27. Small ones fill the chip where there are few entries: 2 M
// merged entries 20.9 us with 15, 25.0 with 11. They give way where they are more than can be at work at once: a second wave of
// them costs more than places that stay empty in one of large tiles. Sums of 1.2, 1.5, 2, 2.6 M entries per operand 26.7, 30.7, 35.0, 41.1 us with
// 15 and 23.0, 26.5, 31.2, 38.3 with 31, products of 1.3 and 2.3 M 25.0, 34.3 and 21.4, 27.9, trees of 1.5 M 66.4 and 60.9.
// Both are odd: a thread's shares of A and B then start at odd word distances from its neighbour's where
// rows alternate evenly, and the shared-memory banks are hit evenly (16 took twice the time of 18).
constexpr int V_LARGE = V_MOST, V_SMALL = 15;
constexpr int64_t LARGE_FROM = (int64_t)RESIDENT * tile_step(V_SMALL) + 1, LARGE_ALWAYS_FROM = 6000000;
// Up to LARGE_ALWAYS_FROM entries they stay small for two kinds of merge, whose large tiles take longer for an entry:
//   - many rows. A large tile that more rows begin in than it keeps reads their offsets from L2 three times; a small one keeps more than
//     twice as many. While all large tiles are at work at once that weighs less than the second wave of small ones, up to about twice
//     the rows that are kept: sums of 2 M entries per operand in 1.4, 2, 4 and 8 M rows 41.1, 42.8, 56.1, 109 us with small tiles,
//     40.5, 47.4, 74.8, 127 with large ones; of 2.7 M (two waves of large ones) in 1.1, 1.3, 2.7, 5.4 M rows 45.4, 46.0, 55.1, 74.3 and 44.4, 52.1, 70.7,
//     111.7. Rows that are hardly ever filled, 80 M for 2 M entries: 1057 and 1170.
//   - keys of 64 bits, for columns beyond 2^30 or so many rows in a tile that their number and a column take more than 31 bits. Where a small
//     tile gets by with 32 bits it is faster, and beyond one wave of large tiles always. Columns of 20, 22, 25 bits, sums of 1.25 M entries per operand in 0.75, 0.25,
//     0.025 M rows 30.7, 28.5, 27.0 us with small tiles, 42.3, 35.5, 32.5 with large ones; of 2.95 M (two waves) in 0.6 M rows of 22, 25, 28 bits 43.6, 57.4, 57.6 and 76.6, 73.6, 77.5.
//     One wave, 64 bits in either tile: up to the rows that a large tile keeps, sums of 2 M entries 38.1 and 40.3, products 33.8 and 31.0; beyond those small tiles (2 M in 1.2, 1.8 M
//     rows of 25 bits 46.6, 50.9 and 50.4, 58.8). The tiles for short rows and for the levels of a tree give way to small ones of 32 bits alike: trees of 1.9, 2.5 M entries per
//     operand in 0.9, 0.6 M fibres of 21, 22 bits 61.3, 67.4 and 77.8, 87.2 us; of 1.9 M fibres in 0.2 M slices of 23 bits 98.1 and 133.3.
// `rows` is the most there can be where only the device knows how many (row lists; sums of 1.3, 1.9, 2.5, 2.95 M entries per operand in as many rows: 51, 60, 75, 85 us with
// small tiles, 78, 91, 134, 145 with large ones), 0 if the call does not know that either.
inline int tile_v(int64_t total, int64_t rows, int32_t cols, int large = V_LARGE) {
    if (total < LARGE_FROM) return V_SMALL;
    if (total >= LARGE_ALWAYS_FROM) return large;
    const bool one_wave = total <= (int64_t)RESIDENT * tile_step(V_LARGE);
    const int bits = col_bits(cols);
    auto wide = [&](int v, int64_t more) {
        const int64_t average = rows * tile_step(v) / total;
        return bits > 30 || (average + 1 + more * (2 + average / 32)) << bits > int64_t(1) << 31;
    };
    const bool wide_keys = wide(large, 1);  // not the average tile alone
    if (wide_keys && !wide(V_SMALL, 0)) return V_SMALL;
    if (large != V_LARGE) return large;
    if (wide_keys && !one_wave) return V_SMALL;
    return rows * tile_step(V_LARGE) > (one_wave && !wide_keys ? 2 : 1) * TilePlan<V_LARGE, false>::ROWS * total ? V_SMALL : V_LARGE;
}

// Raises the tile kernel's dynamic shared-memory limit once per instantiation and device.
template <int V, int OP, int MODE, bool LEVELS = false, bool OWN = false>
cudaError_t configure_tile_kernel() {
    static bool configured[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(k_csr2_tile<V, OP, MODE, LEVELS, OWN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TilePlan<V, LEVELS>::BYTES);
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    return cudaSuccess;
}

// Launches the tile kernel so that it may take its places while the kernel before it on the stream (the
// partition) still runs; it waits for that kernel's results itself.
template <int V, int OP, int MODE, bool LEVELS = false>
cudaError_t launch_tile_v(const CsrIn &A, const CsrIn &B, const RowCount &rows, const Cuts &cuts, int cbits, int32_t *tile_count,
                          TileWords words, FusedCtl *ctl, const CsrOut &Z, int num_tiles, cudaStream_t stream, const LaunchKnobs &knobs,
                          const LevelOffsets &levels = LevelOffsets()) {
    constexpr size_t smem = TilePlan<V, LEVELS>::BYTES;
    const dim3 grid(num_tiles - knobs.first_tile + cuts.own.cutters);
    if (MODE == MODE_FUSED && cuts.step) {
        constexpr bool OWN = MODE == MODE_FUSED;
        cudaError_t e = configure_tile_kernel<V, OP, MODE, LEVELS, OWN>();
        if (e != cudaSuccess) return e;
        return launch_overlapped(k_csr2_tile<V, OP, MODE, LEVELS, OWN>, grid, dim3(NT), smem, stream, A, B, rows, cuts, cbits, tile_count, words, ctl, Z,
                                 levels, num_tiles, knobs.first_tile, knobs.poll_limit);
    }
    cudaError_t e = configure_tile_kernel<V, OP, MODE, LEVELS>();
    if (e != cudaSuccess) return e;
    return launch_overlapped(k_csr2_tile<V, OP, MODE, LEVELS, false>, grid, dim3(NT), smem, stream, A, B, rows, cuts, cbits, tile_count, words, ctl, Z,
                             levels, num_tiles, knobs.first_tile, knobs.poll_limit);
}

template <int OP, int MODE>
cudaError_t launch_tile(const CsrIn &A, const CsrIn &B, const RowCount &rows, const Cuts &cuts, int cbits, int32_t *tile_count,
                        TileWords words, FusedCtl *ctl, const CsrOut &Z, int num_tiles, int v, cudaStream_t stream,
                        const LaunchKnobs &knobs = LaunchKnobs()) {
    static const char *const names[2][3] = {{"csr_add_count", "csr_add_fill", "csr_add_fused"},
                                            {"csr_mul_count", "csr_mul_fill", "csr_mul_fused"}};
    if (num_tiles - knobs.first_tile <= 0) return cudaSuccess;
    LaunchScope scope(names[OP][MODE], stream);
    return v == V_LARGE ? launch_tile_v<V_LARGE, OP, MODE>(A, B, rows, cuts, cbits, tile_count, words, ctl, Z, num_tiles, stream, knobs)
                        : launch_tile_v<V_SMALL, OP, MODE>(A, B, rows, cuts, cbits, tile_count, words, ctl, Z, num_tiles, stream, knobs);
}

// Eight lanes per cut once a full warp per cut would need more than one wave of the chip: the searches
// then run a few dependent loads longer, but four times fewer warps issue them.
cudaError_t launch_partition(const CsrIn &A, const CsrIn &B, const RowCount &rows, int num_tiles, int step, int4 *cuts,
                             long long *result, uint64_t *zero_block, int zero_words, cudaStream_t stream, const FusedCtl *earlier = nullptr) {
    const int64_t lanes = num_tiles < 8192 ? 32 : 8;
    const int blocks = (int)(((int64_t)(num_tiles + 1) * lanes + NT - 1) / NT);
    return launch_overlapped(lanes == 32 ? k_csr2_partition<32> : k_csr2_partition<8>, dim3(blocks), dim3(NT), 0, stream, A, B, rows, step, num_tiles, cuts,
                             result, zero_block, zero_words, earlier);
}

// Shared driver of add and multiply. When `alloc` is set the result arrays are allocated
// here (one cudaMallocAsync each); otherwise z's arrays are the caller's, `capacity` entries.
//
// With room for the largest possible result (every operand entry for a union, the smaller
// operand for an intersection) the single-pass kernel runs. A caller-provided capacity below
// that bound takes the two-pass route, which knows the exact length before it writes.
//
// `device_result`, when given, makes the call asynchronous: the result length and the device
// status go to those two device words in stream order and the host does not wait (z->nnz stays 0).
// Only the single-pass route can do that; the call refuses a capacity below the bound.
template <int OP>
int csr2_run(const nb200_csr *a, const nb200_csr *b, nb200_csr *z, bool alloc, int64_t capacity, void *stream_v,
             int64_t *device_result = nullptr, const LaunchKnobs &knobs = LaunchKnobs()) {
    int st;
    if ((st = check_csr(a, true)) || (st = check_csr(b, true))) return st;
    if (!z || a->rows != b->rows || a->cols != b->cols) return NB200_E_BADARG;
    if (!alloc && (!z->row_ptr || capacity < 0)) return NB200_E_BADARG;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
    const int32_t rows = a->rows;
    const RowCount row_count{rows};
    const int64_t total = (int64_t)a->nnz + b->nnz;
    const int v = tile_v(total, rows, a->cols), step = tile_step(v);
    const int64_t tiles64 = (total + step - 1) / step;
    if (tiles64 > INT32_MAX - 1) return NB200_E_OVERFLOW;
    const int num_tiles = (int)tiles64;
    const int64_t bound = OP == OP_UNION ? total : std::min<int64_t>(a->nnz, b->nnz);
    // a caller's arrays must exist wherever the kernels may write: capacity > 0 promises col / val
    if (!alloc && capacity > 0 && total > 0 && (!z->col || !z->val)) return NB200_E_BADARG;
    if (device_result && (alloc || capacity < bound)) return NB200_E_CAPACITY;

    z->rows = rows;
    z->cols = a->cols;
    z->nnz = 0;
    if (alloc) {
        z->row_ptr = nullptr;
        z->col = nullptr;
        z->val = nullptr;
        NB200_CUDA(cudaMallocAsync(reinterpret_cast<void **>(&z->row_ptr), sizeof(int32_t) * ((size_t)rows + 1), stream));
    }
    auto fail = [&](int code) {
        if (alloc) {
            cudaFreeAsync(z->row_ptr, stream);
            if (z->col) cudaFreeAsync(z->col, stream);
            if (z->val) cudaFreeAsync(z->val, stream);
            z->row_ptr = z->col = nullptr;
            z->val = nullptr;
        }
        return code;
    };
    if (num_tiles == 0) {  // both operands empty: all-zero offsets, nothing else
        cudaError_t e = cudaMemsetAsync(z->row_ptr, 0, sizeof(int32_t) * ((size_t)rows + 1), stream);
        if (e == cudaSuccess && device_result) {
            const int64_t words[3] = {0, NB200_OK, rows};  // copied before the call returns: pageable source
            e = cudaMemcpyAsync(device_result, words, sizeof(words), cudaMemcpyDefault, stream);  // the words may be mapped host memory
        }
        if (e != cudaSuccess) return fail(note_cuda_error(e, "cudaMemsetAsync"));
        return NB200_OK;
    }

    Carver sizes;
    sizes.take<int4>((size_t)num_tiles + 1);
    sizes.take<int32_t>((size_t)num_tiles + 1);
    sizes.take<uint64_t>(TileWords::needed(num_tiles) + 4);
    Workspace *ws = nullptr;
    if ((st = acquire_workspace(stream, sizes.used(), &ws))) return fail(st);
    Carver carve(ws->dev);
    Cuts cuts;
    cuts.at = carve.take<int4>((size_t)num_tiles + 1);
    int32_t *tile_count = carve.take<int32_t>((size_t)num_tiles + 1);
    // control block (status word, result length) and the tile words of the single-pass kernel, contiguous for the partition
    // kernel, which clears them; the two-pass route uses the control block alone
    uint64_t *fused_block = carve.take<uint64_t>(TileWords::needed(num_tiles) + 4);
    static_assert(sizeof(FusedCtl) <= 4 * sizeof(uint64_t), "control block must fit its slot");
    FusedCtl *ctl = reinterpret_cast<FusedCtl *>(fused_block);
    TileWords words = TileWords::at(fused_block + 4);

    const CsrIn A{a->row_ptr, a->col, a->val, a->nnz}, B{b->row_ptr, b->col, b->val, b->nnz};
    const int cbits = col_bits(a->cols);
    // NACHO_B200_TWO_PASS=1 forces the count -> scan -> fill route (for comparisons).
    static const bool force_two_pass = [] { const char *e = std::getenv("NACHO_B200_TWO_PASS"); return e && e[0] == '1'; }();
    // NACHO_B200_EXACT_ALLOC=1 makes the allocating entry points count first and allocate col / val at
    // exactly nnz(Z), as the reference's drivers do (src/backend/stitch_and_generate.cpp:438-527),
    // instead of at the worst case: for callers short of memory, at the price of a second read of
    // the operands' columns.
    static const bool exact_alloc = [] { const char *e = std::getenv("NACHO_B200_EXACT_ALLOC"); return e && e[0] == '1'; }();
    const bool fused = device_result || (alloc ? !exact_alloc : (capacity >= bound && !force_two_pass));
    cudaError_t e = cudaSuccess;
    if (fused && alloc && bound > 0) {
        e = cudaMallocAsync(reinterpret_cast<void **>(&z->col), sizeof(int32_t) * (size_t)bound, stream);
        if (e == cudaSuccess) e = cudaMallocAsync(reinterpret_cast<void **>(&z->val), sizeof(float) * (size_t)bound, stream);
        if (e != cudaSuccess) return fail(note_cuda_error(e, "cudaMallocAsync"));
    }
    bool tagged = fused && !device_result && num_tiles > 1 && num_tiles <= OWN_CUTS_UP_TO && !profiling_apart();
    OwnWords own;
    if ((st = take_own_words(stream, num_tiles, &tagged, &own))) return fail(st);
    if (tagged) {
        cuts = Cuts{nullptr, step, own};
        ctl = own.ctl, words = own.words;
    } else if (num_tiles == 1) {
        cuts.at = nullptr;  // one tile: no cut to search, and the tile kernel clears the control block itself
    } else {
        LaunchScope scope("csr2_partition", stream);
        e = launch_partition(A, B, row_count, num_tiles, step, cuts.at, reinterpret_cast<long long *>(device_result), fused_block,
                             fused ? (int)TileWords::needed(num_tiles) + 4 : 4, stream);
    }
    if (e != cudaSuccess) return fail(note_cuda_error(e, "k_csr2_partition"));

    // Reads the control block back (one small copy and the call's only wait for the GPU).
    auto read_ctl = [&](FusedCtl &h) -> int {
        cudaError_t c = cudaMemcpyAsync(ws->host, ctl, sizeof(FusedCtl), cudaMemcpyDeviceToHost, stream);
        if (c == cudaSuccess) c = cudaStreamSynchronize(stream);
        if (c != cudaSuccess) return note_cuda_error(c, "read result length");
        std::memcpy(&h, ws->host, sizeof(h));
        return NB200_OK;
    };

    FusedCtl h;
    if (fused) {
        unsigned long long *word = device_result ? nullptr : result_word(ws, 0);
        e = launch_tile<OP, MODE_FUSED>(A, B, row_count, cuts, cbits, nullptr, words, ctl,
                                        CsrOut{z->row_ptr, z->col, z->val, reinterpret_cast<long long *>(device_result), word}, num_tiles, v, stream,
                                        knobs);
        if (e != cudaSuccess && tagged) spoil_tagged(stream);
        if (e != cudaSuccess) return fail(note_cuda_error(e, "k_csr2_tile<fused>"));
        if (device_result) return NB200_OK;  // length, status and rows arrive in the caller's device words, written by the kernels
        int64_t length;
        int device_status;
        if ((st = wait_result_word(word, stream, &length, &device_status))) return fail(st);
        if (device_status != 0) {
            if ((st = read_ctl(h))) return fail(st);
            return fail(note_timeout(h.status.error, h.status.detail, "csr merge"));
        }
        h.total = length;
        if (h.total > INT32_MAX) return fail(NB200_E_OVERFLOW);
        z->nnz = (int32_t)h.total;
        if (alloc && h.total == 0) {  // zero-length arrays are handed over as NULL
            if (z->col) cudaFreeAsync(z->col, stream);
            if (z->val) cudaFreeAsync(z->val, stream);
            z->col = nullptr;
            z->val = nullptr;
        }
        return NB200_OK;
    }

    // count -> scan -> fill. The scan leaves the result length in the control block, whose status
    // word also collects a give-up of either tile launch (a bulk copy that did not land in time).
    e = launch_tile<OP, MODE_COUNT>(A, B, row_count, cuts, cbits, tile_count, TileWords{}, ctl, CsrOut{nullptr, nullptr, nullptr}, num_tiles, v, stream);
    if (e != cudaSuccess) return fail(note_cuda_error(e, "k_csr2_tile<count>"));
    {
        LaunchScope scope("scan_tiles", stream);
        k_scan_tiles<<<1, 1024, 0, stream>>>(tile_count, num_tiles, reinterpret_cast<int64_t *>(&ctl->total));
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) return fail(note_cuda_error(e, "k_scan_tiles"));
    if ((st = read_ctl(h))) return fail(st);
    if (h.status.error != 0) return fail(note_timeout(h.status.error, h.status.detail, "csr merge"));
    if (h.total > INT32_MAX) return fail(NB200_E_OVERFLOW);
    z->nnz = (int32_t)h.total;
    if (alloc) {
        if (h.total > 0) {
            e = cudaMallocAsync(reinterpret_cast<void **>(&z->col), sizeof(int32_t) * (size_t)h.total, stream);
            if (e == cudaSuccess) e = cudaMallocAsync(reinterpret_cast<void **>(&z->val), sizeof(float) * (size_t)h.total, stream);
            if (e != cudaSuccess) return fail(note_cuda_error(e, "cudaMallocAsync"));
        }
    } else if (h.total > capacity) {
        return NB200_E_CAPACITY;
    }
    e = launch_tile<OP, MODE_FILL>(A, B, row_count, cuts, cbits, tile_count, TileWords{}, ctl, CsrOut{z->row_ptr, z->col, z->val}, num_tiles, v, stream);
    if (e != cudaSuccess) return fail(note_cuda_error(e, "k_csr2_tile<fill>"));
    if ((st = read_ctl(h))) return fail(st);
    if (h.status.error != 0) return fail(note_timeout(h.status.error, h.status.detail, "csr merge"));
    return NB200_OK;
}

// ------------------------------------------------------- entry point that allocates nothing ----

// Scratch of nb200_csr_add_f32_noalloc: tile cuts, the single-pass control block and one
// 8-byte word per tile, carved out of one fixed array that lives in the library's device image
// (so every GPU that loads the library holds these bytes until the process exits).
constexpr int64_t NOALLOC_MAX_ENTRIES = 159350784;
constexpr int NOALLOC_MAX_TILES = (int)(NOALLOC_MAX_ENTRIES / tile_step(V_LARGE)) + 1;
static_assert(LARGE_ALWAYS_FROM / tile_step(V_SMALL) + 1 <= NOALLOC_MAX_TILES, "small tiles must fit the scratch too");
constexpr size_t NOALLOC_SCRATCH_BYTES = 1u << 20;
static __device__ __align__(256) unsigned char g_noalloc_scratch[NOALLOC_SCRATCH_BYTES];

// Device address of the array above for each device, looked up once per device. The array's
// name is only a host-side handle; kernels must be given the address from
// cudaGetSymbolAddress, taken while that device is current.
int noalloc_scratch_address(void **out) {
    static void *address[64] = {};
    static std::mutex lock;
    int dev = 0;
    NB200_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return NB200_E_UNSUPPORTED;
    std::lock_guard<std::mutex> g(lock);
    if (!address[dev]) {
        void *p = nullptr;
        NB200_CUDA(cudaGetSymbolAddress(&p, g_noalloc_scratch));
        // the tile kernel needs more dynamic shared memory than the default limit; set that
        // here too so that later calls are launches and nothing else
        NB200_CUDA((configure_tile_kernel<V_LARGE, OP_UNION, MODE_FUSED>()));
        NB200_CUDA((configure_tile_kernel<V_SMALL, OP_UNION, MODE_FUSED>()));
        address[dev] = p;
    }
    *out = address[dev];
    return NB200_OK;
}

int csr_add_noalloc(const nb200_csr *a, const nb200_csr *b, nb200_csr *z, int64_t capacity, void *stream_v) {
    int st;
    if ((st = check_csr(a, true)) || (st = check_csr(b, true))) return st;
    if (!z || !z->row_ptr || capacity < 0 || a->rows != b->rows || a->cols != b->cols) return NB200_E_BADARG;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
    const int32_t rows = a->rows;
    const RowCount row_count{rows};
    const int64_t total = (int64_t)a->nnz + b->nnz;
    const int v = tile_v(total, rows, a->cols), step = tile_step(v);
    const int64_t tiles64 = (total + step - 1) / step;
    if (total > NOALLOC_MAX_ENTRIES) return NB200_E_UNSUPPORTED;
    if (capacity < total) return NB200_E_CAPACITY;  // this entry point has the single-pass route only
    if (total > 0 && (!z->col || !z->val)) return NB200_E_BADARG;
    const int num_tiles = (int)tiles64;
    z->rows = rows;
    z->cols = a->cols;
    z->nnz = 0;
    if (num_tiles == 0) {
        NB200_CUDA(cudaMemsetAsync(z->row_ptr, 0, sizeof(int32_t) * ((size_t)rows + 1), stream));
        return NB200_OK;
    }
    void *scratch = nullptr;
    if ((st = noalloc_scratch_address(&scratch))) return st;
    Carver carve(scratch);
    uint64_t *fused_block = carve.take<uint64_t>(TileWords::needed(NOALLOC_MAX_TILES) + 4);
    Cuts cuts;
    cuts.at = carve.take<int4>((size_t)NOALLOC_MAX_TILES + 1);
    static_assert(8 * (TileWords::needed(NOALLOC_MAX_TILES) + 4) + 16 * (NOALLOC_MAX_TILES + 1) + 512 <= NOALLOC_SCRATCH_BYTES,
                  "scratch layout must fit the fixed array");
    FusedCtl *ctl = reinterpret_cast<FusedCtl *>(fused_block);
    const TileWords words = TileWords::at(fused_block + 4);
    // the array keeps the previous call's contents: the control block and every tile word
    // must start at zero (the partition kernel clears them)

    const CsrIn A{a->row_ptr, a->col, a->val, a->nnz}, B{b->row_ptr, b->col, b->val, b->nnz};
    NB200_CUDA(launch_partition(A, B, row_count, num_tiles, step, cuts.at, nullptr, fused_block, (int)TileWords::needed(num_tiles) + 4, stream));
    const CsrOut Z{z->row_ptr, z->col, z->val};
    NB200_CUDA((v == V_LARGE ? launch_tile_v<V_LARGE, OP_UNION, MODE_FUSED>(A, B, row_count, cuts, col_bits(a->cols), nullptr, words, ctl, Z, num_tiles, stream, LaunchKnobs())
                            : launch_tile_v<V_SMALL, OP_UNION, MODE_FUSED>(A, B, row_count, cuts, col_bits(a->cols), nullptr, words, ctl, Z, num_tiles, stream, LaunchKnobs())));
    FusedCtl h;  // read back into ordinary host memory: no pinned buffer is taken for this
    NB200_CUDA(cudaMemcpyAsync(&h, ctl, sizeof(h), cudaMemcpyDeviceToHost, stream));
    NB200_CUDA(cudaStreamSynchronize(stream));
    if (h.status.error != 0) return note_timeout(h.status.error, h.status.detail, "csr merge (no-alloc)");
    if (h.total > INT32_MAX) return NB200_E_OVERFLOW;
    z->nnz = (int32_t)h.total;
    return NB200_OK;
}

// In the offsets mode a tile needs 8 bytes of shared memory per entry, so its large tile is smaller.
constexpr int V_LEVELS = 23;

}  // namespace

size_t csr2_scratch_bytes(int64_t entries) {
    const size_t tiles = (size_t)(entries / tile_step(V_SMALL)) + 2;  // the smallest tile, whichever will be taken
    Carver sizes;
    sizes.take<int4>(tiles + 1);
    sizes.take<uint64_t>(TileWords::needed(tiles) + 4);
    return sizes.used();
}

int csr2_enqueue(SetOp op, const CsrIn &A, const CsrIn &B, const RowCount &rows, int32_t cols, const CsrOut &Z, const LevelOffsets *levels,
                 void *scratch, cudaStream_t stream, FusedCtl **ctl_out, const LaunchKnobs &knobs) {
    const int64_t total = (int64_t)A.nnz + B.nnz;
    const int large = levels ? V_LEVELS : rows.short_rows && op == OP_UNION ? V_FIBRES : V_LARGE;
    const int v = tile_v(total, rows.value, cols, large), step = tile_step(v);
    const int num_tiles = (int)std::max<int64_t>(1, (total + step - 1) / step);
    Carver carve(scratch);
    Cuts cuts;
    cuts.at = carve.take<int4>((size_t)num_tiles + 1);
    uint64_t *fused_block = carve.take<uint64_t>(TileWords::needed(num_tiles) + 4);
    FusedCtl *ctl = reinterpret_cast<FusedCtl *>(fused_block);
    TileWords words = TileWords::at(fused_block + 4);
    *ctl_out = ctl;
    cudaError_t e = cudaSuccess;
    bool tagged = num_tiles > 1 && num_tiles <= OWN_CUTS_UP_TO && !profiling_apart();
    OwnWords own;
    const int st = take_own_words(stream, num_tiles, &tagged, &own);
    if (st != NB200_OK) return st;
    if (tagged) {
        cuts = Cuts{nullptr, step, own};
        *ctl_out = ctl = own.ctl, words = own.words;
    } else if (num_tiles == 1) {
        cuts.at = nullptr;
    } else {
        LaunchScope scope("csr2_partition", stream);
        e = launch_partition(A, B, rows, num_tiles, step, cuts.at, nullptr, fused_block, (int)TileWords::needed(num_tiles) + 4, stream, Z.earlier);
    }
    if (e != cudaSuccess) return note_cuda_error(e, "k_csr2_partition");
    const int cbits = col_bits(cols);
    if (levels) {
        LaunchScope scope("csr_levels_fused", stream);
        e = v == V_LEVELS ? launch_tile_v<V_LEVELS, OP_UNION, MODE_FUSED, true>(A, B, rows, cuts, cbits, nullptr, words, ctl, Z, num_tiles, stream, knobs, *levels)
                          : launch_tile_v<V_SMALL, OP_UNION, MODE_FUSED, true>(A, B, rows, cuts, cbits, nullptr, words, ctl, Z, num_tiles, stream, knobs, *levels);
    } else if (v == V_FIBRES) {
        LaunchScope scope("csr_add_fused", stream);
        e = launch_tile_v<V_FIBRES, OP_UNION, MODE_FUSED>(A, B, rows, cuts, cbits, nullptr, words, ctl, Z, num_tiles, stream, knobs);
    } else if (op == OP_UNION) {
        e = launch_tile<OP_UNION, MODE_FUSED>(A, B, rows, cuts, cbits, nullptr, words, ctl, Z, num_tiles, v, stream, knobs);
    } else {
        e = launch_tile<OP_INTERSECT, MODE_FUSED>(A, B, rows, cuts, cbits, nullptr, words, ctl, Z, num_tiles, v, stream, knobs);
    }
    if (e != cudaSuccess && tagged) spoil_tagged(stream);
    return e == cudaSuccess ? NB200_OK : note_cuda_error(e, "k_csr2_tile");
}

namespace {

// Three-operand add Z = (A + B) + C as two chained unions. The association is the reference's
// (src/backend/compute.cpp:426-432 builds a + b first), so running the two-operand union twice
// gives bit-identical values to the reference's fused three-way merge: positions present in A
// and C only hold a + c, in B and C only b + c, in all three (a + b) + c, and explicit zeros
// stay. The intermediate A + B, eight bytes per entry of A and of B, lies in the caller's scratch or in the pool, and its
// length stays in device memory: the second union is cut into the tiles that its longest possible input needs (those
// past its end are empty) and nothing waits in between. A kernel that merged three operands in one pass, in two stages
// per tile, took 2.0 ms where this takes 1.17 (three times 67 M entries), although it moves 1.6 GB less.
struct Add3Sizes {
    int64_t bound, total;              // most entries of the intermediate and of the result
    size_t own, first_bytes, all;      // bytes: the intermediate, the first union's scratch, everything
    Add3Sizes(const nb200_csr *a, const nb200_csr *b, const nb200_csr *c) : bound((int64_t)a->nnz + b->nnz), total(bound + c->nnz) {
        Carver sizes;
        sizes.take<int32_t>((size_t)a->rows + 1);
        sizes.take<int32_t>((size_t)bound);
        sizes.take<float>((size_t)bound);
        own = sizes.used(), first_bytes = csr2_scratch_bytes(bound);
        all = own + first_bytes + csr2_scratch_bytes(total);
    }
};

int check_add3(const nb200_csr *a, const nb200_csr *b, const nb200_csr *c) {
    int st;
    if ((st = check_csr(a, true)) || (st = check_csr(b, true)) || (st = check_csr(c, true))) return st;
    return a->rows != b->rows || a->cols != b->cols || a->rows != c->rows || a->cols != c->cols ? NB200_E_BADARG : NB200_OK;
}

// `lent`: scratch of the caller's (Add3Sizes::all bytes), or null for the pool's.
int csr_add3_run(const nb200_csr *a, const nb200_csr *b, const nb200_csr *c, nb200_csr *z, bool alloc, int64_t capacity, void *lent,
                 void *stream_v, const LaunchKnobs &first_knobs = LaunchKnobs()) {
    int st;
    if ((st = check_add3(a, b, c))) return st;
    if (!z) return NB200_E_BADARG;
    if (!alloc && (!z->row_ptr || capacity < 0)) return NB200_E_BADARG;
    const Add3Sizes sizes(a, b, c);
    const int64_t bound = sizes.bound, total = sizes.total;
    if (total > INT32_MAX) return NB200_E_OVERFLOW;
    if (!alloc && capacity > 0 && total > 0 && (!z->col || !z->val)) return NB200_E_BADARG;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
    // pool slot 1: the calls below use slot 0
    Workspace *ws = nullptr;
    if ((st = acquire_workspace(stream, lent ? 0 : sizes.all, &ws, 1))) return st;
    unsigned char *base = static_cast<unsigned char *>(lent ? lent : ws->dev);
    Carver carve(base);
    nb200_csr t{};
    t.row_ptr = carve.take<int32_t>((size_t)a->rows + 1);
    t.col = carve.take<int32_t>((size_t)bound);
    t.val = carve.take<float>((size_t)bound);
    if (alloc || capacity < total || bound == 0) {  // (allocating callers get arrays of the size the second union chooses)
        if ((st = csr2_run<OP_UNION>(a, b, &t, false, bound, stream_v))) return st;
        return csr2_run<OP_UNION>(&t, c, z, alloc, capacity, stream_v);
    }
    unsigned char *scratch = base + sizes.own;
    unsigned long long *word = result_word(ws, 0);
    FusedCtl *first = nullptr, *second = nullptr;
    if ((st = csr2_enqueue(OP_UNION, CsrIn{a->row_ptr, a->col, a->val, a->nnz}, CsrIn{b->row_ptr, b->col, b->val, b->nnz}, RowCount{a->rows}, a->cols,
                           CsrOut{t.row_ptr, t.col, t.val}, nullptr, scratch, stream, &first, first_knobs)))
        return st;
    if ((st = csr2_enqueue(OP_UNION, CsrIn{t.row_ptr, t.col, t.val, (int32_t)bound, &first->total}, CsrIn{c->row_ptr, c->col, c->val, c->nnz},
                           RowCount{a->rows}, a->cols, CsrOut{z->row_ptr, z->col, z->val, nullptr, word, first}, nullptr, scratch + sizes.first_bytes, stream,
                           &second)))
        return st;
    int64_t length;
    int device_status;
    if ((st = wait_result_word(word, stream, &length, &device_status))) return st;
    if (device_status != 0) {
        NB200_CUDA(cudaMemcpyAsync(ws->host, second, sizeof(FusedCtl), cudaMemcpyDeviceToHost, stream));
        NB200_CUDA(cudaStreamSynchronize(stream));
        FusedCtl h;
        std::memcpy(&h, ws->host, sizeof(h));
        return note_timeout(h.status.error, h.status.detail, "csr add3");
    }
    z->rows = a->rows;
    z->cols = a->cols;
    z->nnz = (int32_t)length;
    return NB200_OK;
}

}  // namespace

}  // namespace nb200

using namespace nb200;

extern "C" {

int nb200_csr_add_f32(const nb200_csr *a, const nb200_csr *b, nb200_csr *z, int32_t, int32_t, void *stream) {
    return csr2_run<OP_UNION>(a, b, z, true, 0, stream);
}

int nb200_csr_add_f32_into(const nb200_csr *a, const nb200_csr *b, nb200_csr *z, int64_t capacity, void *stream) {
    return csr2_run<OP_UNION>(a, b, z, false, capacity, stream);
}

int nb200_csr_mul_f32(const nb200_csr *a, const nb200_csr *b, nb200_csr *z, int32_t, int32_t, void *stream) {
    return csr2_run<OP_INTERSECT>(a, b, z, true, 0, stream);
}

int nb200_csr_mul_f32_into(const nb200_csr *a, const nb200_csr *b, nb200_csr *z, int64_t capacity, void *stream) {
    return csr2_run<OP_INTERSECT>(a, b, z, false, capacity, stream);
}

int nb200_csr_add_3_f32(const nb200_csr *a, const nb200_csr *b, const nb200_csr *c, nb200_csr *z, int32_t, int32_t,
                        void *stream) {
    return csr_add3_run(a, b, c, z, true, 0, nullptr, stream);
}

int nb200_csr_add_3_f32_into(const nb200_csr *a, const nb200_csr *b, const nb200_csr *c, nb200_csr *z,
                             int64_t capacity, void *stream) {
    return csr_add3_run(a, b, c, z, false, capacity, nullptr, stream);
}

int64_t nb200_csr_add_3_f32_scratch(const nb200_csr *a, const nb200_csr *b, const nb200_csr *c) {
    return check_add3(a, b, c) == NB200_OK ? (int64_t)Add3Sizes(a, b, c).all : 0;
}

int nb200_csr_add_3_f32_lent(const nb200_csr *a, const nb200_csr *b, const nb200_csr *c, nb200_csr *z, int64_t capacity, void *scratch,
                             int64_t scratch_bytes, void *stream) {
    if (check_add3(a, b, c) == NB200_OK && (!scratch || scratch_bytes < (int64_t)Add3Sizes(a, b, c).all)) return NB200_E_BADARG;
    return csr_add3_run(a, b, c, z, false, capacity, scratch, stream);
}

int nb200_csr_add_f32_noalloc(const nb200_csr *a, const nb200_csr *b, nb200_csr *z, int64_t capacity, void *stream) {
    return csr_add_noalloc(a, b, z, capacity, stream);
}

int nb200_csr_add_f32_async(const nb200_csr *a, const nb200_csr *b, nb200_csr *z, int64_t capacity, int64_t *device_result,
                            void *stream) {
    if (!device_result) return NB200_E_BADARG;
    return csr2_run<OP_UNION>(a, b, z, false, capacity, stream, device_result);
}

int nb200_csr_mul_f32_async(const nb200_csr *a, const nb200_csr *b, nb200_csr *z, int64_t capacity, int64_t *device_result,
                            void *stream) {
    if (!device_result) return NB200_E_BADARG;
    return csr2_run<OP_INTERSECT>(a, b, z, false, capacity, stream, device_result);
}

int nb200_selftest_lookback_timeout(const nb200_csr *a, const nb200_csr *b, nb200_csr *z, int64_t capacity, int32_t polls,
                                    void *stream) {
    if (polls < 1 || !a || !b || capacity < (int64_t)a->nnz + b->nnz) return NB200_E_BADARG;
    LaunchKnobs knobs;
    knobs.first_tile = 1;
    knobs.poll_limit = polls;
    return csr2_run<OP_UNION>(a, b, z, false, capacity, stream, nullptr, knobs);
}

int nb200_selftest_chain_timeout(const nb200_csr *a, const nb200_csr *b, const nb200_csr *c, nb200_csr *z, int64_t capacity, int32_t polls,
                                 void *stream) {
    if (polls < 1 || !a || !b || !c || capacity < (int64_t)a->nnz + b->nnz + c->nnz || (int64_t)a->nnz + b->nnz < SELFTEST_ENTRIES) return NB200_E_BADARG;
    LaunchKnobs knobs;
    knobs.first_tile = 1;
    knobs.poll_limit = polls;
    return csr_add3_run(a, b, c, z, false, capacity, nullptr, stream, knobs);
}

int nb200_selftest_late_give_up(const nb200_csr *a, const nb200_csr *b, nb200_csr *z, int64_t capacity, int32_t polls, void *stream) {
    if (polls < 1 || !a || !b || capacity < (int64_t)a->nnz + b->nnz) return NB200_E_BADARG;
    LaunchKnobs knobs;
    knobs.poll_limit = polls;
    return csr2_run<OP_UNION>(a, b, z, false, capacity, stream, nullptr, knobs);
}

}  // extern "C"
