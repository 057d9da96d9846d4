// COO3 tensor add: sorted union of two 3-mode tensors stored as parallel (i, j, k) coordinate
// arrays, as one flat merge-path over lexicographic coordinate order.
//
// The reference flattens the three COO levels into one merged coordinate and compares
// tuples (src/Compile.cpp:66-154, src/backend/tensor.cpp:447-560); its partition is the 2-way
// merge-path with the rule that equal coordinates are never split
// (src/backend/partition.cpp:813-993, :964-983). Here each coordinate is packed into one
// 64-bit key, i in the top bits, then j, then k, using just enough bits for each extent, so
// that tuple order is integer order; inside a tile the keys are counted from its smallest and then nearly
// always fit 32 bits. Tensors whose three extents need more than 63 bits in total take a second, simpler
// tile kernel that compares (i, j) and k as a 64-bit and a 32-bit word, i.e. the full three-int32 tuple
// compare of the reference for any extents.
//
// Kernels: k_coo3_partition (tile cuts) and k_coo3_tile (one CTA per tile: stage and pack the coordinates,
// bring the values in their place, split by merge-path, merge VT entries per thread, rank survivors, obtain the output base -- single pass
// with the cross-tile scan, or from the scanned counts of a first pass -- store coalesced).
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <type_traits>

#include "merge_common.cuh"
#include "tma.cuh"

namespace nb200 {

namespace {

constexpr int NT = 256;

struct Coo3In {
    const int32_t *i, *j, *k;
    const float *val;
    int32_t nnz;
};

struct Coo3Out {
    int32_t *i, *j, *k;
    float *val;
    unsigned long long *host = nullptr;  // result word: the length, or for a reduction that it is done
    float *scalar = nullptr;             // result of a reduction
};

struct Packing {
    using Key = uint64_t;
    int bj, bk;  // bits of j and k; i takes the rest
    __host__ __device__ uint64_t pack(int32_t i, int32_t j, int32_t k) const {
        return ((((uint64_t)(uint32_t)i << bj) | (uint32_t)j) << bk) | (uint32_t)k;
    }
    __host__ __device__ int32_t i_of(uint64_t key) const { return (int32_t)(key >> (bj + bk)); }
    __host__ __device__ int32_t j_of(uint64_t key) const { return (int32_t)((key >> bk) & ((1ull << bj) - 1ull)); }
    __host__ __device__ int32_t k_of(uint64_t key) const { return (int32_t)(key & ((1ull << bk) - 1ull)); }
};

// Coordinates too wide for one 64-bit word: (i, j) in one word, k in another, compared in that
// order -- the three-int32 tuple order of the reference (src/backend/tensor.cpp:447-560).
struct Key96 {
    uint64_t ij;
    uint32_t k;
    __device__ bool operator<=(const Key96 &o) const { return ij < o.ij || (ij == o.ij && k <= o.k); }
    __device__ bool operator==(const Key96 &o) const { return ij == o.ij && k == o.k; }
};
struct WidePacking {
    using Key = Key96;
    __device__ Key96 pack(int32_t i, int32_t j, int32_t k) const {
        return Key96{((uint64_t)(uint32_t)i << 32) | (uint32_t)j, (uint32_t)k};
    }
};

// Tile cuts: positions in A and B. Without them the tiles find their cuts themselves, every `step` merged entries, with words of their own
// (no step: a single tile).
struct Cuts2 {
    int32_t *a = nullptr, *b = nullptr;
    int32_t step = 0;
    OwnWords own;
};

template <typename PK>
__device__ __forceinline__ typename PK::Key key_at(const Coo3In &T, const PK &pk, int64_t p) {
    return pk.pack(ld_nc(T.i + p), ld_nc(T.j + p), ld_nc(T.k + p));
}

// Whether A's entry m orders before B's entry p or is the same position, by tuple order; j and k are read only
// where i (and j) do not decide: most probes of a search end after two loads instead of six.
__device__ __forceinline__ bool at_or_before(const Coo3In &A, int64_t m, const Coo3In &B, int64_t p) {
    const int32_t ia = ld_nc(A.i + m), ib = ld_nc(B.i + p);
    if (ia != ib) return ia < ib;
    const int32_t ja = ld_nc(A.j + m), jb = ld_nc(B.j + p);
    if (ja != jb) return ja < jb;
    return ld_nc(A.k + m) <= ld_nc(B.k + p);
}

// The cut at merged position d, equal coordinates on one side of it, between positions x_lo and x_hi of A, by G neighbouring lanes; all
// lanes of a warp call this together. Returns the positions in A and B.
template <int G>
__device__ __forceinline__ int2 find_cut(const Coo3In &A, const Coo3In &B, const int64_t d, const int64_t x_lo, const int64_t x_hi, const bool mine) {
    const int64_t x = group_count_true<G>((uint32_t)x_lo, (uint32_t)(mine ? x_hi : x_lo), [&](uint32_t m) { return at_or_before(A, m, B, d - 1 - m); });
    int64_t y = d - x;
    if (mine && x > 0 && y < B.nnz && ld_nc(A.i + x - 1) == ld_nc(B.i + y) && ld_nc(A.j + x - 1) == ld_nc(B.j + y) && ld_nc(A.k + x - 1) == ld_nc(B.k + y)) ++y;
    return make_int2((int32_t)x, (int32_t)y);
}

// Cut t of a merge by a warp, over the whole range of A.
__device__ __forceinline__ int2 tile_cut(const Coo3In &A, const Coo3In &B, const int32_t step, const int t, const int num_tiles) {
    const int64_t total = (int64_t)A.nnz + B.nnz, d = min((int64_t)t * step, total);
    const bool inner = t > 0 && t < num_tiles;
    const int2 cut = find_cut<32>(A, B, d, max((int64_t)0, d - B.nnz), min(d, (int64_t)A.nnz), inner);
    return inner ? cut : t == 0 ? make_int2(0, 0) : make_int2(A.nnz, B.nnz);
}

// Tile cuts, G lanes per cut. Cut t sits at merged position min(t * tile_step, total); equal coordinates stay on one
// side of a cut. `stride` > 1: only every stride-th cut (and the last) is made. `between` > 0: only the cuts that
// a launch with that stride left out, each searched between its two neighbours among those. The control block and
// the tile words of the tile kernel are cleared on the way.
template <int G>
__global__ void __launch_bounds__(NT) k_coo3_partition(Coo3In A, Coo3In B, int64_t total, int32_t tile_step, int32_t num_tiles, int stride, int between,
                                                       Cuts2 cuts, uint64_t *zero_block, int zero_words) {
    trigger_dependents();
    const int64_t gid = (int64_t)blockIdx.x * NT + threadIdx.x;
    for (int64_t z = gid; z < zero_words; z += (int64_t)gridDim.x * NT) zero_block[z] = 0;
    if (between) wait_for_previous();           // the cuts made so far
    const int64_t t64 = gid / G * stride;
    const int t = (int)min(t64, (int64_t)num_tiles);  // spare groups repeat the last cut
    const bool mine = t64 < num_tiles + stride && !(between && (t % between == 0 || t == num_tiles));
    const int64_t d = min((int64_t)t * tile_step, total);
    const bool inner = t > 0 && t < num_tiles;
    int64_t x_lo = max((int64_t)0, d - B.nnz), x_hi = min(d, (int64_t)A.nnz);
    if (between && mine) {
        const int before = t / between * between;
        x_lo = max(x_lo, (int64_t)cuts.a[before]);
        x_hi = min(x_hi, (int64_t)cuts.a[min(before + between, num_tiles)]);
    }
    int2 cut = find_cut<G>(A, B, d, x_lo, x_hi, inner && mine);
    if (!inner) cut = t == 0 ? make_int2(0, 0) : make_int2(A.nnz, B.nnz);
    if ((threadIdx.x & (G - 1)) == 0 && mine) {
        cuts.a[t] = cut.x;
        cuts.b[t] = cut.y;
    }
}

constexpr int RW_COO3 = 8;  // index of the result word (the callers that lend their workspace use lower ones)
constexpr int MBAR_POLL_LIMIT = 1 << 24;
constexpr int ERR_COPY_TIMEOUT = 2;

// Number of 4-byte elements from `p` up to the next 16-byte boundary (0..3).
__device__ __forceinline__ int head_elems(const void *p) {
    return (int)(((16u - (unsigned)(reinterpret_cast<uintptr_t>(p) & 15u)) & 15u) >> 2);
}

// The last tile has its base: the result length (negative after a give-up of any tile) goes to the control block and the host.
__device__ __forceinline__ void coo3_finish(FusedCtl *ctl, const Coo3Out &Z, long long total) {
    if (total >= 0) ctl->total = total;
    publish_result_word(Z.host, total < 0 ? NB200_E_TIMEOUT : NB200_OK, total < 0 ? 0 : total);
}

// One thread per tile, after the tile's sum: the last tile to get here writes the reduction's result.
__device__ __forceinline__ void coo3_reduce_done(FusedCtl *ctl, const Coo3Out &Z, int num_tiles) {
    __threadfence();
    if (atomicAdd(&ctl->hollow, 1) != num_tiles - 1) return;
    __threadfence();
    *Z.scalar = (float)__longlong_as_double(*(volatile long long *)&ctl->total);
    publish_result_word(Z.host, ld_relaxed_gpu_i32(&ctl->status.error) != 0 ? NB200_E_TIMEOUT : NB200_OK, 0);
}

// Shared-memory plan of the tile body, in 4-byte words: three raw arrays (i, j, k), in which A's entry e sits
// at word oa + e and B's at word ob + e, chosen so that 16-byte boundaries of global memory fall on 16-byte
// boundaries here (what a bulk copy needs). Every entry's coordinates are packed in place: the key takes the
// place of i (and, for 64-bit keys, of j), and the 16-bit source indices of the result take the place of j (of k).
template <int VT>
struct Coo3Plan {
    static constexpr int CAP = NT * VT;
    static constexpr int SLOTS = CAP + 16;
    static constexpr size_t BYTES = 12 * (size_t)SLOTS;
    static_assert(4 * SLOTS < 32768, "byte offsets of entries are kept in 15 bits");
};
// A tile asks for the coordinates of one that starts a few microseconds later, so that they wait in L2. 100 M entries per
// operand: 1061 us without, 1184, 1042, 1031 and 1036 with those 592, 296, 148 and 64 tiles ahead. Not for a tile that starts with
// the first ones: 3 M entries per operand 77.1 -> 75.5 us.
constexpr int TILES_AHEAD = 148;

struct Coo3Shared {
    uint64_t mbar;
    long long base;  // output base of the tile
    int2 cut[2];     // where it begins and ends, if it finds that out itself
    int wtotal[NT / 32];
    double partial[NT / 32];
};

// x << s, nothing where s is 32 or more.
__device__ __forceinline__ uint32_t shl32(uint32_t x, int s) {
    uint32_t r;
    asm("shl.b32 %0, %1, %2;" : "=r"(r) : "r"(x), "r"(s));
    return r;
}

// Brings the tile's values into shared memory, entry e of A to word oa + e of `to` and B's to ob + e: aligned interiors by bulk
// copy on the second phase of the tile's mbarrier, ragged ends by plain loads, arrays whose alignment differs word by word, on their way during the
// merge too (copies_landed; sums of 16 M and 60 M entries of that kind took 263 and 680 us a call with plain loads, which the merge waits for, 233 and 630 with values
// gathered from L2 behind it, 219 and 581 so). Called by all threads after a barrier behind the last use of the words.
// Returns, to all of them, whether copies_landed has to be called; where it is not needed it is left out (100 M entries 1031 -> 1027).
__device__ __forceinline__ bool coo3_stage_values(const float *a_val, const float *b_val, const int na, const int nb, const int oa, const int ob, uint32_t *to,
                                                  Coo3Shared &sh) {
    const int tid = threadIdx.x;
    const float *const src[2] = {a_val, b_val};
    const int count[2] = {na, nb}, at[2] = {oa, ob};
    int head[2], nv[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        head[q] = min(count[q], head_elems(src[q]));
        nv[q] = ((at[q] + head[q]) & 3) == 0 ? (count[q] - head[q]) >> 2 : 0;
    }
    if (tid == 0) {
        fence_async_shared();  // the words were read and written by the threads so far
        mbar_arrive_expect_tx(&sh.mbar, 16u * (uint32_t)(nv[0] + nv[1]));
#pragma unroll
        for (int q = 0; q < 2; ++q)
            if (nv[q]) bulk_load(to + at[q] + head[q], src[q] + head[q], 16u * nv[q], &sh.mbar);
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        // the ends of q: a warp each; nothing but ends where no vector is copied
        if (nv[q] == 0) {
            for (int e = tid; e < count[q]; e += NT) copy_word(to + at[q] + e, src[q] + e);
        } else if ((tid >> 5) == 1 + q && (tid & 31) < 6) {
            const int e = tid & 31, idx = e < 3 ? e : head[q] + 4 * nv[q] + (e - 3);
            if (e < 3 ? e < head[q] : idx < count[q]) to[at[q] + idx] = __float_as_uint(__ldg(src[q] + idx));
        }
    }
    return nv[0] == 0 || nv[1] == 0;
}

// One tile. NARROW: the keys of the tile, counted from its smallest, fit 32 bits (true of nearly every tile of
// a tensor of millions of entries); otherwise they are kept as a low and a high word.
//
// The structure is that of the CSR tile kernel (csr_merge.cu), without rows: one result entry per step of a sequential merge; a 16-bit
// source index per result entry is compacted. REDUCE (inner product): only the products of the coordinates that both operands hold are summed.
//
// Bound by instruction issue (0.65 of the slots where this was counted) and the latency of a tile's barrier-separated phases beside HBM. 32-bit keys
// leave the words of k free: the values are copied there during the merge, the sum of a twin is made in place by the thread that merged it, and
// results are fetched from shared memory alone, without a test or an address per entry. 100 M entries per operand: values gathered from L2 and a
// test for twins per result 1208 us a call, this 1098; inner product of 4 M 58.4 -> 54.8.
template <int VT, int MODE, bool NARROW>
__device__ __forceinline__ void coo3_tile(const Coo3In &A, const Coo3In &B, const Packing &pk, const int32_t a0, const int32_t b0, const int na,
                                          const int nb, const int oa, const int ob, const uint64_t key0, const int t, const int num_tiles,
                                          int32_t *tile_count, const TileWords &words, FusedCtl *ctl, const Coo3Out &Z,
                                          unsigned char *smem_raw, Coo3Shared &sh) {
    using P = Coo3Plan<VT>;
    using Key = typename std::conditional<NARROW, uint32_t, uint64_t>::type;
    constexpr Key END = (Key)~(Key)0;
    constexpr bool REDUCE = MODE == MODE_REDUCE;
    constexpr bool STAGED = NARROW && MODE != MODE_COUNT;  // values in shared memory (64-bit keys leave no room for them)
    constexpr uint32_t HIGH = 4 * P::SLOTS;   // byte distance from a key's low to its high word
    constexpr uint32_t VALUE = 8 * P::SLOTS;  // ... from a 32-bit key to its entry's value
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, n = na + nb;
    uint32_t *raw = reinterpret_cast<uint32_t *>(smem_raw);
    uint16_t *src_of = reinterpret_cast<uint16_t *>(raw + (NARROW ? 1 : 2) * P::SLOTS);
    auto word_at = [&](uint32_t byte) -> uint32_t & { return *reinterpret_cast<uint32_t *>(smem_raw + byte); };
    auto key_at_byte = [&](uint32_t byte) -> Key {
        return NARROW ? (Key)word_at(byte) : (Key)((uint64_t)word_at(byte + HIGH) << 32 | word_at(byte));
    };

    // ---- pack, four staged words at a time, whatever they hold: padding packs to something that nobody reads, and the words
    // behind each operand become its sentinel.
    {
        uint4 *w4 = reinterpret_cast<uint4 *>(smem_raw);
        constexpr int S4 = P::SLOTS / 4;
        const int end_a = oa + na, end_b = ob + nb;
        for (int v = tid; 4 * v <= end_b; v += NT) {
            const uint4 i4 = w4[v], j4 = w4[S4 + v], k4 = w4[2 * S4 + v];
            if (NARROW) {  // the low words of the packed coordinates are enough
                auto low = [&](uint32_t i, uint32_t j, uint32_t k) { return (shl32(i, pk.bj + pk.bk) | shl32(j, pk.bk) | k) - (uint32_t)key0; };
                w4[v] = make_uint4(low(i4.x, j4.x, k4.x), low(i4.y, j4.y, k4.y), low(i4.z, j4.z, k4.z), low(i4.w, j4.w, k4.w));
            } else {
                auto full = [&](uint32_t i, uint32_t j, uint32_t k) { return pk.pack((int32_t)i, (int32_t)j, (int32_t)k) - key0; };
                const uint64_t a = full(i4.x, j4.x, k4.x), b = full(i4.y, j4.y, k4.y), c = full(i4.z, j4.z, k4.z), d = full(i4.w, j4.w, k4.w);
                w4[v] = make_uint4((uint32_t)a, (uint32_t)b, (uint32_t)c, (uint32_t)d);
                w4[S4 + v] = make_uint4((uint32_t)(a >> 32), (uint32_t)(b >> 32), (uint32_t)(c >> 32), (uint32_t)(d >> 32));
            }
            if (end_a >> 2 == v || end_b >> 2 == v) {
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    if (4 * v + c == end_a || 4 * v + c == end_b) {
                        raw[4 * v + c] = 0xffffffffu;
                        if (!NARROW) raw[P::SLOTS + 4 * v + c] = 0xffffffffu;
                    }
            }
        }
    }
    __syncthreads();
    // ---- the values take the place of the k coordinates; they land during the merge
    const bool word_by_word = STAGED && coo3_stage_values(A.val + a0, B.val + b0, na, nb, oa, ob, raw + 2 * P::SLOTS, sh);

    // ---- where this thread's share begins: merge-path diagonal tid * VT (ties take A first; a coordinate that
    // both operands hold stays on one side)
    const int diag = min(tid * VT, n);
    int x, y;
    {
        int lo = max(0, diag - nb), up = min(diag, na);
        const uint32_t ca = 4u * (uint32_t)oa, cb = 4u * (uint32_t)(ob + diag - 1);
        while (lo < up) {
            const int mid = (lo + up) >> 1;
            if (key_at_byte(ca + 4u * mid) <= key_at_byte(cb - 4u * mid)) lo = mid + 1; else up = mid;
        }
        x = lo;
        y = diag - lo;
        if (x > 0 && y < nb && key_at_byte(4u * (uint32_t)(oa + x - 1)) == key_at_byte(4u * (uint32_t)(ob + y))) ++y;
    }

    // ---- merge, one result entry per step; src[i]: the entry step i took (A's where both)
    const uint32_t pa0 = 4u * (uint32_t)(oa + x), pb0 = 4u * (uint32_t)(ob + y);
    uint32_t src[VT];
    unsigned twin = 0;
    int steps;
    {
        // (as in the CSR tile kernel: VT steps for everybody, cut to the thread's share afterwards, and the key behind each
        // head a step ahead. Past its end a list reads other words of the tile's shared memory.)
        uint32_t pa = pa0, pb = pb0;
        Key ka = key_at_byte(pa), kb = key_at_byte(pb);
        Key next_a = key_at_byte(pa + 4), next_b = key_at_byte(pb + 4);
#pragma unroll
        for (int i = 0; i < VT; ++i) {
            const bool ta = ka <= kb, tb = kb <= ka;
            src[i] = ta ? pa : pb;
            if (ta && tb) twin |= 1u << i;
            if (ta) {
                pa += 4;
                ka = next_a;
                next_a = key_at_byte(pa + 4);
            }
            if (tb) {
                pb += 4;
                kb = next_b;
                next_b = key_at_byte(pb + 4);
            }
        }
        // step i is the thread's where the entries taken before it, i + (twins before it), are fewer than its share
        const int share = min(tid * VT + VT, n) - (x + y);
        steps = share;
        if (__any_sync(FULL_MASK, twin != 0u)) {
            int lo = 0, hi = max(share, 0);
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (mid + __popc(twin & ((1u << mid) - 1u)) >= share) hi = mid; else lo = mid + 1;
            }
            steps = lo;
        }
        twin &= (1u << steps) - 1u;
    }

    // byte offset of the B word of the twin at step i, whose A word is `at` (step i began at pa0 + pb0 + 4 (i + twins before it))
    auto partner = [&](int i, uint32_t at) { return pa0 + pb0 + 4u * (uint32_t)(i + __popc(twin & ((1u << i) - 1u))) - at; };
    auto report_copy = [&]() {
        if (atomicCAS(&ctl->status.error, 0, ERR_COPY_TIMEOUT) == 0) ctl->status.detail = t;
        __threadfence();
    };
    const char *va = reinterpret_cast<const char *>(A.val + a0) - 4 * (int64_t)oa, *vb = reinterpret_cast<const char *>(B.val + b0) - 4 * (int64_t)ob;

    if (REDUCE) {
        // ---- inner product: products in float32 as the reference's, summed in double; one atomic per tile into
        // the control block (the order of the tiles' sums is not fixed, as with the reference's atomic
        // accumulation, src/backend/compute.cpp:498-525). A thread notes its twins in a part of its own of the source indices.
        uint16_t *own = src_of + tid * VT, *to = own;
#pragma unroll
        for (int i = 0; i < VT; ++i)
            if ((twin >> i) & 1u) *to++ = (uint16_t)src[i];
        if (word_by_word) copies_landed();
        const bool landed = !STAGED || wid > 0 || mbar_wait_bounded(&sh.mbar, 1, MBAR_POLL_LIMIT);
        if (!__syncthreads_and(landed)) {
            if (tid == 0) {
                report_copy();
                mbar_wait_bounded(&sh.mbar, 1, MBAR_POLL_LIMIT);  // second bounded wait for copies in flight
            }
            return;
        }
        double sum = 0.0;
        for (unsigned left = twin; left; left &= left - 1u) {
            const uint32_t at = *own++, other = partner(__ffs(left) - 1, at);
            if (STAGED) sum += (double)(__uint_as_float(word_at(at + VALUE)) * __uint_as_float(word_at(other + VALUE)));
            else sum += (double)(__ldg(reinterpret_cast<const float *>(va + at)) * __ldg(reinterpret_cast<const float *>(vb + other)));
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(FULL_MASK, sum, o);
        if (lane == 0) sh.partial[wid] = sum;
        __syncthreads();
        if (tid == 0) {
            double s = 0.0;
            for (int w = 0; w < NT / 32; ++w) s += sh.partial[w];
            if (s != 0.0) atomicAdd(reinterpret_cast<double *>(&ctl->total), s);
        }
        return;
    }

    // ---- rank the survivors inside the tile
    const int incl = warp_incl_sum(steps);
    if (lane == 31) sh.wtotal[wid] = incl;
    if (word_by_word) copies_landed();
    const bool landed = !STAGED || wid > 0 || mbar_wait_bounded(&sh.mbar, 1, MBAR_POLL_LIMIT);
    if (!__syncthreads_and(landed)) {  // the values did not land in time: report, touch nothing
        if (tid == 0) {
            report_copy();
            if (MODE == MODE_FUSED) {
                publish_failure(words, t);
                if (t == num_tiles - 1) publish_result_word(Z.host, NB200_E_TIMEOUT, 0);
            }
            mbar_wait_bounded(&sh.mbar, 1, MBAR_POLL_LIMIT);  // second bounded wait for copies in flight
        }
        return;
    }
    int total = 0, wbase = 0;
#pragma unroll
    for (int w = 0; w < NT / 32; ++w) {
        const int c = sh.wtotal[w];
        wbase += w < wid ? c : 0;
        total += c;
    }
    const int rank = wbase + incl - steps;
    if (MODE == MODE_COUNT) {
        if (tid == 0) tile_count[t] = total;
        return;
    }
    if (MODE == MODE_FUSED && tid == 0) publish_count(words, t, total);

    // ---- compact; the value of a twin's A entry becomes the sum (64-bit keys: its A word now points to its B word)
    {
        uint16_t *to = src_of + rank;
#pragma unroll
        for (int i = 0; i < VT; ++i)
            if (i < steps) to[i] = (uint16_t)src[i];
        for (unsigned left = twin; left; left &= left - 1u) {
            const int i = __ffs(left) - 1;
            const uint32_t at = to[i], other = partner(i, at);
            if (STAGED) {
                word_at(at + VALUE) = __float_as_uint(__uint_as_float(word_at(at + VALUE)) + __uint_as_float(word_at(other + VALUE)));
            } else {
                word_at(at) = other;
                to[i] = (uint16_t)(at | 0x8000u);
            }
        }
    }

    auto live = [&](int q) { return q < VT && q * NT + tid < total; };
    const uint32_t first_b = 4u * (uint32_t)ob;
    constexpr int GATHER = STAGED ? VT : 8;
    Key key[GATHER];
    float val[GATHER];
    auto gather = [&](const int q0) {
        uint32_t s[GATHER];
#pragma unroll
        for (int g = 0; g < GATHER; ++g) s[g] = live(q0 + g) ? (uint32_t)src_of[(q0 + g) * NT + tid] : 4u * (uint32_t)oa;
#pragma unroll
        for (int g = 0; g < GATHER; ++g) {
            if (STAGED) {
                key[g] = key_at_byte(s[g]);
                val[g] = __uint_as_float(word_at(s[g] + VALUE));
            } else {
                const bool both = (s[g] & 0x8000u) != 0u;
                const uint32_t at = s[g] & 0x7fffu, other = both ? word_at(at) : at;
                key[g] = key_at_byte(other);
                float v = 0.0f;
                if (live(q0 + g)) v = __ldg(reinterpret_cast<const float *>((at >= first_b ? vb : va) + at));
                if (both) v = v + __ldg(reinterpret_cast<const float *>(vb + other));
                val[g] = v;
            }
        }
    };
    __syncthreads();
    gather(0);

    // ---- output base of the tile
    if (MODE == MODE_FUSED && wid == 0) {
        const int64_t b = tile_base(words, t, total, &ctl->status, LOOKBACK_POLL_LIMIT);
        if (lane == 0) {
            sh.base = b;
            if (t == num_tiles - 1) coo3_finish(ctl, Z, b < 0 ? b : b + total);
        }
    }
    __syncthreads();
    const long long base = MODE == MODE_FILL ? (long long)tile_count[t] : sh.base;
    if (base < 0) return;  // a bounded wait gave up; the host reports it

    // ---- unpack and store, coalesced
    int32_t *zi = Z.i + base + tid, *zj = Z.j + base + tid, *zk = Z.k + base + tid;
    float *zv = Z.val + base + tid;
#pragma unroll
    for (int q0 = 0; q0 < VT; q0 += GATHER) {
        if (q0 > 0) {
            if (q0 * NT >= total) break;
            gather(q0);
        }
#pragma unroll
        for (int g = 0; g < GATHER; ++g) {
            if (live(q0 + g)) {
                const uint64_t full = key0 + key[g];
                zi[(q0 + g) * NT] = pk.i_of(full);
                zj[(q0 + g) * NT] = pk.j_of(full);
                zk[(q0 + g) * NT] = pk.k_of(full);
                zv[(q0 + g) * NT] = val[g];
            }
        }
    }
}

template <int VT, int MODE>
__global__ void __launch_bounds__(NT, 4) k_coo3_tile(const __grid_constant__ Coo3In A, const __grid_constant__ Coo3In B, const Packing pk,
                                                     const Cuts2 cuts, int32_t *tile_count, const __grid_constant__ TileWords words, FusedCtl *ctl,
                                                     const __grid_constant__ Coo3Out Z, int num_tiles) {
    using P = Coo3Plan<VT>;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ Coo3Shared sh;
    const int tid = threadIdx.x;
    if (tid == 0) {
        mbar_init(&sh.mbar, 1);
        mbar_fence_init();
    }
    __syncthreads();
    wait_for_previous();  // the cuts
    // tiles are numbered by CTA index: CTAs are dispatched in increasing index order, so a tile
    // only waits on CTAs dispatched before it (and every such wait is bounded)
    const int t = blockIdx.x;
    int32_t a0 = 0, b0 = 0;
    int na = A.nnz, nb = B.nnz;
    if (cuts.step) {
        if (t == 0 && tid == 0) *cuts.own.clear = FusedCtl{};
        const int w = tid >> 5;
        if (w < 2) {
            const int2 cut = tile_cut(A, B, cuts.step, t + w, num_tiles);
            if ((tid & 31) == 0) sh.cut[w] = cut;
        }
        __syncthreads();
        a0 = sh.cut[0].x, b0 = sh.cut[0].y;
        na = sh.cut[1].x - a0, nb = sh.cut[1].y - b0;
    } else if (cuts.a) {
        a0 = cuts.a[t], b0 = cuts.b[t];
        na = cuts.a[t + 1] - a0, nb = cuts.b[t + 1] - b0;
        if (tid == 96 && t + TILES_AHEAD >= RESIDENT && t + TILES_AHEAD < num_tiles) {
            const int32_t a1 = cuts.a[t + TILES_AHEAD], b1 = cuts.b[t + TILES_AHEAD], n_a = cuts.a[t + TILES_AHEAD + 1] - a1, n_b = cuts.b[t + TILES_AHEAD + 1] - b1;
            prefetch_l2(A.i + a1, n_a), prefetch_l2(A.j + a1, n_a), prefetch_l2(A.k + a1, n_a);
            prefetch_l2(B.i + b1, n_b), prefetch_l2(B.j + b1, n_b), prefetch_l2(B.k + b1, n_b);
        }
    } else if (tid == 0) {  // a single tile: no partition kernel ran, so this clears the control block
        *ctl = FusedCtl{};
    }

    // ---- stage the six coordinate arrays: aligned interiors by bulk copy, ragged ends (at most three entries
    // each side) and arrays whose alignment differs from their i array's by plain loads
    uint32_t *raw = reinterpret_cast<uint32_t *>(smem_raw);
    const int ha = head_elems(A.i + a0), hb = head_elems(B.i + b0);
    const int oa = (4 - ha) & 3;
    const int ob = ((oa + na + 1 + 3) & ~3) + ((4 - hb) & 3);  // A's sentinel lies before it
    {
        const int32_t *src[6] = {A.i + a0, A.j + a0, A.k + a0, B.i + b0, B.j + b0, B.k + b0};
        const int head_a = min(na, ha), head_b = min(nb, hb);
        const int nva = (na - head_a) >> 2, nvb = (nb - head_b) >> 2;
        bool bulk[6];
#pragma unroll
        for (int q = 0; q < 6; ++q) bulk[q] = head_elems(src[q]) == (q < 3 ? ha : hb);
        if (tid == 0) {
            uint32_t bytes = 0;
#pragma unroll
            for (int q = 0; q < 6; ++q) bytes += bulk[q] ? 16u * (q < 3 ? nva : nvb) : 0u;
            mbar_arrive_expect_tx(&sh.mbar, bytes);
#pragma unroll
            for (int q = 0; q < 6; ++q) {
                const int nv = q < 3 ? nva : nvb, head = q < 3 ? head_a : head_b;
                if (bulk[q] && nv) bulk_load(raw + (q % 3) * P::SLOTS + (q < 3 ? oa : ob) + head, src[q] + head, 16u * nv, &sh.mbar);
            }
            if (MODE != MODE_COUNT) {
                prefetch_l2(A.val + a0, na);
                prefetch_l2(B.val + b0, nb);
            }
        }
        if (tid >= 32 && tid < 32 + 36) {  // ragged ends: 6 arrays x (3 head + 3 tail)
            const int q = (tid - 32) / 6, e = (tid - 32) % 6;
            const int count = q < 3 ? na : nb, head = q < 3 ? head_a : head_b, nv = q < 3 ? nva : nvb;
            const int idx = e < 3 ? e : head + 4 * nv + (e - 3);
            bool is_bulk = false;
            const int32_t *g = nullptr;
#pragma unroll
            for (int qq = 0; qq < 6; ++qq)
                if (qq == q) is_bulk = bulk[qq], g = src[qq];
            if (is_bulk && (e < 3 ? e < head : idx < count)) raw[(q % 3) * P::SLOTS + (q < 3 ? oa : ob) + idx] = (uint32_t)ld_nc(g + idx);
        }
#pragma unroll
        for (int q = 0; q < 6; ++q)
            if (!bulk[q])
                for (int e = tid; e < (q < 3 ? na : nb); e += NT) raw[(q % 3) * P::SLOTS + (q < 3 ? oa : ob) + e] = (uint32_t)ld_nc(src[q] + e);
    }
    const bool landed = tid >= 32 || mbar_wait_bounded(&sh.mbar, 0, MBAR_POLL_LIMIT);  // one warp polls; the others' issue slots are worth more
    if (!__syncthreads_and(landed)) {  // the copies did not land in time: report, touch nothing
        if (tid == 0) {
            if (atomicCAS(&ctl->status.error, 0, ERR_COPY_TIMEOUT) == 0) ctl->status.detail = t;
            __threadfence();
            if (MODE == MODE_FUSED) {
                publish_failure(words, t);
                if (t == num_tiles - 1) publish_result_word(Z.host, NB200_E_TIMEOUT, 0);
            }
            if (MODE == MODE_REDUCE) coo3_reduce_done(ctl, Z, num_tiles);
            mbar_wait_bounded(&sh.mbar, 0, MBAR_POLL_LIMIT);  // second bounded wait for copies in flight
        }
        return;
    }
    // ---- smallest and largest key of the tile
    auto staged_key = [&](int w) { return pk.pack((int32_t)raw[w], (int32_t)raw[P::SLOTS + w], (int32_t)raw[2 * P::SLOTS + w]); };
    uint64_t key0 = ~0ull, key1 = 0;
    if (na > 0) key0 = staged_key(oa), key1 = staged_key(oa + na - 1);
    if (nb > 0) key0 = min(key0, staged_key(ob)), key1 = max(key1, staged_key(ob + nb - 1));
    __syncthreads();  // everybody has read them: packing overwrites them
    if (key1 - key0 < 0xffffffffull)
        coo3_tile<VT, MODE, true>(A, B, pk, a0, b0, na, nb, oa, ob, key0, t, num_tiles, tile_count, words, ctl, Z, smem_raw, sh);
    else
        coo3_tile<VT, MODE, false>(A, B, pk, a0, b0, na, nb, oa, ob, key0, t, num_tiles, tile_count, words, ctl, Z, smem_raw, sh);
    if (MODE == MODE_REDUCE && tid == 0) coo3_reduce_done(ctl, Z, num_tiles);
}

// ---------------------------------------------------------------- wide coordinates ----

// Tile kernel for extents that need more than 63 bits together. One CTA of WNT threads per tile of
// WNT * WVT - 1 merged entries: (i, j) words and k words staged in shared memory with plain loads,
// merge-path split with the two-word compare, sequential merge of WVT entries per thread, values
// fetched from global memory, compaction through shared memory, coalesced stores. Single pass with
// bounded look-back, or count / fill around a scan, like the packed-key kernel.
constexpr int WNT = 256, WVT = 7, WCAP = WNT * WVT, WKS = WCAP + 2 + WVT;

template <int MODE>
__global__ void __launch_bounds__(WNT) k_coo3_tile_wide(Coo3In A, Coo3In B, Cuts2 cuts, int32_t *tile_count, uint64_t *tile_state_raw,
                                                         FusedCtl *ctl, Coo3Out Z) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ int scan_tmp[40];
    __shared__ long long s_base;
    volatile uint64_t *tile_state = tile_state_raw;
    const WidePacking pk;
    const int tid = threadIdx.x;
    const int t = blockIdx.x;  // CTAs are dispatched in index order; waits on earlier tiles are bounded
    const int32_t a0 = cuts.a[t], b0 = cuts.b[t];
    const int na = cuts.a[t + 1] - a0, nb = cuts.b[t + 1] - b0;
    const int n = na + nb;
    uint64_t *hx = reinterpret_cast<uint64_t *>(smem_raw), *hy = hx + na + 1;
    uint32_t *lx = reinterpret_cast<uint32_t *>(hx + WKS), *ly = lx + na + 1;
    float *out_val = reinterpret_cast<float *>(lx + WKS);
    for (int e = tid; e < na; e += WNT) {
        const Key96 q = key_at(A, pk, (int64_t)a0 + e);
        hx[e] = q.ij;
        lx[e] = q.k;
    }
    for (int e = tid; e < nb; e += WNT) {
        const Key96 q = key_at(B, pk, (int64_t)b0 + e);
        hy[e] = q.ij;
        ly[e] = q.k;
    }
    if (tid < WVT + 1) hy[nb + tid] = ~0ull, ly[nb + tid] = ~0u;  // all-ones orders after every coordinate
    if (tid == 0) hx[na] = ~0ull, lx[na] = ~0u;
    __syncthreads();
    auto kx = [&](int p) { return Key96{hx[p], lx[p]}; };
    auto ky = [&](int p) { return Key96{hy[p], ly[p]}; };

    // ---- split the tile among threads: merge-path diagonal tid * WVT, ties take A first
    const int diag = min(tid * WVT, n);
    int x, y;
    {
        int lo = max(0, diag - nb), hi = min(diag, na);
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (kx(mid) <= ky(diag - 1 - mid)) lo = mid + 1; else hi = mid;
        }
        x = lo;
        y = diag - lo;
    }
    const int x0 = x, y0 = y;

    // ---- merge WVT entries; bit i of `from_a`: entry i came from A; of `twin`: the same
    // coordinate is in B too; of `emit`: the entry goes to the result
    Key96 key[WVT];
    unsigned from_a = 0, twin = 0, emit = 0;
    {
        const int valid = min(WVT, n - diag);
        Key96 cx = kx(x), cy = ky(y);
        Key96 last_x = x > 0 ? kx(x - 1) : Key96{~0ull, ~0u};
#pragma unroll
        for (int i = 0; i < WVT; ++i) {
            const bool tx = cx <= cy;
            const bool both = cx == cy;
            key[i] = tx ? cx : cy;
            from_a |= (unsigned)tx << i;
            twin |= (unsigned)(tx && both) << i;
            emit |= (unsigned)(i < valid && (tx || !(cy == last_x))) << i;
            last_x = tx ? cx : last_x;
            x += tx;
            y += !tx;
            cx = kx(x);
            cy = ky(y);
        }
    }
    int total;
    const int rank = block_excl_sum<WNT>(__popc(emit), scan_tmp, total);  // syncs: key reads are done
    if (MODE == MODE_COUNT) {
        if (tid == 0) tile_count[t] = total;
        return;
    }
    if (MODE == MODE_FUSED && warp_id() == 0) {
        const int64_t b = lookback_exclusive(tile_state, t, total, &ctl->status);
        if (lane_id() == 0) {
            s_base = b;
            if (b >= 0 && t == (int)gridDim.x - 1) ctl->total = b + total;
        }
    }
    // ---- compact through shared memory (the staging arrays reuse the key words), store coalesced
    {
        int r = rank, xi = x0, yi = y0;
#pragma unroll
        for (int i = 0; i < WVT; ++i) {
            const bool tx = (from_a >> i) & 1u;
            if ((emit >> i) & 1u) {
                float v = tx ? ld_nc(A.val + a0 + xi) : ld_nc(B.val + b0 + yi);
                if ((twin >> i) & 1u) v = v + ld_nc(B.val + b0 + yi);
                hx[r] = key[i].ij;
                lx[r] = key[i].k;
                out_val[r] = v;
                ++r;
            }
            xi += tx;
            yi += !tx;
        }
    }
    __syncthreads();
    const long long base = MODE == MODE_FILL ? (long long)tile_count[t] : s_base;
    if (base < 0) return;  // a bounded wait gave up; the host reports it
    for (int e = tid; e < total; e += WNT) {
        const uint64_t ij = hx[e];
        Z.i[base + e] = (int32_t)(ij >> 32);
        Z.j[base + e] = (int32_t)(uint32_t)ij;
        Z.k[base + e] = (int32_t)lx[e];
        Z.val[base + e] = out_val[e];
    }
}

constexpr size_t coo3_wide_smem_bytes() { return 12 * (size_t)WKS + 4 * (size_t)WCAP; }

template <int MODE>
cudaError_t launch_coo3_tile_wide(const Coo3In &A, const Coo3In &B, const Cuts2 &cuts, int32_t *tile_count, uint64_t *tile_state,
                                  FusedCtl *ctl, const Coo3Out &Z, int num_tiles, cudaStream_t stream) {
    static const char *const names[3] = {"coo3_add_wide_count", "coo3_add_wide_fill", "coo3_add_wide_fused"};
    LaunchScope scope(names[MODE], stream);
    k_coo3_tile_wide<MODE><<<num_tiles, WNT, coo3_wide_smem_bytes(), stream>>>(A, B, cuts, tile_count, tile_state, ctl, Z);
    return cudaGetLastError();
}

static_assert(coo3_wide_smem_bytes() <= 48 * 1024, "the wide tile kernel stays within the default shared-memory limit");


int bits_for(int32_t extent) {
    int b = 1;
    while (b < 32 && (int64_t(1) << b) < (int64_t)extent) ++b;
    return b;
}

constexpr int tile_step_of(int v) { return NT * v - 1; }  // a twin may add one entry

// Merged entries per worker thread: large tiles amortise the searches and the wait for the earlier counts, small
// ones fill the chip when there are few entries, up to the number that can be at work at once (as in the CSR kernel). 100 M entries per operand, whole call: 1122 us with 13, 1065
// with 15, 1027 with 17 (52 KB of shared memory: the most of which four CTAs fit an SM), 1098 with 19. Sums of 0.4, 0.6, 1, 1.3 M entries per
// operand, whole call: 21.9, 32.2, 41.3, 48.2 us with 7, 21.3, 25.4, 39.7, 44.8 with 11, 32.4 and 42.4 the latter two with 17. A reduction has nothing
// but the merge behind the staging: 0.1, 0.3, 0.6, 1 M 17.5, 18.6, 24.0, 31.5 with 7, 18.2, 18.9, 20.3, 29.1 with 11, 21.6 and 26.9 the latter two with 17.
constexpr int V_LARGE = 17, V_SMALL = 11, V_REDUCE = 7;
constexpr int tile_v(int64_t total, int small = V_SMALL) { return total > (int64_t)RESIDENT * tile_step_of(small) ? V_LARGE : small; }

template <int VT, int MODE>
cudaError_t launch_coo3_tile_v(const Coo3In &A, const Coo3In &B, const Packing &pk, const Cuts2 &cuts, int32_t *tile_count, const TileWords &words,
                               FusedCtl *ctl, const Coo3Out &Z, int num_tiles, cudaStream_t stream) {
    auto kernel = k_coo3_tile<VT, MODE>;
    constexpr size_t smem = Coo3Plan<VT>::BYTES;
    static bool configured[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    const dim3 grid(num_tiles);
    if ((MODE == MODE_FUSED || MODE == MODE_REDUCE) && cuts.a)
        return launch_overlapped(kernel, grid, dim3(NT), smem, stream, A, B, pk, cuts, tile_count, words, ctl, Z, num_tiles);
    kernel<<<grid, NT, smem, stream>>>(A, B, pk, cuts, tile_count, words, ctl, Z, num_tiles);
    return cudaGetLastError();
}

template <int MODE>
cudaError_t launch_coo3_tile(const Coo3In &A, const Coo3In &B, const Packing &pk, const Cuts2 &cuts, int32_t *tile_count, const TileWords &words,
                             FusedCtl *ctl, const Coo3Out &Z, int num_tiles, int v, cudaStream_t stream) {
    static const char *const names[4] = {"coo3_add_count", "coo3_add_fill", "coo3_add_fused", "coo3_inner_prod"};
    LaunchScope scope(names[MODE], stream);
    constexpr int SMALL = MODE == MODE_REDUCE ? V_REDUCE : V_SMALL;
    return v == V_LARGE ? launch_coo3_tile_v<V_LARGE, MODE>(A, B, pk, cuts, tile_count, words, ctl, Z, num_tiles, stream)
                        : launch_coo3_tile_v<SMALL, MODE>(A, B, pk, cuts, tile_count, words, ctl, Z, num_tiles, stream);
}

// Queues the cuts; `zero_words` words of control block and tile words are cleared on the way. Up to about a wave of
// warps, a warp per cut. Beyond that the bytes that the probes touch count (a sector each, far apart): a warp for
// every 32nd cut, then four lanes for every other one between its two neighbours. 46 000 cuts (100 M entries per
// operand): 87 us so, 104 with eight lanes, 83 with two, 166 with eight lanes over the whole range; 5500 cuts: 33
// with four lanes, 44 with two, a chain of dependent loads by then.
cudaError_t launch_coo3_partition(const Coo3In &A, const Coo3In &B, int64_t total, int32_t step, int num_tiles, const Cuts2 &cuts, uint64_t *zero_block,
                                  int zero_words, cudaStream_t stream) {
    constexpr int COARSE = 32, FINE = 4;
    LaunchScope scope("coo3_partition", stream);
    auto ctas = [&](int64_t groups, int lanes) { return (unsigned)((groups * lanes + NT - 1) / NT); };
    if (num_tiles <= 4096) {
        k_coo3_partition<32><<<ctas(num_tiles + 1, 32), NT, 0, stream>>>(A, B, total, step, num_tiles, 1, 0, cuts, zero_block, zero_words);
        return cudaGetLastError();
    }
    k_coo3_partition<32><<<ctas(num_tiles / COARSE + 2, 32), NT, 0, stream>>>(A, B, total, step, num_tiles, COARSE, 0, cuts, nullptr, 0);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    return launch_overlapped(k_coo3_partition<FINE>, dim3(ctas(num_tiles + 1, FINE)), dim3(NT), 0, stream, A, B, total, step, num_tiles, 1, COARSE, cuts,
                             zero_block, zero_words);
}

int check_coo3(const nb200_coo3 *t) {
    if (!t || t->nnz < 0 || t->dims[0] < 0 || t->dims[1] < 0 || t->dims[2] < 0) return NB200_E_BADARG;
    if (t->nnz > 0 && (!t->i || !t->j || !t->k || !t->val)) return NB200_E_BADARG;
    return NB200_OK;
}

}  // namespace

// Shared by the COO3 entry points and the CSF3 add (which merges expanded coordinates).
// When `alloc` is set the four result arrays are allocated here (one cudaMallocAsync each, at
// the worst-case length nnz(A) + nnz(B)); otherwise they are the caller's, `capacity` entries.
//
// `scratch` / `ws`, when given, replace the library's pooled workspace (the caller then owns a block of
// coo3_add_scratch_bytes() bytes; result words and copies go to the pinned slots of `ws`); the CSF3 kernels use
// this to keep their own temporaries and this function's in one pool block.
// (Both sized for the smallest tile of the kernels here, an upper bound for the others.)
static_assert(WCAP - 1 <= tile_step_of(V_REDUCE), "scratch is sized for the smallest tile");
int64_t coo3_add_tiles(int64_t total_entries) { return (total_entries + (WCAP - 1) - 1) / (WCAP - 1); }

size_t coo3_add_scratch_bytes(int64_t total_entries) {
    const int64_t tiles = coo3_add_tiles(total_entries);
    Carver sizes;
    sizes.take<int32_t>((size_t)tiles + 1);
    sizes.take<int32_t>((size_t)tiles + 1);
    sizes.take<int32_t>((size_t)tiles + 1);
    sizes.take<uint64_t>(TileWords::needed((size_t)tiles) + 8);
    return sizes.used();
}

int coo3_add_run(const nb200_coo3 *a, const nb200_coo3 *b, nb200_coo3 *z, bool alloc, int64_t capacity, void *stream_v,
                 void *scratch, Workspace *ws) {
    int st;
    if ((st = check_coo3(a)) || (st = check_coo3(b))) return st;
    if (!z || a->dims[0] != b->dims[0] || a->dims[1] != b->dims[1] || a->dims[2] != b->dims[2]) return NB200_E_BADARG;
    if (!alloc && capacity < 0) return NB200_E_BADARG;
    const int bi = bits_for(a->dims[0]), bj = bits_for(a->dims[1]), bk = bits_for(a->dims[2]);
    const bool wide = bi + bj + bk > 63;  // the coordinates do not pack into one 64-bit key
    cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
    const int64_t total = (int64_t)a->nnz + b->nnz;
    const int v = tile_v(total), tile_step = wide ? WCAP - 1 : tile_step_of(v);
    const int64_t tiles64 = (total + tile_step - 1) / tile_step;
    if (tiles64 > INT32_MAX - 1) return NB200_E_OVERFLOW;
    const int num_tiles = (int)tiles64;
    for (int d = 0; d < 3; ++d) z->dims[d] = a->dims[d];
    z->nnz = 0;
    if (alloc) z->i = z->j = z->k = nullptr, z->val = nullptr;
    if (num_tiles == 0) return NB200_OK;
    if (!alloc && capacity > 0 && (!z->i || !z->j || !z->k || !z->val)) return NB200_E_BADARG;

    auto fail = [&](int code) {
        if (alloc) {
            if (z->i) cudaFreeAsync(z->i, stream);
            if (z->j) cudaFreeAsync(z->j, stream);
            if (z->k) cudaFreeAsync(z->k, stream);
            if (z->val) cudaFreeAsync(z->val, stream);
            z->i = z->j = z->k = nullptr;
            z->val = nullptr;
        }
        return code;
    };

    if (!scratch) {
        if ((st = acquire_workspace(stream, coo3_add_scratch_bytes(total), &ws))) return st;
        scratch = ws->dev;
    }
    int64_t *host_slot = ws->host;
    Carver carve(scratch);
    Cuts2 cuts;
    cuts.a = carve.take<int32_t>((size_t)num_tiles + 1);
    cuts.b = carve.take<int32_t>((size_t)num_tiles + 1);
    int32_t *tile_count = carve.take<int32_t>((size_t)num_tiles + 1);
    uint64_t *fused_block = carve.take<uint64_t>(TileWords::needed((size_t)num_tiles) + 4);
    FusedCtl *ctl = reinterpret_cast<FusedCtl *>(fused_block);
    TileWords words = TileWords::at(fused_block + 4);

    const Coo3In A{a->i, a->j, a->k, a->val, a->nnz}, B{b->i, b->j, b->k, b->val, b->nnz};
    const Packing pk{bj, bk};
    static const bool force_two_pass = [] { const char *e = std::getenv("NACHO_B200_TWO_PASS"); return e && e[0] == '1'; }();
    const bool fused = alloc || (capacity >= total && !force_two_pass);
    cudaError_t e = cudaSuccess;
    if (fused && alloc) {
        void **arrays[4] = {reinterpret_cast<void **>(&z->i), reinterpret_cast<void **>(&z->j),
                            reinterpret_cast<void **>(&z->k), reinterpret_cast<void **>(&z->val)};
        for (auto p : arrays) {
            e = cudaMallocAsync(p, 4 * (size_t)total, stream);
            if (e != cudaSuccess) return fail(note_cuda_error(e, "cudaMallocAsync"));
        }
    }
    bool tagged = fused && !wide && num_tiles > 1 && num_tiles <= RESIDENT && !profiling_apart();
    OwnWords own;
    if ((st = take_own_words(stream, num_tiles, &tagged, &own))) return fail(st);
    if (tagged) {
        cuts = Cuts2{nullptr, nullptr, tile_step, own};
        ctl = own.ctl, words = own.words;
    } else if (num_tiles == 1 && fused && !wide) {
        cuts = Cuts2{};  // one tile: no cut to search, and the tile kernel clears the control block itself
    } else {
        e = launch_coo3_partition(A, B, total, tile_step, num_tiles, cuts, fused_block, fused ? (int)TileWords::needed((size_t)num_tiles) + 4 : 4, stream);
    }
    if (e != cudaSuccess) return fail(note_cuda_error(e, "k_coo3_partition"));
    const Coo3Out Z{z->i, z->j, z->k, z->val, result_word(ws, RW_COO3)};
    // Reads the control block back (one small copy and a wait for the GPU).
    auto read_ctl = [&](FusedCtl &h) -> int {
        cudaError_t c = cudaMemcpyAsync(host_slot, ctl, sizeof(FusedCtl), cudaMemcpyDeviceToHost, stream);
        if (c == cudaSuccess) c = cudaStreamSynchronize(stream);
        if (c != cudaSuccess) return note_cuda_error(c, "read result length");
        std::memcpy(&h, host_slot, sizeof(h));
        return NB200_OK;
    };
    FusedCtl h;
    if (fused && !wide) {
        e = launch_coo3_tile<MODE_FUSED>(A, B, pk, cuts, nullptr, words, ctl, Z, num_tiles, v, stream);
        if (e != cudaSuccess && tagged) spoil_tagged(stream);
        if (e != cudaSuccess) return fail(note_cuda_error(e, "k_coo3_tile<fused>"));
        int64_t length;
        int device_status;
        if ((st = wait_result_word(Z.host, stream, &length, &device_status))) return fail(st);
        if (device_status != 0) {
            if ((st = read_ctl(h))) return fail(st);
            return fail(note_timeout(h.status.error, h.status.detail, "coo3 merge"));
        }
        if (length > INT32_MAX) return fail(NB200_E_OVERFLOW);
        z->nnz = (int32_t)length;
        return NB200_OK;
    }
    if (fused) {
        e = launch_coo3_tile_wide<MODE_FUSED>(A, B, cuts, nullptr, words.word, ctl, Z, num_tiles, stream);
        if (e != cudaSuccess) return fail(note_cuda_error(e, "k_coo3_tile_wide<fused>"));
        if ((st = read_ctl(h))) return fail(st);
        if (h.status.error != 0) return fail(note_timeout(h.status.error, h.status.detail, "coo3 merge"));
        if (h.total > INT32_MAX) return fail(NB200_E_OVERFLOW);
        z->nnz = (int32_t)h.total;
        return NB200_OK;
    }
    // count -> scan -> fill. The scan leaves the result length in the control block, whose status
    // word also collects a give-up of either tile launch (a bulk copy that did not land in time).
    e = wide ? launch_coo3_tile_wide<MODE_COUNT>(A, B, cuts, tile_count, nullptr, ctl, Coo3Out{}, num_tiles, stream)
             : launch_coo3_tile<MODE_COUNT>(A, B, pk, cuts, tile_count, TileWords{}, ctl, Coo3Out{}, num_tiles, v, stream);
    if (e != cudaSuccess) return note_cuda_error(e, "k_coo3_tile<count>");
    {
        LaunchScope scope("scan_tiles", stream);
        k_scan_tiles<<<1, 1024, 0, stream>>>(tile_count, num_tiles, reinterpret_cast<int64_t *>(&ctl->total));
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) return note_cuda_error(e, "k_scan_tiles");
    if ((st = read_ctl(h))) return st;
    if (h.status.error != 0) return note_timeout(h.status.error, h.status.detail, "coo3 merge");
    if (h.total > INT32_MAX) return NB200_E_OVERFLOW;
    z->nnz = (int32_t)h.total;
    if (h.total > capacity) return NB200_E_CAPACITY;
    e = wide ? launch_coo3_tile_wide<MODE_FILL>(A, B, cuts, tile_count, nullptr, ctl, Z, num_tiles, stream)
             : launch_coo3_tile<MODE_FILL>(A, B, pk, cuts, tile_count, TileWords{}, ctl, Z, num_tiles, v, stream);
    if (e != cudaSuccess) return note_cuda_error(e, "k_coo3_tile<fill>");
    if ((st = read_ctl(h))) return st;
    if (h.status.error != 0) return note_timeout(h.status.error, h.status.detail, "coo3 merge");
    return NB200_OK;
}

// Inner product of two COO3 tensors: sum over the coordinates both hold of a * b, written as one
// float32 to the device word `z` (the reference returns a one-element tensor: compiler.cpp:141-143,
// append-reduction src/backend/compute.cpp:498-525). The same partition and tile kernel as the add,
// in a mode that writes no tensor. Products are float32 (as the reference's), their sum is kept in
// double until the end. Extents that do not pack into 64 bits are not supported here.
// `scratch` / `ws` as for coo3_add_run.
int coo3_inner_run(const nb200_coo3 *a, const nb200_coo3 *b, float *z, void *stream_v, void *scratch, Workspace *ws) {
    int st;
    if ((st = check_coo3(a)) || (st = check_coo3(b))) return st;
    if (!z || a->dims[0] != b->dims[0] || a->dims[1] != b->dims[1] || a->dims[2] != b->dims[2]) return NB200_E_BADARG;
    const int bi = bits_for(a->dims[0]), bj = bits_for(a->dims[1]), bk = bits_for(a->dims[2]);
    if (bi + bj + bk > 63) return NB200_E_UNSUPPORTED;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
    const int64_t total = (int64_t)a->nnz + b->nnz;
    const int v = tile_v(total, V_REDUCE), tile_step = tile_step_of(v);
    const int64_t tiles64 = (total + tile_step - 1) / tile_step;
    if (tiles64 > INT32_MAX - 1) return NB200_E_OVERFLOW;
    const int num_tiles = (int)tiles64;
    if (a->nnz == 0 || b->nnz == 0) {
        NB200_CUDA(cudaMemsetAsync(z, 0, sizeof(float), stream));
        return NB200_OK;
    }
    if (!scratch) {
        if ((st = acquire_workspace(stream, coo3_add_scratch_bytes(total), &ws))) return st;
        scratch = ws->dev;
    }
    Carver carve(scratch);
    Cuts2 cuts;
    cuts.a = carve.take<int32_t>((size_t)num_tiles + 1);
    cuts.b = carve.take<int32_t>((size_t)num_tiles + 1);
    uint64_t *block = carve.take<uint64_t>(4);
    FusedCtl *ctl = reinterpret_cast<FusedCtl *>(block);
    const Coo3In A{a->i, a->j, a->k, a->val, a->nnz}, B{b->i, b->j, b->k, b->val, b->nnz};
    cudaError_t e = cudaSuccess;
    bool tagged = num_tiles > 1 && num_tiles <= RESIDENT && !profiling_apart();
    OwnWords own;
    if ((st = take_own_words(stream, num_tiles, &tagged, &own))) return st;
    if (tagged) {
        cuts = Cuts2{nullptr, nullptr, tile_step, own};
        ctl = own.ctl;
    } else if (num_tiles == 1) cuts = Cuts2{};
    else e = launch_coo3_partition(A, B, total, tile_step, num_tiles, cuts, block, 4, stream);
    if (e != cudaSuccess) return note_cuda_error(e, "k_coo3_partition");
    Coo3Out Z{};
    Z.host = result_word(ws, RW_COO3);
    Z.scalar = z;
    e = launch_coo3_tile<MODE_REDUCE>(A, B, Packing{bj, bk}, cuts, nullptr, TileWords{}, ctl, Z, num_tiles, v, stream);
    if (e != cudaSuccess && tagged) spoil_tagged(stream);
    if (e != cudaSuccess) return note_cuda_error(e, "k_coo3_tile<reduce>");
    int64_t done;
    int device_status;
    if ((st = wait_result_word(Z.host, stream, &done, &device_status))) return st;
    return device_status != 0 ? note_timeout(ERR_COPY_TIMEOUT, 0, "coo3 inner product") : NB200_OK;
}

}  // namespace nb200

using namespace nb200;

extern "C" {

int nb200_coo3d_add_f32(const nb200_coo3 *a, const nb200_coo3 *b, nb200_coo3 *z, int32_t, int32_t, void *stream) {
    return coo3_add_run(a, b, z, true, 0, stream, nullptr, nullptr);
}

int nb200_coo3d_add_f32_into(const nb200_coo3 *a, const nb200_coo3 *b, nb200_coo3 *z, int64_t capacity, void *stream) {
    return coo3_add_run(a, b, z, false, capacity, stream, nullptr, nullptr);
}

int nb200_inner_prod_coo_f32(const nb200_coo3 *a, const nb200_coo3 *b, float *z, void *stream) {
    return coo3_inner_run(a, b, z, stream, nullptr, nullptr);
}

}  // extern "C"
