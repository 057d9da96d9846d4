// Shared host/device plumbing of the nacho_b200 library: status handling, the per-stream
// scratch pool, the launch counter and the optional per-kernel event timing.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "nacho_b200.h"

namespace nb200 {

// ---- status ---------------------------------------------------------------------------

// Records a failing CUDA call for nb200_last_cuda_error() and returns NB200_E_CUDA
// (NB200_E_NOMEM for allocation failures). Replaces the throwing CHECK_CUDA of
// runtime/cuda_utils/cuda_utils.h:13-20 with a status code.
int note_cuda_error(cudaError_t e, const char *what);
// Records which bounded device-side wait gave up (site code and tile of a DeviceStatus) in the
// message nb200_last_cuda_error returns; the value is NB200_E_TIMEOUT.
int note_timeout(int site, int tile, const char *where);

#define NB200_CUDA(call)                                               \
    do {                                                               \
        cudaError_t nb200_e_ = (call);                                 \
        if (nb200_e_ != cudaSuccess) return ::nb200::note_cuda_error(nb200_e_, #call); \
    } while (0)

// ---- scratch pool ---------------------------------------------------------------------

// Grow-only device scratch keyed by (device, stream). The returned block stays valid until
// the next acquire with the same key or nb200_release_workspaces(); calls on one stream are
// ordered by the stream, so reuse across calls is safe. Also carries a small pinned host
// block for result-length read-backs.
struct Workspace {
    void *dev = nullptr;
    size_t dev_bytes = 0;
    int64_t *host = nullptr;  // pinned, device-visible: 32 int64 slots for copies, then 32 result words that kernels write
    uint64_t generation = 0;  // bumped by every acquire: a holder can tell whether the block was handed out again
    uint32_t tag = 0;         // acquire_tagged: the last tag or piece handed out, 0 while the block has to be cleared first
};

// `slot` selects one of several independent blocks per (device, stream): a driver that keeps an
// intermediate alive across calls into other drivers takes slot 1 for it.
int acquire_workspace(cudaStream_t stream, size_t bytes, Workspace **out, int slot = 0);

// Words that are written with a tag, 1 .. 2^28 - 1, which rises with every call: what an earlier call left there has a lower one, so nothing is
// cleared between calls. The tag is part of a launch, so what is launched again without this call (a captured graph) must not use them. They
// lie in a block of their own per (device, stream), which a later call may replace by a larger one. `mine`: eight zeroed words in a
// block that stays, one of eight such pieces in turn; the launch has to clear `later`, which is handed out four calls on.
struct Tagged {
    uint64_t *words, *mine, *later;
    uint32_t tag;
};
constexpr int TAGGED_SLOT = 6, RING_SLOT = 7;
int acquire_tagged(cudaStream_t stream, size_t words, Tagged *out);
// A launch that was given a piece did not run, or ended with an error: all pieces are cleared before one is used again. (wait_result_word
// says so itself where it fails or the word reports an error.)
void spoil_tagged(cudaStream_t stream);

// Gives the device memory of one block back once the work queued on `stream` is done with it. Returns whether there was any.
bool drop_workspace(cudaStream_t stream, int slot);

// Counts the calls of nb200_release_workspaces(): a Workspace pointer obtained under an earlier
// value is dangling.
uint64_t workspace_epoch();

// ---- result words ---------------------------------------------------------------------

// How an operator learns a result length without a copy queued behind its kernels: the last tile
// stores one 8-byte word {valid, status, value} straight into pinned host memory and the host polls
// it. A copy plus a stream synchronisation costs 10 us more on a call that computes for 6.
// The value is complete when the word arrives; the arrays it describes are complete in stream order.
constexpr unsigned long long RW_VALID = 1ull << 63;
constexpr int RW_STATUS_SHIFT = 56;
constexpr unsigned long long RW_VALUE_MASK = (1ull << RW_STATUS_SHIFT) - 1;
constexpr int RW_SLOTS = 32;

// Clears result word `k` (0 .. RW_SLOTS - 1) of a workspace; to be called before the launch that writes it.
inline unsigned long long *result_word(Workspace *ws, int k) {
    volatile unsigned long long *w = reinterpret_cast<volatile unsigned long long *>(ws->host) + 32 + k;
    *w = 0;
    return const_cast<unsigned long long *>(w);
}

// Polls a result word until a kernel of `stream` has written it. Returns NB200_OK with the value and
// the kernel's status, or an error if the stream failed or ran dry without writing the word.
int wait_result_word(const unsigned long long *word, cudaStream_t stream, int64_t *value, int *device_status);

// Carves 256-byte-aligned sub-blocks out of a Workspace.
class Carver {
public:
    explicit Carver(void *base) : p_(reinterpret_cast<uintptr_t>(base)), used_(0) {}
    Carver() : p_(0), used_(0) {}
    template <typename T>
    T *take(size_t count) {
        size_t bytes = (count * sizeof(T) + 255) & ~size_t(255);
        T *r = p_ ? reinterpret_cast<T *>(p_ + used_) : nullptr;
        used_ += bytes;
        return r;
    }
    size_t used() const { return used_; }

private:
    uintptr_t p_;
    size_t used_;
};

// ---- launches and timing --------------------------------------------------------------

// Brackets one kernel launch: counts it and, while profiling is on, records a start/stop
// event pair on `stream` under `name`.
class LaunchScope {
public:
    LaunchScope(const char *name, cudaStream_t stream);
    ~LaunchScope();

private:
    const char *name_;
    cudaStream_t stream_;
    cudaEvent_t start_;
    bool timed_;
};

// Whether launches are being timed in which the searches for the cuts are to show apart from the merge.
bool profiling_apart();

// Launches `kernel` so that its CTAs may take their places while the kernel before it on the stream still
// runs (programmatic dependent launch; that kernel says when, with trigger_dependents). A kernel that reads
// what the one before it writes calls wait_for_previous first; one that does not calls it in its last CTA
// before it ends (finish_after_previous), so that "this kernel is complete" still means that everything
// before it is.
template <typename... P, typename... A>
cudaError_t launch_overlapped(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute early{};
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &early;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// Error word shared by kernels with bounded waits: 0 = fine, otherwise a site code.
struct DeviceStatus {
    int error;
    int detail;
};

// ---- device helpers -------------------------------------------------------------------

#ifdef __CUDACC__
__device__ __forceinline__ int lane_id() { return threadIdx.x & 31; }
__device__ __forceinline__ int warp_id() { return threadIdx.x >> 5; }

// The two sides of launch_overlapped; both do nothing where a kernel was launched without it.
__device__ __forceinline__ void trigger_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void finish_after_previous() {
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) wait_for_previous();
}

// Publishes a result word (see above). The store is a single 8-byte one, so it needs no fence.
__device__ __forceinline__ void publish_result_word(unsigned long long *word, int status, long long value) {
    if (word) *reinterpret_cast<volatile unsigned long long *>(word) = RW_VALID | ((unsigned long long)status << RW_STATUS_SHIFT) |
                                                                       ((unsigned long long)value & RW_VALUE_MASK);
}

// For memory that nothing writes while the kernel runs: from the moment it could start, that is, which for a kernel
// of launch_overlapped lies before the end of the kernel in front of it.
template <typename T>
__device__ __forceinline__ T ld_nc(const T *p) {
    return __ldg(p);
}

// For what a kernel of launch_overlapped reads of the work in front of it, operands that an earlier call may still be
// writing among it: a plain load, which the compiler keeps behind wait_for_previous. (ld_nc tells it that the memory never
// changes, and it may then ask for it before the wait; so does a const __restrict__ parameter.)
template <typename T>
__device__ __forceinline__ T ld_late(const T *p) {
    return *p;
}
#endif

}  // namespace nb200
