// Host-side runtime pieces shared by the entry points: tensor-map encoding through the
// driver entry point (no link-time dependency on libcuda), launch-attribute helpers.
#pragma once
#include <cuda.h>
#include <atomic>
#include "common.cuh"

namespace of3 {

// Encodes a tiled bf16 tensor map. dims/strides are innermost-first; strides_bytes has
// rank-1 entries (stride of dim 1.., the innermost is dense). Returns OF3_OK or an error code.
// swizzle: 0 none, 1 (or true) 128-byte, 2 64-byte. Encoded maps are kept in a per-thread cache keyed
// by every argument, so a steady-state launch costs a lookup instead of a driver call per operand.
int make_tmap_bf16(CUtensorMap* out, const void* base, int rank, const uint64_t* dims,
                   const uint64_t* strides_bytes, const uint32_t* box, int swizzle);

// Per-kernel launch accounting. Every launch site of this library opens a LaunchScope with its
// kernel id: launches are always counted; when timing is enabled (of3_profile_enable) a CUDA event
// pair is recorded around the launch on the launching stream, and of3_profile_read sums their
// elapsed times. Ids: 0 the launches of any kind that were chained to the one ahead (count only), 1 contract, 2 trimul_in, 3 trimul_out, 4 transition, 5 triattn_proj,
// 6 triattn_core, 7 triattn_out, 8 single-track kernels, 9 pair-bias projection, 10 linear layers of the
// single track, 11 single-track attention core, 20 the shape-generic SIMT kernels, 30 / 31 peer
// barrier / pull.
constexpr int kMaxKernelIds = 32;
struct LaunchScope {
    int kid;
    cudaStream_t stream;
    void* rec;
    LaunchScope(int kernel_id, cudaStream_t st);
    ~LaunchScope();
};

// Work enqueued on `waiter` from now on starts after everything enqueued on `signaler` so far.
int stream_wait(cudaStream_t waiter, cudaStream_t signaler);

// One per call of an entry point that launches. Chained kernels load weights before umma::grid_wait(), which alone makes
// the writes of the kernel ahead visible: so the first launch of a call, behind whatever the caller enqueued (an in-place
// update of the weights, a conversion), is an ordinary one, and only launches behind a kernel of the same call are chained.
// `continues`: the caller says that the kernel ahead is that of another call and no parameter was written since.
struct CallScope {
    explicit CallScope(bool continues = false);
};
bool take_chain();   // whether this thread's next launch may be chained

// Launches a kernel that calls umma::grid_wait() before it touches anything another kernel wrote: its prologue (barrier
// set-up, tensor-memory allocation, weight loads) overlaps the end of the kernel before it in the stream, where that is one
// of the same call.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_chained(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                                  Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = take_chain() ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

// Number of SMs of the current device (cached per device).
int sm_count();

// Function attributes (e.g. the dynamic shared-memory limit) are per device: a launch site asks whether
// its kernels (identified by `key`, one per launch site, < 32) are configured on the CURRENT device and
// marks them once cudaFuncSetAttribute has succeeded there. Guarded by the runtime's mutex.
bool device_configured(int key);
void device_mark_configured(int key);

// The same for launch sites that are templates: a static object of one instantiation.
class PerDeviceOnce {
    std::atomic<unsigned long long> bits_{0};
    static int device() {
        int dev = 0;
        return cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 64 ? dev : -1;
    }

  public:
    bool done() const {
        const int d = device();
        return d >= 0 && ((bits_.load(std::memory_order_acquire) >> d) & 1ull);
    }
    void mark() {
        const int d = device();
        if (d >= 0) bits_.fetch_or(1ull << d, std::memory_order_release);
    }
};

}  // namespace of3
