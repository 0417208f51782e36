// Launch accounting and optional per-kernel timing (CUDA events on the launching stream).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>

namespace sfm {

enum KernelClass { kClsLayout = 0, kClsRStep = 1, kClsLStep = 2, kClsLIter = 3, kClsDense = 4, kClsBackward = 5, kNumClasses = 6 };

// Counts one launch of `cls`; when profiling is enabled also brackets the launch with events.
struct LaunchScope {
    LaunchScope(int cls, cudaStream_t stream);
    ~LaunchScope();
    int cls_;
    cudaStream_t stream_;
    int slot_;
};

// Host-side facts that do not change, asked of the runtime once per device: the number of SMs of the current device,
// and a kernel's opt-in to `bytes` of dynamic shared memory.
int device_sms();
int opt_in_smem(const void* kernel, int bytes);
// Held while a call's kernels are launched: they pass their results through its workspace, so the launches of two threads
// that share one (and a stream) must not mix.  A few mutexes serve all workspaces.
constexpr int kLaunchMutexes = 64;
// Which of them an address has.  Large buffers start on 2 MiB boundaries, and those of several streams or GPUs lie a multiple
// of that apart: the bits that tell them from one another, 21 and up, all have to count (multiplicative hashing, Knuth,
// vol. 3, 6.4), or threads that share nothing would wait for one another.
constexpr int launch_slot(uint64_t address) {
    const uint64_t x = address >> 8;                   // workspaces are aligned to 256 bytes
    return (int)(((x ^ (x >> 32)) * 0x9E3779B97F4A7C15ull) >> 58);
}
std::mutex& launch_mutex(const void* workspace);

// Launch as a programmatic dependent of the kernel before it in the stream: the grid may be set up while that one
// finishes, and every thread waits (pdl_wait) for its completion before it touches global memory.  Every kernel launched
// this way must wait, or the kernel after it could run ahead of the one before it.  `overlap` is for launches of a few tens
// of microseconds, which gain 3 to 5 us of them (first chunk, 12 heads: 83.4 -> 78.7 us for the call's three kernels);
// long ones gain nothing, and two launches of 0.25 ms each lost 2 %.
template <typename... Params, typename... Args>
int launch_pdl(bool overlap, void (*kernel)(Params...), dim3 grid, unsigned threads, size_t smem, cudaStream_t stream, Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = overlap ? 1 : 0;
    return (int)cudaLaunchKernelEx(&cfg, kernel, Params(args)...);
}
#ifdef __CUDACC__
// The kernel after this one may be set up from here on (once every block has got here or ended).
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// Waits until the kernel before this one has completed and its writes are visible.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
#endif

}  // namespace sfm
