// Host side shared by the launchers: per-device facts, and the construction of TMA tensor maps (driver entry point fetched through the runtime).
#include <cudaTypedefs.h>

#include <atomic>
#include <mutex>
#include <unordered_map>

#include "common.cuh"
#include "profile.cuh"
#include "tc05.cuh"

namespace sfm {

namespace {
constexpr int kMaxDevices = 64;
}

int device_sms() {
    static std::atomic<int> sms[kMaxDevices];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 148;
    int n = sms[dev].load(std::memory_order_relaxed);
    if (n == 0) {
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) return 148;
        sms[dev].store(n, std::memory_order_relaxed);
    }
    return n;
}

int opt_in_smem(const void* kernel, int bytes) {
    static std::mutex mutex;
    static std::unordered_map<const void*, uint64_t> done;       // devices (bits) that know the kernel's size
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    const uint64_t bit = 1ull << (dev & 63);
    std::lock_guard<std::mutex> lock(mutex);
    uint64_t& mask = done[kernel];
    if (mask & bit) return 0;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) mask |= bit;
    return (int)e;
}

std::mutex& launch_mutex(const void* workspace) {
    static std::mutex mutexes[kLaunchMutexes];
    return mutexes[launch_slot(reinterpret_cast<uintptr_t>(workspace))];
}

EncodeTiledFn get_encode_tiled() {
    static EncodeTiledFn fn = nullptr;
    if (fn) return fn;
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) != cudaSuccess ||
        qres != cudaDriverEntryPointSuccess)
        return nullptr;
    fn = reinterpret_cast<EncodeTiledFn>(p);
    return fn;
}

int make_tmap_bf16(CUtensorMap* out, const void* base, int rank, const uint64_t* dims, const uint64_t* strides_bytes,
                   const uint32_t* box) {
    EncodeTiledFn enc = get_encode_tiled();
    if (!enc) return SFM_ERR_NO_DEVICE;
    cuuint64_t gdim[5], gstr[4];
    cuuint32_t bx[5], estr[5];
    for (int i = 0; i < rank; ++i) { gdim[i] = dims[i]; bx[i] = box[i]; estr[i] = 1; }
    for (int i = 0; i + 1 < rank; ++i) gstr[i] = strides_bytes[i];
    auto encode = [&] {
        return enc(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (cuuint32_t)rank, const_cast<void*>(base), gdim, gstr, bx, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    };
    CUresult r = encode();
    if (r != CUDA_SUCCESS) {
        // A driver function wants a context, and a thread has none before its first runtime call that needs one: bind the
        // current device's, then ask again.
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e == cudaSuccess) e = cudaSetDevice(dev);
        if (e != cudaSuccess) return (int)e;
        r = encode();
    }
    return r == CUDA_SUCCESS ? SFM_OK : SFM_ERR_BAD_SHAPE;
}

int make_bridge_tmap(CUtensorMap* out, const void* base, int b2, int n_keys, int groups, int box_cols, int box_keys) {
    const uint64_t row = (uint64_t)kHeadDim * 2;
    const uint64_t dims[4] = {(uint64_t)kHeadDim, (uint64_t)b2, (uint64_t)n_keys, (uint64_t)groups};
    const uint64_t str[3] = {row, b2 * row, (uint64_t)n_keys * b2 * row};
    const uint32_t box[4] = {64, (uint32_t)box_cols, (uint32_t)box_keys, 1};
    return make_tmap_bf16(out, base, 4, dims, str, box);
}

}  // namespace sfm
