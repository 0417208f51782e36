// Dense softmax attention without a mask over the whole key range: the dense-init chunk and the
// "regular" configuration.  Host side of the tensor-core kernel in dense_tc.cu.
//
// Stands in for flash_attention / attention (wan/modules/attention.py:34-187).
#include <atomic>

#include "common.cuh"
#include "profile.cuh"
#include "tc05.cuh"

namespace sfm {
int launch_dense_tc(const CUtensorMap* maps, __nv_bfloat16* out, int B, int H, int n_q, int n_kv, float scale, int* status,
                    int num_sms, cudaStream_t s);
namespace {
// Set (once, by compare-and-swap from 0) by the kernel when one of its bounded waits gives up; 0 = ok.
// One word per device, shared by every stream, never cleared by a launch: it keeps the first failure since
// the last sfm_dense_status call, which reads and clears it.
__device__ int g_dense_status;
}  // namespace

// Every check of a call, and what its launch needs; launches nothing (see prepare_monarch).
int prepare_dense(DenseCall* c, const void* q, int64_t q_batch_stride, const void* k, const void* v, int64_t kv_batch_stride,
                  void* out, int B, int H, int D, int n_q, int n_kv, float sm_scale) {
    if (!q || !k || !v || !out) return SFM_ERR_NULL_POINTER;
    if (D != kHeadDim) return SFM_ERR_UNSUPPORTED;
    if (B <= 0 || H <= 0 || n_q <= 0 || n_kv <= 0) return SFM_ERR_BAD_SHAPE;
    if (!(sm_scale > 0.f)) return SFM_ERR_BAD_SHAPE;       // the row maximum is taken before scaling
    auto mis = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) != 0; };
    if (mis(q) || mis(k) || mis(v) || mis(out) || (q_batch_stride % 8) || (kv_batch_stride % 8)) return SFM_ERR_ALIGNMENT;
    if (reinterpret_cast<uintptr_t>(out) & 31) return SFM_ERR_ALIGNMENT;       // the kernel's stores are 32 bytes wide

    static std::atomic<int*> words[64];                     // the status word's address, looked up once per device
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    int* status = dev >= 0 && dev < 64 ? words[dev].load(std::memory_order_relaxed) : nullptr;
    if (!status) {
        e = cudaGetSymbolAddress(reinterpret_cast<void**>(&status), g_dense_status);
        if (e != cudaSuccess) return (int)e;
        if (dev >= 0 && dev < 64) words[dev].store(status, std::memory_order_relaxed);
    }

    const uint64_t row = (uint64_t)kHeadDim * 2, tok = (uint64_t)H * row;
    uint64_t dq[4] = {(uint64_t)kHeadDim, (uint64_t)H, (uint64_t)n_q, (uint64_t)B};
    uint64_t sq[3] = {row, tok, (uint64_t)q_batch_stride * 2};
    uint64_t dk[4] = {(uint64_t)kHeadDim, (uint64_t)H, (uint64_t)n_kv, (uint64_t)B};
    uint64_t sk[3] = {row, tok, (uint64_t)kv_batch_stride * 2};
    uint32_t box[4] = {64, 1, 128, 1};
    int rc;
    if ((rc = make_tmap_bf16(&c->maps[0], k, 4, dk, sk, box))) return rc;
    if ((rc = make_tmap_bf16(&c->maps[1], v, 4, dk, sk, box))) return rc;
    if ((rc = make_tmap_bf16(&c->maps[2], q, 4, dq, sq, box))) return rc;
    c->out = out; c->status = status;
    c->B = B; c->H = H; c->n_q = n_q; c->n_kv = n_kv;
    c->scale = sm_scale;
    return SFM_OK;
}

int launch_dense(const DenseCall& c, cudaStream_t s) {
    return launch_dense_tc(c.maps, (__nv_bfloat16*)c.out, c.B, c.H, c.n_q, c.n_kv, c.scale, c.status, device_sms(), s);
}
}  // namespace sfm

using namespace sfm;

extern "C" int sfm_dense_fwd(const void* q, int64_t q_batch_stride, const void* k, const void* v,
                             int64_t kv_batch_stride, void* out, int B, int H, int D, int n_q, int n_kv,
                             float sm_scale, void* stream) {
    DenseCall c;
    int rc = prepare_dense(&c, q, q_batch_stride, k, v, kv_batch_stride, out, B, H, D, n_q, n_kv, sm_scale);
    return rc ? rc : launch_dense(c, (cudaStream_t)stream);
}

// Waits for `stream`, then reports (and clears) the status word of the dense-attention kernels on the
// current device: SFM_OK, or SFM_ERR_DEVICE_STATUS if a launch since the last call gave up on a bounded wait.
extern "C" int sfm_dense_status(void* stream) {
    int* status = nullptr;
    cudaError_t e = cudaGetSymbolAddress(reinterpret_cast<void**>(&status), g_dense_status);
    int st = 0;
    if (e == cudaSuccess) e = cudaMemcpyAsync(&st, status, sizeof(int), cudaMemcpyDeviceToHost, (cudaStream_t)stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize((cudaStream_t)stream);
    if (e == cudaSuccess && st != 0) e = cudaMemsetAsync(status, 0, sizeof(int), (cudaStream_t)stream);
    if (e != cudaSuccess) return (int)e;
    return st == 0 ? SFM_OK : SFM_ERR_DEVICE_STATUS;
}
