// Layout maps, rotary table and the fused RoPE + layout + in-place KV-cache write kernel.
#include <math.h>

#include "common.cuh"
#include "profile.cuh"

namespace sfm {

// An item is one token of one of the tensors k, v and q (grid y; grid z = batch): all heads x 16 vectors of 16 bytes (8 bf16 = 4 rotary pairs),
// moved by W warps (W = 1, 2 or 4, a launch constant).  A lane's vectors lie 32 * W apart, so they all carry the same four
// rotary pairs: the token's position arithmetic and its (cos, sin) pairs cost each lane one 32-byte read, and the row stays
// in registers between the sum of squares and the rotation (at most kMaxVec vectors per lane: 12 heads on one warp, 48
// on four; wider tokens take the looping form, which reads them twice).  The kernel is HBM bound: it reads 3 tensors and
// writes 3 (2 when q is absent); beside that, its instructions count: with 64-bit index divisions and separately rounded
// conversions the 4680 tokens of a 12-head chunk, normalised and rotated, took 26 us (0.63 of the issue slots busy),
// now 21 (cold caches, 86 MB moved).  One warp per tensor row instead of one CTA per token keeps 24 warps per SM
// resident, each with its whole row in flight, and lets the eviction's chains of k and v run beside each other.
//
// Sources may be sharded by token over up to kMaxPeers GPUs of one box (head-sharded attention): token n
// then lives in buffer n / src_tokens, a [B, src_tokens, src_heads, 128] tensor of which this GPU takes
// heads [head0, head0 + H).  Buffers of other GPUs are read with plain loads over NVLink.  Unsharded
// input is the case of one buffer with src_tokens = n_new, src_heads = H, head0 = 0.
//
// Sliding-window eviction (causal_model.py:912-926) can ride along: before the new tokens land, the cached
// tokens after the sink move left by `roll_shift` positions, cache[p] = cache[p + roll_shift] for
// roll_dst <= p < start_idx, and the new tokens follow them at start_idx.  The move overlaps itself, but it
// splits into independent chains p, p + shift, p + 2 shift, ... one per residue of p; the chain that ends at
// position start_idx + m is walked, front to back, by the CTA that afterwards writes the new token of slot
// m < shift there (every element is read before the same thread overwrites it), so the whole eviction needs
// no temporary and no ordering between CTAs.
struct PeerSrc {
    const uint4* q[kMaxPeers];
    const uint4* k[kMaxPeers];
    const uint4* v[kMaxPeers];
};

constexpr int kLayoutThreads = 128;
constexpr int kMaxVec = 6;                 // vectors per lane and tensor held in registers

__device__ __forceinline__ __nv_bfloat162 as_bf162(uint32_t w) { return *reinterpret_cast<const __nv_bfloat162*>(&w); }
__device__ __forceinline__ uint32_t as_u32(__nv_bfloat162 v) { return *reinterpret_cast<const uint32_t*>(&v); }
__device__ __forceinline__ float lo_f(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float hi_f(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }

__device__ __forceinline__ float sum_squares(const uint4& v, float acc) {
    const uint32_t* w = reinterpret_cast<const uint32_t*>(&v);
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        const float a = lo_f(w[p]), c = hi_f(w[p]);
        acc = fmaf(a, a, fmaf(c, c, acc));
    }
    return acc;
}
// y = bf16(bf16(x * rs) * weight): the two roundings of the reference (the bf16 product rounds the exact one, once)
__device__ __forceinline__ void norm_vec(uint4& v, const uint4& weight, float rs) {
    uint32_t* w = reinterpret_cast<uint32_t*>(&v);
    const uint32_t* g = reinterpret_cast<const uint32_t*>(&weight);
#pragma unroll
    for (int p = 0; p < 4; ++p)
        w[p] = as_u32(__hmul2(__floats2bfloat162_rn(lo_f(w[p]) * rs, hi_f(w[p]) * rs), as_bf162(g[p])));
}
__device__ __forceinline__ void rotate_vec(uint4& v, const float2 (&cs)[4]) {
    uint32_t* w = reinterpret_cast<uint32_t*>(&v);
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        const float re = lo_f(w[p]), im = hi_f(w[p]);
        w[p] = pack_bf16(re * cs[p].x - im * cs[p].y, re * cs[p].y + im * cs[p].x);
    }
}

// kWarps warps per item.  kRegs: the item's vectors stay in registers between the two passes.
template <int kWarps, bool kRegs>
__global__ void __launch_bounds__(kLayoutThreads, 6)
rope_cache_write_kernel(const __grid_constant__ PeerSrc src, int src_tokens, int src_heads, int head0,
                        uint4* __restrict__ q_out, uint4* k_cache, uint4* v_cache,
                        long long cache_batch_stride_vec, const float2* __restrict__ rope,
                        int B, int n_new, int H, int start_idx, Blocking blk, int start_frame,
                        int monarch_order, int p0, int p1,
                        const __nv_bfloat16* __restrict__ wq, const __nv_bfloat16* __restrict__ wk, float eps,
                        int roll_dst, int roll_shift, int rope_tok0) {
    constexpr int kVecPerRow = kHeadDim / 8;  // 16
    constexpr int kLanes = 32 * kWarps;       // lanes per item
    pdl_trigger();
    pdl_wait();
    __shared__ float red_s[kLayoutThreads / 32];
    const int warp = threadIdx.x >> 5;
    const int l = threadIdx.x & (kLanes - 1);                   // lane within the item's group
    const int n_all = (int)blockIdx.x * (kLayoutThreads / kLanes) + (int)threadIdx.x / kLanes;
    const bool live = n_all < n_new;                            // groups past the end only take part in the barriers
    const int n = live ? n_all : 0, which = blockIdx.y, b = blockIdx.z;     // which = 0: k, 1: v, 2: q
    const int vecs = H * kVecPerRow;

    const int peer = src_tokens == n_new ? 0 : n / src_tokens;
    const uint4* __restrict__ x = (which == 0 ? src.k[peer] : (which == 1 ? src.v[peer] : src.q[peer])) +
                                  (((long long)b * src_tokens + (n - peer * src_tokens)) * src_heads + head0) * kVecPerRow;
    uint4 r[kMaxVec];
    if constexpr (kRegs) {
#pragma unroll
        for (int i = 0; i < kMaxVec; ++i)
            if (live && l + i * kLanes < vecs) r[i] = x[l + i * kLanes];
    }
    const bool rotate = rope && which != 1;
    float2 cs[4];
    if (rotate) {
        const int frame_tokens = blk.h * blk.w;
        const int np = n + rope_tok0;                           // position in the chunk's token grid (token slices)
        const int fr = np / frame_tokens, rem = np - fr * frame_tokens;
        const int rw = rem / blk.w, cl = rem - rw * blk.w;
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            const int m = (l & (kVecPerRow - 1)) * 4 + p;       // rotary pair within the head: the same for all of a lane's vectors
            const int pos = m < p0 ? start_frame + fr : (m < p0 + p1 ? rw : cl);
            cs[p] = rope[pos * (kHeadDim / 2) + m];
        }
    }
    const int dst_tok = start_idx + (monarch_order && which != 2 ? blk.nat2mon(n) : n);
    const long long base = (long long)b * cache_batch_stride_vec;
    uint4* const cache = which == 1 ? v_cache : k_cache;
    uint4* const dst = which == 2 ? q_out + ((long long)b * n_new + n) * vecs : cache + base + (long long)dst_tok * vecs;

    if (live && which != 2 && roll_shift > 0 && dst_tok - start_idx < roll_shift) {
        // this token's slot ends a chain of the eviction shift: walk it (same lane-to-vector mapping as the write below, so
        // the last source element is read by the lane that then overwrites it), one chain element ahead
        const long long step = (long long)roll_shift * vecs;
        const int first = roll_dst + (dst_tok - roll_dst) % roll_shift;
        if (first < dst_tok) {
            for (int t0 = l; t0 < vecs; t0 += kMaxVec * kLanes) {
                uint4 c[kMaxVec];
                uint4* d = cache + base + (long long)first * vecs + t0;
                for (int pos = first; pos < dst_tok; pos += roll_shift, d += step) {
#pragma unroll
                    for (int i = 0; i < kMaxVec; ++i)
                        if (t0 + i * kLanes < vecs) c[i] = d[step + i * kLanes];
#pragma unroll
                    for (int i = 0; i < kMaxVec; ++i)
                        if (t0 + i * kLanes < vecs) d[i * kLanes] = c[i];
                }
            }
        }
    }

    const __nv_bfloat16* const weight = which == 1 ? nullptr : (which == 0 ? wk : wq);
    float rs = 1.f;
    if (wk) {
        // RMS normalisation over the token's full width (all heads)
        float sq = 0.f;
        if constexpr (kRegs) {
#pragma unroll
            for (int i = 0; i < kMaxVec; ++i)
                if (live && l + i * kLanes < vecs) sq = sum_squares(r[i], sq);
        } else if (live && weight) {
            for (int t = l; t < vecs; t += kLanes) sq = sum_squares(x[t], sq);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
        if constexpr (kWarps > 1) {
            if ((threadIdx.x & 31) == 0) red_s[warp] = sq;
            __syncthreads();
            const int w0 = warp & ~(kWarps - 1);
            sq = 0.f;
#pragma unroll
            for (int i = 0; i < kWarps; ++i) sq += red_s[w0 + i];
        }
        rs = rsqrtf(sq / (float)(H * kHeadDim) + eps);
    }
    if (!live) return;

    auto finish = [&](int t, uint4 v) {
        if (weight) norm_vec(v, reinterpret_cast<const uint4*>(weight)[t], rs);
        if (rotate) rotate_vec(v, cs);
        dst[t] = v;
    };
    if constexpr (kRegs) {
#pragma unroll
        for (int i = 0; i < kMaxVec; ++i)
            if (l + i * kLanes < vecs) finish(l + i * kLanes, r[i]);
    } else {
        for (int t = l; t < vecs; t += kLanes) finish(t, x[t]);
    }
}

}  // namespace sfm

using namespace sfm;

extern "C" int sfm_build_maps(int32_t* nat2mon, int32_t* mon2nat, int n_tokens, int f_tied, int h_reduce,
                              int w_reduce, int h, int w) {
    Blocking blk;
    int rc = make_blocking(&blk, f_tied, h_reduce, w_reduce, h, w);
    if (rc) return rc;
    if (n_tokens <= 0 || n_tokens % blk.tied_tokens) return SFM_ERR_BAD_SHAPE;
    for (int n = 0; n < n_tokens; ++n) {
        int m = blk.nat2mon(n);
        if (nat2mon) nat2mon[n] = m;
        if (mon2nat) mon2nat[m] = n;
    }
    return SFM_OK;
}

extern "C" int sfm_rope_table(float* out, int head_dim, int max_len, double theta) {
    if (!out) return SFM_ERR_NULL_POINTER;
    if (head_dim <= 0 || head_dim % 2 || max_len <= 0) return SFM_ERR_BAD_SHAPE;
    int c = head_dim / 2;
    int split[3] = {c - 2 * (c / 3), c / 3, c / 3};
    for (int pos = 0; pos < max_len; ++pos) {
        int m = 0;
        for (int ax = 0; ax < 3; ++ax) {
            for (int mm = 0; mm < split[ax]; ++mm, ++m) {
                double inv = 1.0 / pow(theta, (double)(2 * mm) / (double)(2 * split[ax]));
                double ang = (double)pos * inv;
                out[((size_t)pos * c + m) * 2 + 0] = (float)cos(ang);
                out[((size_t)pos * c + m) * 2 + 1] = (float)sin(ang);
            }
        }
    }
    return SFM_OK;
}

namespace {
int rope_cache_write_impl(const PeerSrc& src, bool have_q, int src_tokens, int src_heads, int head0, void* q_out,
                          void* k_cache, void* v_cache, int64_t cache_batch_stride, const float* rope, int B, int n_new,
                          int H, int D, int start_idx, int f_tied, int h_reduce, int w_reduce, int h, int w,
                          int start_frame, int monarch_order, void* stream, const void* wq = nullptr,
                          const void* wk = nullptr, float eps = 0.f, int roll_dst = 0, int roll_shift = 0,
                          int rope_tok0 = -1) {
    if (!k_cache || !v_cache) return SFM_ERR_NULL_POINTER;
    if ((reinterpret_cast<uintptr_t>(wq) | reinterpret_cast<uintptr_t>(wk)) & 15) return SFM_ERR_ALIGNMENT;
    if (have_q && !q_out) return SFM_ERR_NULL_POINTER;
    if (D != kHeadDim) return SFM_ERR_UNSUPPORTED;
    Blocking blk;
    int rc = make_blocking(&blk, f_tied, h_reduce, w_reduce, h, w);
    if (rc) return rc;
    if (B <= 0 || H <= 0 || n_new <= 0 || start_idx < 0) return SFM_ERR_BAD_SHAPE;
    if (monarch_order && n_new % blk.tied_tokens) return SFM_ERR_BAD_SHAPE;
    if (rope) {
        // whole frames, unless the caller rotates a token slice of a chunk (rope_tok0 >= 0: its first token's
        // index in the chunk's grid)
        if (rope_tok0 < 0 && n_new % (h * w)) return SFM_ERR_BAD_SHAPE;
        const int last_frame = start_frame + ((rope_tok0 < 0 ? 0 : rope_tok0) + n_new - 1) / (h * w);
        if (start_frame < 0 || last_frame >= 1024 || h > 1024 || w > 1024) return SFM_ERR_BAD_SHAPE;
    }
    auto mis = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) != 0; };
    if (mis(q_out) || mis(k_cache) || mis(v_cache) || (cache_batch_stride % 8)) return SFM_ERR_ALIGNMENT;
    if (cache_batch_stride < (int64_t)(start_idx + n_new) * H * D && B > 1) return SFM_ERR_BAD_SHAPE;
    // eviction shift: the moved tokens end where the new ones start, and every chain ends in a new token's slot
    if (roll_shift < 0 || (roll_shift > 0 && (roll_dst > start_idx || roll_shift > n_new))) return SFM_ERR_BAD_SHAPE;
    int c = D / 2;
    int p0 = c - 2 * (c / 3), p1 = c / 3;
    // the narrowest group of warps whose lanes hold a token's row in registers; wider tokens are walked by four warps
    const int vecs = H * (D / 8);
    const int warps = vecs <= 32 * kMaxVec ? 1 : (vecs <= 64 * kMaxVec ? 2 : 4);
    const bool in_regs = vecs <= 32 * warps * kMaxVec;
    const int per_cta = kLayoutThreads / 32 / warps, tensors = have_q ? 3 : 2;
    const dim3 grid((n_new + per_cta - 1) / per_cta, tensors, B);
    if (B > 65535) return SFM_ERR_BAD_SHAPE;
    LaunchScope scope(kClsLayout, (cudaStream_t)stream);
    auto go = [&](auto kernel) {
        return launch_pdl(true, kernel, grid, kLayoutThreads, 0, (cudaStream_t)stream, src, src_tokens, src_heads, head0,
                          (uint4*)q_out, (uint4*)k_cache, (uint4*)v_cache, cache_batch_stride / 8, (const float2*)rope, B, n_new,
                          H, start_idx, blk, start_frame, monarch_order, p0, p1, (const __nv_bfloat16*)wq,
                          (const __nv_bfloat16*)wk, eps, roll_dst, roll_shift, rope_tok0 < 0 ? 0 : rope_tok0);
    };
    if (!in_regs) return go(rope_cache_write_kernel<4, false>);
    if (warps == 1) return go(rope_cache_write_kernel<1, true>);
    if (warps == 2) return go(rope_cache_write_kernel<2, true>);
    return go(rope_cache_write_kernel<4, true>);
}
}  // namespace

extern "C" int sfm_rope_cache_write(const void* q, const void* k, const void* v, void* q_out, void* k_cache,
                                    void* v_cache, int64_t cache_batch_stride, const float* rope, int B,
                                    int n_new, int H, int D, int start_idx, int f_tied, int h_reduce,
                                    int w_reduce, int h, int w, int start_frame, int monarch_order,
                                    void* stream) {
    if (!k || !v) return SFM_ERR_NULL_POINTER;
    auto mis = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) != 0; };
    if (mis(q) || mis(k) || mis(v)) return SFM_ERR_ALIGNMENT;
    PeerSrc src = {};
    src.q[0] = (const uint4*)q; src.k[0] = (const uint4*)k; src.v[0] = (const uint4*)v;
    return rope_cache_write_impl(src, q != nullptr, n_new > 0 ? n_new : 1, H, 0, q_out, k_cache, v_cache,
                                 cache_batch_stride, rope, B, n_new, H, D, start_idx, f_tied, h_reduce, w_reduce, h, w,
                                 start_frame, monarch_order, stream);
}

extern "C" int sfm_norm_rope_cache_write(const void* q, const void* k, const void* v, const void* norm_q_weight,
                                         const void* norm_k_weight, float eps, void* q_out, void* k_cache,
                                         void* v_cache, int64_t cache_batch_stride, const float* rope, int B,
                                         int n_new, int H, int D, int start_idx, int f_tied, int h_reduce,
                                         int w_reduce, int h, int w, int start_frame, int monarch_order,
                                         void* stream) {
    if (!q || !k || !v || !norm_q_weight || !norm_k_weight) return SFM_ERR_NULL_POINTER;
    if (!(eps >= 0.f)) return SFM_ERR_BAD_SHAPE;
    auto mis = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) != 0; };
    if (mis(q) || mis(k) || mis(v)) return SFM_ERR_ALIGNMENT;
    PeerSrc src = {};
    src.q[0] = (const uint4*)q; src.k[0] = (const uint4*)k; src.v[0] = (const uint4*)v;
    return rope_cache_write_impl(src, true, n_new > 0 ? n_new : 1, H, 0, q_out, k_cache, v_cache, cache_batch_stride,
                                 rope, B, n_new, H, D, start_idx, f_tied, h_reduce, w_reduce, h, w, start_frame,
                                 monarch_order, stream, norm_q_weight, norm_k_weight, eps);
}

extern "C" int sfm_rope_cache_write_roll(const void* q, const void* k, const void* v, const void* norm_q_weight,
                                         const void* norm_k_weight, float eps, void* q_out, void* k_cache,
                                         void* v_cache, int64_t cache_batch_stride, const float* rope, int B,
                                         int n_new, int H, int D, int start_idx, int roll_dst, int roll_shift,
                                         int f_tied, int h_reduce, int w_reduce, int h, int w, int start_frame,
                                         int monarch_order, void* stream) {
    if (!q || !k || !v) return SFM_ERR_NULL_POINTER;
    if ((norm_q_weight == nullptr) != (norm_k_weight == nullptr)) return SFM_ERR_NULL_POINTER;
    if (!(eps >= 0.f)) return SFM_ERR_BAD_SHAPE;
    auto mis = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) != 0; };
    if (mis(q) || mis(k) || mis(v)) return SFM_ERR_ALIGNMENT;
    PeerSrc src = {};
    src.q[0] = (const uint4*)q; src.k[0] = (const uint4*)k; src.v[0] = (const uint4*)v;
    return rope_cache_write_impl(src, true, n_new > 0 ? n_new : 1, H, 0, q_out, k_cache, v_cache, cache_batch_stride,
                                 rope, B, n_new, H, D, start_idx, f_tied, h_reduce, w_reduce, h, w, start_frame,
                                 monarch_order, stream, norm_q_weight, norm_k_weight, eps, roll_dst, roll_shift);
}

extern "C" int sfm_norm_rope_token_slice(const void* q, const void* k, const void* v, const void* norm_q_weight,
                                        const void* norm_k_weight, float eps, void* q_out, void* k_out, void* v_out,
                                        const float* rope, int B, int n_tokens, int H, int D, int token0, int h, int w,
                                        int start_frame, void* stream) {
    if (!q || !k || !v || !q_out || !k_out || !v_out || !rope) return SFM_ERR_NULL_POINTER;
    if ((norm_q_weight == nullptr) != (norm_k_weight == nullptr)) return SFM_ERR_NULL_POINTER;
    if (!(eps >= 0.f) || token0 < 0) return SFM_ERR_BAD_SHAPE;
    auto mis = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) != 0; };
    if (mis(q) || mis(k) || mis(v)) return SFM_ERR_ALIGNMENT;
    PeerSrc src = {};
    src.q[0] = (const uint4*)q; src.k[0] = (const uint4*)k; src.v[0] = (const uint4*)v;
    // natural order, slot 0 of a "cache" that is just the output tensors
    return rope_cache_write_impl(src, true, n_tokens > 0 ? n_tokens : 1, H, 0, q_out, k_out, v_out,
                                 (int64_t)n_tokens * H * D, rope, B, n_tokens, H, D, 0, 1, 1, 1, h, w, start_frame, 0,
                                 stream, norm_q_weight, norm_k_weight, eps, 0, 0, token0);
}

extern "C" int sfm_rope_cache_write_gather(const void* const* q_shards, const void* const* k_shards,
                                           const void* const* v_shards, int world, int rank, void* q_out, void* k_cache,
                                           void* v_cache, int64_t cache_batch_stride, const float* rope, int B,
                                           int n_new, int H, int D, int start_idx, int f_tied, int h_reduce,
                                           int w_reduce, int h, int w, int start_frame, int monarch_order,
                                           void* stream) {
    if (!q_shards || !k_shards || !v_shards) return SFM_ERR_NULL_POINTER;
    if (world < 1 || world > kMaxPeers || rank < 0 || rank >= world) return SFM_ERR_BAD_SHAPE;
    if (n_new <= 0 || n_new % world) return SFM_ERR_BAD_SHAPE;
    PeerSrc src = {};
    for (int p = 0; p < world; ++p) {
        if (!q_shards[p] || !k_shards[p] || !v_shards[p]) return SFM_ERR_NULL_POINTER;
        if ((reinterpret_cast<uintptr_t>(q_shards[p]) | reinterpret_cast<uintptr_t>(k_shards[p]) |
             reinterpret_cast<uintptr_t>(v_shards[p])) & 15)
            return SFM_ERR_ALIGNMENT;
        src.q[p] = (const uint4*)q_shards[p]; src.k[p] = (const uint4*)k_shards[p]; src.v[p] = (const uint4*)v_shards[p];
    }
    return rope_cache_write_impl(src, true, n_new / world, H * world, rank * H, q_out, k_cache, v_cache,
                                 cache_batch_stride, rope, B, n_new, H, D, start_idx, f_tied, h_reduce, w_reduce, h, w,
                                 start_frame, monarch_order, stream);
}

namespace sfm {
// Stand-alone rotation of one tensor (same arithmetic as the fused kernel above).
__global__ void __launch_bounds__(256)
rope_apply_kernel(const uint4* __restrict__ x, uint4* __restrict__ out, const float2* __restrict__ rope, int B,
                  int L, int H, int seq, int hgrid, int wgrid, int start_frame, int p0, int p1) {
    constexpr int kVecPerRow = kHeadDim / 8;
    const long long total = (long long)B * L * H * kVecPerRow;
    const int frame_tokens = hgrid * wgrid;
    for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
         idx += (long long)gridDim.x * blockDim.x) {
        int vec = (int)(idx % kVecPerRow);
        long long row = idx / kVecPerRow;
        int n = (int)((row / H) % L);
        uint4 xv = x[idx];
        if (n < seq) {
            int fr = n / frame_tokens, rem = n - fr * frame_tokens;
            int rw = rem / wgrid, cl = rem - rw * wgrid;
            uint32_t* xw = reinterpret_cast<uint32_t*>(&xv);
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                int m = vec * 4 + p;
                int pos = m < p0 ? start_frame + fr : (m < p0 + p1 ? rw : cl);
                float2 cs = rope[pos * (kHeadDim / 2) + m];
                __nv_bfloat162 v2 = *reinterpret_cast<__nv_bfloat162*>(&xw[p]);
                float re = __low2float(v2), im = __high2float(v2);
                xw[p] = pack_bf16(re * cs.x - im * cs.y, re * cs.y + im * cs.x);
            }
        }
        out[idx] = xv;
    }
}
}  // namespace sfm

extern "C" int sfm_rope_apply(const void* x, void* out, const float* rope, int B, int L, int H, int D, int frames,
                              int h, int w, int start_frame, void* stream) {
    if (!x || !out || !rope) return SFM_ERR_NULL_POINTER;
    if (D != kHeadDim) return SFM_ERR_UNSUPPORTED;
    if (B <= 0 || L <= 0 || H <= 0 || frames <= 0 || h <= 0 || w <= 0) return SFM_ERR_BAD_SHAPE;
    if ((long long)frames * h * w > L) return SFM_ERR_BAD_SHAPE;
    if (start_frame < 0 || start_frame + frames > 1024 || h > 1024 || w > 1024) return SFM_ERR_BAD_SHAPE;
    if ((reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(out) & 15)) return SFM_ERR_ALIGNMENT;
    int c = D / 2, p0 = c - 2 * (c / 3), p1 = c / 3;
    long long total = (long long)B * L * H * (D / 8);
    long long want = (total + 255) / 256;
    int blocks = (int)(want < 148LL * 16 ? want : 148LL * 16);
    LaunchScope scope(kClsLayout, (cudaStream_t)stream);
    rope_apply_kernel<<<blocks, 256, 0, (cudaStream_t)stream>>>((const uint4*)x, (uint4*)out, (const float2*)rope, B,
                                                                 L, H, frames * h * w, h, w, start_frame, p0, p1);
    return (int)cudaGetLastError();
}
