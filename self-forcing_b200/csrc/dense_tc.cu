// Dense softmax attention, no mask, on the 5th-generation tensor cores (tcgen05 + TMEM), fed by TMA.
//
// A unit is 128 consecutive queries of one (batch, head); its keys and values stream from the KV cache in tiles of 128:
//   S = Q K^T,  P = exp2(scale S - m),  O += P V          one thread per query row, running max / sum in registers
// Every tile is worked on as two 64-key halves, one for each of two softmax warpgroups with an accumulator of its own
// (split-KV, lazy rescale); the epilogue warpgroup merges the two partial softmaxes, normalises and stores.  The halves rotate
// over three S / P buffers.  The queries go from shared memory to TMEM once per unit and are the S GEMMs' A operand there.
// Units are dealt round-robin, so that the CTAs running at the same time share keys in L2.
//
// Warp roles (16 warps): 0 = query and key tiles, 3 = value tiles, 1 = PV-GEMM issuer (owns the TMEM allocation), 2 =
// S-GEMM issuer (these four run as whole warps with an elected issuing lane), 4..7 / 8..11 = softmax warpgroups, 12..15 =
// epilogue warpgroup, which also moves the next unit's queries to TMEM.  They meet only through mbarriers with bounded waits;
// a timeout records a status code and the CTA unwinds.
//
// What bounds it: the tensor pipe, the exponentials and the chain of a half between them.  By the counters at 4680 queries x
// 18720 keys x 12 heads (434 us) the tensor pipe is busy 66 % of the time (1270 of 1940 cycles a tile of 128 x 128), the
// transcendental pipe, which packs P too, 67 %, shared memory 34 %, DRAM 4 %.  With the queries in shared memory an N = 64 instruction takes 48 cycles instead
// of 32 and the S GEMMs read 96 KB.  4680 queries x 18720 keys x 12 heads, in runs of 40 calls with their cache writes: 457 us
// with the queries in shared memory, four S / P buffers and the tiles dealt to the warpgroups in turn, 429 as it is; in
// long runs, under the power cap, 532 and 503.  Tried and slower: P handed over 32 keys at a time (440), tiles of 96 keys with
// four buffers (450), an issuing warp per warpgroup (457), one N = 128 S GEMM for both halves of a warpgroup (488).
//
// Arithmetic: softmax(q k^T * scale) v (wan/modules/attention.py:177-187).
#include "common.cuh"
#include "profile.cuh"
#include "tc05.cuh"

namespace sfm {

using namespace tc;

namespace {

constexpr int kKStages = 2;                // key tile ring, released as soon as the S GEMMs have read a tile
constexpr int kVStages = 3;                // value tile ring, released after the PV GEMMs
constexpr int kThreads = 512;
constexpr int kKT = 128;                   // keys per tile
constexpr int kHalf = kKT / 2;             // keys per S / P buffer
constexpr uint32_t kTmemCols = 512;
// TMEM columns: three S / P buffers, the queries (bf16 pairs), the accumulators of the two softmax warpgroups
constexpr int kSBufs = 3;
__host__ __device__ constexpr uint32_t col_s(int b) { return (uint32_t)b * kHalf; }
constexpr uint32_t kColQ = kSBufs * kHalf;
__host__ __device__ constexpr uint32_t col_o(int w) { return 256u + (uint32_t)w * 128u; }
static_assert(kColQ + kHeadDim / 2 <= 256, "below the accumulators");
constexpr float kRescaleThreshold = 8.0f;  // log2 units: accumulators are rescaled only past this growth

struct DenseParams {
    __nv_bfloat16* out;        // [B, n_q, H, 128], contiguous
    int H, n_q, n_kv;
    int q_tiles;               // ceil(n_q / 128)
    int n_units;               // B * H * q_tiles
    float scale;
    int* status;
};

struct __align__(8) Barriers {
    float stats[2][2][128];                // [warpgroup][m | l][tile row]
    uint64_t q_full, q_empty;              // query tile in shared memory
    uint64_t qt_full, qt_free;             // and in TMEM
    uint64_t k_full[kKStages], k_empty[kKStages];
    uint64_t v_full[kVStages], v_empty[kVStages];
    uint64_t s_full[kSBufs], p_full[kSBufs], sp_free[kSBufs];
    uint64_t pv_done[2];                   // all PV GEMMs issued so far into accumulator w have completed
    uint64_t o_full, o_free;
    uint32_t tmem_base;
    volatile int abort_flag;
};

constexpr int kTileBytes = 2 * kKT * 128;  // a query, key or value tile: two 64-column halves of 128 rows
constexpr int kSmemBytes = 1024 + (1 + kKStages + kVStages) * kTileBytes + (int)sizeof(Barriers) + 64;

__device__ __forceinline__ void st_global_v8(void* ptr, const uint32_t (&w)[8]) {
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(ptr), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]),
                 "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]) : "memory");
}

// tk, tv, tq: K / V cache and query maps, 4-D (channel, head, token, batch), box 64 x 1 x 128 x 1.
__global__ void __launch_bounds__(kThreads, 1)
dense_tc_kernel(const __grid_constant__ CUtensorMap tk, const __grid_constant__ CUtensorMap tv,
                const __grid_constant__ CUtensorMap tq, DenseParams p) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char* q_s = base;
    unsigned char* k_s = q_s + kTileBytes;
    unsigned char* v_s = k_s + kKStages * kTileBytes;
    Barriers* bars = reinterpret_cast<Barriers*>(v_s + kVStages * kTileBytes);

    const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
    const int n_tiles = (p.n_kv + kKT - 1) / kKT;
    const int u_first = blockIdx.x, u_step = gridDim.x;

    if (warp == 2 && lane == 0) { prefetch_tmap(&tq); prefetch_tmap(&tk); prefetch_tmap(&tv); }
    if (tid == 0) {
        mbar_init(&bars->q_full, 1); mbar_init(&bars->q_empty, 128); mbar_init(&bars->qt_full, 128); mbar_init(&bars->qt_free, 1);
        for (int s = 0; s < kKStages; ++s) { mbar_init(&bars->k_full[s], 1); mbar_init(&bars->k_empty[s], 1); }
        for (int s = 0; s < kVStages; ++s) { mbar_init(&bars->v_full[s], 1); mbar_init(&bars->v_empty[s], 1); }
        for (int s = 0; s < kSBufs; ++s) { mbar_init(&bars->s_full[s], 1); mbar_init(&bars->p_full[s], 128); mbar_init(&bars->sp_free[s], 1); }
        mbar_init(&bars->pv_done[0], 1); mbar_init(&bars->pv_done[1], 1);
        mbar_init(&bars->o_full, 1); mbar_init(&bars->o_free, 128);
        bars->abort_flag = 0;
        mbar_init_fence();
    }
    if (warp == 1) { tmem_alloc(&bars->tmem_base, kTmemCols); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = bars->tmem_base;
    pdl_trigger();
    pdl_wait();

    auto fail = [&](int code) {
        bars->abort_flag = 1;
        atomicCAS(p.status, 0, code);
    };
    // every role counts the key tiles or halves it has gone through: ring slots and phases follow from it

    if (warp == 0) {
        // ------------------------------------------------------------------ query and key tiles
        const uint32_t el = elect_one();
        int gk = 0, uc = 0;
        bool ok = true;
        for (int u = u_first; ok && u < p.n_units; u += u_step, ++uc) {
            const int qt = u % p.q_tiles, bh = u / p.q_tiles, b = bh / p.H, hd = bh - b * p.H;
            if (uc > 0 && !mbar_wait_u(&bars->q_empty, (uc - 1) & 1)) { fail(10); break; }
            mbar_arrive_expect_tx_e(el, &bars->q_full, (uint32_t)kTileBytes);
            tma_load_4d_e(el, q_s, &tq, &bars->q_full, 0, hd, qt * 128, b);
            tma_load_4d_e(el, q_s + 128 * 128, &tq, &bars->q_full, 64, hd, qt * 128, b);
            for (int t = 0; t < n_tiles; ++t, ++gk) {
                const int s = gk % kKStages;
                if (gk >= kKStages && !mbar_wait_u(&bars->k_empty[s], ((gk / kKStages) - 1) & 1)) { fail(11); ok = false; break; }
                unsigned char* d = k_s + s * kTileBytes;
                mbar_arrive_expect_tx_e(el, &bars->k_full[s], (uint32_t)kTileBytes);
                tma_load_4d_e(el, d, &tk, &bars->k_full[s], 0, hd, t * kKT, b);
                tma_load_4d_e(el, d + kKT * 128, &tk, &bars->k_full[s], 64, hd, t * kKT, b);
            }
        }
    } else if (warp == 3) {
        // ------------------------------------------------------------------ value tiles
        const uint32_t el = elect_one();
        int gv = 0;
        bool ok = true;
        for (int u = u_first; ok && u < p.n_units; u += u_step) {
            const int bh = u / p.q_tiles, b = bh / p.H, hd = bh - b * p.H;
            for (int t = 0; t < n_tiles; ++t, ++gv) {
                const int s = gv % kVStages;
                if (gv >= kVStages && !mbar_wait_u(&bars->v_empty[s], ((gv / kVStages) - 1) & 1)) { fail(12); ok = false; break; }
                unsigned char* d = v_s + s * kTileBytes;
                mbar_arrive_expect_tx_e(el, &bars->v_full[s], (uint32_t)kTileBytes);
                tma_load_4d_e(el, d, &tv, &bars->v_full[s], 0, hd, t * kKT, b);
                tma_load_4d_e(el, d + kKT * 128, &tv, &bars->v_full[s], 64, hd, t * kKT, b);
            }
        }
    } else if (warp == 2) {
        // ------------------------------------------------------------------ S-GEMM issuer
        const uint32_t el = elect_one();
        constexpr uint32_t idesc_s = idesc_bf16(128, kHalf, 0, 0);
        const uint64_t k_desc0 = smem_desc_sw128(smem_addr(k_s), 16, 1024);
        int gk = 0, uc = 0, sb = 0, sp = 1;                        // sb, sp: S / P buffer and its phase
        bool ok = true;
        for (int u = u_first; ok && u < p.n_units; u += u_step, ++uc) {
            if (!mbar_wait_u(&bars->qt_full, uc & 1)) { fail(20); break; }
            for (int t = 0; ok && t < n_tiles; ++t, ++gk) {
                const int s = gk % kKStages;
                if (!mbar_wait_u(&bars->k_full[s], (gk / kKStages) & 1)) { fail(21); ok = false; break; }
                const uint64_t kd = k_desc0 + (uint64_t)((s * kTileBytes) >> 4);
                for (int hh = 0; hh < 2; ++hh) {                   // keys [64 hh, 64 hh + 64) of the tile
                    if (!mbar_wait_u(&bars->sp_free[sb], sp)) { fail(25); ok = false; break; }
                    tc_fence_after();
#pragma unroll
                    for (int ks = 0; ks < 8; ++ks) {
                        const uint32_t off = ((ks >> 2) * (128 * 128) + (ks & 3) * 32) >> 4;
                        mma_ts_e(el, tmem + col_s(sb), tmem + kColQ + ks * 8, kd + off + (uint32_t)((hh * kHalf * 128) >> 4), idesc_s, ks > 0);
                    }
                    mma_commit_e(el, &bars->s_full[sb]);
                    if (++sb == kSBufs) { sb = 0; sp ^= 1; }
                }
                mma_commit_e(el, &bars->k_empty[s]);
                if (t + 1 == n_tiles) mma_commit_e(el, &bars->qt_free);
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ PV-GEMM issuer
        const uint32_t el = elect_one();
        constexpr uint32_t idesc_o = idesc_bf16(128, kHeadDim, 0, 1);
        const uint64_t v_desc0 = smem_desc_sw128(smem_addr(v_s), kKT * 128, 1024);
        int gv = 0, uc = 0, sb = 0, sp = 0;
        bool ok = true;
        for (int u = u_first; ok && u < p.n_units; u += u_step, ++uc) {
            for (int t = 0; ok && t < n_tiles; ++t, ++gv) {
                const int s = gv % kVStages;
                // the unit's first GEMM into an accumulator overwrites it: the previous unit's result must have been read
                if (t == 0 && uc > 0 && !mbar_wait_u(&bars->o_free, (uc - 1) & 1)) { fail(23); ok = false; break; }
                if (!mbar_wait_u(&bars->v_full[s], (gv / kVStages) & 1)) { fail(26); ok = false; break; }
                const uint64_t vd = v_desc0 + (uint64_t)((s * kTileBytes) >> 4);
                for (int hh = 0; hh < 2; ++hh) {
                    if (!mbar_wait_u(&bars->p_full[sb], sp)) { fail(22); ok = false; break; }
                    tc_fence_after();
#pragma unroll
                    for (int kk = 0; kk < kHalf / 16; ++kk)
                        mma_ts_e(el, tmem + col_o(hh), tmem + col_s(sb) + kk * 8,
                                 vd + (((hh * (kHalf / 16) + kk) * 2048) >> 4), idesc_o, (t > 0) || (kk > 0));
                    mma_commit_e(el, &bars->pv_done[hh]);
                    mma_commit_e(el, &bars->sp_free[sb]);
                    if (++sb == kSBufs) { sb = 0; sp ^= 1; }
                }
                mma_commit_e(el, &bars->v_empty[s]);
                if (t + 1 == n_tiles) mma_commit_e(el, &bars->o_full);
            }
        }
    } else if (warp >= 4 && warp < 12) {
        // ------------------------------------------------------------------ softmax warpgroups
        const int w = (warp - 4) >> 2;
        const int quad = warp & 3;
        const int row = quad * 32 + lane;
        const uint32_t lane_sel = (uint32_t)(quad * 32) << 16;
        const uint32_t o_t = tmem + lane_sel + col_o(w);
        const float scale_l2 = p.scale * kLog2e;
        const uint64_t scale2 = f2_pack(scale_l2, scale_l2);
        int uc = 0, idx = 0;                  // idx: halves this warpgroup has handled so far
        int sb = w, sp = 0;                   // its next S / P buffer and that one's phase
        bool ok = true;
        for (int u = u_first; ok && u < p.n_units && !bars->abort_flag; u += u_step, ++uc) {
            float m_run = -INFINITY, l_run = 0.f;
            for (int t = 0; ok && t < n_tiles; ++t, ++idx) {
                const uint32_t s_t = tmem + lane_sel + col_s(sb);
                const int valid = p.n_kv - t * kKT - w * kHalf;            // keys of this half that exist (more than 64: all)
                const bool first = t == 0, tail = valid < kHalf;
                if (!mbar_wait(&bars->s_full[sb], sp)) { fail(31); ok = false; break; }
                tc_fence_after();
                float lsum = 0.f;
                bool done = false;
                // After a unit's first half the row maximum rarely moves past the rescale threshold, so a half is first
                // taken in ONE pass against the running reference; the packed P is only stored if every row of the
                // warp stayed below 2^threshold in total (no weight exceeded it then), else the two passes below run on
                // the untouched S.
                if (!first && !tail) {
                    const uint64_t nm2 = f2_pack(-m_run, -m_run);
                    uint64_t ls2 = f2_pack(0.f, 0.f);
                    uint32_t pk0[16], pk1[16];
                    uint32_t r[64];
                    tmem_ld64(s_t, r);
                    tmem_wait_ld();
#pragma unroll
                    for (int c = 0; c < 64; c += 2) {
                        float d0, d1;
                        f2_unpack(f2_fma(f2_pack(__uint_as_float(r[c]), __uint_as_float(r[c + 1])), scale2, nm2), d0, d1);
                        const float e0 = exp2f(d0), e1 = exp2f(d1);
                        ls2 = f2_add(ls2, f2_pack(e0, e1));
                        (c < 32 ? pk0[(c >> 1) & 15] : pk1[(c >> 1) & 15]) = pack_bf16(e0, e1);
                    }
                    float la, lb;
                    f2_unpack(ls2, la, lb);
                    lsum = la + lb;
                    done = !__any_sync(0xffffffffu, !(lsum < 256.0f));   // 2^kRescaleThreshold; also catches inf / nan
                    if (done) {
                        tmem_st16(s_t, pk0);
                        tmem_st16(s_t + 16, pk1);
                    }
                }
                if (!done) {
                    float mx = -INFINITY;
#pragma unroll 1
                    for (int c0 = 0; c0 < kHalf; c0 += 32) {
                        uint32_t r[32];
                        tmem_ld32(s_t + c0, r);
                        tmem_wait_ld();
#pragma unroll
                        for (int c = 0; c < 32; ++c)                     // keys past the end of the cache view do not count
                            mx = fmaxf(mx, c0 + c < valid ? __uint_as_float(r[c]) : -INFINITY);
                    }
                    mx *= scale_l2;
                    // lazy rescale: keep the old reference while the maximum grew by less than the threshold
                    bool rescale = false;
                    float corr = 1.0f;
                    if (first) {
                        m_run = mx;
                    } else if (mx > m_run + kRescaleThreshold) {
                        corr = exp2f(m_run - mx);
                        m_run = mx;
                        l_run *= corr;
                        rescale = true;
                    }
                    if (__any_sync(0xffffffffu, rescale)) {
                        // the accumulator may only be touched once the previous GEMMs into it have finished
                        if (!mbar_wait(&bars->pv_done[w], (idx - 1) & 1)) { fail(32); ok = false; break; }
                        tc_fence_after();
#pragma unroll 1
                        for (int c0 = 0; c0 < kHeadDim; c0 += 32) {
                            uint32_t r[32];
                            tmem_ld32(o_t + c0, r);
                            tmem_wait_ld();
#pragma unroll
                            for (int c = 0; c < 32; ++c) r[c] = __float_as_uint(__uint_as_float(r[c]) * corr);
                            tmem_st32(o_t + c0, r);
                        }
                        tmem_wait_st();
                    }
                    const float neg_m = (m_run == -INFINITY) ? 0.f : -m_run;
                    const uint64_t nm2 = f2_pack(neg_m, neg_m);
                    lsum = 0.f;
#pragma unroll 1
                    for (int c0 = 0; c0 < kHalf; c0 += 32) {             // P over the S columns already consumed
                        uint32_t r[32], pk[16];
                        tmem_ld32(s_t + c0, r);
                        tmem_wait_ld();
#pragma unroll
                        for (int c = 0; c < 32; c += 2) {
                            float d0, d1;
                            f2_unpack(f2_fma(f2_pack(__uint_as_float(r[c]), __uint_as_float(r[c + 1])), scale2, nm2), d0, d1);
                            const float e0 = c0 + c < valid ? exp2f(d0) : 0.f, e1 = c0 + c + 1 < valid ? exp2f(d1) : 0.f;
                            lsum += e0 + e1;
                            pk[c >> 1] = pack_bf16(e0, e1);
                        }
                        tmem_st16(s_t + (c0 >> 1), pk);
                    }
                }
                tmem_wait_st();
                l_run += lsum;
                if (t + 1 == n_tiles) {                      // the unit's last tile: publish (m, l)
                    // the previous unit's statistics must have been consumed
                    if (uc > 0 && !mbar_wait(&bars->o_free, (uc - 1) & 1)) { fail(34); ok = false; break; }
                    bars->stats[w][0][row] = m_run;
                    bars->stats[w][1][row] = l_run;
                }
                tc_fence_before();
                mbar_arrive(&bars->p_full[sb]);
                sb += 2;                                     // every second half
                if (sb >= kSBufs) { sb -= kSBufs; sp ^= 1; }
            }
        }
    } else if (warp >= 12) {
        // ------------------------------------------------------------------ epilogue warpgroup
        const int quad = warp & 3;
        const int row = quad * 32 + lane;
        const uint32_t lane_sel = (uint32_t)(quad * 32) << 16;
        // The queries are the S GEMMs' A operand, from TMEM: a unit's go there as soon as the last S GEMM of the unit before it
        // has completed.
        auto copy_q = [&](int c) -> bool {                       // c: units before this one
            if (!mbar_wait(&bars->q_full, c & 1)) { fail(42); return false; }
            if (c > 0 && !mbar_wait(&bars->qt_free, (c - 1) & 1)) { fail(43); return false; }
            tc_fence_after();
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                uint32_t r[32];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const uint4 v = *reinterpret_cast<const uint4*>(q_s + h * (128 * 128) + row * 128 + ((i ^ (row & 7)) << 4));
                    r[4 * i] = v.x; r[4 * i + 1] = v.y; r[4 * i + 2] = v.z; r[4 * i + 3] = v.w;
                }
                tmem_st32(tmem + lane_sel + kColQ + h * 32, r);
            }
            tmem_wait_st();
            tc_fence_before();
            mbar_arrive(&bars->qt_full);
            mbar_arrive(&bars->q_empty);
            return true;
        };
        int uc = 0;
        if (u_first < p.n_units) copy_q(0);
        for (int u = u_first; u < p.n_units && !bars->abort_flag; u += u_step, ++uc) {
            if (u + u_step < p.n_units && !copy_q(uc + 1)) break;
            if (!mbar_wait(&bars->o_full, uc & 1)) { fail(41); break; }
            tc_fence_after();
            const float m0 = bars->stats[0][0][row], l0 = bars->stats[0][1][row];
            const float m1 = bars->stats[1][0][row], l1 = bars->stats[1][1][row];
            const float ms = fmaxf(m0, m1);
            const float w0 = exp2f(m0 - ms);
            const float w1 = exp2f(m1 - ms);                         // 0 where the second halves hold no key
            const float inv = 1.0f / (w0 * l0 + w1 * l1);
            const int qt = u % p.q_tiles, bh = u / p.q_tiles, b = bh / p.H, hd = bh - b * p.H;
            const long long tok = (long long)qt * 128 + row;
            const bool row_ok = tok < p.n_q;
            __nv_bfloat16* out_row = p.out + (((long long)b * p.n_q + tok) * p.H + hd) * kHeadDim;
#pragma unroll 1
            for (int c0 = 0; c0 < kHeadDim; c0 += 32) {
                uint32_t ra[32], rb[32];
                tmem_ld32(tmem + lane_sel + col_o(0) + c0, ra);
                tmem_ld32(tmem + lane_sel + col_o(1) + c0, rb);
                tmem_wait_ld();
                if (c0 + 32 == kHeadDim) {
                    tc_fence_before();
                    mbar_arrive(&bars->o_free);               // accumulators and statistics are in registers
                }
                if (row_ok) {
#pragma unroll
                    for (int v8 = 0; v8 < 2; ++v8) {
                        uint32_t wv[8];
#pragma unroll
                        for (int e = 0; e < 8; ++e) {
                            const int c = v8 * 16 + 2 * e;
                            float x0 = __uint_as_float(ra[c]) * w0, x1 = __uint_as_float(ra[c + 1]) * w0;
                            x0 = fmaf(__uint_as_float(rb[c]), w1, x0);
                            x1 = fmaf(__uint_as_float(rb[c + 1]), w1, x1);
                            wv[e] = pack_bf16(x0 * inv, x1 * inv);
                        }
                        st_global_v8(out_row + c0 + v8 * 16, wv);
                    }
                }
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, kTmemCols);
}

}  // namespace

// maps = {K, V, q}: 4-D (channel, head, token, batch), box 64 x 1 x 128 x 1.
int launch_dense_tc(const CUtensorMap* maps, __nv_bfloat16* out, int B, int H, int n_q, int n_kv, float scale, int* status,
                    int num_sms, cudaStream_t s) {
    LaunchScope scope(kClsDense, s);
    DenseParams p;
    p.out = out;
    p.H = H; p.n_q = n_q; p.n_kv = n_kv;
    p.q_tiles = (n_q + 127) / 128;
    p.n_units = B * H * p.q_tiles;
    p.scale = scale;
    p.status = status;
    dim3 grid(p.n_units < num_sms ? p.n_units : num_sms);
    if (int rc = opt_in_smem((const void*)dense_tc_kernel, kSmemBytes)) return rc;
    return launch_pdl((long long)p.n_units * n_kv <= 64ll * kKT * num_sms, dense_tc_kernel, grid, kThreads, kSmemBytes, s, maps[0], maps[1], maps[2], p);
}

}  // namespace sfm
