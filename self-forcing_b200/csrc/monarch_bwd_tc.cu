// Backward of the Monarch column step on the 5th-generation tensor cores (tcgen05 + TMEM), fed by TMA.
//
// Forward column step, per slab (batch*head, query group a, column j), query row i, key n = (f, k):
//   s[i,n] = scale * q[a,i,j] . aL[n] - cL[n],   P = softmax_n s,   out[a,i,j] = sum_n P[i,n] Y[n]
// with aL[n] = sum_l R_l K_l and Y[n] = sum_l R_l V_l the row step's results (bf16, in the bridge layout
// [query group][key][column][128]).  Given dOut, lse[i] = log sum_n exp s[i,n] (from a forward column step run just before)
// and delta[i] = dOut[i] . out[i], one sweep over the slab's keys in tiles of 128 gives every gradient:
//   dP[i,n] = dOut[i] . Y[n]                      dS = P (dP - delta)
//   dY[n]  = sum_i P[i,n] dOut[i]                 daL[n] = scale * sum_i dS[i,n] q[i]        dcL[n] = -sum_i dS[i,n]
//   dq[i]  = scale * sum_n dS[i,n] aL[n]          (the row step's share of dQ is added by its own backward)
// The KEYS sit on the M side of the tensor core (TMEM lane = key), the slab's queries on the N side in chunks of
// 32 rows (NC = 1, 2 or 3 chunks: block rows up to 96), so that dY, daL and dcL come out one key per lane, ready
// for row-wise stores.  Per (key tile, chunk of query rows):
//   S^T  = aL_tile Q^T,  dP^T = Y_tile dOut^T               two tcgen05.mma, operands in shared memory
//   P^T, (scale dS)^T as bf16 over the S^T / dP^T columns     one thread per key; dcL from its registers
//   dY_tile = P^T dOut,  daL_tile = (scale dS)^T Q            A from TMEM, B = the query-side rows, MN-major
//   dq^T (+)= aL_tile^T (scale dS)^T                          A = the aL tile read MN-major, B = a bf16 copy of
//                                                             (scale dS)^T in shared memory; accumulates over the slab
// dY and daL accumulate over the chunks of a tile in TMEM, dq^T has 32 columns per chunk and accumulates over the
// tiles.  dY and daL are written over Y and aL in place (a tile is in shared memory before its rows are overwritten).
//
// Warp roles (16 warps): 0 = aL / Y tiles, 1 = MMA issuer (owns TMEM), 2 = query side, 3 idle, 4-7 and 8-11 = two warpgroups that take even
// / odd (tile, chunk) steps (element-wise pass), 12-15 = drain warpgroup: a tile's dY / daL, rounded, into the shared memory of
// its Y / aL tile, which nothing reads any more, and from there by TMA store over Y / aL; dcL; after a slab's last tile its
// dq.  The issuer takes the next step's S GEMMs before this step's gradient GEMMs only if that tile is already there: the tile
// ring has two stages, and a stage is free again when its tile's results have left it.  Persistent CTAs, one slab each a
// round.  All waits are bounded and report through the status word.
//
// What bounds it: the bridge, read and written (378 + 318 MB at 4680 queries, 18720 cached tokens, 12 heads).  With the results
// stored one 256-byte row per lane by the element-wise warpgroups, between two of their steps, and one warp loading tiles and
// query side, where a slab's log-sum-exps held up its tiles, it took 236 us, now 142 (4.9 TB/s); with the drain warpgroup alone, 205.
//
// Stands in for the Triton kernel _z_bwd and its preprocess (wan/modules/monarch_attn.py:852-886, 1034-1222).
#include <algorithm>

#include "monarch_params.cuh"
#include "profile.cuh"
#include "tc05.cuh"

namespace sfm {

using namespace tc;

namespace {

constexpr int kStgB = 2;                     // (aL, Y) tile-pair ring
constexpr int kThreadsB = 512;
constexpr int kKB = 128;                     // keys per tile
constexpr int kNI = 32;                      // query rows per chunk
constexpr int kMaxNC = 3;                    // chunks per slab: block rows up to 96
constexpr uint32_t kTmemColsB = 512;
// TMEM columns: per warpgroup S^T / P^T at w*64, dP^T / dS^T at w*64 + 32; accumulators after them
__host__ __device__ constexpr uint32_t bc_s(int w) { return (uint32_t)w * 64u; }
__host__ __device__ constexpr uint32_t bc_dp(int w) { return (uint32_t)w * 64u + 32u; }
constexpr uint32_t kColDaL = 128, kColDY = 256, kColDq = 384;

struct BwdColParams {
    const float* delta;            // [B, n_q, H]: dOut . out per token and head
    const float* lse;              // [slab][b1]
    const float* cL;               // [slab][n_keys_c]
    float* dcL;                    // [slab][n_keys_c]
    float* dq;                     // natural order [B, n_q, H, 128] fp32
    int H, n_q, A, n_keys, n_keys_c, bh0, nbh;
    int n_units;                   // nbh * A * b2
    int q_box_rows;                // rows per box of the q / dOut row maps (32, or all the grid rows there are)
    float scale;
    Blocking blk;
    int* status;
};

constexpr int kQdHalf = kNI * 128;                 // one 64-column half of a query-side tile (32 rows)
constexpr int kQdTile = 2 * kQdHalf;               // 8 KB
constexpr int kQdBuf = 2 * kQdTile;                // q rows + dOut rows of one chunk
constexpr int kBTile = 2 * kKB * 128;              // one aL or Y tile, 32 KB
constexpr int kBStage = 2 * kBTile;                // aL + Y
constexpr int kDsTile = kKB * 128;                 // (scale dS)^T copy: 128 keys x 64 bf16, 16 KB

struct __align__(16) BBarriers {
    float lse2[2][kMaxNC * kNI];
    float delta[2][kMaxNC * kNI];
    float dsum[4][kMaxNC][kKB];             // [tile & 3][chunk][key]: -dcL shares of the chunks
    uint64_t q_full[2], q_empty[2];
    uint64_t a_full[kStgB], a_empty[kStgB];
    uint64_t s_full[2], p_full[2], sd_free[2];
    uint64_t acc_full, acc_free;
    uint64_t dq_full, dq_free;
    uint32_t tmem_base;
    volatile int abort_flag;
};

// query-side buffers: two slabs of one chunk (the next slab's rows load while this one is worked on), or one slab of NC
__host__ __device__ constexpr int qd_bytes(int nc) { return (nc == 1 ? 2 : nc) * kQdBuf; }
__host__ __device__ constexpr int b_smem_bytes(int nc) {
    return 1024 + qd_bytes(nc) + kStgB * kBStage + 2 * kDsTile + (int)sizeof(BBarriers) + 64;
}

struct BUnit { int bhl, a, j; };
__device__ __forceinline__ BUnit b_decode(const BwdColParams& p, int u) {
    BUnit r;
    r.j = u % p.blk.b2; u /= p.blk.b2;
    r.a = u % p.A;
    r.bhl = u / p.A;
    return r;
}

// tal / ty = bridge maps (box 64 x 1 column x 128 keys), sal / sy the same with boxes of 32 keys; tqr / tdo = query rows of q / dOut (5-D, box of 32 rows).
template <int NC>
__global__ void __launch_bounds__(kThreadsB, 1)
monarch_bwd_col_tc_kernel(const __grid_constant__ CUtensorMap tal, const __grid_constant__ CUtensorMap ty,
                          const __grid_constant__ CUtensorMap sal, const __grid_constant__ CUtensorMap sy,
                          const __grid_constant__ CUtensorMap tqr, const __grid_constant__ CUtensorMap tdo,
                          BwdColParams p) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char* qd_s = base;                                   // [slab buffer][chunk][q rows | dOut rows]
    unsigned char* a_s = qd_s + qd_bytes(NC);                      // [stage][aL tile | Y tile]
    unsigned char* ds_s = a_s + kStgB * kBStage;                   // [warpgroup] (scale dS)^T, 128 rows of 128 bytes
    BBarriers* bars = reinterpret_cast<BBarriers*>(ds_s + 2 * kDsTile);

    const Blocking& blk = p.blk;
    const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
    const int b1 = blk.b1;
    const int n_keys = p.n_keys;
    const int n_tiles = (n_keys + kKB - 1) / kKB;
    // The grid goes through the slabs together, from the last one: neighbouring columns are neighbours in the bridge, what the
    // row step wrote last is read first, and what is written last here the row step's backward reads first
    // (all backward kernels at the size above 289 -> 282 us against a contiguous share per CTA).
    const int n_my = (p.n_units - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
    auto unit_at = [&](int uc) -> int { return p.n_units - 1 - (uc * (int)gridDim.x + (int)blockIdx.x); };
    const int total = n_my * n_tiles * NC;                         // (slab, tile, chunk) steps of this CTA
    constexpr int kQBufs = NC == 1 ? 2 : 1;

    if (tid == 0) {
        for (int s = 0; s < 2; ++s) { mbar_init(&bars->q_full[s], 1); mbar_init(&bars->q_empty[s], 1); }
        for (int s = 0; s < kStgB; ++s) { mbar_init(&bars->a_full[s], 1); mbar_init(&bars->a_empty[s], 4); }
        for (int w = 0; w < 2; ++w) {
            mbar_init(&bars->s_full[w], 1); mbar_init(&bars->p_full[w], 128); mbar_init(&bars->sd_free[w], 1);
        }
        mbar_init(&bars->acc_full, 1); mbar_init(&bars->acc_free, 128);
        mbar_init(&bars->dq_full, 1); mbar_init(&bars->dq_free, 128);
        bars->abort_flag = 0;
        mbar_init_fence();
    }
    // query-side rows no load writes, and the padding columns of the (scale dS)^T copies, must read as zero
    for (int i = tid; i < qd_bytes(NC) / 16; i += kThreadsB) reinterpret_cast<uint4*>(qd_s)[i] = make_uint4(0, 0, 0, 0);
    for (int i = tid; i < 2 * kDsTile / 16; i += kThreadsB) reinterpret_cast<uint4*>(ds_s)[i] = make_uint4(0, 0, 0, 0);
    if (warp == 1) { tmem_alloc(&bars->tmem_base, kTmemColsB); tmem_relinquish(); }
    fence_async_smem();
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

    if (warp == 0) {
        // ------------------------------------------------------------------ tile loads
        const uint32_t el = elect_one();
        prefetch_tmap(&tal); prefetch_tmap(&ty); prefetch_tmap(&sal); prefetch_tmap(&sy);
        int g = 0;                                               // tiles loaded
        bool ok = true;
        for (int uc = 0; ok && uc < n_my && !bars->abort_flag; ++uc) {
            const BUnit un = b_decode(p, unit_at(uc));
            const int grp = un.bhl * p.A + un.a;
            for (int t = 0; t < n_tiles; ++t, ++g) {
                const int s = g % kStgB;
                if (g >= kStgB && !mbar_wait_u(&bars->a_empty[s], ((g / kStgB) - 1) & 1)) { fail(11); ok = false; break; }
                unsigned char* st = a_s + s * kBStage;
                mbar_arrive_expect_tx_e(el, &bars->a_full[s], (uint32_t)kBStage);
                tma_load_4d_e(el, st, &tal, &bars->a_full[s], 0, un.j, t * kKB, grp);
                tma_load_4d_e(el, st + kKB * 128, &tal, &bars->a_full[s], 64, un.j, t * kKB, grp);
                tma_load_4d_e(el, st + kBTile, &ty, &bars->a_full[s], 0, un.j, t * kKB, grp);
                tma_load_4d_e(el, st + kBTile + kKB * 128, &ty, &bars->a_full[s], 64, un.j, t * kKB, grp);
            }
        }
    } else if (warp == 2) {
        // ------------------------------------------------------------------ query side: rows of q and dOut, lse, delta
        const uint32_t el = elect_one();
        prefetch_tmap(&tqr); prefetch_tmap(&tdo);
        for (int uc = 0; uc < n_my && !bars->abort_flag; ++uc) {
            const int u = unit_at(uc);
            const BUnit un = b_decode(p, u);
            const int bh = p.bh0 + un.bhl, b = bh / p.H, hd = bh - b * p.H;
            const int qb = kQBufs == 2 ? (uc & 1) : 0;
            unsigned char* qt = qd_s + qb * kQdBuf;
            const int tok0 = blk.row_token(un.a, 0) + un.j;      // the slab's rows are consecutive rows of the token grid
            float l2[NC], dl[NC];
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const int i = c * kNI + lane;
                l2[c] = INFINITY; dl[c] = 0.f;
                if (i < b1) {
                    l2[c] = kLog2e * p.lse[(long long)u * b1 + i];
                    dl[c] = p.delta[((long long)b * p.n_q + tok0 + i * blk.w) * p.H + hd];
                }
            }
            if (uc >= kQBufs && !mbar_wait_u(&bars->q_empty[qb], ((uc / kQBufs) - 1) & 1)) { fail(10); break; }
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                bars->lse2[qb][c * kNI + lane] = l2[c];
                bars->delta[qb][c * kNI + lane] = dl[c];
            }
            __syncwarp();
            // 32 consecutive rows of the token grid per chunk; rows past the slab's b1 hold other tokens (or the
            // fill value) and are masked by an infinite log-sum-exp
            mbar_arrive_expect_tx_e(el, &bars->q_full[qb], (uint32_t)(NC * 4 * p.q_box_rows * 128));
            const int frow0 = tok0 / blk.w, col = tok0 - frow0 * blk.w;
            for (int c = 0; c < NC; ++c) {
                unsigned char* dq_ = qt + c * kQdBuf;
                tma_load_5d_e(el, dq_, &tqr, &bars->q_full[qb], 0, hd, col, frow0 + c * kNI, b);
                tma_load_5d_e(el, dq_ + kQdHalf, &tqr, &bars->q_full[qb], 64, hd, col, frow0 + c * kNI, b);
                tma_load_5d_e(el, dq_ + kQdTile, &tdo, &bars->q_full[qb], 0, hd, col, frow0 + c * kNI, b);
                tma_load_5d_e(el, dq_ + kQdTile + kQdHalf, &tdo, &bars->q_full[qb], 64, hd, col, frow0 + c * kNI, b);
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer
        {
            const uint32_t el = elect_one();
            constexpr uint32_t idesc_s = idesc_bf16(128, kNI, 0, 0);            // S^T, dP^T
            constexpr uint32_t idesc_o = idesc_bf16(128, kHeadDim, 0, 1);       // dY, daL: A from TMEM, B MN-major
            constexpr uint32_t idesc_q = idesc_bf16(128, 64, 1, 1);             // dq^T: both operands MN-major
            const uint64_t a_k0 = smem_desc_sw128(smem_addr(a_s), 16, 1024);               // aL / Y tile, K-major
            const uint64_t a_mn0 = smem_desc_sw128(smem_addr(a_s), kKB * 128, 1024);        // aL tile, MN-major (M = d)
            const uint64_t q_k0 = smem_desc_sw128(smem_addr(qd_s), 16, 1024);              // q / dOut rows, K-major
            const uint64_t q_mn0 = smem_desc_sw128(smem_addr(qd_s), kQdHalf, 1024);         // q / dOut rows, MN-major
            const uint64_t ds0 = smem_desc_sw128(smem_addr(ds_s), 16, 1024);                // (scale dS)^T copy, MN-major, N = 64
            bool ok = true;
            // step g = ((slab, tile), chunk); its warpgroup is g & 1
            auto issue_s = [&](int g) -> bool {
                const int gt = g / NC, c = g - gt * NC;
                const int uc = gt / n_tiles, t = gt - uc * n_tiles, w = g & 1, s = gt % kStgB;
                const int qb = kQBufs == 2 ? (uc & 1) : 0;
                if (t == 0 && c == 0 && !mbar_wait_u(&bars->q_full[qb], (uc / kQBufs) & 1)) { fail(20); return false; }
                if (c == 0 && !mbar_wait_u(&bars->a_full[s], (gt / kStgB) & 1)) { fail(21); return false; }
                if (g >= 2 && !mbar_wait_u(&bars->sd_free[w], ((g >> 1) - 1) & 1)) { fail(22); return false; }
                tc_fence_after();
                const uint64_t al = a_k0 + (uint64_t)((s * kBStage) >> 4);
                const uint64_t yy = al + (uint64_t)(kBTile >> 4);
                const uint64_t qq = q_k0 + (uint64_t)(((qb + c) * kQdBuf) >> 4);
                const uint64_t dd = qq + (uint64_t)(kQdTile >> 4);
#pragma unroll
                for (int ks = 0; ks < 8; ++ks) {
                    const uint32_t ao = ((ks >> 2) * (kKB * 128) + (ks & 3) * 32) >> 4;
                    const uint32_t qo = ((ks >> 2) * kQdHalf + (ks & 3) * 32) >> 4;
                    mma_ss_e(el, tmem + bc_s(w), al + ao, qq + qo, idesc_s, ks > 0);
                }
#pragma unroll
                for (int ks = 0; ks < 8; ++ks) {
                    const uint32_t ao = ((ks >> 2) * (kKB * 128) + (ks & 3) * 32) >> 4;
                    const uint32_t qo = ((ks >> 2) * kQdHalf + (ks & 3) * 32) >> 4;
                    mma_ss_e(el, tmem + bc_dp(w), yy + ao, dd + qo, idesc_s, ks > 0);
                }
                mma_commit_e(el, &bars->s_full[w]);
                return true;
            };
            // the tile (and, at a slab's start, the query rows) of step g have arrived
            auto ready = [&](int g) -> bool {
                const int gt = g / NC, c = g - gt * NC;
                const int uc = gt / n_tiles, t = gt - uc * n_tiles, s = gt % kStgB;
                if (c != 0) return true;
                return mbar_test_u(&bars->a_full[s], (gt / kStgB) & 1) &&
                       (t != 0 || mbar_test_u(&bars->q_full[kQBufs == 2 ? (uc & 1) : 0], (uc / kQBufs) & 1));
            };
            if (total > 0) ok = issue_s(0);
            for (int g = 0; ok && g < total && !bars->abort_flag; ++g) {
                // The S GEMMs of the next step are issued ahead of this step's, except across a slab boundary when the
                // query-side rows are single buffered: the next slab's rows can only load once this slab's last
                // GEMMs have released the buffer, so waiting for them here would never end.
                // Nor when the next tile is not there yet: it may be waiting for a stage that this step's tile follows.
                const bool ahead = g + 1 < total && !(kQBufs == 1 && (g + 1) % (n_tiles * NC) == 0) && ready(g + 1);
                if (ahead && !issue_s(g + 1)) { ok = false; break; }
                const int gt = g / NC, c = g - gt * NC;
                const int uc = gt / n_tiles, t = gt - uc * n_tiles, w = g & 1, s = gt % kStgB;
                const int qb = kQBufs == 2 ? (uc & 1) : 0;
                if (!mbar_wait_u(&bars->p_full[w], (g >> 1) & 1)) { fail(23); break; }
                // the accumulators are shared by all tiles: the previous tile's must have been drained
                if (c == 0 && gt >= 1 && !mbar_wait_u(&bars->acc_free, (gt - 1) & 1)) { fail(24); break; }
                if (t == 0 && c == 0 && uc >= 1 && !mbar_wait_u(&bars->dq_free, (uc - 1) & 1)) { fail(25); break; }
                tc_fence_after();
                const uint64_t qn = q_mn0 + (uint64_t)(((qb + c) * kQdBuf) >> 4);
                const uint64_t dn = qn + (uint64_t)(kQdTile >> 4);
#pragma unroll
                for (int kk = 0; kk < kNI / 16; ++kk)          // dY_tile (+)= P^T dOut
                    mma_ts_e(el, tmem + kColDY, tmem + bc_s(w) + kk * 8, dn + ((kk * 2048) >> 4), idesc_o, (c > 0 || kk > 0) ? 1u : 0u);
#pragma unroll
                for (int kk = 0; kk < kNI / 16; ++kk)          // daL_tile (+)= (scale dS)^T Q
                    mma_ts_e(el, tmem + kColDaL, tmem + bc_dp(w) + kk * 8, qn + ((kk * 2048) >> 4), idesc_o, (c > 0 || kk > 0) ? 1u : 0u);
                const uint64_t am = a_mn0 + (uint64_t)((s * kBStage) >> 4);
                const uint64_t dsd = ds0 + (uint64_t)((w * kDsTile) >> 4);
                // dq^T of chunk c (+)= aL_tile^T (scale dS)^T: 64 output columns of which the upper 32 receive zeros
                // (and, on a slab's first tile, are set to zero before the next chunk sets its own)
#pragma unroll
                for (int kk = 0; kk < kKB / 16; ++kk)
                    mma_ss_e(el, tmem + kColDq + c * kNI, am + ((kk * 2048) >> 4), dsd + ((kk * 2048) >> 4), idesc_q, (t > 0 || kk > 0) ? 1u : 0u);
                if (c == NC - 1) mma_commit_e(el, &bars->acc_full);
                mma_commit_e(el, &bars->sd_free[w]);
                if (t + 1 == n_tiles && c == NC - 1) { mma_commit_e(el, &bars->dq_full); mma_commit_e(el, &bars->q_empty[qb]); }
                if (g + 1 < total && !ahead && !issue_s(g + 1)) { ok = false; break; }
            }
        }
    } else if (warp >= 4 && warp < 12) {
        // ------------------------------------------------------------------ the two working warpgroups
        const int w = (warp - 4) >> 2;
        const int quad = warp & 3;
        const int row = quad * 32 + lane;                       // TMEM lane: key within the tile
        const uint32_t lane_sel = (uint32_t)(quad * 32) << 16;
        const float scale_l2 = p.scale * kLog2e;
        unsigned char* ds_row = ds_s + w * kDsTile + row * 128;
        auto load_cl = [&](int g) -> float {                    // step g's bias of this thread's key
            const int gt = g / NC, uc = gt / n_tiles, key = (gt - uc * n_tiles) * kKB + row;
            return g < total && key < n_keys ? kLog2e * p.cL[(long long)unit_at(uc) * p.n_keys_c + key] : INFINITY;
        };
        float cl_next = load_cl(w);
        for (int g = w; g < total && !bars->abort_flag; g += 2) {
            const int gt = g / NC, c = g - gt * NC;
            const int uc = gt / n_tiles;
            const int qb = kQBufs == 2 ? (uc & 1) : 0;
            const float cl2 = cl_next;
            cl_next = load_cl(g + 2);
            if (!mbar_wait(&bars->s_full[w], (g >> 1) & 1)) { fail(31); break; }
            tc_fence_after();
            uint32_t rs[kNI], rd[kNI];
            tmem_ld32(tmem + lane_sel + bc_s(w), rs);
            tmem_ld32(tmem + lane_sel + bc_dp(w), rd);
            tmem_wait_ld();
            const float* lse2 = bars->lse2[qb] + c * kNI;
            const float* dlt = bars->delta[qb] + c * kNI;
            float dsum = 0.f;
            uint32_t pp[kNI / 2], pd[kNI / 2];
#pragma unroll
            for (int cc = 0; cc < kNI; cc += 2) {
                const float p0 = exp2f(fmaf(__uint_as_float(rs[cc]), scale_l2, -(cl2 + lse2[cc])));
                const float p1 = exp2f(fmaf(__uint_as_float(rs[cc + 1]), scale_l2, -(cl2 + lse2[cc + 1])));
                const float d0 = p0 * (__uint_as_float(rd[cc]) - dlt[cc]);
                const float d1 = p1 * (__uint_as_float(rd[cc + 1]) - dlt[cc + 1]);
                dsum += d0 + d1;
                pp[cc >> 1] = pack_bf16(p0, p1);
                pd[cc >> 1] = pack_bf16(d0 * p.scale, d1 * p.scale);
            }
            tmem_st16(tmem + lane_sel + bc_s(w), pp);
            tmem_st16(tmem + lane_sel + bc_dp(w), pd);
            // bf16 copy of this key's (scale dS) row for the dq GEMM: 64 bytes of data, 128-byte swizzled row
#pragma unroll
            for (int cc = 0; cc < 4; ++cc)
                *reinterpret_cast<uint4*>(ds_row + ((cc ^ (row & 7)) << 4)) = make_uint4(pd[4 * cc], pd[4 * cc + 1], pd[4 * cc + 2], pd[4 * cc + 3]);
            bars->dsum[gt & 3][c][row] = dsum;
            fence_async_smem();
            tmem_wait_st();
            tc_fence_before();
            mbar_arrive(&bars->p_full[w]);
        }
    } else if (warp >= 12) {
        // ------------------------------------------------------------------ drain warpgroup
        const uint32_t el = elect_one();
        const int quad = warp & 3;
        const int row = quad * 32 + lane;                       // TMEM lane: key within the tile (d for dq)
        const uint32_t lane_sel = (uint32_t)(quad * 32) << 16;
        const int n_gt = n_my * n_tiles;
        for (int gt = 0; gt < n_gt && !bars->abort_flag; ++gt) {
            const int uc = gt / n_tiles, t = gt - uc * n_tiles, s = gt % kStgB;
            const int u = unit_at(uc);
            const BUnit un = b_decode(p, u);
            const int key0 = t * kKB + quad * 32;
            if (!mbar_wait_u(&bars->acc_full, gt & 1)) { fail(41); break; }
            tc_fence_after();
            if (key0 + lane < n_keys) {
                float acc = 0.f;                     // the chunks' shares in a fixed order
#pragma unroll
                for (int cc = 0; cc < NC; ++cc) acc += bars->dsum[gt & 3][cc][row];
                p.dcL[(long long)u * p.n_keys_c + key0 + lane] = -acc;
            }
            // this warp's 32 keys, 64 columns at a time: daL over the aL tile, dY over the Y tile
#pragma unroll 1
            for (int h = 0; h < 4; ++h) {
                unsigned char* const st = a_s + s * kBStage + h * (kKB * 128) + quad * 4096;
                uint32_t ra[32], rb[32];
                const uint32_t col0 = (h < 2 ? kColDaL : kColDY) + (h & 1) * 64;
                tmem_ld32(tmem + lane_sel + col0, ra);
                tmem_ld32(tmem + lane_sel + col0 + 32, rb);
                tmem_wait_ld();
                if (h == 3) {
                    tc_fence_before();
                    mbar_arrive(&bars->acc_free);
                }
                if (key0 >= n_keys) continue;        // keys past the end of the last tile
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const uint32_t (&r)[32] = c < 4 ? ra : rb;
                    uint32_t wv[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        wv[e] = pack_bf16(__uint_as_float(r[(c & 3) * 8 + 2 * e]), __uint_as_float(r[(c & 3) * 8 + 2 * e + 1]));
                    *reinterpret_cast<uint4*>(st + lane * 128 + ((c ^ (lane & 7)) << 4)) = make_uint4(wv[0], wv[1], wv[2], wv[3]);
                }
                fence_async_smem();
                __syncwarp();
                tma_store_4d_e(el, h < 2 ? &sal : &sy, st, (h & 1) * 64, un.j, key0, un.bhl * p.A + un.a);
                tma_store_commit();
            }
            tma_store_wait_read_all();
            __syncwarp();
            if (el) mbar_arrive(&bars->a_empty[s]);
            // ---- last tile of the slab: its dq (TMEM lane = d, column = query row)
            if (t + 1 == n_tiles) {
                if (!mbar_wait_u(&bars->dq_full, uc & 1)) { fail(42); break; }
                tc_fence_after();
                const int bh = p.bh0 + un.bhl, b = bh / p.H, hd = bh - b * p.H;
                const long long pitch = (long long)blk.w * p.H * kHeadDim;
                float* const dq0 = p.dq + (((long long)b * p.n_q + blk.row_token(un.a, 0) + un.j) * p.H + hd) * kHeadDim + row;
#pragma unroll 1
                for (int cc = 0; cc < NC; ++cc) {
                    uint32_t r[kNI];
                    tmem_ld32(tmem + lane_sel + kColDq + cc * kNI, r);
                    tmem_wait_ld();
                    if (cc == NC - 1) {
                        tc_fence_before();
                        mbar_arrive(&bars->dq_free);
                    }
#pragma unroll
                    for (int ii = 0; ii < kNI; ++ii) {
                        const int i = cc * kNI + ii;
                        if (i < b1) dq0[i * pitch] = __uint_as_float(r[ii]);
                    }
                }
            }
        }
        tma_store_wait_all();
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, kTmemColsB);
}

// delta[b, token, head] = sum_d dOut * out.  Half a warp per (token, head) row, eight rows a warp, whose loads are all under way at
// once: what bounds it is the two tensors' trip from memory (29 MB for 4680 queries of 12 heads in 8 to 9 us from cold caches).
constexpr int kDeltaRows = 64;                                 // per CTA
__global__ void __launch_bounds__(256) bwd_delta_kernel(const __nv_bfloat16* __restrict__ dout, const __nv_bfloat16* __restrict__ out,
                                                        float* __restrict__ delta, long long rows) {
    pdl_trigger();
    pdl_wait();
    const int lane = threadIdx.x & 31, l = lane & 15;
    const long long r0 = (long long)blockIdx.x * kDeltaRows + (threadIdx.x >> 5) * 8 + (lane >> 4);
    uint4 a[4], b[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const long long r = r0 + 2 * i;
        a[i] = b[i] = make_uint4(0, 0, 0, 0);
        if (r < rows) {
            a[i] = reinterpret_cast<const uint4*>(dout + r * kHeadDim)[l];
            b[i] = reinterpret_cast<const uint4*>(out + r * kHeadDim)[l];
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t aw[4] = {a[i].x, a[i].y, a[i].z, a[i].w}, bw[4] = {b[i].x, b[i].y, b[i].z, b[i].w};
        float s = 0.f;
#pragma unroll
        for (int c = 0; c < 4; ++c)
            s = fmaf(__uint_as_float(aw[c] << 16), __uint_as_float(bw[c] << 16),
                     fmaf(__uint_as_float(aw[c] & 0xffff0000u), __uint_as_float(bw[c] & 0xffff0000u), s));
#pragma unroll
        for (int o = 8; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (l == 0 && r0 + 2 * i < rows) delta[r0 + 2 * i] = s;
    }
}

}  // namespace

int launch_bwd_delta(const void* dout, const void* out, float* delta, long long rows, cudaStream_t s) {
    LaunchScope scope(kClsBackward, s);
    return launch_pdl(true, bwd_delta_kernel, dim3((unsigned)((rows + kDeltaRows - 1) / kDeltaRows)), 256, 0, s, (const __nv_bfloat16*)dout,
                      (const __nv_bfloat16*)out, delta, rows);
}

// Column-step backward for one slice of (batch, head) pairs.  maps = {q rows, dOut rows}, 5-D (d, head, column, row of the token grid, batch) with boxes of 32 rows.
int launch_bwd_col_tc(const MonarchParams& mp, const CUtensorMap* maps, const float* delta, float* dcL, float* dq,
                      int* status, int num_sms, bool behind_delta, cudaStream_t s) {
    // query rows come by TMA: they must be consecutive rows of the token grid
    if (mp.blk.b1 > kMaxNC * kNI || (mp.blk.f_tied != 1 && mp.blk.h_reduce != 1)) return SFM_ERR_UNSUPPORTED;
    LaunchScope scope(kClsBackward, s);
    BwdColParams p;
    p.delta = delta; p.lse = mp.lse;
    p.cL = mp.cL; p.dcL = dcL; p.dq = dq;
    p.H = mp.H; p.n_q = mp.n_q; p.A = mp.na; p.n_keys = mp.n_keys; p.n_keys_c = mp.n_keys_c;
    p.bh0 = mp.bh0; p.nbh = mp.nbh;
    p.n_units = mp.nbh * mp.na * mp.blk.b2;
    p.q_box_rows = std::min(32, mp.n_q / mp.blk.w);
    p.scale = mp.scale;
    p.blk = mp.blk;
    p.status = status;
    dim3 grid(p.n_units < num_sms ? p.n_units : num_sms);
    const int nc = (mp.blk.b1 + kNI - 1) / kNI;
    CUtensorMap bridge[4];
    if (int rc = make_bridge_tmap(&bridge[0], mp.aL, mp.blk.b2, mp.n_keys, mp.nbh * mp.na, 1, kKB)) return rc;
    if (int rc = make_bridge_tmap(&bridge[1], mp.Y, mp.blk.b2, mp.n_keys, mp.nbh * mp.na, 1, kKB)) return rc;
    if (int rc = make_bridge_tmap(&bridge[2], mp.aL, mp.blk.b2, mp.n_keys, mp.nbh * mp.na, 1, 32)) return rc;
    if (int rc = make_bridge_tmap(&bridge[3], mp.Y, mp.blk.b2, mp.n_keys, mp.nbh * mp.na, 1, 32)) return rc;
    auto go = [&](auto kernel, int smem) -> int {
        if (int rc = opt_in_smem((const void*)kernel, smem)) return rc;
        // set up while the kernel before it drains, if that one is short
        return launch_pdl(behind_delta || (long long)p.n_units * ((p.n_keys + kKB - 1) / kKB) <= 32ll * num_sms, kernel, grid, kThreadsB, smem, s, bridge[0], bridge[1], bridge[2], bridge[3], maps[0], maps[1], p);
    };
    int rc = nc == 1 ? go(monarch_bwd_col_tc_kernel<1>, b_smem_bytes(1))
                     : (nc == 2 ? go(monarch_bwd_col_tc_kernel<2>, b_smem_bytes(2)) : go(monarch_bwd_col_tc_kernel<3>, b_smem_bytes(3)));
    if (rc) return rc;
    return (int)cudaGetLastError();
}

}  // namespace sfm
