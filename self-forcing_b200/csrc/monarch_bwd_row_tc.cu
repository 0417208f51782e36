// Backward of the Monarch row step on the 5th-generation tensor cores (tcgen05 + TMEM), fed by TMA.
//
// Forward row step, per (batch*head, block row k, cached group f) and stacked query row r = (query group a, column j):
//   z_l = scale * q[r] . K[f,k,l],  R = softmax_l z,  aL[r] = sum_l R_l K_l,  Y[r] = sum_l R_l V_l,  cL[r] = sum_l R_l ln R_l
// Given daL[r], dY[r] (bf16, in the bridge layout [query group][key][column][128], left there by the column step's backward) and dcL[r]:
//   dR_l = daL[r] . K_l + dY[r] . V_l + dcL[r] (ln R_l + 1)          dz_l = R_l (dR_l - sum_m R_m dR_m)
//   dQ[r] += scale * sum_l dz_l K_l
//   dK_l  += sum_r (R_l daL[r] + scale dz_l q[r])                      dV_l += sum_r R_l dY[r]
// Units are those of the forward row step: (batch*head, tile of stacked query groups, block row k), each walking
// all cached groups f; per step
//   S  = Q_tile K^T                 dR = daL_tile K^T + dY_tile V^T        three tcgen05.mma chains, operands in shared memory
//   R, dz                           16 rows per warp, read from TMEM as fragments: a quad has a row, whose sums are shuffles
//   dQ (+)= (scale dz) K            A = a bf16 copy of scale dz in shared memory, B = the K tile MN-major; accumulates over f
//   dK = R^T daL_tile + (scale dz)^T Q_tile,   dV = R^T dY_tile
//                                   A = bf16 copies of R / scale dz in shared memory read MN-major, B = the row tiles read
//                                   MN-major; dK on lanes 0 to 63 (M = key l) and dV on the others of the same columns, by output
//                                   masks; only for the cached groups whose dK / dV are wanted, which come first where they are the
//                                   last ones
// dK / dV of a (f, k) get one contribution per tile of query groups: with more than one, each tile writes fp32 partials to its own
// buffer and a small kernel adds them in a fixed order and rounds to bf16 (no atomics).  dQ rows are owned by one
// unit each and added to what the column step's backward left in dq.
//
// Warp roles (16 warps): 0 = daL and dY tiles, 1 = S and dR GEMMs (owns TMEM), 2 = query, K and V tiles, 3 = gradient GEMMs, 4-11 =
// element-wise pass, 12-15 = drain warpgroup (dK / dV per step, dQ per unit).  Every wait is bounded and
// reports through the status word.
//
// What bounds it: 53 KB of daL and dY, 27 KB of K and V a step (two query groups of 52 columns), whose slots are all the shared
// memory there is and wait 1600 to 3000 cycles for a tile; 2600 to 3000 cycles a step, 4500 with dK / dV.  4680
// queries, 18720 cached tokens, 12 heads, dK / dV of the last quarter: 175 us, now 144.  What it took, by the cycles of one CTA (281
// thousand before): a third K tile, which a step holds until its dQ GEMM is done (with two a K tile was waited for at every step); the
// element-wise pass without a shared-memory exchange between the halves of a row and without divisions for the address of
// dcL (a third of its 3500 cycles); a unit's dQ drained behind the dK / dV of the next, from two accumulators (6000 cycles a unit); R
// written ahead of dz, so that a step's row tiles leave when dR is done, and fragments stored as they are (4500 cycles for a dK / dV
// through a transposition, which the next step waited for).
//
// The training call takes dq in bf16 and dk / dv with their tokens in natural order from here: cast and permutation as
// passes of their own over the same rows, and the permutation's table sent from the host (which waits for the GPU) made up
// 125 of the 1050 us of a call with 4680 queries and 18720 cached tokens.
//
// Stands in for the Triton kernel _al_cl_y_bwd (wan/modules/monarch_attn.py:403-596), without its atomic adds.
#include "monarch_params.cuh"
#include "profile.cuh"
#include "tc05.cuh"

namespace sfm {

using namespace tc;

namespace {

constexpr int kThreadsRB = 512;
constexpr int kRows = 128;
// Above 48 block columns the working warps hold three values for each of 32 elements: they take registers that the issuing warps
// leave (the launch's 128 a thread).  Spilled words come back from L2, behind what the drain warps read and write: 190 bytes of them
// in the drain warps cost 8 us of 152.
constexpr int kRegsIssue = 104, kRegsWork = 144, kRegsDrain = 120;
static_assert(kRegsIssue + 2 * kRegsWork + kRegsDrain <= 4 * 128, "registers of the four warpgroups");
constexpr uint32_t kTmemColsRB = 512;
// S, dR, dK (lanes 0 to 63) and dV (64 to 127); dQ of even and odd units
constexpr uint32_t kCS = 0, kCDR = 64, kCDKV = 256;
__host__ __device__ constexpr uint32_t col_dq(int uc) { return uc & 1 ? 384u : 128u; }

struct BwdRowParams {
    MonarchParams mp;              // q, kc, vc, blocking, slice; mp.aL / mp.Y hold daL / dY
    const float* dcL;              // [slab][n_keys_c]
    float* dq;                     // natural order fp32, already holds the column step's share
    __nv_bfloat16* dq_bf16;        // the sum goes here, rounded, instead of back to dq (null: back to dq)
    float* part_k;                 // [tile][nbh][n_sel tokens][128] fp32 partial dK (n_sel = (g1 - g0) * b1 * b2)
    float* part_v;
    __nv_bfloat16* dk;             // the results, written from here when there is one tile (no partials, no merge)
    __nv_bfloat16* dv;
    int natural;                   // their tokens' order
    int g0, g1;                    // cached groups whose dK / dV are wanted
    int rows_per_group, groups_per_tile, tiles, n_units;
    int tile_rows;                 // rows held of a row tile, a multiple of 16: those of its groups (the GEMMs' M is 128)
    int n_rt, n_k;                 // slots for daL / dY tiles, for K tiles
    int* status;
};

// At most.  With four, dR of the step after a kv step can be complete before the gradient warp has looked at the kv step's, behind its
// R copy: dr_full has a barrier for even and one for odd steps.  The parity it looks at would turn back two steps on: that dR waits for
// dr_read of the step between, which the element-wise warps give behind rz_free of the kv step, and that the gradient warp commits last.
constexpr int kRowSlots = 4;
constexpr int kKSlots = 3;                                 // at most
struct __align__(16) RBBarriers {
    uint64_t q_full, q_empty;
    uint64_t k_full[kKSlots], k_empty[kKSlots], v_full, v_empty;
    uint64_t rt_full[kRowSlots], rt_empty[kRowSlots];      // daL and dY tiles in turn
    uint64_t s_full, dr_full[2], s_read, dr_read;          // S, dR (even, odd steps): written; S, dR: in registers
    uint64_t r_full, p_full, rz_free;                      // R copy (kv steps), dz copy: written; both free
    uint64_t dkv_full, dkv_free, dq_full[2], dq_free[2];
    uint32_t tmem_base;
    volatile int abort_flag;
};

constexpr int kStageT = kRows * 128;                 // R or dz copy: 128 rows x 64 bf16 (16 KB)
constexpr int kOutStage = 32 * 64;                   // a drain warp's staging: 32 rows of 16 fp32 columns
// Tiles: queries, daL / dY tiles, R and dz copies, a V tile, K tiles.  A K or V tile is two 64-column halves of N_S rows, a row
// tile two of tile_rows: the rows behind them that a GEMM reads too are another tile's, and what comes of them is not read.
constexpr int kRBTiles = 208 << 10;
constexpr int kRBSmem = 1024 + kRBTiles + 4 * kOutStage + 1024;
static_assert(sizeof(RBBarriers) <= 1024, "barriers");
static_assert(kRBSmem <= 227 * 1024, "shared memory");


// 16 rows x N columns of a TMEM tile, spread over a warp like an mma accumulator: r[4 i + e] is column 8 i + 2 (lane % 4) + (e & 1) of
// row lane / 4 + 8 (e >> 1).
template <int N>
__device__ __forceinline__ void tmem_ld_frag(uint32_t taddr, uint32_t (&r)[N / 2]) {
    if constexpr (N == 64) {
        asm volatile(
            "tcgen05.ld.sync.aligned.16x256b.x8.b32 "
            "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
            "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
              "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
              "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
              "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
            : "r"(taddr) : "memory");
    } else if constexpr (N == 32) {
        asm volatile(
            "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
              "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
            : "r"(taddr) : "memory");
    } else if constexpr (N == 16) {
        asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                     : "r"(taddr) : "memory");
    } else {
        static_assert(N == 48, "a multiple of 16 up to 64");
        tmem_ld_frag<32>(taddr, *reinterpret_cast<uint32_t(*)[16]>(&r[0]));
        tmem_ld_frag<16>(taddr + 32, *reinterpret_cast<uint32_t(*)[8]>(&r[16]));
    }
}

// Four 8 x 8 tiles of bf16 held like mma accumulators; lane l has the address of row l % 8 of tile l / 8.
__device__ __forceinline__ void stmatrix_x4(uint32_t saddr, uint32_t r0, uint32_t r1, uint32_t r2, uint32_t r3) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(saddr), "r"(r0), "r"(r1), "r"(r2), "r"(r3) : "memory");
}

__device__ __forceinline__ void red_add_v4(float* ptr, const float4& v) {
    asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(ptr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}

struct RBUnit { int bhl, tile, k; };
__device__ __forceinline__ RBUnit rb_decode(const BwdRowParams& rp, int u) {
    RBUnit r;
    r.k = u % rp.mp.blk.b1; u /= rp.mp.blk.b1;
    r.tile = u % rp.tiles;
    r.bhl = u / rp.tiles;
    return r;
}

// tq, tk, tv: the forward's maps of q, K, V; tda, tdy: bridge maps of daL / dY (box 64 x rows_per_group columns x 1 key).
// kOneTile: all query groups fit one tile, whose dK / dV are the results (24 x 32 tokens, 2 videos, 12 heads, 6 frames cached:
// training call 380 -> 358 us against partials and a merge).
template <int N_S, bool kOneTile>
__global__ void __launch_bounds__(kThreadsRB, 1)
monarch_bwd_row_tc_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk,
                          const __grid_constant__ CUtensorMap tv, const __grid_constant__ CUtensorMap tda,
                          const __grid_constant__ CUtensorMap tdy, BwdRowParams rp) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    constexpr int kHalf = N_S * 128, kKVTile = 2 * kHalf;
    constexpr bool kSplit = N_S > 48;
    const int q_half = rp.tile_rows * 128, q_tile = 2 * q_half;
    const int n_rt = rp.n_rt, n_ks = rp.n_k;
    unsigned char* q_s = base;
    unsigned char* rt_s = q_s + q_tile;                    // daL / dY tiles
    unsigned char* r_s = rt_s + n_rt * q_tile;             // R copy | dz copy
    unsigned char* z_s = r_s + kStageT;
    unsigned char* v_s = z_s + kStageT;                    // V tile, K tiles
    unsigned char* k_s = v_s + kKVTile;
    unsigned char* o_s = base + kRBTiles;                  // drain staging
    RBBarriers* bars = reinterpret_cast<RBBarriers*>(o_s + 4 * kOutStage);

    const MonarchParams& p = rp.mp;
    const Blocking& blk = p.blk;
    const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
    const int b1 = blk.b1, b2 = blk.b2;
    const int RG = rp.rows_per_group;
    const int F = p.F;

    if (tid == 0) {
        mbar_init(&bars->q_full, 1); mbar_init(&bars->q_empty, 2);
        for (int s = 0; s < kKSlots; ++s) { mbar_init(&bars->k_full[s], 1); mbar_init(&bars->k_empty[s], 1); }
        mbar_init(&bars->v_full, 1); mbar_init(&bars->v_empty, 1);
        for (int s = 0; s < kRowSlots; ++s) { mbar_init(&bars->rt_full[s], 1); mbar_init(&bars->rt_empty[s], 1); }
        mbar_init(&bars->s_full, 1); mbar_init(&bars->s_read, 256); mbar_init(&bars->dr_read, 256);
        mbar_init(&bars->r_full, 256); mbar_init(&bars->p_full, 256); mbar_init(&bars->rz_free, 1);
        mbar_init(&bars->dkv_full, 1); mbar_init(&bars->dkv_free, 128);
        for (int s = 0; s < 2; ++s) { mbar_init(&bars->dr_full[s], 1); mbar_init(&bars->dq_full[s], 1); mbar_init(&bars->dq_free[s], 128); }
        bars->abort_flag = 0;
        mbar_init_fence();
    }
    // tile rows no load writes and the padding of the R / dz copies must read as zero
    for (int i = tid; i < kRBTiles / 16; i += kThreadsRB)
        reinterpret_cast<uint4*>(q_s)[i] = make_uint4(0, 0, 0, 0);
    if (warp == 1) { tmem_alloc(&bars->tmem_base, kTmemColsRB); tmem_relinquish(); }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = bars->tmem_base;
    pdl_trigger();
    pdl_wait();

    auto fail = [&](int code) {
        bars->abort_flag = 1;
        atomicCAS(rp.status, 0, code);
    };
    const int u_first = blockIdx.x, u_stride = gridDim.x;
    // The groups of a unit, last one first: a training call wants dK / dV of the last ones, and the query tile is then free
    // from the last step's S GEMM on.  The order does not depend on which are wanted (nor then does dQ's rounding).
    auto group_of = [&](int i) { return F - 1 - i; };
    auto wants_kv = [&](int i) { const int f = group_of(i); return f >= rp.g0 && f < rp.g1; };

    if (warp < 4) {
    if constexpr (kSplit) reg_dec<kRegsIssue>();
    if (warp == 0) {
        // ------------------------------------------------------------------ daL, dY
        const uint32_t el = elect_one();
        prefetch_tmap(&tda); prefetch_tmap(&tdy);
        int sr = 0, pr = 1;
        bool ok = true;
        for (int u = u_first; ok && u < rp.n_units && !bars->abort_flag; u += u_stride) {
            const RBUnit un = rb_decode(rp, u);
            const int g_first = un.tile * rp.groups_per_tile;
            const int ng = min(rp.groups_per_tile, p.na - g_first);
            for (int i = 0; ok && i < F; ++i) {
                const int key = group_of(i) * b1 + un.k;
                for (int which = 0; which < 2; ++which) {
                    if (!mbar_wait_u(&bars->rt_empty[sr], pr)) { fail(12); ok = false; break; }
                    unsigned char* rt = rt_s + sr * q_tile;
                    mbar_arrive_expect_tx_e(el, &bars->rt_full[sr], (uint32_t)(ng * RG * 256));
                    for (int gi = 0; gi < ng; ++gi) {
                        const int grp = un.bhl * p.na + g_first + gi;
                        tma_load_4d_e(el, rt + gi * RG * 128, which ? &tdy : &tda, &bars->rt_full[sr], 0, 0, key, grp);
                        tma_load_4d_e(el, rt + q_half + gi * RG * 128, which ? &tdy : &tda, &bars->rt_full[sr], 64, 0, key, grp);
                    }
                    if (++sr == n_rt) { sr = 0; pr ^= 1; }
                }
            }
        }
    } else if (warp == 2) {
        // ------------------------------------------------------------------ query, K and V tiles
        const uint32_t el = elect_one();
        prefetch_tmap(&tq); prefetch_tmap(&tk); prefetch_tmap(&tv);
        int uc = 0, g = 0, sk = 0, pk = 1;
        bool ok = true;
        for (int u = u_first; ok && u < rp.n_units && !bars->abort_flag; u += u_stride, ++uc) {
            const RBUnit un = rb_decode(rp, u);
            const int bh = p.bh0 + un.bhl, b = bh / p.H, hd = bh - b * p.H;
            const int g_first = un.tile * rp.groups_per_tile;
            const int ng = min(rp.groups_per_tile, p.na - g_first);
            if (uc > 0 && !mbar_wait_u(&bars->q_empty, (uc - 1) & 1)) { fail(10); break; }
            mbar_arrive_expect_tx_e(el, &bars->q_full, (uint32_t)(ng * b2 * 256));           // the padding rows stay zero
            for (int gi = 0; gi < ng; ++gi) {
                const int tok = blk.row_token(p.a0 + g_first + gi, un.k);
                tma_load_4d_e(el, q_s + gi * RG * 128, &tq, &bars->q_full, 0, hd, tok, b);
                tma_load_4d_e(el, q_s + q_half + gi * RG * 128, &tq, &bars->q_full, 64, hd, tok, b);
            }
            for (int i = 0; i < F; ++i, ++g) {
                const int tok = (group_of(i) * b1 + un.k) * b2;
                if (!mbar_wait_u(&bars->k_empty[sk], pk)) { fail(11); ok = false; break; }
                unsigned char* kt = k_s + sk * kKVTile;
                mbar_arrive_expect_tx_e(el, &bars->k_full[sk], (uint32_t)(2 * b2 * 128));
                tma_load_4d_e(el, kt, &tk, &bars->k_full[sk], 0, hd, tok, b);
                tma_load_4d_e(el, kt + kHalf, &tk, &bars->k_full[sk], 64, hd, tok, b);
                if (++sk == n_ks) { sk = 0; pk ^= 1; }
                if (g >= 1 && !mbar_wait_u(&bars->v_empty, (g - 1) & 1)) { fail(13); ok = false; break; }
                mbar_arrive_expect_tx_e(el, &bars->v_full, (uint32_t)(2 * b2 * 128));
                tma_load_4d_e(el, v_s, &tv, &bars->v_full, 0, hd, tok, b);
                tma_load_4d_e(el, v_s + kHalf, &tv, &bars->v_full, 64, hd, tok, b);
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ S and dR GEMMs
        const uint32_t el = elect_one();
        constexpr uint32_t idesc_s = idesc_bf16(kRows, N_S, 0, 0);
        const uint64_t q_k = smem_desc_sw128(smem_addr(q_s), 16, 1024);
        const uint64_t rt_k0 = smem_desc_sw128(smem_addr(rt_s), 16, 1024);
        const uint64_t k_k0 = smem_desc_sw128(smem_addr(k_s), 16, 1024);
        const uint64_t vd = smem_desc_sw128(smem_addr(v_s), 16, 1024);
        int g = 0, uc = 0, sr = 0, pr = 0, sk = 0, pk = 0;
        bool ok = true;
        for (int u = u_first; ok && u < rp.n_units && !bars->abort_flag; u += u_stride, ++uc) {
            if (!mbar_wait_u(&bars->q_full, uc & 1)) { fail(20); break; }
            for (int i = 0; i < F; ++i, ++g) {
                const bool kvw = wants_kv(i);
                if (!mbar_wait_u(&bars->k_full[sk], pk)) { fail(21); ok = false; break; }
                if (g >= 1 && !mbar_wait_u(&bars->s_read, (g - 1) & 1)) { fail(22); ok = false; break; }
                tc_fence_after();
                const uint64_t kd = k_k0 + (uint64_t)((sk * kKVTile) >> 4);
                if (++sk == n_ks) { sk = 0; pk ^= 1; }
#pragma unroll
                for (int ks = 0; ks < 8; ++ks) {
                    const uint32_t qo = ((ks >> 2) * q_half + (ks & 3) * 32) >> 4;
                    const uint32_t ko = ((ks >> 2) * kHalf + (ks & 3) * 32) >> 4;
                    mma_ss_e(el, tmem + kCS, q_k + qo, kd + ko, idesc_s, ks > 0);
                }
                mma_commit_e(el, &bars->s_full);
                if (i + 1 == F) mma_commit_e(el, &bars->q_empty);
                if (g >= 1 && !mbar_wait_u(&bars->dr_read, (g - 1) & 1)) { fail(28); ok = false; break; }
#pragma unroll 1
                for (int which = 0; which < 2; ++which) {
                    if (!mbar_wait_u(&bars->rt_full[sr], pr)) { fail(23); ok = false; break; }
                    if (which && !mbar_wait_u(&bars->v_full, g & 1)) { fail(27); ok = false; break; }
                    tc_fence_after();
                    const uint64_t rd = rt_k0 + (uint64_t)((sr * q_tile) >> 4);
                    const uint64_t bd = which ? vd : kd;
#pragma unroll
                    for (int ks = 0; ks < 8; ++ks) {
                        const uint32_t qo = ((ks >> 2) * q_half + (ks & 3) * 32) >> 4;
                        const uint32_t ko = ((ks >> 2) * kHalf + (ks & 3) * 32) >> 4;
                        mma_ss_e(el, tmem + kCDR, rd + qo, bd + ko, idesc_s, (which || ks > 0) ? 1u : 0u);
                    }
                    if (!kvw) mma_commit_e(el, &bars->rt_empty[sr]);      // nothing else reads the row tiles this step
                    if (++sr == n_rt) { sr = 0; pr ^= 1; }
                }
                if (!ok) break;
                mma_commit_e(el, &bars->dr_full[g & 1]);
                mma_commit_e(el, &bars->v_empty);
            }
        }
    } else {
        // ------------------------------------------------------------------ gradient GEMMs
        const uint32_t el = elect_one();
        constexpr uint32_t idesc_q = idesc_bf16(kRows, kHeadDim, 0, 1);        // dQ: B MN-major
        constexpr uint32_t idesc_k = idesc_bf16(kRows, kHeadDim, 1, 1);        // dK, dV: both MN-major
        const uint64_t q_mn = smem_desc_sw128(smem_addr(q_s), q_half, 1024);
        const uint64_t rt_mn0 = smem_desc_sw128(smem_addr(rt_s), q_half, 1024);
        const uint64_t k_mn0 = smem_desc_sw128(smem_addr(k_s), kHalf, 1024);
        const uint64_t r_mn = smem_desc_sw128(smem_addr(r_s), kStageT, 1024);
        const uint64_t z_mn = smem_desc_sw128(smem_addr(z_s), kStageT, 1024);
        const uint64_t z_k = smem_desc_sw128(smem_addr(z_s), 16, 1024);
        // dK on lanes 0 to 63, dV on the others of the same columns: its A operand starts a copy's size before R, so that R is
        // the operand's second half
        const uint64_t r_mn_hi = r_mn - (kStageT >> 4);
        const LaneMask lo = lane_mask_rows(0, 64), hi = lane_mask_rows(64, 64);
        const int n_kk = rp.tile_rows / 16;                          // K = 16 steps over a tile's rows
        const int q_last = rp.g1 > rp.g0 ? F - 1 - rp.g0 : 0;        // from here on these GEMMs leave the query tile alone
        int g = 0, uc = 0, gd = 0, sr = 0, sk = 0;
        bool ok = true;
        for (int u = u_first; ok && u < rp.n_units && !bars->abort_flag; u += u_stride, ++uc) {
            const uint32_t dq_t = tmem + col_dq(uc);
            for (int i = 0; i < F; ++i, ++g) {
                const int da = sr, dy = da + 1 == n_rt ? 0 : da + 1;
                sr = dy + 1 == n_rt ? 0 : dy + 1;
                const bool kvw = wants_kv(i);
                if (kvw) {
                    // R is there long before dz: the row tiles leave as soon as dR has been taken from them
                    if (!mbar_wait_u(&bars->r_full, gd & 1)) { fail(29); ok = false; break; }
                    if (!mbar_wait_u(&bars->dr_full[g & 1], (g >> 1) & 1)) { fail(30); ok = false; break; }
                    if (gd >= 1 && !mbar_wait_u(&bars->dkv_free, (gd - 1) & 1)) { fail(26); ok = false; break; }
                    tc_fence_after();
                    const uint64_t da_mn = rt_mn0 + (uint64_t)((da * q_tile) >> 4), dy_mn = rt_mn0 + (uint64_t)((dy * q_tile) >> 4);
#pragma unroll
                    for (int kk = 0; kk < kRows / 16; ++kk)     // dK = R^T daL_tile
                        if (kk < n_kk) mma_ss_masked_e(el, tmem + kCDKV, r_mn + ((kk * 2048) >> 4), da_mn + ((kk * 2048) >> 4), idesc_k, kk > 0, lo);
                    mma_commit_e(el, &bars->rt_empty[da]);
#pragma unroll
                    for (int kk = 0; kk < kRows / 16; ++kk)     // dV = R^T dY_tile
                        if (kk < n_kk) mma_ss_masked_e(el, tmem + kCDKV, r_mn_hi + ((kk * 2048) >> 4), dy_mn + ((kk * 2048) >> 4), idesc_k, kk > 0, hi);
                    mma_commit_e(el, &bars->rt_empty[dy]);
                }
                if (!mbar_wait_u(&bars->p_full, g & 1)) { fail(24); ok = false; break; }
                if (i == 0 && uc >= 2 && !mbar_wait_u(&bars->dq_free[uc & 1], ((uc >> 1) - 1) & 1)) { fail(25); ok = false; break; }
                tc_fence_after();
                const uint64_t kmn = k_mn0 + (uint64_t)((sk * kKVTile) >> 4);
#pragma unroll
                for (int kk = 0; kk < N_S / 16; ++kk)      // dQ (+)= (scale dz) K
                    mma_ss_e(el, dq_t, z_k + ((kk * 32) >> 4), kmn + ((kk * 2048) >> 4), idesc_q, (i > 0 || kk > 0) ? 1u : 0u);
                mma_commit_e(el, &bars->k_empty[sk]);
                if (++sk == n_ks) sk = 0;
                if (kvw) {
#pragma unroll
                    for (int kk = 0; kk < kRows / 16; ++kk)     // dK += (scale dz)^T Q_tile
                        if (kk < n_kk) mma_ss_masked_e(el, tmem + kCDKV, z_mn + ((kk * 2048) >> 4), q_mn + ((kk * 2048) >> 4), idesc_k, 1u, lo);
                    mma_commit_e(el, &bars->dkv_full);
                    ++gd;
                }
                if (i == q_last) mma_commit_e(el, &bars->q_empty);
                mma_commit_e(el, &bars->rz_free);
                if (i + 1 == F) mma_commit_e(el, &bars->dq_full[uc & 1]);
            }
        }
    }
    } else if (warp < 12) {
        if constexpr (kSplit) reg_inc<kRegsWork>();
        // ------------------------------------------------------------------ element-wise pass: 16 query rows per warp
        // A thread has a quarter of the columns of two rows, 8 rows apart; the rows' sums come from its neighbours by shuffles.
        constexpr int kB = N_S / 8;                             // blocks of 8 columns
        const int quad = warp & 3, row0 = quad * 32 + ((warp - 4) >> 2) * 16;
        const uint32_t s_t = tmem + ((uint32_t)row0 << 16) + kCS;
        const uint32_t dr_t = s_t + (kCDR - kCS);
        const float scale_l2 = p.mult0 * kLog2e;
        const uint64_t scale2 = f2_pack(scale_l2, scale_l2);
        int gl[2], j[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int row = row0 + (lane >> 2) + 8 * h;
            gl[h] = row / RG;
            j[h] = row - gl[h] * RG;
        }
        // the copies' rows this lane has the addresses of
        const int st_row = row0 + (lane & 15), st_blk = lane >> 4;
        const uint32_t r_row = smem_addr(r_s) + st_row * 128, z_row = smem_addr(z_s) + st_row * 128;
        auto quad_sums = [&](uint64_t (&v)[2], float (&o)[2]) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float lo, hi;
                f2_unpack(v[h], lo, hi);
                o[h] = quad_sum(lo + hi);
            }
        };
        int g = 0;
        bool ok = true;
        for (int u = u_first; ok && u < rp.n_units && !bars->abort_flag; u += u_stride) {
            const RBUnit un = rb_decode(rp, u);
            const float* dcl_at[2];                             // of this unit's rows; null: no row
            float dcl_next[2] = {0.f, 0.f};
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int al = un.tile * rp.groups_per_tile + gl[h];
                dcl_at[h] = gl[h] < rp.groups_per_tile && al < p.na && j[h] < b2
                                ? rp.dcL + (((long long)un.bhl * p.na + al) * b2 + j[h]) * p.n_keys_c + group_of(0) * b1 + un.k : nullptr;
                if (dcl_at[h]) dcl_next[h] = *dcl_at[h];
            }
            for (int i = 0; i < F; ++i, ++g) {
                float dcl[2];                                   // used only when dR has been summed up: in no hurry to arrive
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    dcl[h] = dcl_next[h];
                    if (i + 1 < F && dcl_at[h]) dcl_next[h] = dcl_at[h][-(i + 1) * b1];
                }
                if (!mbar_wait_u(&bars->s_full, g & 1)) { fail(31); ok = false; break; }
                tc_fence_after();
                uint64_t d2[2][kB], e[2][kB], x[2][kB];         // log2 of the weight over the row's maximum, weight, dR
                {
                    uint32_t r[N_S / 2];
                    tmem_ld_frag<N_S>(s_t, r);
                    tmem_wait_ld();
                    tc_fence_before();
                    mbar_arrive(&bars->s_read);
#pragma unroll
                    for (int c = 0; c < N_S / 2; ++c)           // columns past b2, of the last two blocks at most: weight zero
                        if (c >= N_S / 2 - 8 && 8 * (c >> 2) + 2 * (lane & 3) + (c & 1) >= b2) r[c] = 0xf149f2cau;   // -1e30
#pragma unroll
                    for (int c = 0; c < N_S / 2; c += 2) d2[(c >> 1) & 1][c >> 2] = f2_pack(__uint_as_float(r[c]), __uint_as_float(r[c + 1]));
                }
                uint64_t zz[2], el2[2], ex2[2];                 // sums of e, e log2 e, e (daL . K + dY . V)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
                    for (int c = 0; c < kB; ++c) {
                        float x0, x1;
                        f2_unpack(d2[h][c], x0, x1);
                        mx[c & 1] = max3(mx[c & 1], x0, x1);
                    }
                    const float m2 = quad_max(fmaxf(mx[0], mx[1])) * scale_l2;
                    const uint64_t neg_m2 = f2_pack(-m2, -m2);
                    zz[h] = el2[h] = f2_pack(0.f, 0.f);
#pragma unroll
                    for (int c = 0; c < kB; ++c) {
                        d2[h][c] = f2_fma(d2[h][c], scale2, neg_m2);
                        float x0, x1;
                        f2_unpack(d2[h][c], x0, x1);
                        e[h][c] = f2_pack(exp2f(x0), exp2f(x1));
                        zz[h] = f2_add(zz[h], e[h][c]);
                        el2[h] = f2_fma(e[h][c], d2[h][c], el2[h]);
                    }
                }
                float z[2], el[2], inv_z[2], l2z[2], rs[2];
                quad_sums(zz, z);
                quad_sums(el2, el);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    inv_z[h] = 1.0f / z[h];
                    l2z[h] = __log2f(z[h]);
                    rs[h] = dcl_at[h] ? inv_z[h] : 0.f;         // rows of no unit must not reach dK / dV
                }
                const bool kvw = wants_kv(i);
                if (g >= 1 && !mbar_wait_u(&bars->rz_free, (g - 1) & 1)) { fail(34); ok = false; break; }
                if (kvw) {
#pragma unroll
                    for (int c = 0; c < kB; c += 2) {
                        uint32_t w[4];
#pragma unroll
                        for (int t = 0; t < 4; ++t) {
                            float v0, v1;
                            f2_unpack(f2_mul(e[t & 1][c + (t >> 1)], f2_pack(rs[t & 1], rs[t & 1])), v0, v1);
                            w[t] = pack_bf16(v0, v1);
                        }
                        stmatrix_x4(r_row + (((c + st_blk) ^ (st_row & 7)) << 4), w[0], w[1], w[2], w[3]);
                    }
                    fence_async_smem();
                    mbar_arrive(&bars->r_full);
                }
                if (!mbar_wait_u(&bars->dr_full[g & 1], (g >> 1) & 1)) { fail(32); ok = false; break; }
                tc_fence_after();
                {
                    uint32_t r[N_S / 2];
                    tmem_ld_frag<N_S>(dr_t, r);
                    tmem_wait_ld();
                    tc_fence_before();
                    mbar_arrive(&bars->dr_read);
#pragma unroll
                    for (int c = 0; c < N_S / 2; ++c)
                        if (c >= N_S / 2 - 8 && 8 * (c >> 2) + 2 * (lane & 3) + (c & 1) >= b2) r[c] = 0u;
#pragma unroll
                    for (int c = 0; c < N_S / 2; c += 2) x[(c >> 1) & 1][c >> 2] = f2_pack(__uint_as_float(r[c]), __uint_as_float(r[c + 1]));
                }
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    ex2[h] = f2_pack(0.f, 0.f);
#pragma unroll
                    for (int c = 0; c < kB; ++c) ex2[h] = f2_fma(e[h][c], x[h][c], ex2[h]);
                }
                float ex[2];
                quad_sums(ex2, ex);
                uint64_t zs2[2], dc2[2], off2[2];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    // dR_l = (daL . K_l + dY . V_l) + dcL (ln R_l + 1); the sum of R dR from its parts
                    const float rlr = fmaf(el[h], inv_z[h], -l2z[h]);                  // sum of R log2 R
                    const float dcl2 = dcl[h] * 0.6931471805599453f;
                    const float dot = fmaf(dcl2, rlr, ex[h] * inv_z[h]);
                    const float off = fmaf(dcl2, -l2z[h], -dot);                       // dR - sum = x + dcl2 d2 + off (dcL itself cancels)
                    zs2[h] = f2_pack(rs[h] * p.scale, rs[h] * p.scale);
                    dc2[h] = f2_pack(dcl2, dcl2);
                    off2[h] = f2_pack(off, off);
                }
#pragma unroll
                for (int c = 0; c < kB; c += 2) {
                    uint32_t w[4];
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        const int h = t & 1, cc = c + (t >> 1);
                        float v0, v1;
                        f2_unpack(f2_mul(f2_mul(e[h][cc], zs2[h]), f2_fma(dc2[h], d2[h][cc], f2_add(x[h][cc], off2[h]))), v0, v1);
                        w[t] = pack_bf16(v0, v1);
                    }
                    stmatrix_x4(z_row + (((c + st_blk) ^ (st_row & 7)) << 4), w[0], w[1], w[2], w[3]);
                }
                fence_async_smem();
                mbar_arrive(&bars->p_full);
            }
        }
    } else {
        if constexpr (kSplit) reg_dec<kRegsDrain>();
        // ------------------------------------------------------------------ drain warpgroup
        // Rows come out of TMEM one per lane; through a small transposition in shared memory they go out 64 bytes at a time,
        // four lanes a row, instead of 32 rows per store instruction.
        const int quad = warp & 3;
        const uint32_t lane_sel = (uint32_t)(quad * 32) << 16;
        unsigned char* const st = o_s + quad * kOutStage;
        const int l_row = lane >> 2, l_col = (lane & 3) * 4;     // of each group of 8 rows, of each block of 16 columns
        auto transpose = [&](const uint32_t (&r)[16], float4 (&v)[4]) {
            __syncwarp();
#pragma unroll
            for (int c = 0; c < 4; ++c)
                *reinterpret_cast<uint4*>(st + lane * 64 + ((c ^ ((lane >> 1) & 3)) << 4)) = make_uint4(r[4 * c], r[4 * c + 1], r[4 * c + 2], r[4 * c + 3]);
            __syncwarp();
#pragma unroll
            for (int it = 0; it < 4; ++it) {
                const int rr = it * 8 + l_row;
                v[it] = *reinterpret_cast<const float4*>(st + rr * 64 + (((lane & 3) ^ ((rr >> 1) & 3)) << 4));
            }
        };
        const long long n_sel = (long long)(rp.g1 - rp.g0) * b1 * b2;
        int x = 0, gd = 0;
        bool ok = true;
        // A unit's dQ is drained behind the dK / dV of the unit after it, which that one's next steps wait for.
        for (int u = u_first; ok && u < rp.n_units + u_stride && !bars->abort_flag; u += u_stride, ++x) {
            const RBUnit un = rb_decode(rp, u);
            const int bh = p.bh0 + un.bhl, b = bh / p.H, hd = bh - b * p.H;
            for (int i = 0; i < F && u < rp.n_units; ++i) {
                if (!wants_kv(i)) continue;
                if (!mbar_wait_u(&bars->dkv_full, gd & 1)) { fail(41); ok = false; break; }
                tc_fence_after();
                // The keys of the block, at most 64, are on two warps' lanes each for dK and for dV.  16 rows at a time as fragments: a
                // quad's eight channels of a row are a sector of the fp32 partials (half a one of bf16 results), and the GEMMs have
                // the accumulator back after four loads.
                const int key0 = (quad & 1) * 32;
                if (key0 < b2) {
                    const long long row0 = ((long long)un.tile * p.nbh + un.bhl) * n_sel + ((long long)(group_of(i) - rp.g0) * b1 + un.k) * b2;
                    // with one tile: the results themselves, in the order asked for
                    const int fi = group_of(i) - rp.g0, tok0 = rp.natural ? blk.row_token(fi, un.k) : (fi * b1 + un.k) * b2;
                    const int r0 = key0 + (lane >> 2), ch = (lane & 3) * 2;
                    float* const part = (quad < 2 ? rp.part_k : rp.part_v) + (row0 + r0) * kHeadDim + ch;
                    __nv_bfloat16* const res = (quad < 2 ? rp.dk : rp.dv) + (((long long)b * n_sel + tok0 + r0) * p.H + hd) * kHeadDim + ch;
#pragma unroll 1
                    for (int x4 = 0; x4 < 4; ++x4) {
                        const int rr = (x4 >> 1) * 16, c0 = (x4 & 1) * 64;
                        uint32_t r[32];
                        tmem_ld_frag<64>(tmem + lane_sel + ((uint32_t)rr << 16) + kCDKV + c0, r);
                        tmem_wait_ld();
                        if (x4 == 3) {
                            tc_fence_before();
                            mbar_arrive(&bars->dkv_free);
                        }
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            if (r0 + rr + 8 * h >= b2) continue;
#pragma unroll
                            for (int c = 0; c < 8; ++c) {
                                const float v0 = __uint_as_float(r[4 * c + 2 * h]), v1 = __uint_as_float(r[4 * c + 2 * h + 1]);
                                if constexpr (kOneTile)
                                    *reinterpret_cast<uint32_t*>(res + (long long)(rr + 8 * h) * p.H * kHeadDim + c0 + 8 * c) = pack_bf16(v0, v1);
                                else *reinterpret_cast<float2*>(part + (rr + 8 * h) * kHeadDim + c0 + 8 * c) = make_float2(v0, v1);
                            }
                        }
                    }
                } else mbar_arrive(&bars->dkv_free);
                ++gd;
            }
            if (!ok) break;
            if (x == 0) continue;
            // ---- dQ rows of the unit before: added to the column step's share
            const int uc = x - 1;
            const RBUnit uq = rb_decode(rp, u - u_stride);
            const int bhq = p.bh0 + uq.bhl, bq = bhq / p.H, hq = bhq - bq * p.H;
            const int g_first = uq.tile * rp.groups_per_tile;
            const int ng = min(rp.groups_per_tile, p.na - g_first);
            long long off[4];                                    // of this lane's rows; negative: no row
#pragma unroll
            for (int it = 0; it < 4; ++it) {
                const int row = quad * 32 + it * 8 + l_row, gl = row / RG, j = row - gl * RG;
                const int tok = gl < ng && j < b2 ? blk.row_token(p.a0 + g_first + gl, uq.k) + j : -1;
                off[it] = tok < 0 ? -1 : (((long long)bq * p.n_q + tok) * p.H + hq) * kHeadDim + l_col;
            }
            constexpr int kAhead = 3;                            // blocks of 16 columns whose share is on its way
            float4 share[kAhead][4];
            auto load_share = [&](int blk16) {
#pragma unroll
                for (int it = 0; it < 4; ++it)
                    if (rp.dq_bf16 && off[it] >= 0) share[blk16 % kAhead][it] = *reinterpret_cast<const float4*>(rp.dq + off[it] + blk16 * 16);
            };
#pragma unroll
            for (int c = 0; c < kAhead; ++c) load_share(c);
            if (!mbar_wait_u(&bars->dq_full[uc & 1], (uc >> 1) & 1)) { fail(42); break; }
            tc_fence_after();
            const uint32_t dq_t = tmem + lane_sel + col_dq(uc);
#pragma unroll
            for (int c = 0; c < kHeadDim / 16; ++c) {
                uint32_t r[16];
                float4 v[4];
                tmem_ld16(dq_t + c * 16, r);
                tmem_wait_ld();
                if ((c + 1) * 16 == kHeadDim) {
                    tc_fence_before();
                    mbar_arrive(&bars->dq_free[uc & 1]);
                }
                transpose(r, v);
                if (rp.dq_bf16) {
#pragma unroll
                    for (int it = 0; it < 4; ++it) {
                        const float4 w = share[c % kAhead][it];
                        v[it].x += w.x; v[it].y += w.y; v[it].z += w.z; v[it].w += w.w;
                    }
                    if (c + kAhead < kHeadDim / 16) load_share(c + kAhead);
                }
#pragma unroll
                for (int it = 0; it < 4; ++it) {
                    if (off[it] < 0) continue;
                    if (rp.dq_bf16)
                        *reinterpret_cast<uint2*>(rp.dq_bf16 + off[it] + c * 16) = make_uint2(pack_bf16(v[it].x, v[it].y), pack_bf16(v[it].z, v[it].w));
                    else
                        red_add_v4(rp.dq + off[it] + c * 16, v[it]);     // the only addition to these words
                }
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, kTmemColsRB);
}

// dk / dv [B, n_sel, H, 128] bf16 (Monarch order, or the tokens in natural order) = sum over the tiles' fp32 partials, in tile order.
// A thread has eight channels of a token, a block 16 tokens of a (batch, head) pair.  Bound by the partials' trip from memory
// (144 MB with the results for 4680 tokens, 12 heads, two tiles: 20 us).
__global__ void __launch_bounds__(256) bwd_merge_kv_kernel(const float* __restrict__ part_k, const float* __restrict__ part_v,
                                                           __nv_bfloat16* __restrict__ dk, __nv_bfloat16* __restrict__ dv,
                                                           int tiles, int n_sel, MonarchParams mp, FastDiv by_blocks, FastDiv by_group, int natural) {
    pdl_trigger();
    pdl_wait();
    int block;
    const int bhl = by_blocks.divmod((int)blockIdx.x, block);
    const int tok = block * 16 + (int)(threadIdx.x >> 4), c8 = (threadIdx.x & 15) * 8;
    if (tok >= n_sel) return;
    const long long tile_step = (long long)mp.nbh * n_sel * kHeadDim;
    long long o = ((long long)bhl * n_sel + tok) * kHeadDim + c8;
    float k[8] = {}, v[8] = {};
#pragma unroll 2
    for (int t = 0; t < tiles; ++t, o += tile_step) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float4 a = *reinterpret_cast<const float4*>(part_k + o + 4 * h);
            const float4 c = *reinterpret_cast<const float4*>(part_v + o + 4 * h);
            k[4 * h] += a.x; k[4 * h + 1] += a.y; k[4 * h + 2] += a.z; k[4 * h + 3] += a.w;
            v[4 * h] += c.x; v[4 * h + 1] += c.y; v[4 * h + 2] += c.z; v[4 * h + 3] += c.w;
        }
    }
    int tok_out = tok;
    if (natural) {
        int in_g, j, col;
        const int g = by_group.divmod(tok, in_g), r = mp.by_b2.divmod(in_g, j);
        const int row = mp.first_row(g, j, col) + mp.row_ahead(r);
        tok_out = row * mp.blk.w + col;
    }
    int hd;
    const int b = mp.by_H.divmod(mp.bh0 + bhl, hd);
    const long long out = (((long long)b * n_sel + tok_out) * mp.H + hd) * kHeadDim + c8;
    *reinterpret_cast<uint4*>(dk + out) = make_uint4(pack_bf16(k[0], k[1]), pack_bf16(k[2], k[3]), pack_bf16(k[4], k[5]), pack_bf16(k[6], k[7]));
    *reinterpret_cast<uint4*>(dv + out) = make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
}

}  // namespace

size_t bwd_row_tc_partial_bytes(const MonarchParams& mp, int g0, int g1) {
    const int rows_per_group = (mp.blk.b2 + 7) & ~7;
    const int gpt = kRows / rows_per_group;
    const int tiles = (mp.na + gpt - 1) / gpt;
    return tiles == 1 ? 0 : (size_t)tiles * mp.nbh * (size_t)(g1 - g0) * mp.blk.b1 * mp.blk.b2 * kHeadDim * sizeof(float);
}

// Row-step backward for one slice.  maps = {q, K, V} (the forward's).
int launch_bwd_row_tc(const MonarchParams& mp, const CUtensorMap* maps, const float* dcL, float* dq, float* part_k,
                      float* part_v, __nv_bfloat16* dk, __nv_bfloat16* dv, int g0, int g1, __nv_bfloat16* dq_bf16, int natural,
                      int* status, int num_sms, cudaStream_t s) {
    if (mp.blk.b2 > 64) return SFM_ERR_UNSUPPORTED;
    BwdRowParams rp;
    rp.mp = mp;
    rp.dcL = dcL; rp.dq = dq; rp.dq_bf16 = dq_bf16; rp.part_k = part_k; rp.part_v = part_v;
    rp.dk = dk; rp.dv = dv; rp.natural = natural;
    rp.g0 = g0; rp.g1 = g1;
    rp.rows_per_group = (mp.blk.b2 + 7) & ~7;
    rp.groups_per_tile = kRows / rp.rows_per_group;
    rp.tiles = (mp.na + rp.groups_per_tile - 1) / rp.groups_per_tile;
    rp.n_units = mp.nbh * rp.tiles * mp.blk.b1;
    // The tiles' room: with rows, keys and queries as wide as they are a third K tile fits in for block columns up to 56, and a
    // fourth daL / dY tile for some.
    rp.tile_rows = (rp.rows_per_group * rp.groups_per_tile + 15) & ~15;
    const int kv_tile = ((mp.blk.b2 + 15) & ~15) * 256, row_tile = rp.tile_rows * 256;
    rp.n_k = kRBTiles >= 4 * kv_tile + 2 * kStageT + 4 * row_tile ? 3 : 2;
    const int n_rt = (kRBTiles - (1 + rp.n_k) * kv_tile - 2 * kStageT) / row_tile - 1;
    rp.n_rt = n_rt < kRowSlots ? n_rt : kRowSlots;
    rp.status = status;
    dim3 grid(rp.n_units < num_sms ? rp.n_units : num_sms);
    const int n_s = (mp.blk.b2 + 15) & ~15;
    CUtensorMap bridge[2];
    if (int rc = make_bridge_tmap(&bridge[0], mp.aL, mp.blk.b2, mp.n_keys, mp.nbh * mp.na, rp.rows_per_group, 1)) return rc;
    if (int rc = make_bridge_tmap(&bridge[1], mp.Y, mp.blk.b2, mp.n_keys, mp.nbh * mp.na, rp.rows_per_group, 1)) return rc;
    auto go = [&](auto kernel) -> int {
        if (int rc = opt_in_smem((const void*)kernel, kRBSmem)) return rc;
        // Set up while the column step's backward drains, if that is short.  With the launches before and behind it and the status word's
        // clearing in the row step: training calls of 3 + 3 frames 280 -> 273 us, 2 of 6 frames 45 x 40 tokens 177 -> 173, 2 videos, 20 x 30
        // tokens, 9 frames 187.5 -> 184.3; 12 frames the same (640, with a long one's launch overlapped too 642).
        return launch_pdl((long long)rp.n_units * mp.F <= 32ll * num_sms, kernel, grid, kThreadsRB, kRBSmem, s, maps[0], maps[1], maps[2], bridge[0], bridge[1], rp);
    };
    int rc;
    {
        LaunchScope scope(kClsBackward, s);
        switch (n_s) {
            case 16: rc = rp.tiles == 1 ? go(monarch_bwd_row_tc_kernel<16, true>) : go(monarch_bwd_row_tc_kernel<16, false>); break;
            case 32: rc = rp.tiles == 1 ? go(monarch_bwd_row_tc_kernel<32, true>) : go(monarch_bwd_row_tc_kernel<32, false>); break;
            case 48: rc = rp.tiles == 1 ? go(monarch_bwd_row_tc_kernel<48, true>) : go(monarch_bwd_row_tc_kernel<48, false>); break;
            case 64: rc = rp.tiles == 1 ? go(monarch_bwd_row_tc_kernel<64, true>) : go(monarch_bwd_row_tc_kernel<64, false>); break;
            default: return SFM_ERR_UNSUPPORTED;
        }
        if (rc) return rc;
        if (cudaGetLastError() != cudaSuccess) return SFM_ERR_UNSUPPORTED;
    }
    if (g1 > g0 && rp.tiles > 1) {
        LaunchScope scope(kClsBackward, s);
        const int n_sel = (g1 - g0) * mp.blk.b1 * mp.blk.b2;
        MonarchParams m = mp;
        m.set_divs();
        const int blocks = (n_sel + 15) / 16;                        // of a pair
        if (int e = launch_pdl(true, bwd_merge_kv_kernel, dim3((unsigned)blocks * mp.nbh), 256, 0, s, (const float*)part_k, (const float*)part_v, dk, dv,
                               rp.tiles, n_sel, m, FastDiv::of(blocks), FastDiv::of(mp.blk.b1 * mp.blk.b2), natural))
            return e;
    }
    return SFM_OK;
}

}  // namespace sfm
