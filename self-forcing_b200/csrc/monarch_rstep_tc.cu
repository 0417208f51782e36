// Monarch row step on the 5th-generation tensor cores (tcgen05 + TMEM), fed by TMA.
//
// Work is cut into units (batch*head, tile of stacked query groups, block row k, range of cached
// groups f).  A tile stacks up to 128 query rows r = (query group a, column j); each group takes 16, 32, 64 or 128 tile
// rows, so that the 32 rows of an epilogue warp belong to one group (or are two whole groups of 16).
// CTAs are persistent: each walks the unit list with a fixed stride and, for every (unit, f),
// computes per query row a complete softmax over the b2 keys of K[f,k,:]:
//   S  = Q_tile K[f,k]^T                 tcgen05.mma, both operands from shared memory (K-major)
//   P  = softmax rows of S (scaled)      one thread per row: tcgen05.ld, registers, tcgen05.st (bf16)
//   [aL | Y] = P [K[f,k] | V[f,k]]       one N=256 tcgen05.mma per 16 keys, A = P from TMEM,
//                                        B = the K and V tiles side by side (MN-major)
//   cL = sum_l P ln P                    from the softmax registers
// and streams aL, Y (bf16) and cL to the chunk's bridge.
//
// Warp roles (19 warps): 0 = TMA producer, 1 = issuer of the [aL | Y] GEMMs (owns the TMEM allocation), 2 = issuer of the S
// GEMMs (all three run as whole warps with an elected issuing lane), 3..6 and 7..10 = two softmax warpgroups that take even
// / odd steps (a warp reaches TMEM lane quadrant warp % 4, and four consecutive warps cover all four), 11..14 and 15..18 =
// two epilogue warpgroups (aL half / Y half of the accumulator).  All roles run the same unit loop and meet only through
// mbarriers whose phases follow running step counters, so the pipeline keeps flowing across unit boundaries.  Every wait
// is bounded; on a timeout the CTA records a status code and unwinds.
//
// What bounds it: the bridge rows it writes, 512 bytes per (query row, cached group, block row).  Written by the epilogue
// threads themselves (one 256-byte row per lane in 32-byte pieces) they go out at 25-27 KB per us and SM, 3.8 TB/s in all,
// into L2 or DRAM alike; without the stores the same kernel takes a third to a half of the time.  So each epilogue warp packs
// 32 rows x 64 columns to bf16 into a swizzled 4 KB staging buffer (two, in turn) and one lane hands it to the TMA store
// engine.  With four S / P buffers in TMEM (the S GEMMs then run ahead of the softmax instead of waiting for the last P to
// be consumed), one query tile and four 32 KB K / V stages: framewise, 21 cached frames, 12 heads 0.188 -> 0.167 ms;
// reduce2xh, 9 frames, 4 videos 0.563 -> 0.500 ms; reduce4xw2xh, 21 frames 1.237 -> 1.135 ms (4.6 TB/s of DRAM traffic).
// Tried and slower: 16 epilogue warps with a register split by setmaxnreg, separate accumulator hand-overs for the two
// halves, one K / V tile for two query tiles, L2 prefetch of the K / V tiles.
//
// Arithmetic follows monarch_attn_ref_op (wan/modules/monarch_attn.py:1813-1823, 1828); the sqrt(s)
// scaling of q and k is folded into the softmax scale, so aL here is the reference's aL / sqrt(s).
#include "monarch_params.cuh"
#include "profile.cuh"
#include "tc05.cuh"

namespace sfm {

using namespace tc;

namespace {

constexpr int kStages = 8;            // K/V tile ring, at most
constexpr int kThreads = 608;          // 19 warps, 96 registers a thread
constexpr int kTileRows = 128;
constexpr int kMaxSBufs = 4;
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kColO = 256;        // O = [aL | Y], 256 columns; the S/P buffers lie below it

struct RTcParams {
    MonarchParams mp;
    int rows_per_group;    // b2 padded to 16, 32, 64 or 128: a warp's 32 tile rows belong to one group, or to two whole ones
    int groups_per_tile;   // 128 / rows_per_group
    int tiles;             // tiles per (batch*head) of the chunk
    int fsplit, f_per;     // split of the F loop over units
    int n_units;           // nbh * tiles * b1 * fsplit
    int col_kt;            // keys per tile of the column step (block-causal: it reads whole tiles)
    int* status;           // device status word (0 = ok)
    int clear_status;      // the call's first launch starts it from zero
};


struct RUnit {
    int bhl, tile, k, f_begin, n_it;
    int f_limit;          // block-causal: cached groups the tile may see
};

template <bool kCausal>
__device__ __forceinline__ RUnit decode_unit(const RTcParams& rp, int u) {
    const MonarchParams& p = rp.mp;
    RUnit r;
    int fs = u % rp.fsplit; u /= rp.fsplit;
    r.k = u % p.blk.b1; u /= p.blk.b1;
    r.tile = u % rp.tiles;
    r.bhl = u / rp.tiles;
    r.f_begin = fs * rp.f_per;
    int f_end = min(p.F, r.f_begin + rp.f_per);
    if (kCausal) {
        // block-causal (no-cache path): the tile's last query group sees the most; later groups f are skipped
        const int a_hi = p.a0 + min((r.tile + 1) * rp.groups_per_tile, p.na) - 1;
        r.f_limit = min(p.F, (a_hi / p.causal_groups + 1) * p.causal_groups);
        f_end = min(f_end, r.f_limit);
    }
    r.n_it = max(0, f_end - r.f_begin);               // 0: nothing to do, every role skips the unit
    return r;
}

struct __align__(8) Barriers {
    uint64_t q_full[2], q_empty[2];   // single pass: buffer 0, once per unit; iterative variant: one per step, alternating
    uint64_t kv_full[kStages];
    uint64_t kv_empty[kStages];
    uint64_t s_full[kMaxSBufs];
    uint64_t p_full[kMaxSBufs];
    uint64_t sp_free[kMaxSBufs];   // PV GEMM has consumed the P operand held in this S/P buffer
    uint64_t o_full;
    uint64_t o_free;
    uint32_t tmem_base;
    volatile int abort_flag;
};

// shared memory carve-up (bytes from a 1024-aligned base)
constexpr int kQBytes = 2 * kTileRows * 128;               // two 64-column halves
constexpr int kOutBytes = 8 * 2 * 32 * 128;                    // result staging: 32 rows x 64 columns per epilogue warp
constexpr int kSmemData = 224 << 10;                       // query tiles | K / V ring | staging
constexpr int kSmemBytes = 1024 + kSmemData + 512;
static_assert(sizeof(Barriers) <= 512, "barriers follow the tiles");

// kIter: a pass of the iterative variant after the first one.  The query operand is no longer the chunk's q
// (one tile per unit) but the state aR[a,f,k,j,:] of the previous pass, which differs for every cached group f:
// one tile per STEP, loaded through `tq` = a 3-D map of aR ([bh*F*b1][na*b2][128]) into two alternating
// buffers, and every row's logits are divided by its cR (monarch_attn.py:1716-1719).
template <int N_S, bool kCausal, bool kIter>
__global__ void __launch_bounds__(kThreads, 1)
monarch_r_tc_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk,
                    const __grid_constant__ CUtensorMap tv, const __grid_constant__ CUtensorMap tal,
                    const __grid_constant__ CUtensorMap ty, RTcParams rp) {
    static_assert(!kIter || (N_S <= 64 && !kCausal), "the iterative variant exists for block columns up to 64, no mask");
    extern __shared__ unsigned char smem_raw[];
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const MonarchParams& p = rp.mp;
    const Blocking& blk = p.blk;
    const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
    const int b1 = blk.b1, b2 = blk.b2;
    const int RG = rp.rows_per_group;
    constexpr int kHalf = N_S * 128;                    // bytes of one 64-column half of a K or V tile
    // Block columns above 64 (wide grids): 128-row K / V stages (two of them fit), S/P buffers and the
    // accumulator move up in TMEM, and the softmax walks its row in 32-column chunks (see below).
    constexpr bool kWide = N_S > 64;
    // a stage holds K lo, K hi, V lo, V hi of N_S rows each: 16 KB up to 32 block columns, 32 KB up to 64, 64 KB beyond
    constexpr int kStgBytes = kWide ? 65536 : (N_S <= 32 ? 16384 : 32768);
    constexpr int kSBufs = kWide ? 2 : 4;
    constexpr uint32_t kSCols = kColO / kSBufs;          // TMEM columns per S/P buffer
    constexpr int kQBufs = kIter ? 2 : 1;               // a query tile per unit, or per step
    constexpr int kStg = (kSmemData - kQBufs * kQBytes - kOutBytes) / kStgBytes;
    static_assert(kStg >= 2 && kStg <= kStages, "K / V ring");
    unsigned char* q_s = base;
    unsigned char* kv_s = q_s + kQBufs * kQBytes;
    unsigned char* o_s = kv_s + kStg * kStgBytes;            // two 4 KB staging buffers per epilogue warp
    Barriers* bars = reinterpret_cast<Barriers*>(base + kSmemData);

    if (warp == 2 && lane == 0) { prefetch_tmap(&tq); prefetch_tmap(&tk); prefetch_tmap(&tv); prefetch_tmap(&tal); prefetch_tmap(&ty); }
    if (tid == 0) {
        for (int s = 0; s < 2; ++s) { mbar_init(&bars->q_full[s], 1); mbar_init(&bars->q_empty[s], 1); }
        for (int s = 0; s < kStg; ++s) { mbar_init(&bars->kv_full[s], 1); mbar_init(&bars->kv_empty[s], 1); }
        for (int s = 0; s < kSBufs; ++s) { mbar_init(&bars->s_full[s], 1); mbar_init(&bars->p_full[s], 128); mbar_init(&bars->sp_free[s], 1); }
        mbar_init(&bars->o_full, 1);
        mbar_init(&bars->o_free, 256);
        bars->abort_flag = 0;
        mbar_init_fence();
    }
    if (warp == 1) { tmem_alloc(&bars->tmem_base, kTmemCols); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = bars->tmem_base;

    auto fail = [&](int code) {
        bars->abort_flag = 1;
        atomicCAS(rp.status, 0, code);
    };
    pdl_trigger();
    pdl_wait();
    // no wait can run out before block 0 has started
    if (rp.clear_status && blockIdx.x == 0 && tid == 0) *rp.status = 0;
    const int u_first = blockIdx.x, u_stride = gridDim.x;

    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer
        {
            const uint32_t el = elect_one();
            int g = 0, uc = 0;
            for (int u = u_first; u < rp.n_units && !bars->abort_flag; u += u_stride) {
                const RUnit un = decode_unit<kCausal>(rp, u);
                if (kCausal && un.n_it == 0) continue;
                const int bh = p.bh0 + un.bhl, b = bh / p.H, hd = bh - b * p.H;
                const int g_first = un.tile * rp.groups_per_tile;
                const int ng = min(rp.groups_per_tile, p.na - g_first);
                for (int i = 0; i < un.n_it; ++i, ++g) {
                    const int s = g % kStg;
                    if (g >= kStg && !mbar_wait_u(&bars->kv_empty[s], ((g / kStg) - 1) & 1)) { fail(11); break; }
                    const int tok = ((un.f_begin + i) * b1 + un.k) * b2;
                    unsigned char* st = kv_s + s * kStgBytes;
                    mbar_arrive_expect_tx_e(el, &bars->kv_full[s], (uint32_t)(4 * kHalf));
                    tma_load_4d_e(el, st, &tk, &bars->kv_full[s], 0, hd, tok, b);
                    tma_load_4d_e(el, st + kHalf, &tk, &bars->kv_full[s], 64, hd, tok, b);
                    tma_load_4d_e(el, st + 2 * kHalf, &tv, &bars->kv_full[s], 0, hd, tok, b);
                    tma_load_4d_e(el, st + 3 * kHalf, &tv, &bars->kv_full[s], 64, hd, tok, b);
                    if (!kIter && i > 0) continue;
                    // the query tile: the unit's rows of q, or this step's state rows (a, j) of (f, k), group by group
                    const int qc = kIter ? g : uc, qb = qc % kQBufs;
                    if (qc >= kQBufs && !mbar_wait_u(&bars->q_empty[qb], ((qc / kQBufs) - 1) & 1)) { fail(10); break; }
                    unsigned char* qd = q_s + qb * kQBytes;
                    mbar_arrive_expect_tx_e(el, &bars->q_full[qb], (uint32_t)(ng * b2 * 256));
                    for (int gi = 0; gi < ng; ++gi, qd += RG * 128) {
                        if constexpr (kIter) {
                            const int fk = (un.bhl * p.F + un.f_begin + i) * b1 + un.k;
                            tma_load_3d_e(el, qd, &tq, &bars->q_full[qb], 0, (g_first + gi) * b2, fk);
                            tma_load_3d_e(el, qd + kTileRows * 128, &tq, &bars->q_full[qb], 64, (g_first + gi) * b2, fk);
                        } else {
                            const int qtok = blk.row_token(p.a0 + g_first + gi, un.k);
                            tma_load_4d_e(el, qd, &tq, &bars->q_full[qb], 0, hd, qtok, b);
                            tma_load_4d_e(el, qd + kTileRows * 128, &tq, &bars->q_full[qb], 64, hd, qtok, b);
                        }
                    }
                }
                ++uc;
            }
        }
    } else if (warp == 2) {
        // ------------------------------------------------------------------ S-GEMM issuer
        {
            const uint32_t el = elect_one();
            constexpr uint32_t idesc_s = idesc_bf16(kTileRows, N_S, 0, 0);
            // Descriptors differ from step to step only in the start-address field (16-byte units
            // in the low word), so they are built once and advanced with integer adds.
            const uint64_t q_desc = smem_desc_sw128(smem_addr(q_s), 16, 1024);
            const uint64_t k_desc0 = smem_desc_sw128(smem_addr(kv_s), 16, 1024);
            int g = 0, uc = 0;
            bool ok = true;
            for (int u = u_first; ok && u < rp.n_units && !bars->abort_flag; u += u_stride) {
                const RUnit un = decode_unit<kCausal>(rp, u);
                if (kCausal && un.n_it == 0) continue;
                if constexpr (!kIter) {
                    if (!mbar_wait_u(&bars->q_full[0], uc & 1)) { fail(20); break; }
                }
                for (int i = 0; i < un.n_it; ++i, ++g) {
                    const int s = g % kStg;
                    if constexpr (kIter) {
                        if (!mbar_wait_u(&bars->q_full[g & 1], (g >> 1) & 1)) { fail(20); ok = false; break; }
                    }
                    if (!mbar_wait_u(&bars->kv_full[s], (g / kStg) & 1)) { fail(21); ok = false; break; }
                    if (g >= kSBufs && !mbar_wait_u(&bars->sp_free[g % kSBufs], ((g / kSBufs) - 1) & 1)) { fail(25); ok = false; break; }
                    tc_fence_after();
                    const uint64_t kd = k_desc0 + (uint64_t)((s * kStgBytes) >> 4);
                    const uint32_t d = tmem + (g % kSBufs) * kSCols;
#pragma unroll
                    for (int ks = 0; ks < 8; ++ks) {
                        const uint32_t q_off = ((ks >> 2) * (kTileRows * 128) + (ks & 3) * 32) >> 4;
                        const uint32_t k_off = ((ks >> 2) * kHalf + (ks & 3) * 32) >> 4;
                        mma_ss_e(el, d, q_desc + (uint32_t)(((kIter ? g & 1 : 0) * kQBytes) >> 4) + q_off, kd + k_off, idesc_s, ks > 0);
                    }
                    mma_commit_e(el, &bars->s_full[g % kSBufs]);
                    if constexpr (kIter) {
                        mma_commit_e(el, &bars->q_empty[g & 1]);                 // this step's query tile has been read
                    } else {
                        if (i + 1 == un.n_it) mma_commit_e(el, &bars->q_empty[0]);   // last read of this unit's Q tile
                    }
                }
                ++uc;
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ PV-GEMM issuer
        {
            const uint32_t el = elect_one();
            // [aL | Y] in one N = 256 GEMM; the passes of the iterative variant that only need aL and cL stop at N = 128
            const uint32_t idesc_o = p.write_Y ? idesc_bf16(kTileRows, 2 * kHeadDim, 0, 1) : idesc_bf16(kTileRows, kHeadDim, 0, 1);
            constexpr int ksteps_pv = N_S / 16;
            const uint64_t kv_desc_mn0 = smem_desc_sw128(smem_addr(kv_s), kHalf, 1024);   // 4 column blocks: K lo, K hi, V lo, V hi
            int g = 0;
            bool ok = true;
            for (int u = u_first; ok && u < rp.n_units && !bars->abort_flag; u += u_stride) {
                const RUnit un = decode_unit<kCausal>(rp, u);
                for (int i = 0; i < un.n_it; ++i, ++g) {
                    if (!mbar_wait_u(&bars->p_full[g % kSBufs], (g / kSBufs) & 1)) { fail(22); ok = false; break; }
                    if (g > 0 && !mbar_wait_u(&bars->o_free, (g - 1) & 1)) { fail(23); ok = false; break; }
                    tc_fence_after();
                    const int s = g % kStg;
                    const uint64_t bd = kv_desc_mn0 + (uint64_t)((s * kStgBytes) >> 4);
                    const uint32_t p_t = tmem + (g % kSBufs) * kSCols;
#pragma unroll
                    for (int kk = 0; kk < ksteps_pv; ++kk)
                        mma_ts_e(el, tmem + kColO, p_t + kk * 8, bd + ((kk * 2048) >> 4), idesc_o, kk > 0);
                    mma_commit_e(el, &bars->o_full);
                    mma_commit_e(el, &bars->kv_empty[s]);
                    mma_commit_e(el, &bars->sp_free[g % kSBufs]);
                }
            }
        }
    } else if (warp >= 3 && warp < 11) {
        // ------------------------------------------------------------------ softmax warpgroups
        const int wg = (warp - 3) >> 2;                 // 0: even steps, 1: odd steps; the S / P buffers rotate over all steps
        const int quad = warp & 3;                      // TMEM lane quadrant this warp may access
        const int row = quad * 32 + lane;               // tile row == TMEM lane
        const int gl = row / RG, j = row - gl * RG;
        const float scale_l2 = p.mult0 * kLog2e;
        const uint32_t s_t0 = tmem + ((uint32_t)(quad * 32) << 16);
        int g = 0;
        bool ok = true;
        for (int u = u_first; ok && u < rp.n_units && !bars->abort_flag; u += u_stride) {
            const RUnit un = decode_unit<kCausal>(rp, u);
            const int g_first = un.tile * rp.groups_per_tile;
            const int ng = min(rp.groups_per_tile, p.na - g_first);
            const bool warp_active = quad * 32 < ng * RG;
            const bool row_ok = gl < ng && j < b2;
            const long long aj = ((long long)un.bhl * p.na + g_first + gl) * b2 + j;
            // block-causal: groups f this row's query group may not see get an infinite bias
            const int f_allowed = kCausal ? ((p.a0 + g_first + gl) / p.causal_groups + 1) * p.causal_groups : p.F;
            for (int i = 0; i < un.n_it; ++i, ++g) {
                if ((g & 1) != wg) continue;
                float scale_row = scale_l2;
                if constexpr (kIter) {
                    // logits are divided by the row's cR of the previous pass (clamped as in the reference)
                    if (row_ok) {
                        const long long ci = (((long long)un.bhl * p.F + un.f_begin + i) * b1 + un.k) * (long long)(p.na * b2) +
                                             (long long)(g_first + gl) * b2 + j;
                        scale_row = p.scale * kLog2e * fminf(1.0f / (p.cR[ci] + 1e-6f), 1e4f);
                    }
                }
                const int sb = g % kSBufs;
                const uint32_t s_t = s_t0 + sb * kSCols;
                if (!mbar_wait(&bars->s_full[sb], (g / kSBufs) & 1)) { fail(31); ok = false; break; }
                tc_fence_after();
                if (warp_active) {
                    if constexpr (!kWide) {
                    uint32_t raw[N_S];
                    if constexpr (N_S == 64) {
                        tmem_ld32(s_t, *reinterpret_cast<uint32_t(*)[32]>(&raw[0]));
                        tmem_ld32(s_t + 32, *reinterpret_cast<uint32_t(*)[32]>(&raw[32]));
                    } else if constexpr (N_S == 32) {
                        tmem_ld32(s_t, *reinterpret_cast<uint32_t(*)[32]>(&raw[0]));
                    } else if constexpr (N_S == 48) {
                        tmem_ld32(s_t, *reinterpret_cast<uint32_t(*)[32]>(&raw[0]));
                        tmem_ld16(s_t + 32, *reinterpret_cast<uint32_t(*)[16]>(&raw[32]));
                    } else {
                        tmem_ld16(s_t, *reinterpret_cast<uint32_t(*)[16]>(&raw[0]));
                    }
                    tmem_wait_ld();
                    // only the last 16 columns can lie beyond b2
#pragma unroll
                    for (int c = N_S - 16; c < N_S; ++c)
                        if (c >= b2) raw[c] = 0xf149f2cau;   // -1e30: exp2 gives 0 and 0 * (finite) stays 0 below
                    float mx = -INFINITY;
#pragma unroll
                    for (int c = 0; c < N_S; c += 2) mx = max3(mx, __uint_as_float(raw[c]), __uint_as_float(raw[c + 1]));
                    const float neg_m = -mx * scale_row;
                    // two columns at a time on the packed fp32 pipe
                    const uint64_t scale2 = f2_pack(scale_row, scale_row), negm2 = f2_pack(neg_m, neg_m);
                    uint64_t z2 = f2_pack(0.f, 0.f), ent2 = z2;
                    uint64_t e2[N_S / 2];
#pragma unroll
                    for (int c = 0; c < N_S / 2; ++c) {
                        const uint64_t d2 = f2_fma(f2_pack(__uint_as_float(raw[2 * c]), __uint_as_float(raw[2 * c + 1])), scale2, negm2);
                        float d0, d1;                         // log2 units, <= 0 (about -1e29 if masked)
                        f2_unpack(d2, d0, d1);
                        e2[c] = f2_pack(exp2f(d0), exp2f(d1));
                        z2 = f2_add(z2, e2[c]);
                        ent2 = f2_fma(e2[c], d2, ent2);       // masked: 0 * (-1e29) = 0
                    }
                    float z, zh, ent, enth;
                    f2_unpack(z2, z, zh);
                    f2_unpack(ent2, ent, enth);
                    z += zh;
                    ent += enth;
                    const float inv_z = 1.0f / z;
                    const uint64_t invz2 = f2_pack(inv_z, inv_z);
                    uint32_t pk[N_S / 2];
#pragma unroll
                    for (int c = 0; c < N_S / 2; ++c) {
                        float p0, p1;
                        f2_unpack(f2_mul(e2[c], invz2), p0, p1);
                        pk[c] = pack_bf16_alu(p0, p1);
                    }
                    if constexpr (N_S == 64) {
                        tmem_st32(s_t, pk);
                    } else if constexpr (N_S == 32) {
                        tmem_st16(s_t, pk);
                    } else if constexpr (N_S == 48) {
                        tmem_st16(s_t, *reinterpret_cast<uint32_t(*)[16]>(&pk[0]));
                        uint32_t p2[16];
#pragma unroll
                        for (int c = 0; c < 16; ++c) p2[c] = c < 8 ? pk[16 + c] : 0u;
                        tmem_st16(s_t + 16, p2);
                    } else {
                        uint32_t p2[16];
#pragma unroll
                        for (int c = 0; c < 16; ++c) p2[c] = c < 8 ? pk[c] : 0u;
                        tmem_st16(s_t, p2);   // 8 packed columns are the operand; the other 8 lie inside the S buffer
                    }
                    tmem_wait_st();
                    if (row_ok) {
                        const int key = (un.f_begin + i) * b1 + un.k;
                        p.cL[aj * p.n_keys_c + key] =
                            (!kCausal || un.f_begin + i < f_allowed) ? 0.6931471805599453f * ent * inv_z - __logf(z) : INFINITY;
                    }
                    } else {
                    // Wide rows: three passes over the row in 32-column chunks read back from TMEM (maximum;
                    // sum and entropy; normalised P written over the S columns already consumed).
                    auto load_chunk = [&](int c0, uint32_t (&r)[32]) {
                        if (c0 + 32 <= N_S) {
                            tmem_ld32(s_t + c0, r);
                        } else {
                            tmem_ld16(s_t + c0, *reinterpret_cast<uint32_t(*)[16]>(&r[0]));
                        }
                        tmem_wait_ld();
#pragma unroll
                        for (int c = 0; c < 32; ++c)
                            if (c0 + c >= b2) r[c] = 0xf149f2cau;          // -1e30, as above
                    };
                    float mx = -INFINITY;
#pragma unroll 1
                    for (int c0 = 0; c0 < N_S; c0 += 32) {
                        uint32_t r[32];
                        load_chunk(c0, r);
#pragma unroll
                        for (int c = 0; c < 32; c += 2) mx = max3(mx, __uint_as_float(r[c]), __uint_as_float(r[c + 1]));
                    }
                    const float neg_m = -mx * scale_l2;
                    const uint64_t scale2 = f2_pack(scale_l2, scale_l2), negm2 = f2_pack(neg_m, neg_m);
                    uint64_t z2 = f2_pack(0.f, 0.f), ent2 = z2;
#pragma unroll 1
                    for (int c0 = 0; c0 < N_S; c0 += 32) {
                        uint32_t r[32];
                        load_chunk(c0, r);
#pragma unroll
                        for (int c = 0; c < 32; c += 2) {
                            const uint64_t d2 = f2_fma(f2_pack(__uint_as_float(r[c]), __uint_as_float(r[c + 1])), scale2, negm2);
                            float d0, d1;
                            f2_unpack(d2, d0, d1);
                            const uint64_t e2 = f2_pack(exp2f(d0), exp2f(d1));
                            z2 = f2_add(z2, e2);
                            ent2 = f2_fma(e2, d2, ent2);
                        }
                    }
                    float z, zh, ent, enth;
                    f2_unpack(z2, z, zh);
                    f2_unpack(ent2, ent, enth);
                    z += zh;
                    ent += enth;
                    const float inv_z = 1.0f / z;
                    const uint64_t invz2 = f2_pack(inv_z, inv_z);
#pragma unroll 1
                    for (int c0 = 0; c0 < N_S; c0 += 32) {
                        uint32_t r[32], pk[16];
                        load_chunk(c0, r);
#pragma unroll
                        for (int c = 0; c < 32; c += 2) {
                            float d0, d1, p0, p1;
                            f2_unpack(f2_fma(f2_pack(__uint_as_float(r[c]), __uint_as_float(r[c + 1])), scale2, negm2), d0, d1);
                            f2_unpack(f2_mul(f2_pack(exp2f(d0), exp2f(d1)), invz2), p0, p1);
                            pk[c >> 1] = pack_bf16_alu(p0, p1);
                        }
                        tmem_st16(s_t + (c0 >> 1), pk);
                    }
                    tmem_wait_st();
                    if (row_ok) {
                        const int key = (un.f_begin + i) * b1 + un.k;
                        p.cL[aj * p.n_keys_c + key] =
                            (!kCausal || un.f_begin + i < f_allowed) ? 0.6931471805599453f * ent * inv_z - __logf(z) : INFINITY;
                    }
                    }
                }
                tc_fence_before();
                mbar_arrive(&bars->p_full[sb]);
            }
        }
    } else if (warp >= 11) {
        // ------------------------------------------------------------------ epilogue warpgroups
        const int which = (warp - 11) >> 2;              // 0: aL (columns 0..127 of O), 1: Y (columns 128..255)
        const int quad = warp & 3;
        const int row = quad * 32 + lane;
        const uint32_t o_t = tmem + ((uint32_t)(quad * 32) << 16) + kColO + which * kHeadDim;
        const uint32_t el = elect_one();
        // this warp's staging: 32 tile rows x 64 columns, 128-byte swizzle; its rows of a group start at column j0
        unsigned char* const st = o_s + (warp - 11) * 8192;
        unsigned char* const st_row = st + lane * 128;
        const int gl0 = quad * 32 / RG, j0 = quad * 32 - gl0 * RG, n_box = RG == 16 ? 2 : 1;
        const CUtensorMap* const om = which ? &ty : &tal;
        int g = 0;
        bool ok = true;
        for (int u = u_first; ok && u < rp.n_units && !bars->abort_flag; u += u_stride) {
            const RUnit un = decode_unit<kCausal>(rp, u);
            const int g_first = un.tile * rp.groups_per_tile;
            const int ng = min(rp.groups_per_tile, p.na - g_first);
            const bool warp_active = quad * 32 < ng * RG;
            for (int i = 0; ok && i < un.n_it; ++i, ++g) {
                if (!mbar_wait(&bars->o_full, g & 1)) { fail(41); ok = false; break; }
                tc_fence_after();
                const int key = (un.f_begin + i) * b1 + un.k;
                const bool work = warp_active && (which == 0 || p.write_Y);
                if (!work) {
                    tc_fence_before();
                    mbar_arrive(&bars->o_free);
                    continue;
                }
                uint32_t ra[32], rb[32];
                // 64 columns from registers to this warp's staging rows, and on to the bridge
                auto put = [&](int h) {
                    tma_store_wait_read();                     // the previous box has been read
                    __syncwarp();
#pragma unroll
                    for (int c = 0; c < 8; ++c) {
                        const uint32_t (&r)[32] = c < 4 ? ra : rb;
                        uint32_t w[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            w[e] = pack_bf16(__uint_as_float(r[(c & 3) * 8 + 2 * e]), __uint_as_float(r[(c & 3) * 8 + 2 * e + 1]));
                        *reinterpret_cast<uint4*>(st_row + h * 4096 + ((c ^ (lane & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
                    }
                    fence_async_smem();
                    __syncwarp();
                    for (int x = 0; x < n_box; ++x)
                        if (gl0 + x < ng)
                            tma_store_4d_e(el, om, st + h * 4096 + x * 2048, h * 64, j0, key, un.bhl * p.na + g_first + gl0 + x);
                    tma_store_commit();
                };
                tmem_ld32(o_t, ra);
                tmem_ld32(o_t + 32, rb);
                tmem_wait_ld();
                put(0);
                tmem_ld32(o_t + 64, ra);
                tmem_ld32(o_t + 96, rb);
                tmem_wait_ld();
                tc_fence_before();
                mbar_arrive(&bars->o_free);                    // accumulator may be overwritten from here on
                put(1);
            }
            if (kCausal && which == 1 && warp_active && un.n_it > 0 && un.f_begin + un.n_it == un.f_limit) {
                // The column step reads whole tiles of col_kt keys and gives the keys past the limit weight zero: their Y
                // rows must hold finite numbers.  The unit that computed the tile's last cached group writes them.
                const int gl = row / RG, j = row - gl * RG;
                const int end = min(p.n_keys, (un.f_limit * b1 + rp.col_kt - 1) / rp.col_kt * rp.col_kt);
                for (int key = un.f_limit * b1 + un.k; key < end; key += b1)
                    if (gl < ng && j < b2) {
                        uint4* y = reinterpret_cast<uint4*>(p.Y + ((((long long)un.bhl * p.na + g_first + gl) * p.n_keys + key) * b2 + j) * kHeadDim);
                        for (int c = 0; c < kHeadDim / 8; ++c) y[c] = make_uint4(0, 0, 0, 0);
                    }
            }
        }
        tma_store_wait_all();
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, kTmemCols);
}

}  // namespace


// Launches the tensor-core row step for one chunk as a persistent grid.  `status` is a device int the
// kernel sets on an internal timeout.
int l_tile_keys(const MonarchParams& p);

int launch_r_step_tc(const MonarchParams& p, const CUtensorMap* maps /* q (or the aR state), k, v */, int n_s, int* status,
                     int clear_status, int num_sms, cudaStream_t s) {
    LaunchScope scope(kClsRStep, s);
    RTcParams rp;
    rp.mp = p;
    const int b2 = p.blk.b2;
    rp.rows_per_group = b2 <= 16 ? 16 : (b2 <= 32 ? 32 : (b2 <= 64 ? 64 : 128));
    rp.groups_per_tile = kTileRows / rp.rows_per_group;
    rp.col_kt = l_tile_keys(p);
    rp.tiles = (p.na + rp.groups_per_tile - 1) / rp.groups_per_tile;
    {
        // Persistent CTAs take whole units round-robin, so the launch lasts (units per CTA, rounded up) x (steps per
        // unit).  Pick the split of the F loop that makes that smallest, with one and a half steps charged per unit for the
        // reload of its query tile.
        long long best = -1;
        for (int fs = 1; fs <= p.F; ++fs) {
            const int per = (p.F + fs - 1) / fs, splits = (p.F + per - 1) / per;
            const long long units = (long long)p.nbh * rp.tiles * p.blk.b1 * splits;
            const long long cost = ((units + num_sms - 1) / num_sms) * (2 * per + 3);
            if (best < 0 || cost < best) { best = cost; rp.f_per = per; rp.fsplit = splits; }
        }
    }
    rp.n_units = p.nbh * rp.tiles * p.blk.b1 * rp.fsplit;
    rp.status = status;
    rp.clear_status = clear_status;
    dim3 grid(rp.n_units < num_sms ? rp.n_units : num_sms);
    const bool iter = p.use_aR != 0;
    if (iter && (n_s > 64 || p.causal_groups > 0)) return SFM_ERR_UNSUPPORTED;
    const int smem_bytes = kSmemBytes;
    // result stores: one box = 64 channels of up to 32 columns of one key
    CUtensorMap out_maps[2];
    for (int i = 0; i < 2; ++i)
        if (int rc = make_bridge_tmap(&out_maps[i], i ? p.Y : p.aL, p.blk.b2, p.n_keys, p.nbh * p.na, rp.rows_per_group < 32 ? rp.rows_per_group : 32, 1)) return rc;
    auto go = [&](auto kernel) -> int {
        if (int rc = opt_in_smem((const void*)kernel, smem_bytes)) return rc;
        return launch_pdl(rp.n_units * rp.f_per <= 32 * num_sms, kernel, grid, kThreads, smem_bytes, s, maps[0], maps[1], maps[2], out_maps[0], out_maps[1], rp);
    };
    int rc;
    const bool causal = p.causal_groups > 0;
    if (iter) {
        switch (n_s) {
            case 16: rc = go(monarch_r_tc_kernel<16, false, true>); break;
            case 32: rc = go(monarch_r_tc_kernel<32, false, true>); break;
            case 48: rc = go(monarch_r_tc_kernel<48, false, true>); break;
            case 64: rc = go(monarch_r_tc_kernel<64, false, true>); break;
            default: return SFM_ERR_UNSUPPORTED;
        }
    } else switch (n_s) {
        case 16: rc = causal ? go(monarch_r_tc_kernel<16, true, false>) : go(monarch_r_tc_kernel<16, false, false>); break;
        case 32: rc = causal ? go(monarch_r_tc_kernel<32, true, false>) : go(monarch_r_tc_kernel<32, false, false>); break;
        case 48: rc = causal ? go(monarch_r_tc_kernel<48, true, false>) : go(monarch_r_tc_kernel<48, false, false>); break;
        case 64: rc = causal ? go(monarch_r_tc_kernel<64, true, false>) : go(monarch_r_tc_kernel<64, false, false>); break;
        case 80: rc = causal ? go(monarch_r_tc_kernel<80, true, false>) : go(monarch_r_tc_kernel<80, false, false>); break;
        case 96: rc = causal ? go(monarch_r_tc_kernel<96, true, false>) : go(monarch_r_tc_kernel<96, false, false>); break;
        case 112: rc = causal ? go(monarch_r_tc_kernel<112, true, false>) : go(monarch_r_tc_kernel<112, false, false>); break;
        case 128: rc = causal ? go(monarch_r_tc_kernel<128, true, false>) : go(monarch_r_tc_kernel<128, false, false>); break;
        default: return SFM_ERR_UNSUPPORTED;
    }
    if (rc) return rc;
    return (int)cudaGetLastError();
}

}  // namespace sfm
