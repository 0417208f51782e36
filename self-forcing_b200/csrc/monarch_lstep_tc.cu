// Monarch column step on the 5th-generation tensor cores (tcgen05 + TMEM).
//
// One unit = (batch*head, query group a, column j): the b1 queries Q[a,:,j] attend the n_keys = F*b1 summary keys
// aL[a,f,j,k] (bias -cL, values Y) produced by the row step.  The MMA tile is 128 rows tall but a unit has only b1
// queries (30 at 480p framewise), so a CTA works on a GROUP of U = min(8, 128 / b1) consecutive units at once: query i of
// unit slot u sits on tile row u*R + i with R = 128 / U.  Keys stream through shared memory in tiles of KT <= 128 per unit:
//   S  = Q_tile aL_tile(u)^T        tcgen05.mma with a lane mask that only updates unit u's rows
//   P  = exp2(scale*S - cL - m)     one thread per tile row, running max / sum in registers
//   O += P Y_tile(u)                tcgen05.mma, A = P (bf16) from TMEM, same lane mask
// Key tiles alternate, across the groups too, between two softmax warpgroups with their own S/P buffer and accumulator
// (split-KV; a group of one tile leaves the other side to the next group); the
// epilogue warpgroup merges the two partial softmaxes, normalises and writes each row to natural token order with
// 32-byte stores (the inverse layout map is the store address).
//
// KT is the number of keys divided evenly over the tiles that 128-key tiles would take, so that short caches (90 keys per
// 3-frame chunk at framewise) load and multiply fewer padding keys, and the two rings hold as many tiles as fit.
//
// Warp roles (16 warps): 0 = bias slices and aL tiles, 3 = Y tiles, 1 = PV-GEMM issuer (owns the TMEM allocation), 2 = the
// groups' query rows and the S GEMMs, 4..7 / 8..11 = softmax warpgroups, 12..15 = epilogue warpgroup.  Roles 0 to 3 run as
// whole warps with an elected issuing lane.  With one buffer of query rows, warp 2 reloads it as soon as its last S GEMM
// of a group has completed, which the softmax and PV GEMMs of that group cover, while warp 0 is already loading the next
// group's keys; groups of few tiles or few units have two.  The code is kept small: a short launch fetches it from L2 or DRAM as it goes (a
// second copy of the query load cost the first chunk 2 us).  All roles meet only through mbarriers with bounded waits; a timeout
// records a status code and the CTA unwinds.
//
// What bounds it: reading the bridge (604 MB in 0.111 ms at framewise, 21 cached frames, 12 heads: 5.4 TB/s with the start-up
// and the uneven last round, 6.3 in between; a bare TMA stream of the same tiles reaches 6.5), and at short caches, whose
// bridge is in L2, the chain of a group (90 keys: 43 -> 29 us).  Against the form with queries spread over the four lane
// quadrants, MMAs issued from one-lane code, two softmax passes and a warpgroup chosen by tile parity within the group:
// a masked MMA took up to 165 cycles to issue, a query tile 32 boxes instead of 8, the bias reads met four-way bank
// conflicts, and groups of one tile ran one after another.  4 videos, reduce2xh, 9 frames: 0.503 -> 0.388 ms;
// reduce4xw2xh, 21 frames: 1.165 -> 1.008 ms.
//
// Arithmetic follows monarch_attn_ref_op (wan/modules/monarch_attn.py:1821-1829).
#include "monarch_params.cuh"
#include "profile.cuh"
#include "tc05.cuh"

namespace sfm {

using namespace tc;

namespace {

constexpr int kMaxStages = 8;              // tiles per ring, at most
constexpr int kThreads = 512;
constexpr int kKT = 128;                   // keys per tile, at most
constexpr int kMaxU = 8;                   // units per group (the bias ring is sized for it)
constexpr int kBiasPitch = kKT + 4;        // the rows of a warp may read two units' slices: different banks
constexpr uint32_t kTmemCols = 512;
// TMEM columns: S / P buffers of the two softmax warpgroups at 0 and 128, their accumulators at 256 and 384
__host__ __device__ constexpr uint32_t col_s(int w) { return (uint32_t)w * 128u; }
__host__ __device__ constexpr uint32_t col_o(int w) { return 256u + (uint32_t)w * 128u; }
constexpr float kRescaleThreshold = 40.0f; // log2 units: the reference of a row moves only past this growth

struct LTcParams {
    MonarchParams mp;
    int n_units;     // nbh * na * b2
    int U;           // units per group
    int R;           // tile rows per unit slot (128 / U, rounded down)
    int kt;          // keys per tile (multiple of 16, <= 128)
    int n_q, n_a, n_y;    // query tiles, tiles in the aL and Y rings
    int q_rows_tma;  // the query rows of a unit are consecutive rows of the token grid: load them with TMA
    int write_lse;   // also store the log-sum-exp of every query row (iterative variant, backward)
    int lse_only;    // nothing but that (no value tiles, no PV GEMMs, no output rows)
    int* status;
};

struct __align__(16) Barriers {
    alignas(16) float cl[4][kMaxU][kBiasPitch];   // bias slices, per unit slot: a ring of four tiles
    float stats[2][2][128];                // [warpgroup][m | l][tile row]
    uint64_t q_full[2], q_empty[2];
    uint64_t q_first;                      // the first group's query rows are there: once a launch
    uint64_t a_full[kMaxStages], a_empty[kMaxStages];
    uint64_t y_full[kMaxStages], y_empty[kMaxStages];
    uint64_t cl_full[4], cl_empty[4];
    uint64_t s_full[2], p_full[2], sp_free[2];
    uint64_t pv_done[2];                   // all PV GEMMs issued so far into accumulator w have completed
    uint64_t o_full[2];                    // by group parity
    uint64_t o_free[2];                    // accumulator and statistics of warpgroup w have been read
    uint32_t tmem_base;
    volatile int abort_flag;
};

constexpr int kQBytes = 2 * 128 * 128;     // query tile, two 64-column halves
constexpr int kTiles = 204 << 10;          // query tiles, aL tiles, Y tiles
constexpr int kSmemBytes = 1024 + kTiles + (int)sizeof(Barriers) + 64;
static_assert(kSmemBytes <= 227 * 1024, "shared memory");

__device__ __forceinline__ void st_global_v8(void* ptr, const uint32_t (&w)[8]) {
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(ptr), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]),
                 "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]) : "memory");
}

struct LUnit { int bhl, al, j; };
__device__ __forceinline__ LUnit decode_unit(const MonarchParams& p, int u) {
    LUnit r;
    u = p.by_b2.divmod(u, r.j);
    r.bhl = p.by_na.divmod(u, r.al);
    return r;
}

// tal / ty = bridge aL / Y maps [group][key][column][128] (box 64 x 1 column x kt keys), tqr = query rows (5-D, box b1 rows).
// kLarge: the bridge is much larger than L2 (MonarchParams::large_bridge).
template <bool kCausal, bool kLarge>
__global__ void __launch_bounds__(kThreads, 1)
monarch_l_tc_kernel(const __grid_constant__ CUtensorMap tal, const __grid_constant__ CUtensorMap ty,
                    const __grid_constant__ CUtensorMap tqr, LTcParams lp) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char* q_s = base;
    unsigned char* a_s = q_s + lp.n_q * kQBytes;
    unsigned char* y_s = a_s + lp.n_a * lp.kt * 256;
    Barriers* bars = reinterpret_cast<Barriers*>(base + kTiles);

    const MonarchParams& p = lp.mp;
    const Blocking& blk = p.blk;
    const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
    const int b1 = blk.b1, b2 = blk.b2, kt = lp.kt;
    const int U = lp.U, R = lp.R;
    const int half = kt * 128, tile_bytes = 2 * half;       // one 64-column half of a key or value tile, the whole tile
    // Keys a unit may see, and the tiles a group of units has to walk.  Block-causal (no-cache path): a unit sees the
    // cached groups up to the end of its own causal block; its tiles past that are neither loaded nor multiplied, and
    // the keys past it within its last tile get weight zero (the row step leaves finite values there).
    auto group_keys = [&](int al) -> int {                 // of query group al of the slice
        return kCausal ? min(p.F, ((p.a0 + al) / p.causal_groups + 1) * p.causal_groups) * b1 : p.n_keys;
    };
    // The units of a group belong to one query group or to two (U <= b2 if block-causal): the second from unit `split` on.
    // Worked out once per group: with four integer divisions per tile and unit in every role, a block-causal clip of 12 frames,
    // 12 heads took 267 us, without 214.
    struct GroupKeys { int first, second, split; __device__ __forceinline__ int of(int us) const { return us < split ? first : second; } };
    auto keys_of = [&](int u0) -> GroupKeys {
        if (!kCausal) return {p.n_keys, p.n_keys, kMaxU};
        int al;
        const int slab = p.by_b2.div(u0);
        p.by_na.divmod(slab, al);
        return {group_keys(al), group_keys(al + 1 == p.na ? 0 : al + 1), b2 - (u0 - slab * b2)};
    };
    auto group_tiles = [&](const GroupKeys& gk, int nu) -> int {
        return ((kCausal && gk.split < nu ? max(gk.first, gk.second) : gk.first) + kt - 1) / kt;
    };
    // This CTA's groups, of U consecutive units each: the grid goes through the unit list together, from its end, one group per
    // CTA a round, and the units left over are dealt out evenly.
    // Neighbouring columns, whose bridge rows are neighbours in memory, are then read at the same time, and what the row step
    // wrote last is read first, partly from L2: against a contiguous share per CTA the clip above went from 502 to 475 us, 40
    // heads with 21 frames from 1052 to 1030, 12 frames from 225 to 222.
    const int round = (int)gridDim.x * U, n_full = lp.n_units / round, rest = lp.n_units - n_full * round;
    const int rest0 = (int)((long long)rest * blockIdx.x / gridDim.x), rest1 = (int)((long long)rest * (blockIdx.x + 1) / gridDim.x);
    const int n_my = n_full + (rest1 > rest0 ? 1 : 0);
    auto group_at = [&](int gi, int& nu) -> int {          // first unit and number of units
        nu = gi < n_full ? U : rest1 - rest0;
        return gi < n_full ? lp.n_units - (gi + 1) * round + (int)blockIdx.x * U : rest0;
    };

    if (warp == 2 && lane == 0) { prefetch_tmap(&tqr); prefetch_tmap(&tal); prefetch_tmap(&ty); }
    if (tid == 0) {
        for (int s = 0; s < 2; ++s) { mbar_init(&bars->q_full[s], 1); mbar_init(&bars->q_empty[s], 1); }
        mbar_init(&bars->q_first, 1);
        for (int s = 0; s < kMaxStages; ++s) {
            mbar_init(&bars->a_full[s], 1); mbar_init(&bars->a_empty[s], 1);
            mbar_init(&bars->y_full[s], 1); mbar_init(&bars->y_empty[s], 1);
        }
        for (int s = 0; s < 4; ++s) { mbar_init(&bars->cl_full[s], 1); mbar_init(&bars->cl_empty[s], 128); }
        for (int w = 0; w < 2; ++w) {
            mbar_init(&bars->s_full[w], 1); mbar_init(&bars->p_full[w], 128); mbar_init(&bars->sp_free[w], 1);
            mbar_init(&bars->pv_done[w], 1); mbar_init(&bars->o_full[w], 1); mbar_init(&bars->o_free[w], 128);
        }
        bars->abort_flag = 0;
        mbar_init_fence();
    }
    // rows of the query tile that no unit writes must still hold finite numbers
    for (int i = tid; i < lp.n_q * kQBytes / 16; i += kThreads) reinterpret_cast<uint4*>(q_s)[i] = make_uint4(0, 0, 0, 0);
    if (warp == 1) { tmem_alloc(&bars->tmem_base, kTmemCols); tmem_relinquish(); }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = bars->tmem_base;
    // tile rows that belong to no unit, and columns past kt, are never written by a GEMM: give their logits a defined value
    if (warp >= 4 && warp < 12) {
        uint32_t z[32];
#pragma unroll
        for (int c = 0; c < 32; ++c) z[c] = 0u;
        const uint32_t s_t = tmem + ((uint32_t)((warp & 3) * 32) << 16) + col_s((warp - 4) >> 2);
#pragma unroll 1
        for (int c0 = 0; c0 < kKT; c0 += 32) tmem_st32(s_t + c0, z);
        tmem_wait_st();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_trigger();
    // The loading warps wait with their first load's coordinates in hand: parameters and instructions come from memory piece by
    // piece, at their first use, and the kernel before this one covers that (the first load went out 2200 cycles after the wait).
    if (warp != 0 && warp != 2 && warp != 3) pdl_wait();

    auto fail = [&](int code) {
        bars->abort_flag = 1;
        atomicCAS(lp.status, 0, code);
    };

    // query rows of a group
    auto load_q = [&](uint32_t el, int qb, int u0, int nu, bool first) {
        unsigned char* const qt = q_s + qb * kQBytes;
        if (lp.q_rows_tma) {
            // the 128-byte swizzle is a function of the shared-memory address, so a box may land on any tile row
            for (int us = 0; us < nu; ++us) {
                const LUnit un = decode_unit(p, u0 + us);
                int hd;
                const int b = p.by_H.divmod(p.bh0 + un.bhl, hd);
                int col;
                const int frow0 = p.first_row(un.al, un.j, col);
                unsigned char* dst = qt + us * R * 128;
                if (us == 0) {
                    if (first) { keep(b + hd + frow0 + col); pdl_wait(); }
                    mbar_arrive_expect_tx_e(el, &bars->q_full[qb], (uint32_t)(nu * b1 * 256));
                }
                tma_load_5d_e(el, dst, &tqr, &bars->q_full[qb], 0, hd, col, frow0, b);
                tma_load_5d_e(el, dst + 128 * 128, &tqr, &bars->q_full[qb], 64, hd, col, frow0, b);
            }
        } else {
            // query rows that are not consecutive rows of the token grid are gathered with plain loads
            if (first) pdl_wait();
            for (int us = 0; us < nu; ++us) {
                const LUnit un = decode_unit(p, u0 + us);
                int hd;
                const int b = p.by_H.divmod(p.bh0 + un.bhl, hd);
                const __nv_bfloat16* src = p.q + (long long)b * p.q_bs + (long long)hd * kHeadDim;
                for (int idx = lane; idx < b1 * 16; idx += 32) {
                    const int i = idx >> 4, ch = idx & 15;
                    const uint4 val = *reinterpret_cast<const uint4*>(
                        src + (long long)(blk.row_token(p.a0 + un.al, i) + un.j) * p.H * kHeadDim + ch * 8);
                    const int r = us * R + i;
                    *reinterpret_cast<uint4*>(qt + (ch >> 3) * (128 * 128) + r * 128 + (((ch & 7) ^ (r & 7)) << 4)) = val;
                }
            }
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars->q_full[qb]);
        }
    };

    if (warp == 0) {
        // ------------------------------------------------------------------ key tiles and bias slices
        const uint32_t el = elect_one();
        const uint64_t policy = kLarge ? l2_evict_first() : 0;
        int sa = 0, pa = 1, gt = 0;       // ring slots and their phases, tiles of all groups so far
        bool ok = true, waiting = true;
        for (int gi = 0; ok && gi < n_my; ++gi) {
            int nu;
            const int u0 = group_at(gi, nu);
            const GroupKeys gk = keys_of(u0);
            const int n_tiles = group_tiles(gk, nu);
            for (int t = 0; ok && t < n_tiles; ++t, ++gt) {
                for (int us = 0; us < nu; ++us) {
                    if (kCausal && t * kt >= gk.of(us)) continue;
                    if (!mbar_wait_u(&bars->a_empty[sa], pa)) { fail(11); ok = false; break; }
                    const LUnit un = decode_unit(p, u0 + us);
                    unsigned char* at = a_s + sa * tile_bytes;
                    if (waiting) { keep(un.j + un.al + un.bhl); pdl_wait(); waiting = false; }
                    mbar_arrive_expect_tx_e(el, &bars->a_full[sa], (uint32_t)tile_bytes);
                    tma_load_halves_e<kLarge>(el, at, half, &tal, &bars->a_full[sa], un.j, t * kt, un.bhl * p.na + un.al, policy);
                    if (++sa == lp.n_a) { sa = 0; pa ^= 1; }
                }
                if (!ok) break;
                const int cslot = gt & 3;
                if (!mbar_wait_u(&bars->cl_empty[cslot], ((gt >> 2) & 1) ^ 1)) { fail(13); ok = false; break; }
                const int have = min(kt, p.n_keys_c - t * kt);                  // floats that exist (multiple of 4)
                mbar_arrive_expect_tx_e(el, &bars->cl_full[cslot], (uint32_t)(nu * have * 4));
                for (int us = 0; us < nu; ++us)
                    bulk_load_e(el, bars->cl[cslot][us], p.cL + (long long)(u0 + us) * p.n_keys_c + t * kt, (uint32_t)(have * 4),
                                &bars->cl_full[cslot]);
            }
        }
    } else if (warp == 3) {
        // ------------------------------------------------------------------ value tiles
        if (!lp.lse_only) {
            const uint32_t el = elect_one();
            const uint64_t policy = kLarge ? l2_evict_first() : 0;
            int sy = 0, py = 1;
            bool ok = true, waiting = true;
            for (int gi = 0; ok && gi < n_my; ++gi) {
                int nu;
                const int u0 = group_at(gi, nu);
                const GroupKeys gk = keys_of(u0);
                const int n_tiles = group_tiles(gk, nu);
                for (int t = 0; ok && t < n_tiles; ++t)
                    for (int us = 0; us < nu; ++us) {
                        if (kCausal && t * kt >= gk.of(us)) continue;
                        if (!mbar_wait_u(&bars->y_empty[sy], py)) { fail(12); ok = false; break; }
                        const LUnit un = decode_unit(p, u0 + us);
                        unsigned char* yt = y_s + sy * tile_bytes;
                        if (waiting) {
                            // a launch's first value tiles go out behind its queries and keys, which are needed first (not by
                            // q_full: groups of one or two tiles fill it again without a value tile)
                            keep(un.j + un.al + un.bhl);
                            pdl_wait();
                            if (!mbar_wait_u(&bars->q_first, 0)) { fail(14); ok = false; break; }
                            waiting = false;
                        }
                        mbar_arrive_expect_tx_e(el, &bars->y_full[sy], (uint32_t)tile_bytes);
                        tma_load_halves_e<kLarge>(el, yt, half, &ty, &bars->y_full[sy], un.j, t * kt, un.bhl * p.na + un.al, policy);
                        if (++sy == lp.n_y) { sy = 0; py ^= 1; }
                    }
            }
        }
    } else if (warp == 2) {
        // ------------------------------------------------------------------ query rows, S GEMMs
        const uint32_t el = elect_one();
        const uint32_t idesc_s = idesc_bf16(128, 0, 0, 0) | ((uint32_t)(kt >> 3) << 17);
        const uint64_t q_desc = smem_desc_sw128(smem_addr(q_s), 16, 1024);
        const uint64_t a_desc0 = smem_desc_sw128(smem_addr(a_s), 16, 1024);
        int sa = 0, pa = 0, gt = 0;
        bool ok = true;
        // with two query tiles a group's rows are asked for before the GEMMs of the group before it, else after them
        const int lead = lp.n_q - 1;
        for (int x = 0; ok && x < n_my + lead; ++x) {
            int nu;
            if (x < n_my) {
                const int qb = x & lead, u0 = group_at(x, nu);
                if (!mbar_wait_u(&bars->q_empty[qb], ((x >> lead) & 1) ^ 1)) { fail(10); break; }
                load_q(el, qb, u0, nu, x == 0);
            }
            const int gi = x - lead;
            if (gi < 0) continue;
            const int qb = gi & lead, u0 = group_at(gi, nu);
            const GroupKeys gk = keys_of(u0);
            const int n_tiles = group_tiles(gk, nu);
            if (!mbar_wait_u(&bars->q_full[qb], (gi >> lead) & 1)) { fail(20); break; }
            if (gi == 0 && lane == 0) mbar_arrive(&bars->q_first);
            const uint64_t qd = q_desc + (uint64_t)((qb * kQBytes) >> 4);
            for (int t = 0; ok && t < n_tiles; ++t, ++gt) {
                const int w = gt & 1;
                if (!mbar_wait_u(&bars->sp_free[w], ((gt >> 1) & 1) ^ 1)) { fail(25); ok = false; break; }
                for (int us = 0; us < nu; ++us) {
                    if (kCausal && t * kt >= gk.of(us)) continue;
                    if (!mbar_wait_u(&bars->a_full[sa], pa)) { fail(21); ok = false; break; }
                    tc_fence_after();
                    const uint64_t ad = a_desc0 + (uint64_t)((sa * tile_bytes) >> 4);
                    const LaneMask m = lane_mask_rows(us * R, R);
#pragma unroll
                    for (int ks = 0; ks < 8; ++ks) {
                        const uint32_t qo = ((ks >> 2) * (128 * 128) + (ks & 3) * 32) >> 4;
                        const uint32_t ao = ((ks >> 2) * half + (ks & 3) * 32) >> 4;
                        mma_ss_masked_e(el, tmem + col_s(w), qd + qo, ad + ao, idesc_s, ks > 0, m);
                    }
                    mma_commit_e(el, &bars->a_empty[sa]);
                    if (++sa == lp.n_a) { sa = 0; pa ^= 1; }
                }
                if (!ok) break;
                mma_commit_e(el, &bars->s_full[w]);
            }
            if (!ok) break;
            mma_commit_e(el, &bars->q_empty[qb]);
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ PV-GEMM issuer
        const uint32_t el = elect_one();
        constexpr uint32_t idesc_o = idesc_bf16(128, kHeadDim, 0, 1);
        const uint64_t y_desc0 = smem_desc_sw128(smem_addr(y_s), half, 1024);
        const int n_k = kt / 16;
        int sy = 0, py = 0, gc = 0, gt = 0, used[2] = {0, 0};     // groups that accumulator w has taken part in
        bool ok = true;
        for (int gi = 0; ok && gi < n_my; ++gi, ++gc) {
            int nu;
            const int u0 = group_at(gi, nu);
            const GroupKeys gk = keys_of(u0);
            const int n_tiles = group_tiles(gk, nu);
            for (int t = 0; ok && t < n_tiles; ++t, ++gt) {
                const int w = gt & 1;
                if (!mbar_wait_u(&bars->p_full[w], (gt >> 1) & 1)) { fail(22); ok = false; break; }
                // first GEMM of the group into this accumulator overwrites it: the last result there must have been read
                if (t < 2 && !mbar_wait_u(&bars->o_free[w], (used[w]++ & 1) ^ 1)) { fail(23); ok = false; break; }
                for (int us = 0; us < nu && !lp.lse_only; ++us) {
                    if (kCausal && t * kt >= gk.of(us)) continue;
                    if (!mbar_wait_u(&bars->y_full[sy], py)) { fail(26); ok = false; break; }
                    tc_fence_after();
                    const uint64_t yd = y_desc0 + (uint64_t)((sy * tile_bytes) >> 4);
                    const LaneMask m = lane_mask_rows(us * R, R);
#pragma unroll
                    for (int kk = 0; kk < kKT / 16; ++kk)
                        if (kk < n_k)
                            mma_ts_masked_e(el, tmem + col_o(w), tmem + col_s(w) + kk * 8, yd + ((kk * 2048) >> 4), idesc_o,
                                            (t >= 2) || (kk > 0), m);
                    mma_commit_e(el, &bars->y_empty[sy]);
                    if (++sy == lp.n_y) { sy = 0; py ^= 1; }
                }
                if (!ok) break;
                mma_commit_e(el, &bars->pv_done[w]);
                mma_commit_e(el, &bars->sp_free[w]);
                if (t + 1 == n_tiles) mma_commit_e(el, &bars->o_full[gc & 1]);
            }
        }
    } else if (warp >= 4 && warp < 12) {
        // ------------------------------------------------------------------ softmax warpgroups
        const int w = (warp - 4) >> 2;
        const int quad = warp & 3;
        const int row = quad * 32 + lane;
        const int us = min(row / R, U - 1);                          // unit slot whose bias this tile row uses
        const uint32_t lane_sel = (uint32_t)(quad * 32) << 16;
        const uint32_t s_t = tmem + lane_sel + col_s(w);
        const uint32_t o_t = tmem + lane_sel + col_o(w);
        const float scale_l2 = p.scale * kLog2e;
        const uint64_t scale2 = f2_pack(scale_l2, scale_l2), nl2 = f2_pack(-kLog2e, -kLog2e);
        int gt0 = 0, used = 0;                // tiles of the groups before this one; groups this warpgroup has taken part in
        bool ok = true;
        for (int gi = 0; ok && gi < n_my && !bars->abort_flag; ++gi) {
            int nu;
            const int u0 = group_at(gi, nu);
            const GroupKeys gk = keys_of(u0);
            const int n_tiles = group_tiles(gk, nu);
            const int my_keys = us < nu ? gk.of(us) : p.n_keys;
            float m_run = -INFINITY, l_run = 0.f;
            int my_tiles = 0;
            for (int t = (gt0 & 1) ^ w; ok && t < n_tiles; t += 2) {
                const int gt = gt0 + t, idx = gt >> 1;
                const int lim = min(kt, my_keys - t * kt);           // keys of this tile that exist for this row
                if (!mbar_wait(&bars->s_full[w], idx & 1)) { fail(31); ok = false; break; }
                const int cslot = gt & 3;
                const float* cs = bars->cl[cslot][us];
                if (!mbar_wait(&bars->cl_full[cslot], (gt >> 2) & 1)) { fail(33); ok = false; break; }
                tc_fence_after();
                // One pass over the tile, 32 keys at a time, against a reference m that is the maximum of the first 32 keys the
                // row has seen: P is bf16 and the accumulators are fp32, so weights may exceed 1 without losing anything,
                // and m only has to move when a logit outgrows it by 2^kRescaleThreshold.  The loop is not unrolled: its
                // instructions are fetched from DRAM, behind the bridge traffic, each time the kernel starts.
                uint64_t sum2 = f2_pack(0.f, 0.f);
#pragma unroll 1
                for (int c0 = 0; c0 < kt; c0 += 32) {
                    uint64_t x[16];                                  // biased logits, log2 units: S * scale - log2(e) * cL
                    {
                        uint32_t r[32];
                        tmem_ld32(s_t + c0, r);
                        tmem_wait_ld();
#pragma unroll
                        for (int c = 0; c < 16; c += 2) {
                            const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(&cs[c0 + 2 * c]);
                            x[c] = f2_fma(f2_pack(__uint_as_float(r[2 * c]), __uint_as_float(r[2 * c + 1])), scale2, f2_mul(nl2, b.x));
                            x[c + 1] = f2_fma(f2_pack(__uint_as_float(r[2 * c + 2]), __uint_as_float(r[2 * c + 3])), scale2, f2_mul(nl2, b.y));
                        }
                    }
                    if (__any_sync(0xffffffffu, c0 + 32 > lim)) {     // keys that do not exist for this row
#pragma unroll
                        for (int c = 0; c < 16; ++c) {
                            float x0, x1;
                            f2_unpack(x[c], x0, x1);
                            x[c] = f2_pack(c0 + 2 * c < lim ? x0 : -INFINITY, c0 + 2 * c + 1 < lim ? x1 : -INFINITY);
                        }
                    }
                    float mx = -INFINITY;
#pragma unroll
                    for (int c = 0; c < 16; ++c) {
                        float x0, x1;
                        f2_unpack(x[c], x0, x1);
                        mx = max3(mx, x0, x1);
                    }
                    if (my_tiles == 0 && c0 == 0) {
                        m_run = mx;
                    } else if (__any_sync(0xffffffffu, mx > m_run + kRescaleThreshold)) {
                        // move the reference of the rows that need it: what they have summed up so far, the P of this
                        // tile's earlier keys and the accumulator are scaled down
                        float corr = 1.0f;
                        if (mx > m_run + kRescaleThreshold) {
                            corr = exp2f(m_run - mx);
                            m_run = mx;
                        }
                        l_run *= corr;
                        sum2 = f2_mul(sum2, f2_pack(corr, corr));
#pragma unroll 1
                        for (int e0 = 0; e0 < c0 >> 1; e0 += 16) {
                            uint32_t r[16];
                            tmem_ld16(s_t + e0, r);
                            tmem_wait_ld();
#pragma unroll
                            for (int c = 0; c < 16; ++c)
                                r[c] = pack_bf16_alu(__uint_as_float(r[c] << 16) * corr, __uint_as_float(r[c] & 0xffff0000u) * corr);
                            tmem_st16(s_t + e0, r);
                        }
                        if (my_tiles > 0) {
                            // the accumulator may only be touched once the previous GEMMs into it have finished
                            if (!mbar_wait(&bars->pv_done[w], (idx - 1) & 1)) { fail(32); ok = false; break; }
                            tc_fence_after();
#pragma unroll 1
                            for (int e0 = 0; e0 < kHeadDim; e0 += 16) {
                                uint32_t r[16];
                                tmem_ld16(o_t + e0, r);
                                tmem_wait_ld();
#pragma unroll
                                for (int c = 0; c < 16; ++c) r[c] = __float_as_uint(__uint_as_float(r[c]) * corr);
                                tmem_st16(o_t + e0, r);
                            }
                        }
                        tmem_wait_st();
                    }
                    // P = exp2(x - m) as packed bf16 over the S columns already consumed, and its (unrounded) sum
                    const float neg_m = m_run == -INFINITY ? 0.f : -m_run;
                    const uint64_t neg_m2 = f2_pack(neg_m, neg_m);
                    uint32_t pk[16];
#pragma unroll
                    for (int c = 0; c < 16; ++c) {
                        float d0, d1;
                        f2_unpack(f2_add(x[c], neg_m2), d0, d1);
                        const float e0 = exp2f(d0), e1 = exp2f(d1);
                        sum2 = f2_add(sum2, f2_pack(e0, e1));
                        pk[c] = pack_bf16_alu(e0, e1);
                    }
                    if (!lp.lse_only) tmem_st16(s_t + (c0 >> 1), pk);
                }
                if (!ok) break;
                tmem_wait_st();
                float lo, hi;
                f2_unpack(sum2, lo, hi);
                mbar_arrive(&bars->cl_empty[cslot]);
                l_run += lo + hi;
                ++my_tiles;
                if (t + 2 >= n_tiles) {                // this warpgroup's last tile of the group: publish (m, l)
                    // the last statistics there must have been consumed
                    if (!mbar_wait(&bars->o_free[w], (used++ & 1) ^ 1)) { fail(34); ok = false; break; }
                    bars->stats[w][0][row] = m_run;
                    bars->stats[w][1][row] = l_run;
                }
                tc_fence_before();
                mbar_arrive(&bars->p_full[w]);
            }
            gt0 += n_tiles;
        }
    } else if (warp >= 12) {
        // ------------------------------------------------------------------ epilogue warpgroup
        const int quad = warp & 3;
        const int row = quad * 32 + lane;
        const int us = row / R, i_row = row - us * R;                // unit slot and query index of this tile row
        const uint32_t lane_sel = (uint32_t)(quad * 32) << 16;
        int gc = 0, gt0 = 0;
        for (int gi = 0; gi < n_my && !bars->abort_flag; ++gi, ++gc) {
            int nu;
            const int u0 = group_at(gi, nu);
            const GroupKeys gk = keys_of(u0);
            const int n_tiles = group_tiles(gk, nu);
            if (!mbar_wait(&bars->o_full[gc & 1], (gc >> 1) & 1)) { fail(41); break; }
            tc_fence_after();
            // the group's first tile went to warpgroup w_a, its second, if any, to the other; a row without a weight there
            // takes nothing from it (its accumulator may never have been written)
            const int w_a = gt0 & 1, w_b = w_a ^ 1;
            gt0 += n_tiles;
            const float m0 = bars->stats[w_a][0][row], l0 = bars->stats[w_a][1][row];
            const float l1 = n_tiles > 1 ? bars->stats[w_b][1][row] : 0.f;
            const bool has1 = l1 > 0.f;
            const float m1 = has1 ? bars->stats[w_b][0][row] : -INFINITY;
            const float ms = fmaxf(m0, m1);
            const float w0 = exp2f(m0 - ms);
            const float w1 = has1 ? exp2f(m1 - ms) : 0.f;
            const float den = w0 * l0 + (has1 ? w1 * l1 : 0.f);
            const float inv = 1.0f / den;
            const bool row_ok = us < nu && i_row < b1;
            __nv_bfloat16* out_row = nullptr;
            if (row_ok) {
                const LUnit un = decode_unit(p, u0 + us);
                int hd;
                const int b = p.by_H.divmod(p.bh0 + un.bhl, hd);
                int col;
                const int frow = p.first_row(un.al, un.j, col) + p.row_ahead(i_row);
                out_row = p.out_row(b, frow * blk.w + col, hd);
                // iterative variant, backward: the softmax's log-sum-exp (natural log)
                if (lp.write_lse) p.lse[(long long)(u0 + us) * b1 + i_row] = (ms + log2f(den)) * 0.6931471805599453f;
            }
            const bool any1 = __any_sync(0xffffffffu, has1);
#pragma unroll 1
            for (int c0 = 0; c0 < kHeadDim; c0 += 32) {
                uint32_t ra[32], rb[32];
                if (!lp.lse_only) {
                    tmem_ld32(tmem + lane_sel + col_o(w_a) + c0, ra);
                    if (any1) tmem_ld32(tmem + lane_sel + col_o(w_b) + c0, rb);
                    tmem_wait_ld();
                }
                if (c0 + 32 == kHeadDim) {
                    tc_fence_before();
                    mbar_arrive(&bars->o_free[w_a]);          // accumulators and statistics are in registers
                    if (n_tiles > 1) mbar_arrive(&bars->o_free[w_b]);
                }
                if (row_ok && !lp.lse_only) {
#pragma unroll
                    for (int v8 = 0; v8 < 2; ++v8) {
                        uint32_t wv[8];
#pragma unroll
                        for (int e = 0; e < 8; ++e) {
                            const int c = v8 * 16 + 2 * e;
                            float x0 = __uint_as_float(ra[c]) * w0, x1 = __uint_as_float(ra[c + 1]) * w0;
                            if (has1) { x0 = fmaf(__uint_as_float(rb[c]), w1, x0); x1 = fmaf(__uint_as_float(rb[c + 1]), w1, x1); }
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

// Keys per tile of the column step: what 128-key tiles would take, divided evenly over them.  Block-causal units see 1, 2, ...
// causal blocks of keys, and the row step writes what the tiles that they reach hold: there the size that holds least, a
// tile counting as 8 keys more than it has (12 frames of 30 x 52 in blocks of three, 90 keys: 96 a tile instead of 128, 17 % less).
int l_tile_keys(const MonarchParams& p) {
    const int even = (p.n_keys + kKT - 1) / kKT;
    int best = (((p.n_keys + even - 1) / even) + 15) & ~15;
    if (p.causal_groups > 0) {
        long long least = 0;
        for (int kt = kKT; kt >= 64; kt -= 16) {
            long long held = 0;
            for (int keys = 0; keys < p.n_keys;) {
                keys = keys + p.causal_groups * p.blk.b1 < p.n_keys ? keys + p.causal_groups * p.blk.b1 : p.n_keys;
                const int tiles = (keys + kt - 1) / kt;
                held += (tiles * kt < p.n_keys ? tiles * kt : p.n_keys) + 8 * tiles;
            }
            if (kt == kKT || held < least) { least = held; best = kt; }
        }
    }
    return best;
}

// Launches the tensor-core column step for one chunk as a persistent grid.  map_qrows = query rows, 5-D, box of b1 rows.
int launch_l_step_tc(const MonarchParams& p, const CUtensorMap* map_qrows, int* status, int num_sms, cudaStream_t s, int write_lse) {
    LaunchScope scope(kClsLStep, s);
    LTcParams lp;
    lp.mp = p;
    lp.mp.set_divs();
    lp.n_units = p.nbh * p.na * p.blk.b2;
    // as many units per group as the tile holds, but no more than it takes to give every SM one: the units of a group
    // follow one another through the MMA pipe and the rings (two heads on a 6 x 8 grid: 18 -> 11 us)
    const int share = (lp.n_units + num_sms - 1) / num_sms;
    lp.U = 128 / p.blk.b1 < kMaxU ? 128 / p.blk.b1 : kMaxU;
    if (lp.U > share) lp.U = share;
    if (p.causal_groups > 0 && lp.U > p.blk.b2) lp.U = p.blk.b2;
    lp.R = 128 / lp.U;
    lp.kt = l_tile_keys(p);
    // A value tile stays until its softmax and GEMM are done, a key tile only until its GEMM: two slots of five for keys
    // Two query tiles where a group has few tiles, or few units: its rows take 2000 to 4000 cycles to arrive, which the GEMMs and
    // softmax of a longer group cover, whose rings need the room.  Calls with one and with two, by tiles times units a group: 4
    // (first chunk) 69.3 -> 68.5 us, 3 (tied3frame, 12 frames) 104.0 -> 101.7; 8 (two tiles, 6 frames, 5 and 12 heads) 58.7 -> 60.0 and
    // 110.2 -> 112.5; 24 (reduce2xh, 9 frames, 4 videos) 858 -> 873.  One or two units, any number of tiles: tied3frame, 18 and 21
    // frames 147.8 -> 142.8 and 160.6 -> 156.9, 45 x 80 tokens, 6 and 12 frames 190.3 -> 188.3 and 181.0 -> 178.4, 64 x 40 tokens, 12
    // frames 294.4 -> 290.1, 16 tiles (96 x 30, 120 x 20 tokens, 21 frames) the same.
    lp.n_q = lp.U <= 2 || lp.U * ((p.n_keys + lp.kt - 1) / lp.kt) <= 4 ? 2 : 1;
    const int slots = (kTiles - lp.n_q * kQBytes) / (lp.kt * 256);
    lp.n_a = (slots * 2 + 4) / 5 < kMaxStages ? (slots * 2 + 4) / 5 : kMaxStages;
    lp.n_y = slots - lp.n_a < kMaxStages ? slots - lp.n_a : kMaxStages;
    lp.status = status;
    // Query rows that are consecutive rows of the token grid come by TMA; other blockings are gathered by the warp.
    lp.q_rows_tma = (p.blk.f_tied == 1 || p.blk.h_reduce == 1) ? 1 : 0;
    lp.write_lse = write_lse != 0;
    lp.lse_only = write_lse == 2;
    CUtensorMap maps[2];
    if (int rc = make_bridge_tmap(&maps[0], p.aL, p.blk.b2, p.n_keys, p.nbh * p.na, 1, lp.kt)) return rc;
    if (int rc = make_bridge_tmap(&maps[1], p.Y, p.blk.b2, p.n_keys, p.nbh * p.na, 1, lp.kt)) return rc;
    const int n_groups = (lp.n_units + lp.U - 1) / lp.U;
    dim3 grid(n_groups < num_sms ? n_groups : num_sms);
    const bool large = p.large_bridge();
    auto kernel = p.causal_groups > 0 ? (large ? monarch_l_tc_kernel<true, true> : monarch_l_tc_kernel<true, false>)
                                      : (large ? monarch_l_tc_kernel<false, true> : monarch_l_tc_kernel<false, false>);
    if (int rc = opt_in_smem((const void*)kernel, kSmemBytes)) return rc;
    const bool is_short = (long long)n_groups * ((p.n_keys + lp.kt - 1) / lp.kt) <= 16ll * num_sms;
    return launch_pdl(is_short, kernel, grid, kThreads, kSmemBytes, s, maps[0], maps[1], *map_qrows, lp);
}

}  // namespace sfm
