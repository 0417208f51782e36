// Monarch row step on the 5th-generation tensor cores (tcgen05 + TMEM), fed by TMA.
//
// Work is cut into units (batch*head, tile of stacked query groups, block row k, range of cached
// groups f).  A tile stacks up to 128 query rows r = (query group a, column j) in four slots of 32, one for each warp of a
// warpgroup: a query group takes one slot for every 32 of its columns, and two groups share one if they have 16 or fewer.
// CTAs are persistent: each walks the unit list with a fixed stride and, for every (unit, f),
// computes per query row a complete softmax over the b2 keys of K[f,k,:]:
//   S  = Q_tile K[f,k]^T                 tcgen05.mma, both operands from shared memory (K-major)
//   P  = softmax rows of S (scaled)      one thread per row: tcgen05.ld, registers, tcgen05.st (bf16)
//   aL = P K[f,k], Y = P V[f,k]          one N=128 tcgen05.mma each per 16 keys, A = P from TMEM, B = the tile (MN-major)
//   cL = sum_l P ln P                    from the softmax registers
// and streams aL, Y (bf16) and cL to the chunk's bridge.
//
// Warp roles (20 warps): 0 = query and K tiles, 3 = V tiles (K tiles where there are none), 1 = issuer of the aL and Y GEMMs (owns the TMEM allocation), 2 =
// issuer of the S GEMMs (all four run as whole warps with an elected issuing lane), 4..7 and 8..11 = two softmax warpgroups
// that take even / odd steps (a warp reaches TMEM lane quadrant warp % 4), 12..15 and 16..19 = two epilogue warpgroups (aL /
// Y).  All roles run the same unit loop and meet only through mbarriers whose phases follow running step counters, so the
// pipeline keeps flowing across unit boundaries.  Every wait is bounded; on a timeout the CTA records a status code and
// unwinds.
//
// What bounds it: the bridge rows it writes, 512 bytes per (query row, cached group, block row).  An SM's TMA engine stores 29
// bytes a cycle at most (loads 82 with all SMs at it, 125 alone) and does one thing at a time, so a step of 104 rows takes 1840
// cycles for its stores and 210 for its K and V; at long caches DRAM takes 5.1 TB/s of stores and what is read beside them (a bare
// stream of the same boxes 6.4).  Written by the epilogue threads themselves, a row a lane or four rows an instruction, they go out
// slower (first chunk 33 -> 39 us), and K / V by cp.async instead do not help (31 -> 35).
// The epilogue's hand-over of an accumulator comes before its stores, aL and Y each have their own, and the working
// warpgroups have 104 registers instead of 96 (a few dozen spilled bytes a thread go through an L1 that is all shared memory:
// 160 -> 190 us), none of which is spilled in any instance (the loading warps of 18 instances spill one word).  framewise,
// 21 cached frames, 12 heads 0.167 -> 0.158 ms; reduce2xh, 9 frames, 4 videos 0.527 -> 0.490;
// reduce4xw2xh, 21 frames 1.15 -> 1.09; a pass of the iterative variant, first chunk, 31.7 -> 25.4 us.
// Tried and slower: results to TMA as 5-D boxes of both halves (158 -> 179 us), three staging buffers a warp (same), all
// columns to registers before the first is stored, two tiles' queries against one K / V tile, L2 prefetch of the K / V tiles.
//
// Arithmetic follows monarch_attn_ref_op (wan/modules/monarch_attn.py:1813-1823, 1828); the sqrt(s)
// scaling of q and k is folded into the softmax scale, so aL here is the reference's aL / sqrt(s).
#include "monarch_params.cuh"
#include "profile.cuh"
#include "tc05.cuh"

namespace sfm {

using namespace tc;

namespace {

constexpr int kKStages = 4, kVStages = 2;    // K and V tiles held, at most
constexpr int kThreads = 640;          // 20 warps, 96 registers a thread when launched
constexpr int kRegsIssue = 56, kRegsWork = 104;     // of the issuing warpgroup and of the four others, from there on
constexpr int kTileRows = 128;
constexpr int kMaxSBufs = 4;
constexpr int kMaxQBufs = 3;
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kColO = 256;        // two accumulators of 128 columns; the S/P buffers lie below them

// A query group of 65 to 96 columns takes three slots, so that tiles cut groups.
__host__ __device__ constexpr bool cuts_groups(int n_s) { return n_s == 80 || n_s == 96; }

// What loads of query rows bring: a group's rows, or a slot's and, in the second map, those of a group's last slot.
template <bool kCut>
struct QueryMaps { CUtensorMap m[kCut ? 2 : 1]; };

struct RTcParams {
    MonarchParams mp;
    int spg;               // slots per query group, 0: two groups in a slot
    int n_slots, tiles;    // slots and tiles per (batch*head) of the chunk
    int per_tile, more;    // tiles that cut groups: slots of each, tiles from the first on that have one more
    int n_whole;           // units that take all cached groups; of the others each is cut into
    int fsplit, f_per;     // fsplit units of f_per cached groups
    int n_units;           // of both kinds
    FastDiv by_fsplit, by_b1, by_tiles, by_spg, by_H;
    int col_kt;            // keys per tile of the column step (block-causal: it reads whole tiles)
    int* status;           // device status word (0 = ok)
    int clear_status;      // the call's first launch starts it from zero
};

struct RUnit {
    int bhl, slot0, ns, k, f_begin, n_it;
    int f_limit;          // block-causal: cached groups the tile may see
};

// First query group (of the chunk) and first column of a slot.
__device__ __forceinline__ int slot_group(const RTcParams& rp, int s, int& j0) {
    if (rp.spg == 0) { j0 = 0; return 2 * s; }
    int x;
    const int g = rp.by_spg.divmod(s, x);
    j0 = x * 32;
    return g;
}

template <bool kCausal, bool kCut>
__device__ __forceinline__ RUnit decode_unit(const RTcParams& rp, int u) {
    const MonarchParams& p = rp.mp;
    RUnit r;
    r.f_begin = 0;
    int f_end = p.F, tile;
    if (u >= rp.n_whole) {
        int fs;
        u = rp.n_whole + rp.by_fsplit.divmod(u - rp.n_whole, fs);
        r.f_begin = fs * rp.f_per;
        f_end = min(p.F, r.f_begin + rp.f_per);
    }
    u = rp.by_b1.divmod(u, r.k);
    r.bhl = rp.by_tiles.divmod(u, tile);
    // Groups of three slots are cut by tiles of four, the slots divided evenly over the tiles; with a tile for each group a quarter
    // of its rows stood empty (clip of 12 frames, 24 x 70 tokens, 6 heads 388 -> 317 us, this and the spills).  Tiles of fours
    // otherwise: even ones (3 + 3 for three groups of two slots) load their queries in more boxes (20 passes 805 -> 831 us).
    if constexpr (kCut) {
        r.slot0 = tile * rp.per_tile + min(tile, rp.more);
        r.ns = rp.per_tile + (tile < rp.more ? 1 : 0);
    } else {
        r.slot0 = 4 * tile;
        r.ns = min(4, rp.n_slots - r.slot0);
    }
    if (kCausal) {
        // block-causal (no-cache path): the tile's last query group sees the most; later groups f are skipped
        int j0;
        const int a_hi = p.a0 + min(slot_group(rp, r.slot0 + r.ns - 1, j0) + (rp.spg == 0 ? 1 : 0), p.na - 1);
        r.f_limit = min(p.F, (a_hi / p.causal_groups + 1) * p.causal_groups);
        f_end = min(f_end, r.f_limit);
    }
    r.n_it = max(0, f_end - r.f_begin);               // 0: nothing to do, every role skips the unit
    return r;
}

struct __align__(8) Barriers {
    uint64_t q_full[kMaxQBufs], q_empty[kMaxQBufs];   // query tiles in turn: one per unit, iterative variant: one per step
    uint64_t k_full[kKStages], k_empty[kKStages];
    uint64_t v_full[kVStages], v_empty[kVStages];
    uint64_t s_full[kMaxSBufs];
    uint64_t p_full[kMaxSBufs];
    uint64_t sp_free[kMaxSBufs];   // PV GEMM has consumed the P operand held in this S/P buffer
    uint64_t o_full[2], o_free[2];    // accumulator: aL / Y, or of the even / odd steps
    uint32_t tmem_base;
    volatile int abort_flag;
};

// shared memory carve-up (bytes from a 1024-aligned base)
constexpr int kQBytes = 2 * kTileRows * 128;               // two 64-column halves
constexpr int kOutBytes = 8 * 2 * 32 * 128;                        // result staging: 32 rows x 64 columns per epilogue warp
constexpr int kSmemData = 224 << 10;                       // query tiles | K / V ring | staging
constexpr int kSmemBytes = 1024 + kSmemData + 512;
static_assert(sizeof(Barriers) <= 512, "barriers follow the tiles");

// kIter: a pass of the iterative variant after the first one.  The query operand is no longer the chunk's q
// (one tile per unit) but the state aR[a,f,k,j,:] of the previous pass, which differs for every cached group f:
// one tile per STEP, loaded through `tq` = a 3-D map of aR ([bh*F*b1][na*b2][128]) into two or three buffers in
// turn, and every row's logits are divided by its cR (monarch_attn.py:1716-1719).
// kY: Y is wanted.  The passes of the iterative variant before the last need aL and cL only: their stages hold K alone, and
// the two epilogue warpgroups take whole steps in turn, each with a 128-column accumulator of its own.
// kLarge: the bridge is much larger than L2 (MonarchParams::large_bridge).
template <int N_S, bool kCausal, bool kIter, bool kY, bool kLarge>
__global__ void __launch_bounds__(kThreads, 1)
monarch_r_tc_kernel(const __grid_constant__ QueryMaps<cuts_groups(N_S)> tq, const __grid_constant__ CUtensorMap tk,
                    const __grid_constant__ CUtensorMap tv, const __grid_constant__ CUtensorMap tal,
                    const __grid_constant__ CUtensorMap ty, RTcParams rp) {
    static_assert(!(kIter || !kY) || (N_S <= 64 && !kCausal), "the iterative variant exists for block columns up to 64, no mask");
    extern __shared__ unsigned char smem_raw[];
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const MonarchParams& p = rp.mp;
    const Blocking& blk = p.blk;
    const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
    const int b1 = blk.b1, b2 = blk.b2;
    constexpr int kHalf = N_S * 128;                    // bytes of one 64-column half of a K or V tile
    // Block columns above 64 (wide grids): two S/P buffers, and the softmax walks its row in 32-column chunks (see below).
    constexpr bool kWide = N_S > 64;
    constexpr bool kCut = cuts_groups(N_S);
    constexpr int kTile = 2 * kHalf;                     // a K or V tile: two halves
    constexpr int kSBufs = kWide ? 2 : 4;
    constexpr uint32_t kSCols = kColO / kSBufs;          // TMEM columns per S/P buffer
    // A query tile per unit, or per step.
    constexpr int kQBufs = kWide ? 1 : (kIter && !kY ? 3 : 2);
    // A K tile stays from its S GEMM to its PV GEMM, two to three steps later, a V tile for its PV GEMM only.  21 frames, 12 heads,
    // 52 columns, K / V slots of 16 KB: 3 / 1 195 us, 3 / 2 162, 4 / 2 159, 4 / 4 162, 5 / 3 171: copies share the TMA engine
    // with the result stores, and those asked for earlier than needed hold them up.  Other slot sizes, whole calls with 3 / 2,
    // 4 / 2, 4 / 3 slots: 30 columns (8 KB), 3 frames 41, 38, 38 us; 32 columns, 21 frames 168, 168, 171; 46 columns (12 KB), 12
    // frames 165, 161, 158; 16 columns (4 KB), 40 heads, 3 frames 71, 64, 64, 21 frames 308, 305, 292.  Above 80 columns room for
    // two or three K slots is all there is (3 / 3 instead of 4 / 2 at 52: first chunk 62 -> 65, block-causal clip 470 -> 487).
    constexpr int kSlots = (kSmemData - kQBufs * kQBytes - kOutBytes) / kTile;
    constexpr int kVStg = kY ? kVStages : 0, kKStg = kSlots - kVStg < kKStages ? kSlots - kVStg : kKStages;
    static_assert(kKStg >= 2 && kQBufs <= kMaxQBufs, "K ring, query tiles");
    unsigned char* q_s = base;
    unsigned char* k_s = q_s + kQBufs * kQBytes;
    unsigned char* v_s = k_s + kKStg * kTile;
    unsigned char* o_s = v_s + kVStg * kTile;                // staging of the epilogue warps
    Barriers* bars = reinterpret_cast<Barriers*>(base + kSmemData);

    if (warp == 2 && lane == 0) { prefetch_tmap(tq.m); prefetch_tmap(&tq.m[kCut]); prefetch_tmap(&tk); prefetch_tmap(&tv); prefetch_tmap(&tal); prefetch_tmap(&ty); }
    if (tid == 0) {
        for (int s = 0; s < kQBufs; ++s) { mbar_init(&bars->q_full[s], 1); mbar_init(&bars->q_empty[s], 1); }
        for (int s = 0; s < kKStg; ++s) { mbar_init(&bars->k_full[s], 1); mbar_init(&bars->k_empty[s], 1); }
        for (int s = 0; s < kVStg; ++s) { mbar_init(&bars->v_full[s], 1); mbar_init(&bars->v_empty[s], 1); }
        for (int s = 0; s < kSBufs; ++s) { mbar_init(&bars->s_full[s], 1); mbar_init(&bars->p_full[s], 128); mbar_init(&bars->sp_free[s], 1); }
        for (int w = 0; w < 2; ++w) { mbar_init(&bars->o_full[w], 1); mbar_init(&bars->o_free[w], 128); }
        bars->abort_flag = 0;
        mbar_init_fence();
    }
    // The copies bring the b2 rows of a block and no more (64 for every 52 were 20 % of what the TMA engine loaded); the GEMMs
    // read N_S, with weight zero past b2: those rows must hold finite numbers.
    for (int i = tid; i < (kKStg + kVStg) * 2 * (N_S - b2) * 8; i += kThreads) {
        const int r = i >> 3, h = r / (N_S - b2);
        reinterpret_cast<uint4*>(k_s + h * kHalf + (b2 + r - h * (N_S - b2)) * 128)[i & 7] = make_uint4(0, 0, 0, 0);
    }
    fence_async_smem();
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
    if (warp != 0 && warp != 3) pdl_wait();              // the loading warps wait with their first load's coordinates in hand
    const int u_first = blockIdx.x, u_stride = gridDim.x;
    // First token of block row k of cached group f.  Keys in natural order are for the instances without a cache alone: the divisions
    // a step, and parameters of their own, cost the others 0.1 us a launch (20 passes 788 -> 792 us).
    auto kv_token = [&](int f, int k) -> int {
        if constexpr (!kCausal) return (f * b1 + k) * b2;
        if (!p.kv_natural) return (f * b1 + k) * b2;
        int col;
        const int row = p.first_row(f - p.a0, 0, col) + p.row_ahead(k);
        return row * blk.w + col;
    };
    auto load_k = [&](uint32_t el, int g, int hd, int tok, int b, uint64_t policy) -> bool {      // K tile of step g
        const int s = g % kKStg;
        if (g >= kKStg && !mbar_wait_u(&bars->k_empty[s], ((g / kKStg) - 1) & 1)) return false;
        mbar_arrive_expect_tx_e(el, &bars->k_full[s], (uint32_t)(2 * b2 * 128));
        tma_load_halves_e<kLarge>(el, k_s + s * kTile, kHalf, &tk, &bars->k_full[s], hd, tok, b, policy);
        return true;
    };

    // Each branch of a role takes its registers itself: where branches of both counts meet, the compiler has the smaller one.
    if (warp < 4) {
    reg_dec<kRegsIssue>();
    if (warp == 0) {
        // ------------------------------------------------------------------ query and K tiles
        {
            const uint32_t el = elect_one();
            const uint64_t policy = kLarge ? l2_evict_last() : 0;
            const int q_pitch = (rp.spg == 0 ? 16 : 32 * rp.spg) * 128;            // of a group's rows
            int g = 0, uc = 0;
            for (int u = u_first; u < rp.n_units && !bars->abort_flag; u += u_stride) {
                const RUnit un = decode_unit<kCausal, kCut>(rp, u);
                if (kCausal && un.n_it == 0) continue;
                int hd;
                const int b = rp.by_H.divmod(p.bh0 + un.bhl, hd);
                // loads of query rows: by whole groups, or slot by slot
                int j0;
                const int g_first = slot_group(rp, un.slot0, j0);
                const int n_q = kCut ? un.ns : (rp.spg == 0 ? min(2 * un.ns, p.na - g_first) : rp.by_spg.div(un.ns));
                for (int i = 0; i < un.n_it; ++i, ++g) {
                    const int tok = kv_token(un.f_begin + i, un.k);
                    if constexpr (kY && kQBufs == 1) {       // the one query tile may be in use for a while yet
                        if (g == 0) { keep(tok + hd + b); pdl_wait(); }
                        if (!load_k(el, g, hd, tok, b, policy)) { fail(11); break; }
                    }
                    if (kIter || i == 0) {
                        // the query tile: the unit's rows of q, or this step's state rows (a, j) of (f, k)
                        const int qc = kIter ? g : uc, qb = qc % kQBufs;
                        if (qc >= kQBufs && !mbar_wait_u(&bars->q_empty[qb], ((qc / kQBufs) - 1) & 1)) { fail(10); break; }
                        unsigned char* qd = q_s + qb * kQBytes;
                        int q_rows = n_q * b2;
                        if constexpr (kCut) {
                            q_rows = 0;
                            for (int x = 0; x < n_q; ++x) {
                                slot_group(rp, un.slot0 + x, j0);
                                q_rows += min(32, b2 - j0);
                            }
                        }
                        for (int x = 0; x < n_q; ++x, qd += kCut ? 32 * 128 : q_pitch) {
                            const CUtensorMap* m = tq.m;
                            int gr = g_first + x;
                            j0 = 0;
                            if constexpr (kCut) {
                                gr = slot_group(rp, un.slot0 + x, j0);
                                if (j0 == 64) m = &tq.m[1];
                            }
                            if (x == 0) {
                                if (g == 0) {
                                    // A launch's parameters and instructions come from memory piece by piece, at their first use: what
                                    // leads to the first load does so while the kernel before this one still runs.  With the wait
                                    // ahead of the roles the first load went out 2700 cycles after it, the queries another 700 later.
                                    keep((kIter ? 0 : blk.row_token(p.a0 + gr, un.k)) + j0 + hd + b + tok);
                                    pdl_wait();
                                    // no wait can run out before block 0 has started
                                    if (rp.clear_status && blockIdx.x == 0 && lane == 0) *rp.status = 0;
                                }
                                mbar_arrive_expect_tx_e(el, &bars->q_full[qb], (uint32_t)(q_rows * 256));
                            }
                            if constexpr (kIter) {
                                const int fk = (un.bhl * p.F + un.f_begin + i) * b1 + un.k;
                                tma_load_3d_e(el, qd, m, &bars->q_full[qb], 0, gr * b2 + j0, fk);
                                tma_load_3d_e(el, qd + kTileRows * 128, m, &bars->q_full[qb], 64, gr * b2 + j0, fk);
                            } else {
                                const int qtok = blk.row_token(p.a0 + gr, un.k) + j0;
                                tma_load_4d_e(el, qd, m, &bars->q_full[qb], 0, hd, qtok, b);
                                tma_load_4d_e(el, qd + kTileRows * 128, m, &bars->q_full[qb], 64, hd, qtok, b);
                            }
                        }
                    }
                    if constexpr (kY && kQBufs > 1)
                        if (!load_k(el, g, hd, tok, b, policy)) { fail(11); break; }
                }
                ++uc;
            }
        }
    } else if (warp == 3) {
        // ------------------------------------------------------------------ V tiles, or the K tiles if there are none
        {
            const uint32_t el = elect_one();
            const uint64_t policy = kLarge ? l2_evict_last() : 0;
            int g = 0;
            bool ok = true;
            for (int u = u_first; ok && u < rp.n_units && !bars->abort_flag; u += u_stride) {
                const RUnit un = decode_unit<kCausal, kCut>(rp, u);
                int hd;
                const int b = rp.by_H.divmod(p.bh0 + un.bhl, hd);
                for (int i = 0; i < un.n_it; ++i, ++g) {
                    const int tok = kv_token(un.f_begin + i, un.k);
                    if constexpr (kY) {
                        const int s = g % kVStages;
                        if (g >= kVStages && !mbar_wait_u(&bars->v_empty[s], ((g / kVStages) - 1) & 1)) { fail(12); ok = false; break; }
                        unsigned char* st = v_s + s * kTile;
                        if (g == 0) { keep(tok + hd + b); pdl_wait(); }
                        mbar_arrive_expect_tx_e(el, &bars->v_full[s], (uint32_t)(2 * b2 * 128));
                        tma_load_halves_e<kLarge>(el, st, kHalf, &tv, &bars->v_full[s], hd, tok, b, policy);
                    } else {
                        if (g == 0) { keep(tok + hd + b); pdl_wait(); }
                        if (!load_k(el, g, hd, tok, b, policy)) { fail(11); ok = false; break; }
                    }
                }
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
            const uint64_t k_desc0 = smem_desc_sw128(smem_addr(k_s), 16, 1024);
            int g = 0, uc = 0;
            bool ok = true;
            for (int u = u_first; ok && u < rp.n_units && !bars->abort_flag; u += u_stride) {
                const RUnit un = decode_unit<kCausal, kCut>(rp, u);
                if (kCausal && un.n_it == 0) continue;
                if constexpr (!kIter) {
                    if (!mbar_wait_u(&bars->q_full[uc % kQBufs], (uc / kQBufs) & 1)) { fail(20); break; }
                }
                for (int i = 0; i < un.n_it; ++i, ++g) {
                    const int s = g % kKStg, qb = (kIter ? g : uc) % kQBufs;
                    if constexpr (kIter) {
                        if (!mbar_wait_u(&bars->q_full[qb], (g / kQBufs) & 1)) { fail(20); ok = false; break; }
                    }
                    if (!mbar_wait_u(&bars->k_full[s], (g / kKStg) & 1)) { fail(21); ok = false; break; }
                    if (g >= kSBufs && !mbar_wait_u(&bars->sp_free[g % kSBufs], ((g / kSBufs) - 1) & 1)) { fail(25); ok = false; break; }
                    tc_fence_after();
                    const uint64_t kd = k_desc0 + (uint64_t)((s * kTile) >> 4);
                    const uint64_t qd = q_desc + (uint64_t)((qb * kQBytes) >> 4);
                    const uint32_t d = tmem + (g % kSBufs) * kSCols;
#pragma unroll
                    for (int ks = 0; ks < 8; ++ks) {
                        const uint32_t q_off = ((ks >> 2) * (kTileRows * 128) + (ks & 3) * 32) >> 4;
                        const uint32_t k_off = ((ks >> 2) * kHalf + (ks & 3) * 32) >> 4;
                        mma_ss_e(el, d, qd + q_off, kd + k_off, idesc_s, ks > 0);
                    }
                    mma_commit_e(el, &bars->s_full[g % kSBufs]);
                    if (kIter || i + 1 == un.n_it) mma_commit_e(el, &bars->q_empty[qb]);   // last read of the query tile
                }
                ++uc;
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ PV-GEMM issuer
        {
            const uint32_t el = elect_one();
            constexpr uint32_t idesc_o = idesc_bf16(kTileRows, kHeadDim, 0, 1);
            constexpr int ksteps_pv = N_S / 16;
            const uint64_t k_desc_mn0 = smem_desc_sw128(smem_addr(k_s), kHalf, 1024);     // column blocks: lo, hi
            const uint64_t v_desc_mn0 = smem_desc_sw128(smem_addr(v_s), kHalf, 1024);
            int g = 0;
            bool ok = true;
            for (int u = u_first; ok && u < rp.n_units && !bars->abort_flag; u += u_stride) {
                const RUnit un = decode_unit<kCausal, kCut>(rp, u);
                for (int i = 0; i < un.n_it; ++i, ++g) {
                    if (!mbar_wait_u(&bars->p_full[g % kSBufs], (g / kSBufs) & 1)) { fail(22); ok = false; break; }
                    const int ob = kY ? 0 : g & 1, og = kY ? g : g >> 1;         // accumulator, its uses before this one
                    if (og > 0 && !mbar_wait_u(&bars->o_free[ob], (og - 1) & 1)) { fail(23); ok = false; break; }
                    tc_fence_after();
                    const int s = g % kKStg;
                    const uint64_t kd = k_desc_mn0 + (uint64_t)((s * kTile) >> 4);
                    const uint32_t p_t = tmem + (g % kSBufs) * kSCols;
#pragma unroll
                    for (int kk = 0; kk < ksteps_pv; ++kk)
                        mma_ts_e(el, tmem + kColO + ob * kHeadDim, p_t + kk * 8, kd + ((kk * 2048) >> 4), idesc_o, kk > 0);
                    mma_commit_e(el, &bars->o_full[ob]);
                    mma_commit_e(el, &bars->k_empty[s]);
                    if constexpr (kY) {
                        const int sv = g % kVStages;
                        const uint64_t vd = v_desc_mn0 + (uint64_t)((sv * kTile) >> 4);
                        if (!mbar_wait_u(&bars->v_full[sv], (g / kVStages) & 1)) { fail(24); ok = false; break; }
                        if (g > 0 && !mbar_wait_u(&bars->o_free[1], (g - 1) & 1)) { fail(26); ok = false; break; }
                        tc_fence_after();
#pragma unroll
                        for (int kk = 0; kk < ksteps_pv; ++kk)
                            mma_ts_e(el, tmem + kColO + kHeadDim, p_t + kk * 8, vd + ((kk * 2048) >> 4), idesc_o, kk > 0);
                        mma_commit_e(el, &bars->o_full[1]);
                        mma_commit_e(el, &bars->v_empty[sv]);
                    }
                    mma_commit_e(el, &bars->sp_free[g % kSBufs]);
                }
            }
        }
    }
    } else if (warp < 12) {
        reg_inc<kRegsWork>();
        // ------------------------------------------------------------------ softmax warpgroups
        const int wg = (warp - 4) >> 2;                 // 0: even steps, 1: odd steps; the S / P buffers rotate over all steps
        const int quad = warp & 3;                      // TMEM lane quadrant this warp may access
        const float scale_l2 = p.mult0 * kLog2e;
        const uint32_t s_t0 = tmem + ((uint32_t)(quad * 32) << 16);
        int g = 0;
        bool ok = true;
        for (int u = u_first; ok && u < rp.n_units && !bars->abort_flag; u += u_stride) {
            const RUnit un = decode_unit<kCausal, kCut>(rp, u);
            const bool warp_active = quad < un.ns;
            int j;
            int gl = slot_group(rp, un.slot0 + quad, j);                // this row's query group and column
            if (rp.spg == 0) { gl += lane >> 4; j = lane & 15; } else { j += lane; }
            const bool row_ok = warp_active && gl < p.na && j < b2;
            const long long aj = ((long long)un.bhl * p.na + gl) * b2 + j;
            // block-causal: groups f this row's query group may not see get an infinite bias
            const int f_allowed = kCausal ? ((p.a0 + gl) / p.causal_groups + 1) * p.causal_groups : p.F;
            // iterative variant: this row's cR at the unit's first cached group
            const float* const cr = p.cR + (((long long)un.bhl * p.F + un.f_begin) * b1 + un.k) * (p.na * b2) + gl * b2 + j;
            for (int i = 0; i < un.n_it; ++i, ++g) {
                if ((g & 1) != wg) continue;
                float scale_row = scale_l2;
                if constexpr (kIter) {
                    // logits are divided by the row's cR of the previous pass (clamped as in the reference)
                    if (row_ok) scale_row = p.scale * kLog2e * fminf(1.0f / (cr[(long long)i * b1 * (p.na * b2)] + 1e-6f), 1e4f);
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
                        tmem_ld32(s_t + c0, r);           // the buffer has 128 columns, whatever lies past N_S is masked
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
    } else {
        reg_inc<kRegsWork>();
        // ------------------------------------------------------------------ epilogue warpgroups
        // with Y: 0 takes aL (columns 0..127 of the accumulator), 1 takes Y (128..255); without: even, odd steps
        const int which = (warp - 12) >> 2;
        const int quad = warp & 3;
        const uint32_t o_t = tmem + ((uint32_t)(quad * 32) << 16) + kColO + which * kHeadDim;
        const uint32_t el = elect_one();
        // This warp's staging, 128-byte swizzle: 32 tile rows x 64 columns, twice; with two groups in a slot, 16 x 64 twice for each.
        const bool pair = rp.spg == 0;
        unsigned char* const st = o_s + (warp - 12) * 8192;
        const int half_bytes = pair ? 2048 : 4096;
        unsigned char* const st_row = st + (pair ? (lane >> 4) * 4096 + (lane & 15) * 128 : lane * 128);
        const CUtensorMap* const om = kY && which ? &ty : &tal;
        uint64_t* const o_full = &bars->o_full[which];
        uint64_t* const o_free = &bars->o_free[which];
        int g = 0;
        bool ok = true;
        for (int u = u_first; ok && u < rp.n_units && !bars->abort_flag; u += u_stride) {
            const RUnit un = decode_unit<kCausal, kCut>(rp, u);
            const bool warp_active = quad < un.ns;
            int j0;
            const int gl0 = slot_group(rp, un.slot0 + quad, j0), n_box = pair && gl0 + 1 < p.na ? 2 : 1;
            for (int i = 0; ok && i < un.n_it; ++i, ++g) {
                if (!kY && (g & 1) != which) continue;
                if (!mbar_wait(o_full, (kY ? g : g >> 1) & 1)) { fail(41); ok = false; break; }
                tc_fence_after();
                const int key = (un.f_begin + i) * b1 + un.k;
                if (!warp_active) {
                    tc_fence_before();
                    mbar_arrive(o_free);
                    continue;
                }
                uint32_t ra[32], rb[32];
                // 64 columns from registers to this warp's staging rows
                auto put = [&](int h) {
#pragma unroll
                    for (int c = 0; c < 8; ++c) {
                        const uint32_t (&r)[32] = c < 4 ? ra : rb;
                        uint32_t w[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            w[e] = pack_bf16(__uint_as_float(r[(c & 3) * 8 + 2 * e]), __uint_as_float(r[(c & 3) * 8 + 2 * e + 1]));
                        *reinterpret_cast<uint4*>(st_row + h * half_bytes + ((c ^ (lane & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
                    }
                };
                tmem_ld32(o_t, ra);
                tmem_ld32(o_t + 32, rb);
                tma_store_wait_read_all();                     // the rows of the step before have been read
                __syncwarp();
                tmem_wait_ld();
                put(0);
                tmem_ld32(o_t + 64, ra);
                tmem_ld32(o_t + 96, rb);
                tmem_wait_ld();
                tc_fence_before();
                mbar_arrive(o_free);                           // accumulator may be overwritten from here on
                put(1);
                fence_async_smem();
                __syncwarp();
                for (int x = 0; x < n_box; ++x) {
                    tma_store_4d_e(el, om, st + x * 4096, 0, j0, key, un.bhl * p.na + gl0 + x);
                    tma_store_4d_e(el, om, st + x * 4096 + half_bytes, 64, j0, key, un.bhl * p.na + gl0 + x);
                }
                tma_store_commit();
            }
            if (kCausal && which == 1 && warp_active && un.n_it > 0 && un.f_begin + un.n_it == un.f_limit) {
                // The column step reads whole tiles of col_kt keys and gives the keys past the limit weight zero: their Y
                // rows must hold finite numbers.  The unit that computed the tile's last cached group writes them.
                const int gl = gl0 + (pair ? lane >> 4 : 0), j = pair ? lane & 15 : j0 + lane;
                const int end = min(p.n_keys, (un.f_limit * b1 + rp.col_kt - 1) / rp.col_kt * rp.col_kt);
                for (int key = un.f_limit * b1 + un.k; key < end; key += b1)
                    if (gl < p.na && j < b2) {
                        uint4* y = reinterpret_cast<uint4*>(p.Y + ((((long long)un.bhl * p.na + gl) * p.n_keys + key) * b2 + j) * kHeadDim);
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

// Columns of a query group that one load brings: all, unless tiles cut groups (three slots); then a slot's, and the last slot's.
int r_load_columns(int b2, bool last) { return b2 <= 64 || b2 > 96 ? b2 : (last ? b2 - 64 : 32); }

// Launches the tensor-core row step for one chunk as a persistent grid.  `status` is a device int the
// kernel sets on an internal timeout.
int l_tile_keys(const MonarchParams& p);

int launch_r_step_tc(const MonarchParams& p, const CUtensorMap* maps /* q (box of r_load_columns tokens) or the aR state, K, V */, int n_s, int* status,
                     int clear_status, int num_sms, cudaStream_t s) {
    LaunchScope scope(kClsRStep, s);
    RTcParams rp;
    rp.mp = p;
    if (p.kv_natural) rp.mp.set_divs();
    const int b2 = p.blk.b2;
    rp.spg = b2 <= 16 ? 0 : (b2 + 31) / 32;
    rp.col_kt = l_tile_keys(p);
    rp.n_slots = b2 <= 16 ? (p.na + 1) / 2 : p.na * rp.spg;
    rp.tiles = (rp.n_slots + 3) / 4;
    rp.per_tile = rp.n_slots / rp.tiles; rp.more = rp.n_slots % rp.tiles;
    const long long whole = (long long)p.nbh * rp.tiles * p.blk.b1;       // units, not cut
    {
        // Persistent CTAs take units round-robin, so a launch lasts as long as its fullest CTA.  Either all units are cut in the same
        // way, or only those past the last full round, whose steps then go to all CTAs: 40 heads, 21 frames 16 rounds of 21 steps and
        // one of 5 instead of 17 of 21 (963 -> 945 us a call); reduce4xw2xh, 21 frames 1830 -> 1785.  A unit costs its steps and one
        // and a half for the reload of its query tile.  Block-causal units differ in length anyway: cut all alike.
        long long best = -1;
        for (int full = 0; full < 2; ++full) {
            const long long rounds = full && p.causal_groups == 0 ? whole / num_sms : 0, rest = whole - rounds * num_sms;
            if (full && rounds == 0) break;                // as cut alike
            for (int fs = 1; fs <= p.F; ++fs) {
                const int per = (p.F + fs - 1) / fs, splits = (p.F + per - 1) / per;
                const long long cost = rounds * (2 * p.F + 3) + ((rest * splits + num_sms - 1) / num_sms) * (2 * per + 3);
                if (best < 0 || cost < best) { best = cost; rp.f_per = per; rp.fsplit = splits; rp.n_whole = (int)(rounds * num_sms); }
            }
        }
    }
    rp.n_units = rp.n_whole + (int)(whole - rp.n_whole) * rp.fsplit;
    rp.by_fsplit = FastDiv::of(rp.fsplit); rp.by_b1 = FastDiv::of(p.blk.b1); rp.by_spg = FastDiv::of(rp.spg ? rp.spg : 1);
    rp.by_tiles = FastDiv::of(rp.tiles); rp.by_H = FastDiv::of(p.H);
    rp.status = status;
    rp.clear_status = clear_status;
    dim3 grid(rp.n_units < num_sms ? rp.n_units : num_sms);
    const bool iter = p.use_aR != 0;
    if (iter && (n_s > 64 || p.causal_groups > 0)) return SFM_ERR_UNSUPPORTED;
    const int smem_bytes = kSmemBytes;
    // result stores: one box = the 128 channels of up to 32 columns of one key
    CUtensorMap out_maps[2];
    const int box_cols = b2 <= 16 ? 16 : 32;
    for (int i = 0; i < 2; ++i)
        if (int rc = make_bridge_tmap(&out_maps[i], i ? p.Y : p.aL, p.blk.b2, p.n_keys, p.nbh * p.na, box_cols, 1)) return rc;
    auto go = [&](auto kernel, auto q_maps) -> int {
        q_maps.m[0] = maps[0];
        if constexpr (sizeof(q_maps) > sizeof(CUtensorMap)) {
            const uint64_t row = (uint64_t)kHeadDim * 2;
            const uint64_t dims[4] = {(uint64_t)kHeadDim, (uint64_t)p.H, (uint64_t)p.n_q, (uint64_t)((p.bh0 + p.nbh - 1) / p.H + 1)};
            const uint64_t strides[3] = {row, row * p.H, (uint64_t)p.q_bs * 2};
            const uint32_t box[4] = {64, 1, (uint32_t)r_load_columns(b2, true), 1};
            if (int rc = make_tmap_bf16(&q_maps.m[1], p.q, 4, dims, strides, box)) return rc;
        }
        if (int rc = opt_in_smem((const void*)kernel, smem_bytes)) return rc;
        return launch_pdl(whole * p.F <= 32 * num_sms, kernel, grid, kThreads, smem_bytes, s, q_maps, maps[1], maps[2], out_maps[0],
                          out_maps[1], rp);
    };
    int rc;
    // Unmasked clips whose keys are in natural order take the block-causal instances, with one block: 3 videos, 12 heads, 3 frames in
    // three bands of rows 383 -> 355 us against copies in Monarch order, 5 heads, 4 frames in two bands 67.6 -> 61.2, 2 videos, 12
    // heads, 6 x 8 tokens 32 -> 26.
    const bool causal = p.causal_groups > 0 || p.kv_natural, large = p.large_bridge();
    if (causal && p.causal_groups == 0) rp.mp.causal_groups = p.A > p.F ? p.A : p.F;
#define SFM_R_GO(...) go(monarch_r_tc_kernel<__VA_ARGS__>, QueryMaps<cuts_groups(N)>())
    if (iter || !p.write_Y) {
        switch (n_s) {
#define SFM_R_CASE(n)                                                     \
    case n: {                                                             \
        constexpr int N = n;                                              \
        rc = !iter       ? SFM_R_GO(N, false, false, false, false)        \
             : p.write_Y ? SFM_R_GO(N, false, true, true, false)          \
                         : SFM_R_GO(N, false, true, false, false);        \
        break;                                                            \
    }
            SFM_R_CASE(16)
            SFM_R_CASE(32)
            SFM_R_CASE(48)
            SFM_R_CASE(64)
#undef SFM_R_CASE
            default: return SFM_ERR_UNSUPPORTED;
        }
    } else {
        switch (n_s) {
#define SFM_R_CASE(n)                                                                                       \
    case n: {                                                                                               \
        constexpr int N = n;                                                                                \
        rc = causal ? (large ? SFM_R_GO(N, true, false, true, true) : SFM_R_GO(N, true, false, true, false))    \
                    : (large ? SFM_R_GO(N, false, false, true, true) : SFM_R_GO(N, false, false, true, false)); \
        break;                                                                                              \
    }
            SFM_R_CASE(16)
            SFM_R_CASE(32)
            SFM_R_CASE(48)
            SFM_R_CASE(64)
            SFM_R_CASE(80)
            SFM_R_CASE(96)
            SFM_R_CASE(112)
            SFM_R_CASE(128)
#undef SFM_R_CASE
            default: return SFM_ERR_UNSUPPORTED;
        }
    }
#undef SFM_R_GO
    if (rc) return rc;
    return (int)cudaGetLastError();
}

}  // namespace sfm
