// dQ, dK, dV at D <= 32 (evo_bwd.cu has the interface, and what the dQ/dK/dV kernels share: transposed products, whole
// pairs or single segments, the drain of dQ).
//
//   warps 0-15 (compute)  group g = warp / 4 owns q columns 32g .. 32g+31 of the tile; groups 0 and 1 are the first half
//                         of the q columns, 2 and 3 the second, and a half has its own S', dP', bias and barriers
//   warps 16-19 (drain)   32 rows of dQ each, after a segment dK and dV as bf16 stores
//   warp 20 (producer)    TMA: per step Q, dO, the extra tile of the q rows, two halves of the pair-bias tile; per
//                         segment K, V and the extra tile of the kv rows
//   warps 21, 22, 23      MMA issuers: S'^T and dP'^T by halves; dV and dK by halves; dQ
//
// What bounded the kernel with one phase of sixteen warps a step was that they did the same thing at the same time: 128
// to 340 clocks of tensor-memory loads, 1024 of exponentials, 500 of stores, 200 to 300 for every barrier of 16 arrivals
// and the round trip to an issuer, one after another, 3300 clocks a step, and no unit busy for more than half of it.  So
//   - a half reads all of its S' and dP' at once and hands the columns back, so that the next step's are formed during
//     its arithmetic, and P and dS are complete in registers before they wait for the previous step's products;
//   - the halves run at their own pace;
//   - accumulator fragments (8 x 8 blocks, evo_ptx.cuh) take the bias transposed by ldmatrix: 4 loads a warp and step
//     instead of 32, each a 16-bit value, and a release of the bias that costs one word per load;
//   - dK takes dS^T from the dS tile in shared memory (40 clocks a block, where tensor memory had 16).  That frees the
//     columns of two more dQ accumulators: rows of up to 512 residues keep dQ in tensor memory, where 384 residues had
//     a scratch area, and the drain of the last kv tile (a bulk copy's completion, two fences and a read back per step)
//     was slower than the step;
//   - dK and dV are both read out before the first is packed and stored.
// Kernel alone: B=1, S=512, N=384, H=8 441 -> 349 us; S=384, N=384, H=4 177 -> 148; S=256, N=768, H=8 848 -> 765;
// S=256, N=512, H=8 387 -> 304; S=256, N=256, H=8 108 -> 96; S=200, N=200, H=4 48 -> 46; N = 128 the same (70).
//
// Tried, against 356 at the first shape then: two dS tiles (428: issuers and LSU then meet on shared memory more often, the
// matrix unit has its operands first and loads take five times as long); half-steps of all warps with the next one
// prefetched into registers (637: twice the barriers); one issuer for dV, dK and dQ (433); loops around the issuers'
// MMAs instead of straight code (404); the waits' slow path as it was (373: two halves at different places of the code
// compete for the instruction cache; with the short one 0.4 warps a scheduler wait for instructions per issue).
#pragma once

namespace evo {

// The walk of Segments one segment after another, without a division but where the pair changes.
template <int WALK>
struct SegmentWalk {
    int bs = 0, h = 0, j, pair;
    __device__ __forceinline__ SegmentWalk(const Segments<WALK>& s, int sg) { seek(s, sg); }
    __device__ __forceinline__ void seek(const Segments<WALK>& s, int sg) { s.decode(sg, bs, h, j); pair = bs * s.H + h; }
    __device__ __forceinline__ void next(const Segments<WALK>& s, int sg, const BwdParams& p) {     // to segment sg
        if (WALK == WALK_BOTH && sg == s.n_ws) { seek(s, sg); return; }
        int dp;
        if (s.whole(sg)) {
            dp = 0;
            if (++j == s.NT) { j = 0; dp = s.stride; }
        } else {
            j += p.seg_dj;
            dp = p.seg_dp;
            if (j >= s.NT) { j -= s.NT; ++dp; }
        }
        if (dp) {
            pair += dp;
            bs = pair / s.H;
            h = pair - bs * s.H;
        }
    }
};


struct BwdHalvesCfg {
    static constexpr int DH = 32;
    static constexpr int NG = 4;                       // compute groups
    static constexpr int NCW = 4 * NG;
    static constexpr int W_DRAIN = NCW, W_PROD = NCW + 4, W_MMA = NCW + 5;
    static constexpr int THREADS = (NCW + 8) * 32;
    // setmaxnreg budgets: the CTA's register pool is the launch count (the cap ptxas derives from the
    // launch bound) times the threads; an increase that the pool cannot satisfy blocks for ever
    static constexpr int REGS_LAUNCH = (65536 / THREADS) & ~7;
    static constexpr int REGS_COMPUTE = 88, REGS_OTHER = 48;       // drain warps: as launched
    static_assert((REGS_COMPUTE * NCW + (REGS_LAUNCH + REGS_OTHER) * 4) * 32 <= REGS_LAUNCH * THREADS, "register pool");
    static constexpr int QS = 3;                       // Q/dO stages
    static constexpr int NKV = 2;                      // K/V buffers
    static constexpr int NB = 4;                       // halves of bias tiles
    static constexpr int DQ_BUFS = 4;
    static constexpr uint32_t ROWT = RowTile<DH>::BYTES;
    static constexpr uint32_t ST_Q = 0, ST_DO = ROWT, ST_XQ = 2 * ROWT;
    static constexpr uint32_t STAGE_BYTES = 2 * ROWT + XT_BYTES;
    static constexpr uint32_t KV_K = 0, KV_V = ROWT, KV_XK = 2 * ROWT, KV_BYTES = 2 * ROWT + XT_BYTES;
    static constexpr uint32_t OFF_STAGE = 0;
    static constexpr uint32_t OFF_KV = OFF_STAGE + QS * STAGE_BYTES;
    static constexpr uint32_t OFF_BIAS = OFF_KV + NKV * KV_BYTES;
    static constexpr uint32_t OFF_DS = OFF_BIAS + NB * SQ_SUB_BYTES;
    // per drain warp: WSLOTS slots of [32 rows][32 fp32], for bulk copies of dQ, dK and dV
    static constexpr uint32_t WQ_BYTES = 32 * 32 * 4;
    static constexpr int WSLOTS = 2;
    static constexpr uint32_t OFF_WSTG = OFF_DS + SQ_BYTES;
    // constant extra tiles, above every tile that refers to the zero tile
    static constexpr uint32_t OFF_XDP = OFF_WSTG + 4 * WSLOTS * WQ_BYTES;            // row selector of -delta
    static constexpr uint32_t OFF_ZERO = OFF_XDP + XT_BYTES;
    static constexpr uint32_t OFF_BARS = OFF_ZERO + XT_BYTES;
    static constexpr uint32_t NUM_BARS = 2 * QS + 2 * NKV + 2 * NB + 2 * DQ_BUFS + 9;
    static constexpr uint32_t OFF_MISC = OFF_BARS + NUM_BARS * 8;
    static constexpr uint32_t SMEM_BYTES = OFF_MISC + 16 + 1024;            // + alignment slack
    static constexpr uint32_t TMEM_S = 0, TMEM_DP = 128, TMEM_P = 256;       // S', dP', P^T (bf16)
    static constexpr uint32_t TMEM_DQ = 320;                                // DQ_BUFS accumulators
    static constexpr uint32_t TMEM_DK = TMEM_DQ + DQ_BUFS * DH, TMEM_DV = TMEM_DK + DH;
    static_assert(TMEM_DV + DH <= BWD_TMEM_COLS, "tensor memory budget");
    static_assert(SMEM_BYTES <= 232448, "shared memory budget");
    static_assert(STAGE_BYTES % 1024 == 0 && KV_BYTES % 1024 == 0 && WQ_BYTES % 1024 == 0, "tile alignment");
};

template <int WALK, int DBIAS_HERE>
__global__ void __launch_bounds__(BwdHalvesCfg::THREADS, 1)
evo_bwd_halves_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
               const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_do,
               const __grid_constant__ CUtensorMap tm_bias, const __grid_constant__ CUtensorMap tm_dq,
               const __grid_constant__ CUtensorMap tm_dk, const __grid_constant__ CUtensorMap tm_dv,
               const __grid_constant__ CUtensorMap tm_acc, const BwdParams p) {
    using C = BwdHalvesCfg;
    constexpr int DH = C::DH;
    using RT = RowTile<DH>;
    using RD = RowDesc<DH>;
    constexpr int QS = C::QS, NKV = C::NKV, NB = C::NB, DQB = C::DQ_BUFS;

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::OFF_BARS);
    uint64_t* st_full = bars;                  // [QS]
    uint64_t* st_empty = st_full + QS;         // [QS]
    uint64_t* kv_full = st_empty + QS;         // [NKV]
    uint64_t* kv_empty = kv_full + NKV;        // [NKV]
    uint64_t* bias_full = kv_empty + NKV;      // [NB]
    uint64_t* bias_empty = bias_full + NB;     // [NB]
    uint64_t* dq_full = bias_empty + NB;       // [DQB]
    uint64_t* dq_free = dq_full + DQB;         // [DQB]
    uint64_t* ds_free = dq_free + DQB;         // P^T and the dS tile are consumed: dV, dK and dQ of the step are complete
    // by half of the q columns
    uint64_t* s_full = ds_free + 1;            // [2] S', dP' are complete
    uint64_t* s_free = s_full + 2;             // [2] ... and read
    uint64_t* ds_ready = s_free + 2;           // [2] P^T and dS are written
    uint64_t* dkv_full = ds_ready + 2;         // dK, dV of the segment are complete
    uint64_t* dkv_free = dkv_full + 1;         // ... and read out
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + C::OFF_MISC);
    volatile uint32_t* abort_flag = tmem_slot + 1;

    const int tid = threadIdx.x;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);      // uniform
    const int lane = tid & 31;
    const int NT = p.NT;
    WaitCtx wc{abort_flag, p.status};

    if (tid == 0) {
        *abort_flag = 0;
        tmem_slot[3] = 0;                      // the abort word of the waits before exit
        for (int i = 0; i < QS; ++i) { mbar_init(&st_full[i], 1); mbar_init(&st_empty[i], 1); }
        for (int i = 0; i < NKV; ++i) { mbar_init(&kv_full[i], 1); mbar_init(&kv_empty[i], 2); }
        for (int i = 0; i < NB; ++i) { mbar_init(&bias_full[i], 1); mbar_init(&bias_empty[i], C::NCW / 2); }
        for (int i = 0; i < DQB; ++i) { mbar_init(&dq_full[i], 1); mbar_init(&dq_free[i], 4); }
        mbar_init(ds_free, 2);
        for (int i = 0; i < 2; ++i) { mbar_init(&s_full[i], 1); mbar_init(&s_free[i], C::NCW / 2); mbar_init(&ds_ready[i], C::NCW / 2); }
        mbar_init(dkv_full, 1);
        mbar_init(dkv_free, 4);
        fence_mbar_init();
    }
    if (warp == C::W_MMA) {
        tmem_alloc(tmem_slot, BWD_TMEM_COLS);
        tmem_relinquish();
    }
    if (warp == C::W_PROD && lane == 0) {
        prefetch_tmap(&tm_q); prefetch_tmap(&tm_k); prefetch_tmap(&tm_v); prefetch_tmap(&tm_do);
        prefetch_tmap(&tm_bias); prefetch_tmap(&tm_dq); prefetch_tmap(&tm_dk); prefetch_tmap(&tm_dv);
        prefetch_tmap(&tm_acc);
    }
    // constant extra tiles: row n of the -delta selector is (0,0,0,0,1,1,0,0); the zero tile
    if (tid < 128) {
        *reinterpret_cast<uint4*>(smem + C::OFF_XDP + tid * 16) = make_uint4(0u, 0u, 0x3f803f80u, 0u);
        *reinterpret_cast<uint4*>(smem + C::OFF_ZERO + tid * 16) = make_uint4(0u, 0u, 0u, 0u);
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    const Segments<WALK> seg(p);
    const int n_segs = seg.n;
    const bool res_ok = NT <= DQB;       // dQ of a whole pair stays in tensor memory
    // dQ accumulators in order of use: one per step, or (resident) one per q tile of a pair
    auto dq_event = [&](bool resident, int sg, int j, int i) {
        return resident ? (sg - j) + i : sg * NT + i - (res_ok ? seg.n_ws * (NT - 1) : 0);
    };

    if (warp >= C::W_PROD) {
    reg_dec<C::REGS_OTHER>();
    if (warp == C::W_PROD) {
        // ------------------------------ producer ------------------------------
        bool ok = true;
        int gs = 0, n_st = 0, n_bias = 0, n_kv = 0;      // steps; loads issued
        SegmentWalk<WALK> at(seg, 0);
#pragma unroll 1
        for (int sg = 0; sg < n_segs && ok; ++sg) {
            if (sg > 0) at.next(seg, sg, p);
            const int bs = at.bs, h = at.h, j = at.j;
            const int b = bs / p.S;
            const __nv_bfloat16* xq = p.xq + (static_cast<size_t>(bs) * p.H + h) * p.NTP * 8;
            {
                const int kb = sg % NKV;
                if (sg >= NKV) ok = warp_all(mbar_wait(&kv_empty[kb], ((sg / NKV) - 1) & 1, wc, 0x40));
                if (!ok) break;
                if (elect_one()) {
                    uint8_t* kvb = smem + C::OFF_KV + kb * C::KV_BYTES;
                    mbar_arrive_expect_tx(&kv_full[kb], C::KV_BYTES);
                    tma_load_row_tile<DH>(kvb + C::KV_K, &tm_k, &kv_full[kb], h, j * TILE, bs);
                    tma_load_row_tile<DH>(kvb + C::KV_V, &tm_v, &kv_full[kb], h, j * TILE, bs);
                    bulk_load(kvb + C::KV_XK, p.xk + (static_cast<size_t>(bs) * p.NTP + j * TILE) * 8, XT_BYTES, &kv_full[kb]);
                }
                __syncwarp();
                ++n_kv;
            }
#pragma unroll 1
            for (int i = 0; i < NT && ok; ++i, ++gs) {
                const int st = gs % QS;
                uint8_t* sb = smem + C::OFF_STAGE + st * C::STAGE_BYTES;
                if (gs >= QS) ok = warp_all(mbar_wait(&st_empty[st], ((gs / QS) - 1) & 1, wc, 0x42));
                if (!ok) break;
                if (elect_one()) {
                    mbar_arrive_expect_tx(&st_full[st], C::STAGE_BYTES);
                    tma_load_row_tile<DH>(sb + C::ST_Q, &tm_q, &st_full[st], h, i * TILE, bs);
                    tma_load_row_tile<DH>(sb + C::ST_DO, &tm_do, &st_full[st], h, i * TILE, bs);
                    bulk_load(sb + C::ST_XQ, xq + static_cast<size_t>(i) * TILE * 8, XT_BYTES, &st_full[st]);
                }
                __syncwarp();
                ++n_st;
#pragma unroll 1
                for (int hf = 0; hf < 2 && ok; ++hf, ++n_bias) {
                    const int bb = n_bias % NB;
                    if (n_bias >= NB) ok = warp_all(mbar_wait(&bias_empty[bb], ((n_bias / NB) - 1) & 1, wc, 0x41));
                    if (!ok) break;
                    if (elect_one()) {
                        uint8_t* bt = smem + C::OFF_BIAS + bb * SQ_SUB_BYTES;
                        mbar_arrive_expect_tx(&bias_full[bb], SQ_SUB_BYTES);
                        tma_load_4d(bt, &tm_bias, &bias_full[bb], j * TILE, i * TILE + 64 * hf, h, b);
                        tma_load_4d(bt + SQ_SUB_BYTES / 2, &tm_bias, &bias_full[bb], j * TILE + 64, i * TILE + 64 * hf, h, b);
                    }
                    __syncwarp();
                }
            }
        }
        // the last loads have landed before the CTA exits, also if a wait gave up
        const WaitCtx dc{tmem_slot + 3, p.status};
        for (int k = (n_st > QS ? n_st - QS : 0); k < n_st; ++k) mbar_wait_landed(&st_full[k % QS], (k / QS) & 1, dc, 0x43);
        for (int k = (n_kv > NKV ? n_kv - NKV : 0); k < n_kv; ++k) mbar_wait_landed(&kv_full[k % NKV], (k / NKV) & 1, dc, 0x45);
        for (int k = (n_bias > NB ? n_bias - NB : 0); k < n_bias; ++k) mbar_wait_landed(&bias_full[k % NB], (k / NB) & 1, dc, 0x44);
    } else {
        // ------------------------------ mma issuers ------------------------------
        // Each warp runs its loop with all lanes (uniform control flow: operand descriptors stay in
        // uniform registers) and elects one lane to issue.
        constexpr uint32_t IDESC_SDP = make_idesc_bf16(128, 64, 0, 0);
        // N = the head-dim columns that hold data (the rest of a wider kernel's tile is zero fill)
        const uint32_t IDESC_DKV = make_idesc_bf16(128, 16 * p.KB, 0, 1);
        const uint32_t IDESC_DQ = make_idesc_bf16(128, 16 * p.KB, 1, 1);
        const uint32_t aSt = smem_u32(smem + C::OFF_STAGE), aKV = smem_u32(smem + C::OFF_KV);
        const uint32_t aZero = smem_u32(smem + C::OFF_ZERO);
        const int role = warp - C::W_MMA;          // 0: S/dP, 1: dV/dK, 2: dQ
        bool ok = true;
        int gs = 0;
#pragma unroll 1
        for (int sg = 0; sg < n_segs && ok; ++sg) {
            const int kb = sg % NKV;
            const uint32_t kvb = aKV + kb * C::KV_BYTES;
#pragma unroll 1
            for (int i = 0; i < NT && ok; ++i, ++gs) {
                const int st = gs % QS;
                const uint32_t sb = aSt + st * C::STAGE_BYTES;
                if (role == 0) {
                    ok = warp_all(mbar_wait(&st_full[st], (gs / QS) & 1, wc, 0x50));
                    if (ok && i == 0) ok = warp_all(mbar_wait(&kv_full[kb], (sg / NKV) & 1, wc, 0x51));
#pragma unroll
                    for (int t = 0; t < 4; ++t) {          // S', then dP' of one half, then of the other
                        const int hf = t >> 1, part = t & 1;
                        if (ok && gs > 0 && part == 0) ok = warp_all(mbar_wait(&s_free[hf], (gs - 1) & 1, wc, 0x52));
                        if (!ok) break;
                        tc_fence_after();
                        if (elect_one()) {
                            // K and V, and Q and dO, lie side by side
                            static_assert(C::KV_V == C::KV_K + C::ROWT && C::ST_DO == C::ST_Q + C::ROWT, "order of the tiles");
                            const uint32_t a_lo = RD::kmajor_lo(kvb + C::KV_K + part * C::ROWT);
                            const uint32_t b_lo = RD::kmajor_lo(sb + C::ST_Q + part * C::ROWT + hf * 64 * RT::ROW_BYTES);
                            const uint32_t d = tmem + C::TMEM_S + 128 * part + 64 * hf;
#pragma unroll
                            for (int kk = 0; kk < RT::KBLOCKS; ++kk)
                                if (kk < p.KB)      // the others are zero-filled blocks past the true head dim
                                    umma_ss(d, RD::kmajor(a_lo, kk), RD::kmajor(b_lo, kk), IDESC_SDP, kk > 0);
                            // the extra contraction block: + (mask - LSE) / scale, - delta
                            umma_ss(d, xt_desc(part ? smem_u32(smem + C::OFF_XDP) : kvb + C::KV_XK, aZero),
                                    xt_desc(sb + C::ST_XQ + hf * 64 * 16, aZero), IDESC_SDP, 1u);
                            if (part) umma_commit(&s_full[hf]);
                        }
                        __syncwarp();
                    }
                } else if (role == 1) {
                    // the first MMA of a segment overwrites dK / dV: the previous one's must be out
                    if (i == 0 && sg > 0) ok = warp_all(mbar_wait(dkv_free, (sg - 1) & 1, wc, 0x55));
#pragma unroll 1
                    for (int hf = 0; hf < 2; ++hf) {
                        if (ok) ok = warp_all(mbar_wait(&ds_ready[hf], gs & 1, wc, 0x5a));
                        if (!ok) break;
                        tc_fence_after();
                        if (elect_one()) {
                            const uint32_t row0 = hf * 64 * RT::ROW_BYTES;
                            const uint32_t do_lo = RD::mnmajor_lo(sb + C::ST_DO + row0), q_lo = RD::mnmajor_lo(sb + C::ST_Q + row0);
                            const uint32_t ds_lo = SqDesc::kmajor_lo(smem_u32(smem + C::OFF_DS) + hf * SQ_SUB_BYTES);
                            const uint32_t t_p = tmem + C::TMEM_P + 32 * hf, acc = (hf > 0 || i > 0) ? 1u : 0u;
#pragma unroll
                            for (int kk = 0; kk < 4; ++kk)
                                umma_ts(tmem + C::TMEM_DV, t_p + 8 * kk, RD::mnmajor(do_lo, kk), IDESC_DKV, kk > 0 ? 1u : acc);
#pragma unroll
                            for (int kk = 0; kk < 4; ++kk)
                                umma_ss(tmem + C::TMEM_DK, SqDesc::kmajor(ds_lo, kk), RD::mnmajor(q_lo, kk), IDESC_DKV, kk > 0 ? 1u : acc);
                            if (hf == 1) {
                                umma_commit(ds_free);
                                umma_commit(&st_empty[st]);
                                if (i == NT - 1) {
                                    umma_commit(dkv_full);
                                    umma_commit(&kv_empty[kb]);
                                }
                            }
                        }
                        __syncwarp();
                    }
                } else {
                    const bool whole = seg.whole(sg), resident = whole && res_ok;
                    const int j = whole ? sg % NT : 0, ev = dq_event(resident, sg, j, i);
                    if (ev >= DQB && !(resident && j > 0)) ok = warp_all(mbar_wait(&dq_free[ev % DQB], ((ev / DQB) - 1) & 1, wc, 0x54));
                    if (ok) ok = warp_all(mbar_wait_both(&ds_ready[0], gs & 1, &ds_ready[1], gs & 1, wc, 0x5b));
                    if (!ok) break;
                    tc_fence_after();
                    if (elect_one()) {
                        const uint32_t ds_lo = SqDesc::mnmajor_lo(smem_u32(smem + C::OFF_DS));
                        const uint32_t k_lo = RD::mnmajor_lo(kvb + C::KV_K);
                        const uint32_t t_dq = tmem + C::TMEM_DQ + (ev % DQB) * DH;
                        const uint32_t acc = (resident && j > 0) ? 1u : 0u;
#pragma unroll
                        for (int kk = 0; kk < 8; ++kk)
                            umma_ss(t_dq, SqDesc::mnmajor(ds_lo, kk), RD::mnmajor(k_lo, kk), IDESC_DQ, kk > 0 ? 1u : acc);
                        umma_commit(ds_free);
                        if (!resident || j == NT - 1) umma_commit(&dq_full[ev % DQB]);
                        if (i == NT - 1) umma_commit(&kv_empty[kb]);
                    }
                    __syncwarp();
                }
            }
        }
    }
    } else if (warp >= C::W_DRAIN) {
        // ------------------------------ drain warps ------------------------------
        // (The loops over DH / 32 run once.  Written without them the mixed walk spills in other places, and is slower with
        // one S row: B=38, N=392, H=8 83 -> 89 us.)
        const int w4 = warp & 3;
        const int wrow0 = w4 * 32;           // tensor-memory lanes (tile rows) of this warp
        const uint32_t lane_base = tmem + (static_cast<uint32_t>(wrow0) << 16);
        uint8_t* const wslot = smem + C::OFF_WSTG + w4 * C::WSLOTS * C::WQ_BYTES;
        // where the next bulk copy (one group each) is staged: two slots in turn, once the copy before last has read its own
        int pos = 0;
        auto next_slot = [&]() -> uint8_t* {
            if (lane == 0) tma_wait_group_read<1>();
            __syncwarp();
            pos ^= 1;
            return wslot + pos * C::WQ_BYTES;
        };
        // 32 columns of 32 rows as bf16, by a bulk tensor store (which clips rows past N and columns past Dt)
        auto store_rows = [&](const CUtensorMap* tm, const uint4 (&u)[4], int h, int row0, int col0, int bs) {
            uint8_t* sl = next_slot();
#pragma unroll
            for (int c = 0; c < 4; ++c) *reinterpret_cast<uint4*>(sl + swz_off<64>(lane, c)) = u[c];
            fence_async_smem();
            __syncwarp();
            if (lane == 0) {
                tma_store_4d(tm, sl, col0, h, row0, bs);
                tma_commit_group();
            }
        };
        auto pack_rows = [](uint4 (&u)[4], const float (&v)[32], float sc) {
#pragma unroll
            for (int c8 = 0; c8 < 4; ++c8)
                u[c8] = make_uint4(pack_bf16(v[c8 * 8 + 0] * sc, v[c8 * 8 + 1] * sc), pack_bf16(v[c8 * 8 + 2] * sc, v[c8 * 8 + 3] * sc),
                                   pack_bf16(v[c8 * 8 + 4] * sc, v[c8 * 8 + 5] * sc), pack_bf16(v[c8 * 8 + 6] * sc, v[c8 * 8 + 7] * sc));
        };
        // whole pairs: the partial sums of this CTA, in units of 4 KB: 32 rows x 32 columns as [16-byte word][row]
        float4* part = reinterpret_cast<float4*>(p.dq_scratch) + static_cast<size_t>(blockIdx.x) * p.scratch_stride;
        bool ok = true;
        auto drain = [&](auto whole_c, int sg0, int sg1) {
            constexpr bool whole = decltype(whole_c)::value;
            if (sg0 >= sg1) return;
            SegmentWalk<WALK> at(seg, sg0);
#pragma unroll 1
            for (int sg = sg0; sg < sg1 && ok; ++sg) {
                if (sg > sg0) at.next(seg, sg, p);
                const int bs = at.bs, h = at.h, j = at.j;
                const bool resident = whole && res_ok;
#pragma unroll 1
                for (int i = 0; i < NT && ok; ++i) {
                    if (resident && j < NT - 1) break;             // dQ is still being summed
                    const int ev = dq_event(resident, sg, j, i), b = ev % DQB;
                    const bool rows = i * TILE + wrow0 < p.N;     // warp-uniform: some row of this warp exists
                    const bool final_sum = whole && j == NT - 1, add = final_sum && j > 0 && !resident && rows;
                    float4* ps = part + static_cast<size_t>(i * 4 + w4) * (DH / 4) * 32;
                    float4 old[8];
                    // The bulk copy that last wrote this part of the scratch area, a segment ago, is complete
                    // before the sum is added to or read: two or more were issued after it (NT > DQB).
                    if (whole && j > 0 && !resident) {
                        if (lane == 0) tma_wait_group<2>();
                        if (add) fence_async_all();
                        __syncwarp();
                    }
                    ok = warp_all(mbar_wait(&dq_full[b], (ev / DQB) & 1, wc, 0x68));
                    if (!ok) break;
                    tc_fence_after();
#pragma unroll
                    for (int rd = 0; rd < DH / 32; ++rd) {
                        float dqv[32];
                        tmem_ld_f32<32>(lane_base + C::TMEM_DQ + b * DH + rd * 32, dqv);
                        if (rd == DH / 32 - 1) {
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0) mbar_arrive(&dq_free[b]);
                        }
                        if (!rows || rd * 32 >= p.Dt) continue;    // warp-uniform
                        if (final_sum) {
                            if (add) {
#pragma unroll
                                for (int c = 0; c < 8; ++c) old[c] = __ldcg(ps + (rd * 8 + c) * 32 + lane);
#pragma unroll
                                for (int c = 0; c < 8; ++c) {
                                    dqv[4 * c] += old[c].x; dqv[4 * c + 1] += old[c].y;
                                    dqv[4 * c + 2] += old[c].z; dqv[4 * c + 3] += old[c].w;
                                }
                            }
                            uint4 u[4];
                            pack_rows(u, dqv, p.scale);
                            store_rows(&tm_dq, u, h, i * TILE + wrow0, rd * 32, bs);
                            continue;
                        }
                        uint8_t* wq = next_slot();
                        const float sc = whole ? 1.0f : p.scale;
#pragma unroll
                        for (int c = 0; c < 8; ++c)
                            *reinterpret_cast<float4*>(wq + (whole ? (c * 32 + lane) * 16 : swz_off<128>(lane, c))) =
                                make_float4(dqv[c * 4 + 0] * sc, dqv[c * 4 + 1] * sc, dqv[c * 4 + 2] * sc, dqv[c * 4 + 3] * sc);
                        fence_async_smem();
                        __syncwarp();
                        if (lane == 0) {
                            if (!whole)
                                tma_reduce_add_4d(&tm_acc, wq, rd * 32, h, i * TILE + wrow0, bs - p.acc_row0);
                            else if (j == 0)
                                bulk_store(ps + rd * 8 * 32, wq, C::WQ_BYTES);
                            else
                                bulk_reduce_add_f32(ps + rd * 8 * 32, wq, C::WQ_BYTES);
                            tma_commit_group();
                        }
                    }
                }
                if (!ok) break;
                ok = warp_all(mbar_wait(dkv_full, sg & 1, wc, 0x69));
                if (!ok) break;
                tc_fence_after();
                const bool some = j * TILE + wrow0 < p.N;      // warp-uniform
                uint4 u[2][DH / 32][4];
#pragma unroll
                for (int t = 0; t < 2; ++t)                     // dK, then dV
#pragma unroll
                    for (int c = 0; c < DH / 32; ++c) {
                        float v[32];
                        __syncwarp();
                        tmem_ld_f32<32>(lane_base + (t ? C::TMEM_DV : C::TMEM_DK) + c * 32, v);
                        pack_rows(u[t][c], v, t ? 1.0f : p.scale);
                    }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(dkv_free);
#pragma unroll
                for (int t = 0; t < 2; ++t)
#pragma unroll
                    for (int c = 0; c < DH / 32; ++c)
                        if (some && c * 32 < p.Dt) store_rows(t ? &tm_dv : &tm_dk, u[t][c], h, j * TILE + wrow0, c * 32, bs);
            }
        };
        if (WALK != WALK_SEGMENTS) drain(std::true_type{}, 0, seg.n_ws);
        if (WALK != WALK_WHOLE) drain(std::false_type{}, seg.n_ws, n_segs);
        if (lane == 0) tma_wait_group<0>();
    } else {
        // ------------------------------ compute groups ------------------------------
        reg_inc<C::REGS_COMPUTE>();
        const int g = warp >> 2;             // q columns 32g .. 32g+31 of the tile
        const int row = tid & 127;           // kv row within the tile == TMEM lane
        const uint32_t lane_base = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16);
        const int hf = g >> 1;               // half of the q columns
        const uint32_t tS = lane_base + C::TMEM_S + 32 * g, tDP = lane_base + C::TMEM_DP + 32 * g, tP = lane_base + C::TMEM_P + 16 * g;
        const uint32_t aDS = smem_u32(smem + C::OFF_DS);
        // Blocks of 8 x 8 (tmem_ld_frag32): bias from its half tile [64 q][kv], transposed on the way; the 16-byte
        // chunks of row q are swizzled by q & 7.  Lane 8 m + r addresses kv 8 m .. of row r of a block.
        const int w4 = warp & 3;
        const uint32_t aBias = smem_u32(smem + C::OFF_BIAS) + (w4 >> 1) * (SQ_SUB_BYTES / 2) + (32 * (g & 1) + (lane & 7)) * 128 +
                               ((((w4 & 1) * 4 + (lane >> 3)) ^ (lane & 7)) << 4);
        const uint32_t scratch_w = smem_u32(tmem_slot + 2);       // a word nobody reads
        bool ok = true;
        int gs = 0;
        const float2 c1x2 = make_float2(p.c1, p.c1), l2e2 = make_float2(LOG2E, LOG2E);

        // Word b of lane c of each four lanes goes to lane b as its word c.
        auto quad_transpose = [&](uint32_t (&a)[4]) {
            const bool odd = lane & 1, high = lane & 2;
            const uint32_t s0 = __shfl_xor_sync(0xffffffffu, odd ? a[0] : a[1], 1);
            const uint32_t s1 = __shfl_xor_sync(0xffffffffu, odd ? a[2] : a[3], 1);
            const uint32_t n0 = odd ? s0 : a[0], n1 = odd ? a[1] : s0, n2 = odd ? s1 : a[2], n3 = odd ? a[3] : s1;
            const uint32_t t0 = __shfl_xor_sync(0xffffffffu, high ? n0 : n2, 2);
            const uint32_t t1 = __shfl_xor_sync(0xffffffffu, high ? n1 : n3, 2);
            a[0] = high ? t0 : n0; a[1] = high ? t1 : n1; a[2] = high ? n2 : t0; a[3] = high ? n3 : t1;
        };
        // One S row: a step's dS tile is the dBias tile (q tile i, kv tile j).  Stored when the issuers have their operands, and
        // by whole rows: four-lane transposes leave lane c with the block of kv 8 c .. 8 c + 7, so that a store takes 128 bytes
        // of one q row (fp32) or 64 of eight (bf16).  Inside the arithmetic, and straight from the fragments, with 32 bytes of
        // four or eight rows, the addresses and values did not fit the registers, and the stores were what a step waited for:
        // B=4, S=1, N=1024, H=16, D=32 fp32 116 -> 91 us, bf16 85 -> 75 (one thread per kv row, as at D = 64: 101 and 82).
        // out: this lane's place in q row 32 g of the tile
        auto store_dbias = [&](auto* out, int q0, uint32_t (&pkd)[16], float2 (&dsv)[16]) {
            if constexpr (DBIAS_HERE != DBIAS_NO) {
#pragma unroll
                for (int cb = 0; cb < 4; ++cb) {
                    const bool rows = q0 + 8 * cb < p.N;          // (N is a multiple of 8)
                    if constexpr (DBIAS_HERE == DBIAS_F32) {
                        uint32_t x[2][4];
#pragma unroll
                        for (int b = 0; b < 4; ++b) { x[0][b] = __float_as_uint(dsv[4 * cb + b].x); x[1][b] = __float_as_uint(dsv[4 * cb + b].y); }
                        quad_transpose(x[0]);
                        quad_transpose(x[1]);
                        if (rows)
#pragma unroll
                            for (int r = 0; r < 8; ++r) out[static_cast<size_t>(8 * cb + r) * p.N] = __uint_as_float(x[r & 1][r >> 1]);
                    } else {
                        uint32_t w[4];
#pragma unroll
                        for (int b = 0; b < 4; ++b) w[b] = movmatrix_trans(pkd[8 * (b >> 1) + 2 * cb + (b & 1)]);
                        quad_transpose(w);
                        if (rows) *reinterpret_cast<uint4*>(out + static_cast<size_t>(8 * cb) * p.N) = make_uint4(w[0], w[1], w[2], w[3]);
                    }
                }
            }
        };

#pragma unroll 1
        for (int sg = 0; sg < n_segs && ok; ++sg) {
            using DBias = std::conditional_t<DBIAS_HERE == DBIAS_F32, float, __nv_bfloat16>;
            DBias* out = nullptr;
            bool cols = false;
            if constexpr (DBIAS_HERE != DBIAS_NO) {
                int bs, h, j;
                seg.decode(sg, bs, h, j);
                const int kv0 = j * TILE + 32 * w4 + 8 * (lane & 3), r = lane >> 2;
                cols = kv0 < p.N;
                out = static_cast<DBias*>(p.dbias) + ((static_cast<size_t>(bs) * p.H + h) * p.N + 32 * g + (DBIAS_HERE == DBIAS_F32 ? 0 : r)) * p.N +
                      kv0 + (DBIAS_HERE == DBIAS_F32 ? r : 0);
            }
#pragma unroll 1
            for (int i = 0; i < NT && ok; ++i, ++gs) {
                // Per element x = S' c1 + bias log2e (S' already carries mask and -LSE through the extra contraction
                // block), P = exp2(x), dS = P dP' (dP' already carries -delta).
                const int u = 2 * gs + hf, slot = u % NB;
                ok = warp_all(mbar_wait_both(&s_full[hf], gs & 1, &bias_full[slot], (u / NB) & 1, wc, 0x63));
                if (!ok) break;
                tc_fence_after();
                uint32_t sv[32], dv[32], bq[4][4], pkp[16], pkd[16];
                float2 dsv[16];
                tmem_ld_frag32(tS, sv);
                tmem_ld_frag32(tDP, dv);
#pragma unroll
                for (int cb = 0; cb < 4; ++cb) ldmatrix4_trans(bq[cb], aBias + slot * SQ_SUB_BYTES + cb * 1024);
                // everything is in registers: S' and dP' of the next step are formed during this one's arithmetic
                tmem_wait_ld();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&s_free[hf]);
#pragma unroll
                for (int cb = 0; cb < 4; ++cb) {              // 8 columns: four blocks of 8 kv
#pragma unroll
                    for (int b = 0; b < 4; ++b) {             // block (8 b, 8 cb)
                        const int r = 16 * (b >> 1) + 4 * cb + 2 * (b & 1), w = 8 * (b >> 1) + 2 * cb + (b & 1);
                        const float2 b2 = fmul2(bf16x2_f2(bq[cb][b]), l2e2);
                        const float2 x2 = ffma2(u2f2(sv[r], sv[r + 1]), c1x2, b2);
                        const float2 e2 = make_float2(ex2(x2.x), ex2(x2.y));
                        const float2 d2 = fmul2(e2, u2f2(dv[r], dv[r + 1]));
                        pkp[w] = pack_bf16(e2.x, e2.y);
                        pkd[w] = pack_bf16(d2.x, d2.y);
                        dsv[4 * cb + b] = d2;
                    }
#pragma unroll
                    for (int b = 0; b < 4; ++b) {             // formed here, not behind the wait below
                        const int w = 8 * (b >> 1) + 2 * cb + (b & 1);
                        asm volatile("" : "+r"(pkp[w]), "+r"(pkd[w]));
                    }
                }
                mbar_release_after_loads(&bias_empty[slot], pkp[0] ^ pkp[2] ^ pkp[4] ^ pkp[6], scratch_w);
                if (gs > 0) {
                    ok = warp_all(mbar_wait(ds_free, (gs - 1) & 1, wc, 0x61));
                    if (!ok) break;
                    tc_fence_after();
                }
                tmem_st_frag16(tP, pkp);
#pragma unroll
                for (int cb = 0; cb < 4; ++cb)
                    stmatrix4(aDS + sq_chunk_off(row, 4 * g + cb), pkd[2 * cb], pkd[2 * cb + 1], pkd[8 + 2 * cb], pkd[8 + 2 * cb + 1]);
                tmem_wait_st();
                tc_fence_before();
                fence_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(&ds_ready[hf]);
                if constexpr (DBIAS_HERE != DBIAS_NO) {
                    store_dbias(out, cols ? i * TILE + 32 * g : p.N, pkd, dsv);
                    out += static_cast<size_t>(TILE) * p.N;
                }
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (tid == 0) { report_abort(wc); report_abort(WaitCtx{tmem_slot + 3, p.status}); }
    if (warp == C::W_MMA) tmem_dealloc(tmem, BWD_TMEM_COLS);
}

}  // namespace evo
