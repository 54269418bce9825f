// dQ, dK, dV at D <= 64 (evo_bwd.cu has the interface, and what the dQ/dK/dV kernels share: transposed products, whole
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
// D = 64.  A kernel with two phases of sixteen warps a step (P, then dS) measured the same as halves that shared its loads:
// what bounded both was that two Q/dO stages and one K/V buffer were freed by a step's last products, 1900 clocks before what
// replaced them had landed (a wait of 1500 clocks a step for Q and dO and of 3900 a segment for K and V), and the drain warps,
// which staged the partial sums of dQ for bulk copies (3400 of a step's 4300 clocks).  Here Q, dO, K and V have rings and
// barriers of their own (dO is free with dV, V with the last dP', so that two and one buffers do), a half hands its bias back
// as soon as it is in registers, and the partial sums of a whole pair go from registers to the CTA's scratch area as vector
// reductions, coalesced and unstaged.  With one dQ accumulator there is room for P^T beside S'; pairs of two tiles then use the
// scratch area, which costs them less than a second accumulator over S' did.  Kernel alone: B=1, S=256, N=1024, H=4 1147 -> 999 us
// (37 rows 166 -> 140); S=74, N=640 137 -> 120, N=384 66 -> 56; S=148, N=256 58 -> 52; S=200, N=200 77 -> 73; B=4, S=1, N=1024,
// H=16 109 -> 106, with an fp32 bias 124 -> 112.  D = 32 with more than four tiles, for the reductions: S=256, N=768, H=8
// 784 -> 718.  (D = 32 with rings of their own for Q, dO, K and V: S=200, N=200, H=4 46 -> 51, N=384 350 -> 360; it keeps the pairs.)
//
// Tried at D = 32, against 356 at the first shape then: two dS tiles (428: issuers and LSU then meet on shared memory more often, the
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


template <int DH_>
struct BwdHalvesCfg {
    static constexpr int DH = DH_;
    static_assert(DH == 32 || DH == 64, "D = 96 and 128 are in evo_bwd_wide.cuh");
    static constexpr int NG = 4;                       // compute groups
    static constexpr int NCW = 4 * NG;
    static constexpr int W_DRAIN = NCW, W_PROD = NCW + 4, W_MMA = NCW + 5;
    static constexpr int THREADS = (NCW + 8) * 32;
    // setmaxnreg budgets: the CTA's register pool is the launch count (the cap ptxas derives from the
    // launch bound) times the threads; an increase that the pool cannot satisfy blocks for ever
    static constexpr int REGS_LAUNCH = (65536 / THREADS) & ~7;
    static constexpr int REGS_COMPUTE = 88, REGS_OTHER = 48;       // drain warps: as launched
    static_assert((REGS_COMPUTE * NCW + (REGS_LAUNCH + REGS_OTHER) * 4) * 32 <= REGS_LAUNCH * THREADS, "register pool");
    // Buffers of Q (with the extra tile of its rows), dO, K (with its extra tile), V, halves of bias tiles.  D = 32: Q and
    // dO, and K and V, come and go together, which is fewer barriers for the producer; D = 64 has no room for that.
    static constexpr bool PAIRED = DH == 32;
    static constexpr int NQ = 3, NDO = PAIRED ? NQ : 2, NK = 2, NV = PAIRED ? NK : 1, NB = (DH == 32) ? 4 : 2;
    static constexpr int DQ_BUFS = (DH == 32) ? 4 : 1;             // dQ accumulators
    static constexpr uint32_t ROWT = RowTile<DH>::BYTES;
    static constexpr uint32_t OFF_Q = 0, OFF_DO = OFF_Q + NQ * ROWT, OFF_K = OFF_DO + NDO * ROWT, OFF_V = OFF_K + NK * ROWT;
    static constexpr uint32_t OFF_BIAS = OFF_V + NV * ROWT;
    static constexpr uint32_t OFF_DS = OFF_BIAS + NB * SQ_SUB_BYTES;
    // per drain warp: WSLOTS slots of [32 rows][32 fp32], for bulk copies of dQ, dK and dV
    static constexpr uint32_t WQ_BYTES = 32 * 32 * 4;
    static constexpr int WSLOTS = (DH == 32) ? 2 : 1;
    static constexpr uint32_t OFF_WSTG = OFF_DS + SQ_BYTES;
    static constexpr uint32_t OFF_XQ = OFF_WSTG + 4 * WSLOTS * WQ_BYTES, OFF_XK = OFF_XQ + NQ * XT_BYTES;
    // constant extra tiles, above every tile that refers to the zero tile
    static constexpr uint32_t OFF_XDP = OFF_XK + NK * XT_BYTES;            // row selector of -delta
    static constexpr uint32_t OFF_ZERO = OFF_XDP + XT_BYTES;
    static constexpr uint32_t OFF_BARS = OFF_ZERO + XT_BYTES;
    static constexpr uint32_t NUM_BARS = 2 * (NQ + NDO + NK + NV + NB + DQ_BUFS) + 9;
    static constexpr uint32_t OFF_MISC = OFF_BARS + NUM_BARS * 8;
    static constexpr uint32_t SMEM_BYTES = OFF_MISC + 16 + 1024;            // + alignment slack
    static constexpr uint32_t TMEM_S = 0, TMEM_DP = 128, TMEM_P = 256;       // S', dP', P^T (bf16)
    static constexpr uint32_t TMEM_DQ = 320;                                // accumulators
    static constexpr uint32_t TMEM_DK = TMEM_DQ + DQ_BUFS * DH, TMEM_DV = TMEM_DK + DH;
    static_assert(TMEM_DV + DH <= BWD_TMEM_COLS, "tensor memory budget");
    static_assert(SMEM_BYTES <= 232448, "shared memory budget");
    static_assert(ROWT % 1024 == 0 && WQ_BYTES % 1024 == 0, "tile alignment");
};

template <int DH, int WALK, int DBIAS_HERE>
__global__ void __launch_bounds__(BwdHalvesCfg<DH>::THREADS, 1)
evo_bwd_halves_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
               const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_do,
               const __grid_constant__ CUtensorMap tm_bias, const __grid_constant__ CUtensorMap tm_dq,
               const __grid_constant__ CUtensorMap tm_dk, const __grid_constant__ CUtensorMap tm_dv,
               const __grid_constant__ CUtensorMap tm_acc, const BwdParams p) {
    using C = BwdHalvesCfg<DH>;
    using RT = RowTile<DH>;
    using RD = RowDesc<DH>;
    constexpr int NQ = C::NQ, NDO = C::NDO, NK = C::NK, NV = C::NV, NB = C::NB, DQB = C::DQ_BUFS;

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::OFF_BARS);
    uint64_t* q_full = bars;                   // [NQ]: Q and the extra tile of its rows
    uint64_t* q_empty = q_full + NQ;           // [NQ]
    uint64_t* do_full = q_empty + NQ;          // [NDO]
    uint64_t* do_empty = do_full + NDO;        // [NDO]
    uint64_t* k_full = do_empty + NDO;         // [NK]: K and the extra tile of its rows
    uint64_t* k_empty = k_full + NK;           // [NK]
    uint64_t* v_full = k_empty + NK;           // [NV]
    uint64_t* v_empty = v_full + NV;           // [NV]
    uint64_t* bias_full = v_empty + NV;       // [NB]
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
    const bool own_prep = WALK == WALK_WHOLE && (DBIAS_HERE == DBIAS_F32 || DBIAS_HERE == DBIAS_BF16) && p.own_prep;
    WaitCtx wc{abort_flag, p.status};

    if (tid == 0) {
        *abort_flag = 0;
        tmem_slot[3] = 0;                      // the abort word of the waits before exit
        const uint32_t full = own_prep ? 5 : 1;      // the loads, and the drain warps for the extra tiles
        for (int i = 0; i < NQ; ++i) { mbar_init(&q_full[i], full); mbar_init(&q_empty[i], 1); }
        for (int i = 0; i < NDO; ++i) { mbar_init(&do_full[i], 1); mbar_init(&do_empty[i], 1); }
        for (int i = 0; i < NK; ++i) { mbar_init(&k_full[i], full); mbar_init(&k_empty[i], 1); }
        for (int i = 0; i < NV; ++i) { mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1); }
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
    chain_wait();

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
        int gs = 0, n_q = 0, n_do = 0, n_k = 0, n_v = 0, n_bias = 0;      // steps; loads issued
        SegmentWalk<WALK> at(seg, 0);
#pragma unroll 1
        for (int sg = 0; sg < n_segs && ok; ++sg) {
            if (sg > 0) at.next(seg, sg, p);
            const int bs = at.bs, h = at.h, j = at.j;
            const int b = bs / p.S;
            const __nv_bfloat16* xq = p.xq + (static_cast<size_t>(bs) * p.H + h) * p.NTP * 8;
            const int kb = sg % NK, vb = sg % NV;
            if (sg >= NK) ok = warp_all(mbar_wait(&k_empty[kb], ((sg / NK) - 1) & 1, wc, 0x40));
            if (!ok) break;
            if (elect_one()) {
                mbar_arrive_expect_tx(&k_full[kb], (C::PAIRED ? 2 : 1) * C::ROWT + (own_prep ? 0 : XT_BYTES));
                tma_load_row_tile<DH>(smem + C::OFF_K + kb * C::ROWT, &tm_k, &k_full[kb], h, j * TILE, bs);
                if (C::PAIRED) tma_load_row_tile<DH>(smem + C::OFF_V + kb * C::ROWT, &tm_v, &k_full[kb], h, j * TILE, bs);
                if (!own_prep) bulk_load(smem + C::OFF_XK + kb * XT_BYTES, p.xk + (static_cast<size_t>(bs) * p.NTP + j * TILE) * 8, XT_BYTES, &k_full[kb]);
            }
            __syncwarp();
            ++n_k;
#pragma unroll 1
            for (int i = 0; i < NT && ok; ++i, ++gs) {
                const int qb = gs % NQ, db = gs % NDO;
                if (gs >= NQ) ok = warp_all(mbar_wait(&q_empty[qb], ((gs / NQ) - 1) & 1, wc, 0x42));
                if (!ok) break;
                if (elect_one()) {
                    mbar_arrive_expect_tx(&q_full[qb], (C::PAIRED ? 2 : 1) * C::ROWT + (own_prep ? 0 : XT_BYTES));
                    tma_load_row_tile<DH>(smem + C::OFF_Q + qb * C::ROWT, &tm_q, &q_full[qb], h, i * TILE, bs);
                    if (C::PAIRED) tma_load_row_tile<DH>(smem + C::OFF_DO + qb * C::ROWT, &tm_do, &q_full[qb], h, i * TILE, bs);
                    if (!own_prep) bulk_load(smem + C::OFF_XQ + qb * XT_BYTES, xq + static_cast<size_t>(i) * TILE * 8, XT_BYTES, &q_full[qb]);
                }
                __syncwarp();
                ++n_q;
                if constexpr (!C::PAIRED) {
                    if (gs >= NDO) ok = warp_all(mbar_wait(&do_empty[db], ((gs / NDO) - 1) & 1, wc, 0x46));
                    if (!ok) break;
                    if (elect_one()) {
                        mbar_arrive_expect_tx(&do_full[db], C::ROWT);
                        tma_load_row_tile<DH>(smem + C::OFF_DO + db * C::ROWT, &tm_do, &do_full[db], h, i * TILE, bs);
                    }
                    __syncwarp();
                    ++n_do;
                    if (i == 0) {
                        // V is free with the last dP' of its segment, K with the last dQ
                        if (sg >= NV) ok = warp_all(mbar_wait(&v_empty[vb], ((sg / NV) - 1) & 1, wc, 0x47));
                        if (!ok) break;
                        if (elect_one()) {
                            mbar_arrive_expect_tx(&v_full[vb], C::ROWT);
                            tma_load_row_tile<DH>(smem + C::OFF_V + vb * C::ROWT, &tm_v, &v_full[vb], h, j * TILE, bs);
                        }
                        __syncwarp();
                        ++n_v;
                    }
                }
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
        for (int k = (n_q > NQ ? n_q - NQ : 0); k < n_q; ++k) mbar_wait_landed(&q_full[k % NQ], (k / NQ) & 1, dc, 0x43);
        // (n_do, n_v: 0 where they come with Q and K)
        for (int k = (n_do > NDO ? n_do - NDO : 0); k < n_do; ++k) mbar_wait_landed(&do_full[k % NDO], (k / NDO) & 1, dc, 0x48);
        for (int k = (n_k > NK ? n_k - NK : 0); k < n_k; ++k) mbar_wait_landed(&k_full[k % NK], (k / NK) & 1, dc, 0x45);
        for (int k = (n_v > NV ? n_v - NV : 0); k < n_v; ++k) mbar_wait_landed(&v_full[k % NV], (k / NV) & 1, dc, 0x49);
        for (int k = (n_bias > NB ? n_bias - NB : 0); k < n_bias; ++k) mbar_wait_landed(&bias_full[k % NB], (k / NB) & 1, dc, 0x44);
    } else {
        // ------------------------------ mma issuers ------------------------------
        // Each warp runs its loop with all lanes (uniform control flow: operand descriptors stay in
        // uniform registers) and elects one lane to issue.
        constexpr uint32_t IDESC_SDP = make_idesc_bf16(128, 64, 0, 0);
        // N = the head-dim columns that hold data (the rest of a wider kernel's tile is zero fill)
        const uint32_t IDESC_DKV = make_idesc_bf16(128, 16 * p.KB, 0, 1);
        const uint32_t IDESC_DQ = make_idesc_bf16(128, 16 * p.KB, 1, 1);
        const uint32_t aQ = smem_u32(smem + C::OFF_Q), aDO = smem_u32(smem + C::OFF_DO), aK = smem_u32(smem + C::OFF_K);
        const uint32_t aZero = smem_u32(smem + C::OFF_ZERO);
        const int role = warp - C::W_MMA;          // 0: S/dP, 1: dV/dK, 2: dQ
        bool ok = true;
        int gs = 0;
#pragma unroll 1
        for (int sg = 0; sg < n_segs && ok; ++sg) {
            const int kb = sg % NK, vb = sg % NV;
#pragma unroll 1
            for (int i = 0; i < NT && ok; ++i, ++gs) {
                const int qb = gs % NQ, db = gs % NDO;
                if (role == 0) {
                    ok = warp_all(mbar_wait(&q_full[qb], (gs / NQ) & 1, wc, 0x50));
                    if (ok && i == 0) ok = warp_all(mbar_wait(&k_full[kb], (sg / NK) & 1, wc, 0x51));
#pragma unroll
                    for (int t = 0; t < 4; ++t) {          // S', then dP' of one half, then of the other
                        const int hf = t >> 1, part = t & 1;
                        if (ok && gs > 0 && part == 0) ok = warp_all(mbar_wait(&s_free[hf], (gs - 1) & 1, wc, 0x52));
                        if (!C::PAIRED && ok && t == 1) ok = warp_all(mbar_wait(&do_full[db], (gs / NDO) & 1, wc, 0x56));
                        if (!C::PAIRED && ok && t == 1 && i == 0) ok = warp_all(mbar_wait(&v_full[vb], (sg / NV) & 1, wc, 0x57));
                        if (!ok) break;
                        tc_fence_after();
                        if (elect_one()) {
                            const uint32_t a_lo = RD::kmajor_lo(part ? smem_u32(smem + C::OFF_V) + vb * C::ROWT : aK + kb * C::ROWT);
                            const uint32_t b_lo = RD::kmajor_lo((part ? aDO + db * C::ROWT : aQ + qb * C::ROWT) + hf * 64 * RT::ROW_BYTES);
                            const uint32_t d = tmem + C::TMEM_S + 128 * part + 64 * hf;
#pragma unroll
                            for (int kk = 0; kk < RT::KBLOCKS; ++kk)
                                if (kk < p.KB)      // the others are zero-filled blocks past the true head dim
                                    umma_ss(d, RD::kmajor(a_lo, kk), RD::kmajor(b_lo, kk), IDESC_SDP, kk > 0);
                            // the extra contraction block: + (mask - LSE) / scale, - delta
                            umma_ss(d, xt_desc(part ? smem_u32(smem + C::OFF_XDP) : smem_u32(smem + C::OFF_XK) + kb * XT_BYTES, aZero),
                                    xt_desc(smem_u32(smem + C::OFF_XQ) + qb * XT_BYTES + hf * 64 * 16, aZero), IDESC_SDP, 1u);
                            if (part) umma_commit(&s_full[hf]);
                            if (!C::PAIRED && t == 3 && i == NT - 1) umma_commit(&v_empty[vb]);
                        }
                        __syncwarp();
                    }
                } else if (role == 1) {
                    // the first MMA of a segment overwrites dK / dV: the previous one's must be out
                    if (i == 0 && sg > 0) ok = warp_all(mbar_wait(dkv_free, (sg - 1) & 1, wc, 0x55));
#pragma unroll 1
                    for (int hf = 0; hf < 2; ++hf) {
                        if (ok) ok = warp_all(mbar_wait(&ds_ready[hf], gs & 1, wc, 0x5a));      // (Q and dO have landed: dP' read them)
                        if (!ok) break;
                        tc_fence_after();
                        if (elect_one()) {
                            const uint32_t row0 = hf * 64 * RT::ROW_BYTES;
                            const uint32_t do_lo = RD::mnmajor_lo(aDO + db * C::ROWT + row0), q_lo = RD::mnmajor_lo(aQ + qb * C::ROWT + row0);
                            const uint32_t ds_lo = SqDesc::kmajor_lo(smem_u32(smem + C::OFF_DS) + hf * SQ_SUB_BYTES);
                            const uint32_t t_p = tmem + C::TMEM_P + 32 * hf, acc = (hf > 0 || i > 0) ? 1u : 0u;
#pragma unroll
                            for (int kk = 0; kk < 4; ++kk)
                                umma_ts(tmem + C::TMEM_DV, t_p + 8 * kk, RD::mnmajor(do_lo, kk), IDESC_DKV, kk > 0 ? 1u : acc);
                            if (!C::PAIRED && hf == 1) umma_commit(&do_empty[db]);
#pragma unroll
                            for (int kk = 0; kk < 4; ++kk)
                                umma_ss(tmem + C::TMEM_DK, SqDesc::kmajor(ds_lo, kk), RD::mnmajor(q_lo, kk), IDESC_DKV, kk > 0 ? 1u : acc);
                            if (hf == 1) {
                                umma_commit(ds_free);
                                umma_commit(&q_empty[qb]);
                                if (i == NT - 1) umma_commit(dkv_full);
                            }
                        }
                        __syncwarp();
                    }
                } else {
                    const bool whole = seg.whole(sg), resident = whole && res_ok;
                    const int j = whole ? sg % NT : 0, ev = dq_event(resident, sg, j, i), buf = ev % DQB, use = ev / DQB;
                    if (use > 0 && !(resident && j > 0)) ok = warp_all(mbar_wait(&dq_free[buf], (use - 1) & 1, wc, 0x54));
                    if (ok) ok = warp_all(mbar_wait_both(&ds_ready[0], gs & 1, &ds_ready[1], gs & 1, wc, 0x5b));
                    if (!ok) break;
                    tc_fence_after();
                    if (elect_one()) {
                        const uint32_t ds_lo = SqDesc::mnmajor_lo(smem_u32(smem + C::OFF_DS));
                        const uint32_t k_lo = RD::mnmajor_lo(aK + kb * C::ROWT);
                        const uint32_t t_dq = tmem + C::TMEM_DQ + buf * DH;
                        const uint32_t acc = (resident && j > 0) ? 1u : 0u;
#pragma unroll
                        for (int kk = 0; kk < 8; ++kk)
                            umma_ss(t_dq, SqDesc::mnmajor(ds_lo, kk), RD::mnmajor(k_lo, kk), IDESC_DQ, kk > 0 ? 1u : acc);
                        umma_commit(ds_free);
                        if (!resident || j == NT - 1) umma_commit(&dq_full[buf]);
                        if (i == NT - 1) umma_commit(&k_empty[kb]);
                    }
                    __syncwarp();
                }
            }
        }
    }
    } else if (warp >= C::W_DRAIN) {
        // ------------------------------ drain warps ------------------------------
        // (The loops over DH / 32 run once at D = 32, twice at 64.  Written without them for D = 32 the mixed walk spills in other places, and is slower with
        // one S row: B=38, N=392, H=8 83 -> 89 us.)
        const int w4 = warp & 3;
        const int wrow0 = w4 * 32;           // tensor-memory lanes (tile rows) of this warp
        const uint32_t lane_base = tmem + (static_cast<uint32_t>(wrow0) << 16);
        uint8_t* const wslot = smem + C::OFF_WSTG + w4 * C::WSLOTS * C::WQ_BYTES;
        // Where the next bulk copy (one group each) is staged: two slots in turn, once the copy before last has read its own;
        // or one slot, or its halves in turn for copies of half its size.
        int pos = 0;
        bool last_half = false;
        auto next_slot = [&](bool half) -> uint8_t* {
            if (lane == 0) {
                if (C::WSLOTS == 2 || (half && last_half)) tma_wait_group_read<1>();
                else tma_wait_group_read<0>();
            }
            __syncwarp();
            last_half = half;
            pos ^= 1;
            return wslot + (C::WSLOTS == 2 ? pos * C::WQ_BYTES : (half ? pos * (C::WQ_BYTES / 2) : 0));
        };
        // 32 columns of 32 rows as bf16, by a bulk tensor store (which clips rows past N and columns past Dt)
        auto store_rows = [&](const CUtensorMap* tm, const uint4 (&u)[4], int h, int row0, int col0, int bs) {
            uint8_t* sl = next_slot(true);
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
                    const int ev = dq_event(resident, sg, j, i), buf = ev % DQB;
                    const bool rows = i * TILE + wrow0 < p.N;     // warp-uniform: some row of this warp exists
                    const bool final_sum = whole && j == NT - 1, add = final_sum && j > 0 && !resident && rows;
                    float4* ps = part + static_cast<size_t>(i * 4 + w4) * (DH / 4) * 32;
                    float4 old[8];
                    ok = warp_all(mbar_wait(&dq_full[buf], (ev / DQB) & 1, wc, 0x68));
                    if (!ok) break;
                    tc_fence_after();
#pragma unroll
                    for (int rd = 0; rd < DH / 32; ++rd) {
                        float dqv[32];
                        tmem_ld_f32<32>(lane_base + C::TMEM_DQ + buf * DH + rd * 32, dqv);
                        if (rd == DH / 32 - 1) {
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0) mbar_arrive(&dq_free[buf]);
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
                        if (whole) {
                            // (the thread that reads the sum in the last segment is the same)
#pragma unroll
                            for (int c = 0; c < 8; ++c) {
                                float4* at = ps + (rd * 8 + c) * 32 + lane;
                                if (j == 0) __stcg(at, make_float4(dqv[c * 4], dqv[c * 4 + 1], dqv[c * 4 + 2], dqv[c * 4 + 3]));
                                else red_add_v4(reinterpret_cast<float*>(at), dqv[c * 4], dqv[c * 4 + 1], dqv[c * 4 + 2], dqv[c * 4 + 3]);
                            }
                            continue;
                        }
                        uint8_t* wq = next_slot(false);
#pragma unroll
                        for (int c = 0; c < 8; ++c)
                            *reinterpret_cast<float4*>(wq + swz_off<128>(lane, c)) =
                                make_float4(dqv[c * 4 + 0] * p.scale, dqv[c * 4 + 1] * p.scale, dqv[c * 4 + 2] * p.scale, dqv[c * 4 + 3] * p.scale);
                        fence_async_smem();
                        __syncwarp();
                        if (lane == 0) {
                            tma_reduce_add_4d(&tm_acc, wq, rd * 32, h, i * TILE + wrow0, bs - p.acc_row0);
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
                auto store = [&](int t) {
#pragma unroll
                    for (int c = 0; c < DH / 32; ++c)
                        if (some && c * 32 < p.Dt) store_rows(t ? &tm_dv : &tm_dk, u[t][c], h, j * TILE + wrow0, c * 32, bs);
                };
#pragma unroll
                for (int t = 0; t < 2; ++t) {                   // dK, then dV
#pragma unroll
                    for (int c = 0; c < DH / 32; ++c) {
                        float v[32];
                        __syncwarp();
                        tmem_ld_f32<32>(lane_base + (t ? C::TMEM_DV : C::TMEM_DK) + c * 32, v);
                        pack_rows(u[t][c], v, t ? 1.0f : p.scale);
                    }
                    if (DH == 64 && t == 0) store(0);          // (no registers for both)
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(dkv_free);
                if (DH == 32) store(0);
                store(1);
            }
        };
        if (own_prep && n_segs > 0) {
            // what the prep kernel does (evo_bwd.cu), for the one step of this CTA: thread = row
            int bs, h, j;
            seg.decode(0, bs, h, j);
            const int row = wrow0 + lane;
            const float inv_scale = 1.0f / p.scale;
            uint4 xq = make_uint4(0x3f803f80u, split_bf16(-1e30f), 0u, 0u), xk = make_uint4(split_bf16(-1e30f), 0x3f803f80u, 0u, 0u);
            if (row < p.N) {
                const size_t off = bs * p.lay_out.row + row * p.lay_out.n + h * p.lay_out.h;
                const float lse = __ldg(p.lse + (static_cast<size_t>(bs) * p.H + h) * p.N + row);
                const float m = __bfloat162float(p.mask[static_cast<size_t>(bs) * p.N + row]);
                float s[DH / 8];                   // by chunks of eight columns, and these in pairs: the prep kernel's sum to the bit
#pragma unroll
                for (int c0 = 0; c0 < DH; c0 += 32) {
                    uint4 a[4], b[4], r[4];
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        a[c] = b[c] = r[c] = make_uint4(0u, 0u, 0u, 0u);
                        if (c0 + 8 * c >= p.Dt) continue;
                        a[c] = __ldg(reinterpret_cast<const uint4*>(p.o + off + c0 + 8 * c));
                        b[c] = __ldg(reinterpret_cast<const uint4*>(p.d_o + off + c0 + 8 * c));
                        if (p.o_resid) r[c] = __ldg(reinterpret_cast<const uint4*>(p.o_resid + off + c0 + 8 * c));
                    }
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const uint32_t aw[4] = {a[c].x, a[c].y, a[c].z, a[c].w}, bw[4] = {b[c].x, b[c].y, b[c].z, b[c].w}, rw[4] = {r[c].x, r[c].y, r[c].z, r[c].w};
                        float& sc = s[c0 / 8 + c];
                        sc = 0.f;
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            sc = fmaf(bf16_lo(aw[e]) + bf16_lo(rw[e]), bf16_lo(bw[e]), sc);
                            sc = fmaf(bf16_hi(aw[e]) + bf16_hi(rw[e]), bf16_hi(bw[e]), sc);
                        }
                    }
                }
#pragma unroll
                for (int w = 1; w < DH / 8; w *= 2)
#pragma unroll
                    for (int c = 0; c < DH / 8; c += 2 * w) s[c] += s[c + w];
                xq = make_uint4(0x3f803f80u, split_bf16(-lse * inv_scale), split_bf16(-s[0]), 0u);
                xk.x = split_bf16(m * inv_scale);
            }
            *reinterpret_cast<uint4*>(smem + C::OFF_XQ + row * 16) = xq;
            *reinterpret_cast<uint4*>(smem + C::OFF_XK + row * 16) = xk;
            fence_async_smem();
            __syncwarp();
            if (lane == 0) { mbar_arrive(&q_full[0]); mbar_arrive(&k_full[0]); }
        }
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
        // B=4, S=1, N=1024, H=16, D=32 fp32 116 -> 91 us, bf16 85 -> 75 (one thread per kv row: 101 and 82).
        // out: this lane's place in q row 32 g of the tile
        auto store_dbias = [&](auto* out, int q0, uint32_t (&pkd)[16], float2 (&dsv)[16]) {
            if constexpr (DBIAS_HERE != DBIAS_NO) {
#pragma unroll
                for (int cb = 0; cb < 4; ++cb) {
                    const bool rows = q0 + 8 * cb < p.N;          // (N is a multiple of 8)
                    if constexpr (DBIAS_HERE != DBIAS_BF16) {
                        uint32_t x[2][4];
#pragma unroll
                        for (int b = 0; b < 4; ++b) { x[0][b] = __float_as_uint(dsv[4 * cb + b].x); x[1][b] = __float_as_uint(dsv[4 * cb + b].y); }
                        quad_transpose(x[0]);
                        quad_transpose(x[1]);
                        if (rows)
#pragma unroll
                            for (int r = 0; r < 8; ++r) {
                                const float v = __uint_as_float(x[r & 1][r >> 1]);
                                if constexpr (DBIAS_HERE == DBIAS_ADD) red_add(&out[static_cast<size_t>(8 * cb + r) * p.N], v);
                                else out[static_cast<size_t>(8 * cb + r) * p.N] = v;
                            }
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

        // DBIAS_ADD: this warp's part of the tile has one row more; with the last one it becomes the bf16 result.
        auto count_row = [&](const float* at, int part, int q0) {
            if constexpr (DBIAS_HERE == DBIAS_ADD) {
                if (p.dbias_done == nullptr) return;
                __threadfence();
                __syncwarp();
                int before = 0;
                if (lane == 0) {
                    before = atomicAdd(p.dbias_done + part, 1);
                    __threadfence();                          // behind the counts of the other warps, for all lanes:
                }
                before = __shfl_sync(0xffffffffu, before, 0);
                __syncwarp();                                 // a shuffle orders no memory
                if (before != p.S - 1) return;
                __nv_bfloat16* res = static_cast<__nv_bfloat16*>(p.dbias) + (at - p.dbias_acc);
                if (q0 >= p.N) return;
                const int rows = p.N - q0 < 32 ? p.N - q0 : 32;
                float v[32];                                  // (all loads in flight at once)
#pragma unroll
                for (int r = 0; r < 32; ++r) v[r] = __ldcg(at + static_cast<size_t>(r < rows ? r : 0) * p.N);
#pragma unroll
                for (int r = 0; r < 32; ++r)
                    if (r < rows) res[static_cast<size_t>(r) * p.N] = __float2bfloat16_rn(v[r]);
            }
        };

#pragma unroll 1
        for (int sg = 0; sg < n_segs && ok; ++sg) {
            using DBias = std::conditional_t<DBIAS_HERE != DBIAS_BF16, float, __nv_bfloat16>;
            DBias* out = nullptr;
            bool cols = false;
            int part = 0;
            if constexpr (DBIAS_HERE != DBIAS_NO) {
                int bs, h, j;
                seg.decode(sg, bs, h, j);
                if (DBIAS_HERE == DBIAS_ADD) bs /= p.S;             // (else S = 1)
                part = ((bs * p.H + h) * NT * NT + j) * 16 + warp;
                const int kv0 = j * TILE + 32 * w4 + 8 * (lane & 3), r = lane >> 2;
                cols = kv0 < p.N;
                constexpr bool BF = DBIAS_HERE == DBIAS_BF16;
                out = static_cast<DBias*>(DBIAS_HERE == DBIAS_ADD ? p.dbias_acc : p.dbias) +
                      ((static_cast<size_t>(bs) * p.H + h) * p.N + 32 * g + (BF ? r : 0)) * p.N + kv0 + (BF ? 0 : r);
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
                if (DH == 64) mbar_release_after_loads(&bias_empty[slot], bq[0][0] ^ bq[1][0] ^ bq[2][0] ^ bq[3][0], scratch_w);
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
                        if constexpr (DBIAS_HERE == DBIAS_ADD && DBIAS_POLY_EVERY<DH> > 0) {
                            // dBias from the dBias kernel's exponentials: polynomials in the same kv columns, this thread's rows
                            const float2 a2 = ex2_poly2<3>(x2);
                            const bool poly = use_poly<DBIAS_POLY_EVERY<DH>>(lane >> 3);
                            float2 p2 = make_float2(poly ? a2.x : e2.x, poly ? a2.y : e2.y);
                            asm volatile("" : "+f"(p2.x), "+f"(p2.y));      // chosen here: 40 bytes of spills, 184 with the choice put off
                            dsv[4 * cb + b] = fmul2(p2, u2f2(dv[r], dv[r + 1]));
                            asm volatile("" : "+f"(dsv[4 * cb + b].x), "+f"(dsv[4 * cb + b].y));
                        }
                    }
#pragma unroll
                    for (int b = 0; b < 4; ++b) {             // formed here, not behind the wait below
                        const int w = 8 * (b >> 1) + 2 * cb + (b & 1);
                        asm volatile("" : "+r"(pkp[w]), "+r"(pkd[w]));
                    }
                }
                if (DH != 64) mbar_release_after_loads(&bias_empty[slot], pkp[0] ^ pkp[2] ^ pkp[4] ^ pkp[6], scratch_w);
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
                    if (DBIAS_HERE == DBIAS_ADD) count_row(reinterpret_cast<float*>(out), part + i * NT * 16, cols ? i * TILE + 32 * g : p.N);
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
