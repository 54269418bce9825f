// dQ, dK, dV at D = 96 and 128 (evo_bwd.cu has the interface and what the dQ/dK/dV kernels share: transposed
// products, whole pairs or single segments).  Tensor memory holds S', dP', dK and dV and
// nothing else: P^T and dS^T overwrite the columns they were computed from, and dQ takes the columns of S'
// once dV, which reads P^T from them, is complete.  A step is then one chain
//
//   S' -> P, dS -> dV -> dQ -> dQ read out -> S' of the next step        (dK and the next dP' beside it)
//
// so what bounds it is that chain, and the 16 compute warps, idle while the products are formed, read
// out dQ (32 columns each, a 600-clock pass; four drain warps took 2900) and, after a segment, dK and dV.
//
// A step takes 8000 clocks (B=1, S=128, N=768, H=4).  Measured in it: 1400 of arithmetic, 3400 in which the compute warps wait for
// their reductions of dQ (64 KB a step; an SM sends them at 18 bytes a clock in rows of 64 bytes, 25 contiguous), 2100 for dQ.
// Without its reductions it is 11 % shorter, no more.  What takes their place is shared memory: 270 KB of operands a step at 128
// bytes a clock beside 100 KB of loads and the compute warps' accesses.  Tried, kernel alone at that shape against 552 us: the reductions
// on four drain warps (554); with that, Q in halves through a ring of three, K and V on barriers of their own and the bias by ldmatrix
// (586); and with that, dQ in the columns of dP', so that S' waits for dV alone, dK from the dS tile, and 32 columns of dQ read by the
// compute warps (589).
//
//   warps 0-15 (compute)  group g = warp / 4 owns q columns 32g .. 32g+31 of the tile, and head-dim columns
//                         32g .. 32g+31 of dQ, dK and dV
//   warp 16 (producer)    TMA: dO with the extra tile of the q rows, Q, the pair-bias tile per step; K, V and
//                         the extra tile of the kv rows per segment
//   warps 17, 18, 19      MMA issuers: S'^T and dP'^T; dV, then dK; dQ
#pragma once

namespace evo {

template <int DH>
struct BwdWideCfg {
    static_assert(DH == 128, "D <= 64 is in evo_bwd_halves.cuh");
    static constexpr int NG = 4;                       // compute groups
    static constexpr int NCW = 4 * NG;
    static constexpr int W_PROD = NCW, W_MMA = NCW + 1;
    static constexpr int THREADS = (NCW + 4) * 32;
    static constexpr uint32_t ROWT = RowTile<DH>::BYTES;
    static constexpr uint32_t ST_Q = 0, ST_DO = ROWT, ST_XQ = 2 * ROWT;
    static constexpr uint32_t STAGE_BYTES = 2 * ROWT + XT_BYTES;
    static constexpr uint32_t KV_K = 0, KV_V = ROWT, KV_XK = 2 * ROWT, KV_BYTES = 2 * ROWT + XT_BYTES;
    static constexpr uint32_t OFF_STAGE = 0;
    static constexpr uint32_t OFF_KV = OFF_STAGE + STAGE_BYTES;
    static constexpr uint32_t OFF_BIAS = OFF_KV + KV_BYTES;
    static constexpr uint32_t OFF_DS = OFF_BIAS + SQ_BYTES;
    // constant extra tiles, above every tile that refers to the zero tile
    static constexpr uint32_t OFF_XDP = OFF_DS + SQ_BYTES;            // row selector of -delta
    static constexpr uint32_t OFF_ZERO = OFF_XDP + XT_BYTES;
    static constexpr uint32_t OFF_BARS = OFF_ZERO + XT_BYTES;
    static constexpr uint32_t NUM_BARS = 15;
    static constexpr uint32_t OFF_MISC = OFF_BARS + NUM_BARS * 8;
    static constexpr uint32_t SMEM_BYTES = OFF_MISC + 16 + 1024;            // + alignment slack
    static constexpr uint32_t TMEM_S = 0, TMEM_DP = 128, TMEM_DQ = TMEM_S, TMEM_DK = 256, TMEM_DV = 384;
    // column of contraction block kk (16 q) of P^T / dS^T, inside the columns of its own group
    __device__ static __forceinline__ uint32_t p_col(int kk) { return TMEM_S + 32 * (kk >> 1) + 8 * (kk & 1); }
    __device__ static __forceinline__ uint32_t ds_col(int kk) { return p_col(kk) + 128; }
    static_assert(TMEM_DV + DH <= BWD_TMEM_COLS, "tensor memory budget");
    static_assert(SMEM_BYTES <= 232448, "shared memory budget");
    static_assert(STAGE_BYTES % 1024 == 0 && KV_BYTES % 1024 == 0, "tile alignment");
};

template <int DH, int WALK, int DBIAS_HERE>
__global__ void __launch_bounds__(BwdWideCfg<DH>::THREADS, 1)
evo_bwd_wide_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
               const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_do,
               const __grid_constant__ CUtensorMap tm_bias, const BwdParams p) {
    using C = BwdWideCfg<DH>;
    using RT = RowTile<DH>;
    using RD = RowDesc<DH>;

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::OFF_BARS);
    uint64_t* do_full = bars;            // dO and the extra tile of the q rows
    uint64_t* do_empty = bars + 1;
    uint64_t* q_full = bars + 2;
    uint64_t* q_empty = bars + 3;
    uint64_t* kv_full = bars + 4;
    uint64_t* kv_empty = bars + 5;
    uint64_t* sdp_full = bars + 6;       // S', dP' complete and the bias tile landed
    uint64_t* bias_empty = bars + 7;
    uint64_t* pds_ready = bars + 8;      // P^T, dS^T and the dS tile are written
    uint64_t* dv_done = bars + 9;        // dV of the step is complete
    uint64_t* dk_done = bars + 10;       // dK of the step is complete
    uint64_t* dq_full = bars + 11;
    uint64_t* dq_free = bars + 12;       // dQ of the step is read out
    uint64_t* dkv_full = bars + 13;      // dK, dV of the segment are complete
    uint64_t* dkv_free = bars + 14;      // ... and read out
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
        for (uint64_t* b : {do_full, do_empty, q_full, q_empty, kv_full, dv_done, dk_done, dq_full, dkv_full}) mbar_init(b, 1);
        for (uint64_t* b : {kv_empty, sdp_full}) mbar_init(b, 2);
        for (uint64_t* b : {bias_empty, pds_ready, dq_free, dkv_free}) mbar_init(b, C::NCW);
        fence_mbar_init();
    }
    if (warp == C::W_MMA) {
        tmem_alloc(tmem_slot, BWD_TMEM_COLS);
        tmem_relinquish();
    }
    if (warp == C::W_PROD && lane == 0) {
        prefetch_tmap(&tm_q); prefetch_tmap(&tm_k); prefetch_tmap(&tm_v); prefetch_tmap(&tm_do);
        prefetch_tmap(&tm_bias);
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

    static_assert(WALK != WALK_BOTH, "all pairs whole, or none");
    const Segments<WALK> seg(p);
    const int n_segs = seg.n;

    if (warp == C::W_PROD) {
        // ------------------------------ producer ------------------------------
        bool ok = true;
        int gs = 0, n_do = 0, n_q = 0, n_bias = 0, n_kv = 0;      // steps; loads issued
        for (int sg = 0; sg < n_segs && ok; ++sg) {
            int bs, h, j;
            seg.decode(sg, bs, h, j);
            const int b = bs / p.S;
            const __nv_bfloat16* xq = p.xq + (static_cast<size_t>(bs) * p.H + h) * p.NTP * 8;
            if (sg > 0) ok = warp_all(mbar_wait(kv_empty, (sg - 1) & 1, wc, 0x40));
            if (!ok) break;
            if (elect_one()) {
                uint8_t* kvb = smem + C::OFF_KV;
                mbar_arrive_expect_tx(kv_full, C::KV_BYTES);
                tma_load_row_tile<DH>(kvb + C::KV_V, &tm_v, kv_full, h, j * TILE, bs);
                tma_load_row_tile<DH>(kvb + C::KV_K, &tm_k, kv_full, h, j * TILE, bs);
                bulk_load(kvb + C::KV_XK, p.xk + (static_cast<size_t>(bs) * p.NTP + j * TILE) * 8, XT_BYTES, kv_full);
            }
            __syncwarp();
            ++n_kv;
            for (int i = 0; i < NT && ok; ++i, ++gs) {
                uint8_t* sb = smem + C::OFF_STAGE;
                if (gs > 0) ok = warp_all(mbar_wait(do_empty, (gs - 1) & 1, wc, 0x42));
                if (!ok) break;
                if (elect_one()) {
                    mbar_arrive_expect_tx(do_full, C::ROWT + XT_BYTES);
                    tma_load_row_tile<DH>(sb + C::ST_DO, &tm_do, do_full, h, i * TILE, bs);
                    bulk_load(sb + C::ST_XQ, xq + static_cast<size_t>(i) * TILE * 8, XT_BYTES, do_full);
                }
                __syncwarp();
                ++n_do;
                if (gs > 0) ok = warp_all(mbar_wait(bias_empty, (gs - 1) & 1, wc, 0x41));
                if (!ok) break;
                if (elect_one()) {
                    uint8_t* bt = smem + C::OFF_BIAS;
                    mbar_arrive_expect_tx(sdp_full, SQ_BYTES);
                    tma_load_4d(bt, &tm_bias, sdp_full, j * TILE, i * TILE, h, b);
                    tma_load_4d(bt + SQ_SUB_BYTES, &tm_bias, sdp_full, j * TILE + 64, i * TILE, h, b);
                }
                __syncwarp();
                ++n_bias;
                if (gs > 0) ok = warp_all(mbar_wait(q_empty, (gs - 1) & 1, wc, 0x46));
                if (!ok) break;
                if (elect_one()) {
                    mbar_arrive_expect_tx(q_full, C::ROWT);
                    tma_load_row_tile<DH>(sb + C::ST_Q, &tm_q, q_full, h, i * TILE, bs);
                }
                __syncwarp();
                ++n_q;
            }
        }
        // The last loads have landed before the CTA exits, also if a wait gave up (a bias load shares its
        // barrier with an MMA commit, which may then never come: a bounded pause instead).
        const WaitCtx dc{tmem_slot + 3, p.status};
        if (n_do > 0) mbar_wait_landed(do_full, (n_do - 1) & 1, dc, 0x43);
        if (n_q > 0) mbar_wait_landed(q_full, (n_q - 1) & 1, dc, 0x47);
        if (n_kv > 0) mbar_wait_landed(kv_full, (n_kv - 1) & 1, dc, 0x45);
        if (!ok && n_bias > 0)
            for (int k = 0; k < 64; ++k) __nanosleep(1000);
    } else if (warp >= C::W_MMA) {
        // ------------------------------ mma issuers ------------------------------
        // Each warp runs its loop with all lanes (uniform control flow: operand descriptors stay in
        // uniform registers) and elects one lane to issue.
        constexpr uint32_t IDESC_SDP = make_idesc_bf16(128, 128, 0, 0);
        // N = the head-dim columns that hold data (the rest of a wider kernel's tile is zero fill)
        const uint32_t IDESC_DKV = make_idesc_bf16(128, 16 * p.KB, 0, 1);
        const uint32_t IDESC_DQ = make_idesc_bf16(128, 16 * p.KB, 1, 1);
        const uint32_t sb = smem_u32(smem + C::OFF_STAGE), kvb = smem_u32(smem + C::OFF_KV);
        const uint32_t aZero = smem_u32(smem + C::OFF_ZERO);
        const int role = warp - C::W_MMA;          // 0: S/dP, 1: dV/dK, 2: dQ
        bool ok = true;
        int gs = 0;
        for (int sg = 0; sg < n_segs && ok; ++sg) {
            for (int i = 0; i < NT && ok; ++i, ++gs) {
                if (role == 0) {
                    ok = warp_all(mbar_wait(do_full, gs & 1, wc, 0x50));
                    if (ok && i == 0) ok = warp_all(mbar_wait(kv_full, sg & 1, wc, 0x51));
                    // dK has consumed dS^T in the columns of dP'
                    if (ok && gs > 0) ok = warp_all(mbar_wait(dk_done, (gs - 1) & 1, wc, 0x52));
                    if (!ok) break;
                    tc_fence_after();
                    const uint64_t d_xq = xt_desc(sb + C::ST_XQ, aZero);
                    if (elect_one()) {
                        const uint32_t do_lo = RD::kmajor_lo(sb + C::ST_DO), v_lo = RD::kmajor_lo(kvb + C::KV_V);
#pragma unroll
                        for (int kk = 0; kk < RT::KBLOCKS; ++kk)
                            if (kk < p.KB)      // the others are zero-filled blocks past the true head dim
                                umma_ss(tmem + C::TMEM_DP, RD::kmajor(v_lo, kk), RD::kmajor(do_lo, kk), IDESC_SDP, kk > 0);
                        // - delta: the extra contraction block
                        umma_ss(tmem + C::TMEM_DP, xt_desc(smem_u32(smem + C::OFF_XDP), aZero), d_xq, IDESC_SDP, 1u);
                    }
                    __syncwarp();
                    ok = warp_all(mbar_wait(q_full, gs & 1, wc, 0x57));
                    // dQ of the previous step, in the columns of S', is read
                    if (ok && gs > 0) ok = warp_all(mbar_wait(dq_free, (gs - 1) & 1, wc, 0x56));
                    if (!ok) break;
                    tc_fence_after();
                    if (elect_one()) {
                        const uint32_t q_lo = RD::kmajor_lo(sb + C::ST_Q), k_lo = RD::kmajor_lo(kvb + C::KV_K);
#pragma unroll
                        for (int kk = 0; kk < RT::KBLOCKS; ++kk)
                            if (kk < p.KB)
                                umma_ss(tmem + C::TMEM_S, RD::kmajor(k_lo, kk), RD::kmajor(q_lo, kk), IDESC_SDP, kk > 0);
                        // + (mask - LSE) / scale
                        umma_ss(tmem + C::TMEM_S, xt_desc(kvb + C::KV_XK, aZero), d_xq, IDESC_SDP, 1u);
                        umma_commit(sdp_full);
                    }
                    __syncwarp();
                } else if (role == 1) {
                    // the first MMA of a segment overwrites dK / dV: the previous one's must be out
                    if (i == 0 && sg > 0) ok = warp_all(mbar_wait(dkv_free, (sg - 1) & 1, wc, 0x55));
                    if (ok) ok = warp_all(mbar_wait(pds_ready, gs & 1, wc, 0x53));
                    if (!ok) break;
                    tc_fence_after();
                    if (elect_one()) {
                        const uint32_t q_lo = RD::mnmajor_lo(sb + C::ST_Q), do_lo = RD::mnmajor_lo(sb + C::ST_DO);
                        const uint32_t acc = (i > 0) ? 1u : 0u;
#pragma unroll
                        for (int kk = 0; kk < 8; ++kk)      // dV first: dQ waits for its columns
                            umma_ts(tmem + C::TMEM_DV, tmem + C::p_col(kk), RD::mnmajor(do_lo, kk), IDESC_DKV, kk > 0 ? 1u : acc);
                        umma_commit(dv_done);
                        umma_commit(do_empty);
#pragma unroll
                        for (int kk = 0; kk < 8; ++kk)
                            umma_ts(tmem + C::TMEM_DK, tmem + C::ds_col(kk), RD::mnmajor(q_lo, kk), IDESC_DKV, kk > 0 ? 1u : acc);
                        umma_commit(dk_done);
                        umma_commit(q_empty);
                        if (i == NT - 1) {
                            umma_commit(dkv_full);
                            umma_commit(kv_empty);
                        }
                    }
                    __syncwarp();
                } else {
                    ok = warp_all(mbar_wait(dv_done, gs & 1, wc, 0x58));      // implies pds_ready
                    if (!ok) break;
                    tc_fence_after();
                    if (elect_one()) {
                        const uint32_t ds_lo = SqDesc::mnmajor_lo(smem_u32(smem + C::OFF_DS));
                        const uint32_t k_lo = RD::mnmajor_lo(kvb + C::KV_K);
#pragma unroll
                        for (int kk = 0; kk < 8; ++kk)
                            umma_ss(tmem + C::TMEM_DQ, SqDesc::mnmajor(ds_lo, kk), RD::mnmajor(k_lo, kk), IDESC_DQ, kk > 0);
                        umma_commit(dq_full);
                        if (i == NT - 1) umma_commit(kv_empty);
                    }
                    __syncwarp();
                }
            }
        }
    } else {
        // ------------------------------ compute groups ------------------------------
        const int g = warp >> 2;             // q columns 32g .. 32g+31 of the tile
        const int row = tid & 127;           // kv row within the tile == TMEM lane
        const uint32_t lane_base = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16);
        const uint32_t tS = lane_base + C::TMEM_S + 32 * g, tDP = lane_base + C::TMEM_DP + 32 * g;
        const uint32_t aDS = smem_u32(smem + C::OFF_DS);
        // this thread's column of the bias tile ([q][kv], swizzled by q & 7), first row of the group
        const uint32_t aBias = smem_u32(smem + C::OFF_BIAS) + (row >> 6) * SQ_SUB_BYTES + 32 * g * 128 + (row & 7) * 2;
        const uint32_t bchunk = (row & 63) >> 3;
        const uint32_t scratch_w = smem_u32(tmem_slot + 2);       // a word nobody reads
        // whole pairs: this thread's 16-byte words of the partial sums of dQ, 32 lanes side by side
        float4* part = reinterpret_cast<float4*>(p.dq_scratch) + static_cast<size_t>(blockIdx.x) * p.scratch_stride + lane;
        const int w4 = warp & 3, wrow0 = 32 * w4;
        const bool has_cols = 32 * g < p.Dt;      // warp-uniform: head-dim columns of this group that exist
        // 32 columns of 32 rows as bf16: lane t of a quad of rows stores chunk t of each of the four, 64
        // contiguous bytes per row
        auto store_rows = [&](__nv_bfloat16* out, const float (&v)[32], float sc, int row0) {
            uint4 u[4];
#pragma unroll
            for (int c8 = 0; c8 < 4; ++c8)
                u[c8] = make_uint4(pack_bf16(v[c8 * 8 + 0] * sc, v[c8 * 8 + 1] * sc), pack_bf16(v[c8 * 8 + 2] * sc, v[c8 * 8 + 3] * sc),
                                   pack_bf16(v[c8 * 8 + 4] * sc, v[c8 * 8 + 5] * sc), pack_bf16(v[c8 * 8 + 6] * sc, v[c8 * 8 + 7] * sc));
            quad_transpose(u);
            const int r0 = row0 + (lane & ~3), col = 32 * g + (lane & 3) * 8;
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (r0 + e < p.N) *reinterpret_cast<uint4*>(out + (r0 + e) * p.lay.n + col) = u[e];
            __syncwarp();
        };
        constexpr bool whole = WALK == WALK_WHOLE;
        bool ok = true;
        int gs = 0;
        const float2 c1x2 = make_float2(p.c1, p.c1), l2e2 = make_float2(LOG2E, LOG2E);

        for (int sg = 0; sg < n_segs && ok; ++sg) {
            int bs, h, j;
            seg.decode(sg, bs, h, j);
            const size_t head = bs * p.lay.row + h * p.lay.h;
            for (int i = 0; i < NT && ok; ++i, ++gs) {
                ok = warp_all(mbar_wait(sdp_full, gs & 1, wc, 0x63));
                if (!ok) break;
                tc_fence_after();
                // Per element: x = S' c1 + bias log2e (S' already carries mask and -LSE through the extra
                // contraction block), P = exp2(x), dS = P dP' (dP' already carries -delta).
                uint32_t dep = 0;
#pragma unroll
                for (int ch = 0; ch < 2; ++ch) {          // 16 columns at a time
                    uint32_t sv[16], dv[16], bq[16];
                    tmem_ld16(tS + 16 * ch, sv);
                    tmem_ld16(tDP + 16 * ch, dv);
#pragma unroll
                    for (int k = 0; k < 16; ++k)
                        bq[k] = lds_u16(aBias + (16 * ch + k) * 128 + ((bchunk ^ (k & 7)) << 4));
                    tmem_wait_ld();
                    uint32_t pkp[8], pkd[8];
                    float2 dsv[8];
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        const float2 b2 = fmul2(make_float2(__uint_as_float(bq[2 * k] << 16), __uint_as_float(bq[2 * k + 1] << 16)), l2e2);
                        const float2 x2 = ffma2(u2f2(sv[2 * k], sv[2 * k + 1]), c1x2, b2);
                        const float2 p2 = make_float2(ex2(x2.x), ex2(x2.y));
                        const float2 ds2 = fmul2(p2, u2f2(dv[2 * k], dv[2 * k + 1]));
                        pkp[k] = pack_bf16(p2.x, p2.y);
                        pkd[k] = pack_bf16(ds2.x, ds2.y);
                        dsv[k] = ds2;
                    }
#pragma unroll
                    for (int k = 0; k < 8; ++k) dep ^= pkp[k];     // depends on every bias value read
                    if (ch == 1) mbar_release_after_loads(bias_empty, dep, scratch_w);
                    // (the dS tile and the columns are free: S' of this step waited for dQ of the previous one)
                    tmem_st8(lane_base + C::p_col(2 * g + ch), pkp);
                    tmem_st8(lane_base + C::ds_col(2 * g + ch), pkd);
#pragma unroll
                    for (int c = 0; c < 2; ++c)
                        sts128(aDS + sq_chunk_off(row, 4 * g + 2 * ch + c),
                               make_uint4(pkd[4 * c], pkd[4 * c + 1], pkd[4 * c + 2], pkd[4 * c + 3]));
                    if constexpr (DBIAS_HERE != DBIAS_NO) {
                        // one S row: this step's dS tile is the dBias tile (q tile i, kv tile j)
                        const int kv = j * TILE + row, q0 = i * TILE + 32 * g + 16 * ch;
                        const size_t at = ((static_cast<size_t>(bs) * p.H + h) * p.N + q0) * p.N + kv;
                        if constexpr (DBIAS_HERE == DBIAS_F32) {
                            float* out = static_cast<float*>(p.dbias) + at;
#pragma unroll
                            for (int k = 0; k < 8; ++k) {
                                if (kv < p.N && q0 + 2 * k < p.N) out[static_cast<size_t>(2 * k) * p.N] = dsv[k].x;
                                if (kv < p.N && q0 + 2 * k + 1 < p.N) out[static_cast<size_t>(2 * k + 1) * p.N] = dsv[k].y;
                            }
                        } else {
                            // lanes 2n and 2n+1 exchange halves: the even one stores both kv of the even q row, the
                            // odd one those of the odd row
                            const bool odd = lane & 1;
                            uint32_t* out = reinterpret_cast<uint32_t*>(static_cast<__nv_bfloat16*>(p.dbias) + at - (odd ? 1 : 0));
#pragma unroll
                            for (int k = 0; k < 8; ++k) {
                                const uint32_t other = __shfl_xor_sync(0xffffffffu, pkd[k], 1);
                                const uint32_t w = odd ? __byte_perm(other, pkd[k], 0x7632) : __byte_perm(pkd[k], other, 0x5410);
                                const int q = q0 + 2 * k + (odd ? 1 : 0);
                                if (kv < p.N && q < p.N) out[static_cast<size_t>(2 * k + (odd ? 1 : 0)) * (p.N >> 1)] = w;
                            }
                        }
                    }
                }
                if (!ok) break;
                tmem_wait_st();
                tc_fence_before();
                fence_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(pds_ready);

                // dQ of the step: 32 rows, 32 head-dim columns
                const bool rows = has_cols && i * TILE + wrow0 < p.N;      // warp-uniform
                float4* ps = part + static_cast<size_t>((i * 4 + w4) * (DH / 4) + 8 * g) * 32;
                float4 old[8];
                if (whole && j > 0 && j == NT - 1 && rows) {   // requested before the wait
#pragma unroll
                    for (int c = 0; c < 8; ++c) old[c] = __ldcg(ps + c * 32);
                }
                ok = warp_all(mbar_wait(dq_full, gs & 1, wc, 0x68));
                if (!ok) break;
                tc_fence_after();
                float dqv[32];
                tmem_ld_f32<32>(lane_base + C::TMEM_DQ + 32 * g, dqv);
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(dq_free);
                if (rows) {
                    if (whole && j == NT - 1) {
                        if (j > 0) {
#pragma unroll
                            for (int c = 0; c < 8; ++c) {
                                dqv[4 * c] += old[c].x; dqv[4 * c + 1] += old[c].y;
                                dqv[4 * c + 2] += old[c].z; dqv[4 * c + 3] += old[c].w;
                            }
                        }
                        store_rows(p.dq + head, dqv, p.scale, i * TILE + wrow0);
                    } else if (whole && j == 0) {
#pragma unroll
                        for (int c = 0; c < 8; ++c)
                            __stcg(ps + c * 32, make_float4(dqv[4 * c], dqv[4 * c + 1], dqv[4 * c + 2], dqv[4 * c + 3]));
                    } else if (whole) {
                        // added in L2, nothing to wait for here; the thread that reads the sum in the last segment is
                        // the same (loaded, added and stored by each segment instead: S=37, N=768, H=4 186 -> 194 us)
#pragma unroll
                        for (int c = 0; c < 8; ++c)
                            red_add_v4(reinterpret_cast<float*>(ps + c * 32), dqv[4 * c], dqv[4 * c + 1], dqv[4 * c + 2], dqv[4 * c + 3]);
                    } else {
                        // fp32 accumulator [B*S][N][H][DH]: lane t of a quad adds chunks t and 4 + t of four rows
                        const int r0 = i * TILE + wrow0 + (lane & ~3);
                        float* acc = p.dq_acc + ((static_cast<size_t>(bs) * p.N + r0) * p.H + h) * DH + 32 * g + 4 * (lane & 3);
#pragma unroll
                        for (int hf = 0; hf < 2; ++hf) {
                            uint4 u[4];
#pragma unroll
                            for (int c = 0; c < 4; ++c)
                                u[c] = make_uint4(__float_as_uint(dqv[16 * hf + 4 * c] * p.scale), __float_as_uint(dqv[16 * hf + 4 * c + 1] * p.scale),
                                                  __float_as_uint(dqv[16 * hf + 4 * c + 2] * p.scale), __float_as_uint(dqv[16 * hf + 4 * c + 3] * p.scale));
                            quad_transpose(u);
#pragma unroll
                            for (int e = 0; e < 4; ++e)
                                if (r0 + e < p.N)
                                    red_add_v4(acc + static_cast<size_t>(e) * p.H * DH + 16 * hf, __uint_as_float(u[e].x),
                                               __uint_as_float(u[e].y), __uint_as_float(u[e].z), __uint_as_float(u[e].w));
                        }
                        __syncwarp();
                    }
                }
            }
            if (!ok) break;
            // dK and dV of the segment, 32 columns of each
            ok = warp_all(mbar_wait(dkv_full, sg & 1, wc, 0x69));
            if (!ok) break;
            tc_fence_after();
#pragma unroll
            for (int t = 0; t < 2; ++t) {      // 0: dK, 1: dV
                float v[32];
                tmem_ld_f32<32>(lane_base + (t ? C::TMEM_DV : C::TMEM_DK) + 32 * g, v);
                if (t == 1) {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(dkv_free);
                }
                if (has_cols) store_rows((t ? p.dv : p.dk) + head, v, t ? 1.0f : p.scale, j * TILE + wrow0);
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (tid == 0) { report_abort(wc); report_abort(WaitCtx{tmem_slot + 3, p.status}); }
    if (warp == C::W_MMA) tmem_dealloc(tmem, BWD_TMEM_COLS);
}

}  // namespace evo
