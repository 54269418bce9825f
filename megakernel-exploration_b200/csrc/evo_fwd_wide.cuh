// EvoAttention forward, D = 96 and 128 (see evo_fwd.cu for the interface and the D <= 64 kernel).
//
// Two item streams per CTA, as at D = 64, but two streams with Q, K and V of their own do not fit shared
// memory.  So the streams are two q tiles of one (row, head) and share its K and V tiles:
//
//   warps 0-3, 4-7   softmax of stream 0 and 1: thread = one q row, all 128 columns of a tile; x stays in
//                    registers, P (bf16) overwrites the S columns it came from
//   warp 8           producer: Q of each stream, K (two buffers) with its mask tile, V (one buffer)
//   warps 9, 10      one MMA warp per stream: S' = Q K^T + mask block, then PV (+)= P V, in turn
//   warp 11          bias: half tiles of 64 columns through a ring of three, in the order in which the streams
//                    read them (stream 0 left, right, stream 1 left, right, next tile)
//
// A row of one q tile (N <= 128) has no second one to share with: the streams are then two items, each
// with its own K buffer, and V follows K into that buffer as soon as S' is complete (OWN).  A stream
// without an item (an odd number of q tiles, or the last item) computes on zero-filled tiles and stores nothing.
//
// What bounds it: a stream's chain PV -> S' -> softmax (2400 clocks of tensor core and barriers, 3400 of
// softmax per tile), of which two are in flight, so 3000 clocks per tile against 1024 for its exponentials
// and 1100 for its products; and 6000 clocks per item for the stores, which all SMs issue at about the same
// time (128 KB each).  Measured against two groups of 64 columns on one item, which waited for each
// other on every tile: B=1, S=128, N=768, H=4, D=128 0.301 -> 0.244 ms; S=1024, N=64, H=16 0.509 -> 0.358;
// S=300, N=600, H=8, D=96 1.04 -> 0.83.  Without turns on the exp2 pass the streams fall into step and queue
// for the tensor core together (0.272); handing the turn on halfway through the pass 0.279.
#pragma once
#include "evo_bias_ring.cuh"

namespace evo {

struct FwdWideCfg {
    static constexpr int DH = 128;
    static constexpr int NSW = 8;                              // softmax warps
    static constexpr int W_PROD = NSW, W_MMA = NSW + 1, W_BIAS = NSW + 3;
    static constexpr int THREADS = (NSW + 4) * 32;
    // setmaxnreg budgets: the pool is the launch count (the cap ptxas derives from the launch bound) times the threads
    static constexpr int REGS_LAUNCH = (65536 / THREADS) & ~7;
    static constexpr int REGS_SOFTMAX = 216, REGS_OTHER = 72;
    static_assert((REGS_SOFTMAX * NSW + REGS_OTHER * 4) * 32 <= REGS_LAUNCH * THREADS, "register pool");
    static constexpr uint32_t ROWT = RowTile<DH>::BYTES;       // one [128][128] bf16 tile
    static constexpr int NK = 2;                               // K buffers
    static constexpr int NR = WideBiasRing::SLOTS, NF = WideBiasRing::PER_ROUND;   // half tiles of bias, their "full" barriers
    static constexpr uint32_t OFF_Q = 0, OFF_K = 2 * ROWT, OFF_V = OFF_K + NK * ROWT, OFF_BIAS = OFF_V + ROWT;
    static constexpr uint32_t OFF_XK = OFF_BIAS + NR * SQ_SUB_BYTES;
    // constant extra tiles, above every tile that refers to the zero tile
    static constexpr uint32_t OFF_XQ = OFF_XK + NK * XT_BYTES; // rows (1, 1, 1, 0, ...)
    static constexpr uint32_t OFF_ZERO = OFF_XQ + XT_BYTES;
    static constexpr uint32_t OFF_BARS = OFF_ZERO + XT_BYTES;
    static constexpr int BARS = 3 * 2 + 1 + 2 * NK + 3 * 2 + NF + NR + 16;
    static constexpr uint32_t OFF_MISC = OFF_BARS + BARS * 8;
    static constexpr uint32_t SMEM_BYTES = OFF_MISC + 16 + 1024;   // + alignment slack
    static constexpr uint32_t TMEM_S = 0, TMEM_PV = 256;       // + 128 s; P: 64 columns over S
    static constexpr uint32_t TMEM_COLS = 512;
    static_assert(SMEM_BYTES <= 232448, "shared memory budget");
    static_assert(OFF_BIAS % 1024 == 0, "tile alignment");
};

template <bool GATED>
__global__ void __launch_bounds__(FwdWideCfg::THREADS, 1)
evo_fwd_wide_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                    const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_bias, const FwdParams p) {
    using C = FwdWideCfg;
    constexpr int DH = C::DH, NK = C::NK, NR = C::NR, NF = C::NF;
    using RT = RowTile<DH>;
    using RD = RowDesc<DH>;

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::OFF_BARS);
    uint64_t* q_full = bars;                 // [stream]
    uint64_t* q_empty = q_full + 2;          // [stream]
    uint64_t* v_full = q_empty + 2;          // [0], or [stream] (OWN)
    uint64_t* v_empty = v_full + 2;          // not OWN: both PV of a tile are complete
    uint64_t* k_full = v_empty + 1;          // [buffer]: K and mask tile
    uint64_t* k_empty = k_full + NK;         // [buffer]
    uint64_t* s_full = k_empty + NK;         // [stream]
    uint64_t* p_ready = s_full + 2;          // [stream]
    uint64_t* pv_done = p_ready + 2;         // [stream]
    uint64_t* bias_full = pv_done + 2;       // [NF]: half tile of the round (evo_bias_ring.cuh)
    uint64_t* bias_empty = bias_full + NF;   // [NR]: slot
    uint64_t* turn = bias_empty + NR;        // [stream][tile parity][warp]: the warp has left its exp2 pass
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + C::OFF_MISC);
    volatile uint32_t* abort_flag = tmem_slot + 1;

    const int tid = threadIdx.x;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);      // uniform: what derives from it stays in uniform registers
    const int lane = tid & 31;
    const int NT = (p.N + TILE - 1) / TILE;
    const bool own = NT == 1;
    WaitCtx wc{abort_flag, p.status};

    if (tid == 0) {
        *abort_flag = 0;
        tmem_slot[3] = 0;                   // the abort word of the waits before exit
        for (int i = 0; i < 2; ++i) {
            mbar_init(&q_full[i], 1); mbar_init(&q_empty[i], 1);
            mbar_init(&v_full[i], 1);
            mbar_init(&s_full[i], 1); mbar_init(&p_ready[i], 4); mbar_init(&pv_done[i], 1);
        }
        mbar_init(v_empty, 2);
        for (int i = 0; i < NK; ++i) { mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], own ? 1 : 2); }
        for (int i = 0; i < NF; ++i) mbar_init(&bias_full[i], 1);
        for (int i = 0; i < NR; ++i) mbar_init(&bias_empty[i], 4);
        for (int i = 0; i < 16; ++i) mbar_init(&turn[i], 1);
        fence_mbar_init();
    }
    if (warp == C::W_PROD) {
        tmem_alloc(tmem_slot, C::TMEM_COLS);
        tmem_relinquish();
        if (lane == 0) { prefetch_tmap(&tm_q); prefetch_tmap(&tm_k); prefetch_tmap(&tm_v); prefetch_tmap(&tm_bias); }
    }
    if (tid < 128) {
        *reinterpret_cast<uint4*>(smem + C::OFF_XQ + tid * 16) = make_uint4(0x3f803f80u, 0x3f80u, 0u, 0u);
        *reinterpret_cast<uint4*>(smem + C::OFF_ZERO + tid * 16) = make_uint4(0u, 0u, 0u, 0u);
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    chain_wait();

    // Items: (head, pair of q tiles, row, batch), or single ones dealt to the streams in turn (OWN).
    const int first = blockIdx.x, stride = gridDim.x, per_cta = stride * (own ? 2 : 1);
    const int n_items = (p.total_items > first) ? (p.total_items - first + per_cta - 1) / per_cta : 0;
    auto items_of = [&](int s) -> FwdItem {
        const FwdStep w = FwdStep::of(first + (own ? s * stride : 0), p.H, p.QT, p.NG);
        return FwdItem{w.h, w.qt, w.g, w.b};
    };
    auto advance = [&](FwdItem& x) { x.next(p.S, 1, p); };
    // the item of stream s: a missing one is the (empty) tile behind the last of row 0
    auto tile_of = [&](const FwdItem& x, int s) -> FwdItem {
        if (!own) return FwdItem{x.h, 2 * x.qt + s, x.row, x.b};
        return x.valid(p) ? x : FwdItem{0, 1, 0, 0};
    };

    if (warp >= C::W_PROD) {
        reg_dec<C::REGS_OTHER>();
        if (warp == C::W_PROD) {
            // ------------------------------ producer ------------------------------
            // The warp runs with all lanes and elects one to issue.
            FwdItem cur0 = items_of(0), cur1 = items_of(1);
            bool ok = true;
            int n_k0 = 0, n_k1 = 0, n_v = 0, n_q0 = 0, n_q1 = 0;   // loads so far
            auto load_q = [&](int s, const FwdItem& x, int& cnt) {
                if (cnt > 0) ok = warp_all(mbar_wait(&q_empty[s], (cnt - 1) & 1, wc, 0x10));
                if (!ok) return;
                if (elect_one()) {
                    mbar_arrive_expect_tx(&q_full[s], C::ROWT);
                    tma_load_row_tile<DH>(smem + C::OFF_Q + s * C::ROWT, &tm_q, &q_full[s], x.h, x.qt * TILE, x.bs(p));
                }
                __syncwarp();
                ++cnt;
            };
            auto load_k = [&](int kb, const FwdItem& x, int j) {
                // four mask values per lane, requested before the wait
                const int c = j * TILE + 4 * lane;
                uint2 mw = make_uint2(0u, 0u);
                if (c < p.N) mw = __ldg(reinterpret_cast<const uint2*>(p.mask + static_cast<size_t>(x.bs(p)) * p.N + c));
                const int cnt = kb ? n_k1 : n_k0;
                if (cnt > 0) ok = warp_all(mbar_wait(&k_empty[kb], (cnt - 1) & 1, wc, 0x11));
                if (!ok) return;
                n_k0 += kb ^ 1;
                n_k1 += kb;
                if (elect_one()) {
                    mbar_expect_tx(&k_full[kb], C::ROWT);
                    tma_load_row_tile<DH>(smem + C::OFF_K + kb * C::ROWT, &tm_k, &k_full[kb], x.h, j * TILE, x.bs(p));
                }
                __syncwarp();
                const float mv[4] = {bf16_lo(mw.x), bf16_hi(mw.x), bf16_lo(mw.y), bf16_hi(mw.y)};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const uint2 w = mask_term(c < p.N ? mv[e] : -INFINITY, p.inv_scale);
                    *reinterpret_cast<uint4*>(smem + C::OFF_XK + kb * XT_BYTES + (4 * lane + e) * 16) = make_uint4(w.x, w.y, 0u, 0u);
                }
                fence_async_smem();
                __syncwarp();
                if (elect_one()) mbar_arrive(&k_full[kb]);
                __syncwarp();
            };
            auto load_v = [&](const FwdItem& x, int j) {
                if (n_v > 0) ok = warp_all(mbar_wait(v_empty, (n_v - 1) & 1, wc, 0x12));
                if (!ok) return;
                if (elect_one()) {
                    mbar_arrive_expect_tx(v_full, C::ROWT);
                    tma_load_row_tile<DH>(smem + C::OFF_V, &tm_v, v_full, x.h, j * TILE, x.bs(p));
                }
                __syncwarp();
                ++n_v;
            };
            if (own) {
                for (int it = 0; it < n_items && ok; ++it) {
                    const FwdItem x0 = tile_of(cur0, 0), x1 = tile_of(cur1, 1);
                    load_q(0, x0, n_q0);
                    if (ok) load_k(0, x0, 0);
                    if (ok) load_q(1, x1, n_q1);
                    if (ok) load_k(1, x1, 0);
                    advance(cur0);
                    advance(cur1);
                }
            } else {
                // V a tile behind K: its buffer is free only when both PV of the tile before are complete
                int r = 0, vj = 0;
                FwdItem vx = cur0;
                for (int it = 0; it < n_items && ok; ++it) {
                    for (int j = 0; j < NT && ok; ++j, ++r) {
                        if (j == 0) load_q(0, tile_of(cur0, 0), n_q0);
                        if (ok) load_k(r & 1, cur0, j);
                        if (ok && r > 0) load_v(vx, vj);
                        if (ok && j == 0) load_q(1, tile_of(cur0, 1), n_q1);
                        vx = cur0;
                        vj = j;
                    }
                    advance(cur0);
                }
                if (ok && r > 0) load_v(vx, vj);
            }
            // the last loads have landed before the CTA exits (also if a wait gave up)
            const WaitCtx dc{tmem_slot + 3, p.status};
            if (n_k0 > 0) mbar_wait_landed(&k_full[0], (n_k0 - 1) & 1, dc, 0x13);
            if (n_k1 > 0) mbar_wait_landed(&k_full[1], (n_k1 - 1) & 1, dc, 0x13);
            if (n_v > 0) mbar_wait_landed(v_full, (n_v - 1) & 1, dc, 0x14);
            if (n_q0 > 0) mbar_wait_landed(&q_full[0], (n_q0 - 1) & 1, dc, 0x15);
            if (n_q1 > 0) mbar_wait_landed(&q_full[1], (n_q1 - 1) & 1, dc, 0x15);
        } else if (warp == C::W_BIAS) {
            // ------------------------------ bias ------------------------------
            FwdItem cur0 = items_of(0), cur1 = items_of(1);
            bool ok = true;
            WideBiasRing ring = WideBiasRing::at(0);
            int n_loads = 0;
            for (int it = 0; it < n_items && ok; ++it) {
                const FwdItem x0 = tile_of(cur0, 0), x1 = tile_of(own ? cur1 : cur0, 1);
                for (int j = 0; j < NT && ok; ++j) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        if (ok && ring.use > 0) ok = warp_all(mbar_wait(&bias_empty[ring.slot], ring.empty_parity(), wc, 0x16));
                        if (!ok) break;
                        const FwdItem& x = i < 2 ? x0 : x1;
                        uint64_t* full = &bias_full[WideBiasRing::full_bar(i >> 1, i & 1)];
                        if (elect_one()) {
                            mbar_arrive_expect_tx(full, SQ_SUB_BYTES);
                            tma_load_4d(smem + C::OFF_BIAS + ring.slot * SQ_SUB_BYTES, &tm_bias, full, j * TILE + 64 * (i & 1),
                                        x.qt * TILE, x.h, x.b);
                        }
                        __syncwarp();
                        ++n_loads;
                        ring.advance(1);
                    }
                }
                advance(cur0);
                advance(cur1);
            }
            const WaitCtx dc{tmem_slot + 3, p.status};
            for (int i = (n_loads > NF ? n_loads - NF : 0); i < n_loads; ++i)
                mbar_wait_landed(&bias_full[i % NF], WideBiasRing::full_parity(i / NF), dc, 0x17);
        } else {
            // ------------------------------ MMA warp of one stream ------------------------------
            const int s = warp - C::W_MMA;
            constexpr uint32_t IDESC_S = make_idesc_bf16(128, 128, 0, 0);
            const uint32_t IDESC_PV = make_idesc_bf16(128, 16 * p.KB, 0, 1);   // N = the head-dim columns that hold data
            const uint32_t aK = smem_u32(smem + C::OFF_K), aZero = smem_u32(smem + C::OFF_ZERO), aXK = smem_u32(smem + C::OFF_XK);
            const uint64_t d_xq = xt_desc(smem_u32(smem + C::OFF_XQ), aZero);
            const uint32_t q_lo = RD::kmajor_lo(smem_u32(smem + C::OFF_Q + s * C::ROWT));
            const uint32_t t_s = tmem + C::TMEM_S + 128 * s, t_pv = tmem + C::TMEM_PV + DH * s;
            uint64_t* vf = own ? &v_full[s] : v_full;
            bool ok = true;
            FwdItem cur = items_of(s);
            int n = 0, n_v = 0;
            for (int it = 0; it < n_items && ok; ++it) {
                for (int j = 0; j < NT && ok; ++j, ++n) {
                    // S' of the tile: its columns are free once PV of the tile before has read P from them
                    const int kb = own ? s : n & 1;
                    if (j == 0) ok = warp_all(mbar_wait(&q_full[s], it & 1, wc, 0x20));
                    if (ok) ok = warp_all(mbar_wait(&k_full[kb], (own ? n : n >> 1) & 1, wc, 0x21));
                    if (ok && n > 0) ok = warp_all(mbar_wait(&pv_done[s], (n - 1) & 1, wc, 0x25));
                    if (!ok) break;
                    tc_fence_after();
                    if (elect_one()) {
                        const uint32_t k_lo = RD::kmajor_lo(aK + kb * C::ROWT);
#pragma unroll
                        for (int kk = 0; kk < RT::KBLOCKS; ++kk)
                            if (kk < p.KB)          // blocks past the true head dim are zero-filled: skipped
                                umma_ss(t_s, RD::kmajor(q_lo, kk), RD::kmajor(k_lo, kk), IDESC_S, kk > 0);
                        umma_ss(t_s, d_xq, xt_desc(aXK + kb * XT_BYTES, aZero), IDESC_S, 1u);
                        umma_commit(&s_full[s]);
                        if (!own) umma_commit(&k_empty[kb]);
                        if (j == NT - 1) umma_commit(&q_empty[s]);
                    }
                    __syncwarp();
                    if (own) {
                        // V takes K's place
                        ok = warp_all(mbar_wait(&s_full[s], n & 1, wc, 0x26));
                        if (!ok) break;
                        const FwdItem x = tile_of(cur, s);
                        if (elect_one()) {
                            mbar_arrive_expect_tx(vf, C::ROWT);
                            tma_load_row_tile<DH>(smem + C::OFF_K + s * C::ROWT, &tm_v, vf, x.h, 0, x.bs(p));
                        }
                        __syncwarp();
                        ++n_v;
                    }
                    ok = warp_all(mbar_wait(vf, n & 1, wc, 0x24));
                    if (ok) ok = warp_all(mbar_wait(&p_ready[s], n & 1, wc, 0x23));
                    if (!ok) break;
                    tc_fence_after();
                    if (elect_one()) {
                        const uint32_t v_lo = RD::mnmajor_lo(own ? aK + s * C::ROWT : smem_u32(smem + C::OFF_V));
#pragma unroll
                        for (int kk = 0; kk < 8; ++kk)
                            umma_ts(t_pv, t_s + kk * 8, RD::mnmajor(v_lo, kk), IDESC_PV, (kk > 0 || j > 0) ? 1u : 0u);
                        umma_commit(&pv_done[s]);
                        umma_commit(own ? &k_empty[s] : v_empty);
                    }
                    __syncwarp();
                }
                advance(cur);
            }
            if (n_v > 0) mbar_wait_landed(vf, (n_v - 1) & 1, WaitCtx{tmem_slot + 3, p.status}, 0x18);
        }
    } else {
        reg_inc<C::REGS_SOFTMAX>();
        // ------------------------------ softmax warps of one stream ------------------------------
        const int s = warp >> 2;
        const int row = tid & 127;           // q row within the tile == TMEM lane
        const uint32_t lane_base = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16);
        const uint32_t tS = lane_base + C::TMEM_S + 128 * s, tPV = lane_base + C::TMEM_PV + DH * s;
        const uint32_t scratch_w = smem_u32(tmem_slot + 2);           // a word nobody reads
        const uint32_t aBias = smem_u32(smem + C::OFF_BIAS);
        const float2 sc2 = make_float2(p.scale, p.scale);
        bool ok = true;
        int n = 0;
        WideBiasRing ring = WideBiasRing::at(2 * s);
        FwdItem cur = items_of(s);
        for (int it = 0; it < n_items && ok; ++it) {
            float m = -INFINITY, l = 0.f;
            for (int j = 0; j < NT; ++j, ++n) {
                ok = warp_all(mbar_wait_both(&bias_full[WideBiasRing::full_bar(s, 0)], WideBiasRing::full_parity(n), &s_full[s], n & 1, wc, 0x31));
                if (!ok) break;
                tc_fence_after();
                // pass 1: x = S' * scale + bias and the row maximum, 32 columns at a time
                float2 xh[64];
                float tmx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
                uint32_t sv[2][32];
                tmem_ld32(tS, sv[0]);
#pragma unroll
                for (int ch = 0; ch < 4; ++ch) {
                    uint32_t (&cv)[32] = sv[ch & 1];
                    if (ch == 2) {
                        ok = warp_all(mbar_wait(&bias_full[WideBiasRing::full_bar(s, 1)], WideBiasRing::full_parity(n), wc, 0x32));
                        if (!ok) break;
                    }
                    uint4 bv[4];
#pragma unroll
                    for (int q4 = 0; q4 < 4; ++q4) bv[q4] = lds128(aBias + ring.slot * SQ_SUB_BYTES + sq_chunk_off(row, (ch & 1) * 4 + q4));
                    tmem_wait_ld();
                    if (ch < 3) tmem_ld32(tS + 32 * (ch + 1), sv[(ch + 1) & 1]);
#pragma unroll
                    for (int q4 = 0; q4 < 4; ++q4) {
                        const uint32_t bw[4] = {bv[q4].x, bv[q4].y, bv[q4].z, bv[q4].w};
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const int k = q4 * 4 + e;
                            const float2 x = ffma2(u2f2(cv[2 * k], cv[2 * k + 1]), sc2, bf16x2_f2(bw[e]));
                            tmx[e] = fmax3_nan(tmx[e], x.x, x.y);
                            xh[ch * 16 + k] = x;
                        }
                    }
                    if (ch & 1) {
                        // the maximum depends on every bias value read: the half tile may be refilled
                        const float dep = fmax_nan(fmax3_nan(tmx[0], tmx[1], tmx[2]), tmx[3]);
                        mbar_release_after_loads(&bias_empty[ring.slot], __float_as_uint(dep), scratch_w);
                        ring.advance(ch == 1 ? 1 : 3);             // to the other half, or past the other stream's two
                    }
                }
                if (!ok) break;
                const float tmax = fmax_nan(fmax3_nan(tmx[0], tmx[1], tmx[2]), tmx[3]);
                // the exact online softmax: the largest P of a row is exp2(0) = 1, which bf16 represents
                // exactly.  When the maximum rises, accumulator and row sum are rescaled.
                const float m_new = fmax_nan(m, tmax);
                const bool need = (j > 0) && (m_new > m);
                const float m_old = m;
                m = m_new;
                const float ms = (m == -INFINITY) ? 0.f : m;
                // Exponentials are 2^(x le - m le), one multiply-add each.  le is log2e, or 1 where |m| is so large that the
                // logits lie 32 and more apart (FWD_FAR).
                const float le = fabsf(m) < FWD_FAR ? LOG2E : 1.f;
                const float nm = -ms * le;
                if (__any_sync(0xffffffffu, need)) {
                    // (the accumulator is at rest: S' of this tile followed PV of the one before)
                    const float alpha = need ? ex2(fmaf(m_old, le, nm)) : 1.0f;
                    const float2 a2 = make_float2(alpha, alpha);
#pragma unroll
                    for (int c = 0; c < DH / 32; ++c) {
                        uint32_t r[32];
                        tmem_ld32(tPV + c * 32, r);
                        tmem_wait_ld();
#pragma unroll
                        for (int i = 0; i < 32; i += 2) {
                            const float2 v2 = fmul2(u2f2(r[i], r[i + 1]), a2);
                            r[i] = __float_as_uint(v2.x);
                            r[i + 1] = __float_as_uint(v2.y);
                        }
                        tmem_st32(tPV + c * 32, r);
                    }
                    l *= alpha;
                }
                // The streams take turns on the exp2 pass, scheduler by scheduler, so that one is in it while the
                // other is in its products and sums: stream 1 after stream 0's pass of this tile, stream 0 after
                // stream 1's of the one before.
                const int t = s ? n : n - 1;
                if (t >= 0) ok = warp_all(mbar_wait(&turn[8 * (s ^ 1) + 4 * (t & 1) + (warp & 3)], (t >> 1) & 1, wc, 0x38));
                if (!ok) break;
                // pass 2: P = exp2(x log2e - m log2e), row sum, bf16 pairs over the S columns
                const float2 nm2 = make_float2(nm, nm), le2 = make_float2(le, le);
                float2 rs[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
                for (int ch = 0; ch < 4; ++ch) {
                    uint32_t pk[16];
#pragma unroll
                    for (int k = 0; k < 16; ++k) {
                        const float2 d2 = ffma2(xh[ch * 16 + k], le2, nm2);
                        const float2 p2 = make_float2(ex2(d2.x), ex2(d2.y));
                        rs[k & 1] = fadd2(rs[k & 1], p2);
                        pk[k] = pack_bf16(p2.x, p2.y);
                    }
                    tmem_st16(tS + 16 * ch, pk);
                    if (ch == 3) {
                        // the turn goes on; the store orders the arrive behind the last exp2
                        __syncwarp();
                        if (lane == 0) {
                            asm volatile("st.shared.u32 [%0], %1;" ::"r"(scratch_w), "r"(pk[15]) : "memory");
                            mbar_arrive(&turn[8 * s + 4 * (n & 1) + (warp & 3)]);
                        }
                    }
                }
                l += (rs[0].x + rs[0].y) + (rs[1].x + rs[1].y);
                tmem_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&p_ready[s]);
            }
            if (!ok) break;
            // epilogue of the item; what does not need the last PV comes before the wait for it
            const FwdItem x = tile_of(cur, s);
            const int bs = x.bs(p), h = x.h, qrow = x.qt * TILE + row;
            if (qrow < p.N) p.lse[(static_cast<size_t>(bs) * p.H + h) * p.N + qrow] = (m == -INFINITY) ? m : m + __logf(l);
            const float inv = (m == -INFINITY) ? __int_as_float(0x7fffffff) : __frcp_rn(l);     // no logit above -inf: NaN
            advance(cur);
            // lane t of a quad of rows stores chunk t of each of the four: 64 contiguous bytes per row
            const int qrow0 = x.qt * TILE + (row & ~3);
            const size_t off0 = bs * p.lay.row + qrow0 * p.lay.n + h * p.lay.h + (lane & 3) * 8;
            ok = warp_all(mbar_wait(&pv_done[s], (n - 1) & 1, wc, 0x34));
            if (!ok) break;
            tc_fence_after();
            if (x.qt * TILE >= p.N) continue;          // a stream without an item
#pragma unroll
            for (int c = 0; c < DH / 32; ++c) {
                float o[32];
                __syncwarp();
                tmem_ld_f32<32>(tPV + c * 32, o);
                const int col = c * 32 + (lane & 3) * 8;
                if (c * 32 >= p.Dt) continue;          // warp-uniform
                uint4 vo[4], vr[4];
#pragma unroll
                for (int c8 = 0; c8 < 4; ++c8) {
                    uint32_t vw[4], rw[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float o0 = o[c8 * 8 + 2 * e] *= inv, o1 = o[c8 * 8 + 2 * e + 1] *= inv;
                        vw[e] = pack_bf16(o0, o1);
                        rw[e] = pack_bf16(o0 - bf16_lo(vw[e]), o1 - bf16_hi(vw[e]));
                    }
                    vo[c8] = make_uint4(vw[0], vw[1], vw[2], vw[3]);
                    vr[c8] = make_uint4(rw[0], rw[1], rw[2], rw[3]);
                }
                quad_transpose(vo);
                if (p.o_resid != nullptr) quad_transpose(vr);
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (qrow0 + e < p.N && col < p.Dt) {
                        *reinterpret_cast<uint4*>(p.o + off0 + e * p.lay.n + c * 32) = vo[e];
                        // rounding residual of O
                        if (p.o_resid != nullptr) *reinterpret_cast<uint4*>(p.o_resid + off0 + e * p.lay.n + c * 32) = vr[e];
                    }
                if constexpr (GATED) {
                    // O * sigmoid(gate), from the unrounded O: the gate's chunks come in transposed
                    uint4 vg[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        vg[e] = make_uint4(0u, 0u, 0u, 0u);
                        if (qrow0 + e < p.N && col < p.Dt) vg[e] = __ldg(reinterpret_cast<const uint4*>(p.gate + off0 + e * p.lay.n + c * 32));
                    }
                    __syncwarp();
                    quad_transpose(vg);
#pragma unroll
                    for (int c8 = 0; c8 < 4; ++c8) {
                        const uint32_t gw[4] = {vg[c8].x, vg[c8].y, vg[c8].z, vg[c8].w};
                        uint32_t ow[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const float s0 = 1.0f / (1.0f + ex2(-bf16_lo(gw[e]) * LOG2E));
                            const float s1 = 1.0f / (1.0f + ex2(-bf16_hi(gw[e]) * LOG2E));
                            ow[e] = pack_bf16(o[c8 * 8 + 2 * e] * s0, o[c8 * 8 + 2 * e + 1] * s1);
                        }
                        vg[c8] = make_uint4(ow[0], ow[1], ow[2], ow[3]);
                    }
                    quad_transpose(vg);
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (qrow0 + e < p.N && col < p.Dt)
                            *reinterpret_cast<uint4*>(p.o_gated + off0 + e * p.lay.n + c * 32) = vg[e];
                }
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (tid == 0) { report_abort(wc); report_abort(WaitCtx{tmem_slot + 3, p.status}); }
    if (warp == C::W_PROD) tmem_dealloc(tmem, C::TMEM_COLS);
}

}  // namespace evo
