// EvoAttention forward for sm_100a.
//
//   O = softmax(q k^T * scale + pair_bias + res_mask) v      per (b, s, h)
//
// replaces evo_fwd_ker (evo_h100/tk_evoattention.cu:102-345) and its host
// launcher (tk_evoattention.cu:911-1043).  Reads q/k/v and writes O directly in
// the caller layout [B][S][N][H][D] through strided TMA tensor maps: no
// transposes, no head-dim padding.
//
// One persistent CTA per SM walks work items (b*s, q-tile of 128 rows, h), h fastest.  D <= 64: two or
// three items at a time, as independent streams (below).  D = 96 and 128: evo_fwd_wide.cuh.
//
// LSE is stored in natural log (tk_evoattention.cu:330-334).
#include "evo_host.cuh"
#include "evo_tiles.cuh"

namespace evo {

// A number of items in mixed radix: heads, q tiles, rows (or groups of rows) of a batch, batches.
struct FwdStep {
    int h, qt, g, b;
    __host__ __device__ static FwdStep of(int w, int H, int QT, int NG) {
        return FwdStep{w % H, w / H % QT, w / H / QT % NG, w / H / QT / NG};
    }
};

struct FwdParams {
    int B, S, N, H;
    int Dt;            // true head dim (16 runs on the D = 32 kernel: loads zero-filled, stores clipped)
    int KB;            // contraction blocks of 16 head-dim columns that hold data: ceil(Dt / 16)
    int QT;            // q tiles (= kv tiles) per row: ceil(N / 128) (D > 64: pairs of them)
    int shared_bias;   // D <= 64: the streams of a CTA work on rows of the same q tile and share its bias tiles
    int NG;            // D <= 64: rows per batch, or groups of G rows if the bias tiles are shared
    int total_items;   // B*S*QT*H, or B*SG*QT*H
    FwdStep step;      // from an item of a stream to its next
    float scale, inv_scale;
    const __nv_bfloat16* mask;   // [B*S][N]
    float* lse;                  // [B*S][H][N]
    __nv_bfloat16* o;            // activation layout `lay`
    __nv_bfloat16* o_resid;      // activation layout `lay`, or nullptr
    const __nv_bfloat16* gate;   // activation layout `lay`, or nullptr: pre-activation gate logits
    __nv_bfloat16* o_gated;      // activation layout `lay` (with gate): O * sigmoid(gate)
    ActLayout lay;               // element strides of the activation tensors
    unsigned int* status;
};

// ---------------------------------------------------------------------------
// D <= 64: independent item streams.
//
// What bounds the kernel at D = 32 is not one unit but the hand-offs: every arrive/wait pair costs
// about 130 clocks, an MMA about 130 more until its commit is seen, and a softmax warp that crosses
// four of them per [128 x 64] tile spends as long waiting as computing.  So a CTA runs G streams that
// share nothing but the bias tiles, the tensor core and the issue slots.  Stream s has four softmax
// warps (thread = one q row, all 128 columns of a tile), its own Q, K, V buffers and tensor-memory
// columns, and one MMA warp; it is a serial chain
//
//   S' = Q K^T + mask block  ->  softmax of the tile  ->  PV (+)= P V  ->  next tile
//
// with two waits per softmax warp and tile; while one stream waits, the others compute.
//
//   D = 32 (G = 3): three warps per scheduler.  x = S' * scale + bias goes back into the S columns
//     and is read again for the exp2 pass (tensor memory moves two columns per clock), so a thread
//     needs no 128 registers for it; P (bf16) overwrites the columns already read, and S' of the
//     next tile follows PV of this one.
//   D = 64 (G = 2; three accumulators of 64 columns do not fit beside three S tiles): x stays in
//     registers, P has columns of its own, so S' of the next tile runs during the exp2 pass.
//
// Bias tiles travel through a ring.  SHARED: the streams of a CTA work on G rows of S at the same
// (b, h, q tile), so one tile serves G streams; otherwise (few rows per batch, or too few items to
// fill the SMs G at a time) every stream has its own items and its own ring slot.
//
// Measured against one item at a time on two groups of 64 columns (what is below included; kernel alone, in one run):
// B=1, S=512, N=384, H=8, D=32 0.358 -> 0.278 ms; S=256, N=768 0.638 -> 0.522; S=256, N=1024, H=4, D=64 0.677 -> 0.585.
// A step takes about 2200 clocks of a CTA: 1024 for its exponentials, 1000 issue slots.  Also tried: the
// epilogue on a warpgroup of its own (its registers cost the softmax warps more than it saves, 0.42 ms),
// two streams in the exp2 pass at a time (0.365), none taking turns (0.39), two streams at D = 32 (0.375).
//
// Between two items a stream's warps wait for the last PV and hand the results over: 3300 clocks, of a
// three-tile item's 18500, when every warp stored its rows itself (32 shuffles to make 64-byte segments).
// Staged in buffers that the item no longer needs, sent by the MMA warp's TMA stores, and with what does
// not depend on the last PV ahead of the wait for it: 2200 (the two shapes at D = 32 0.319 -> 0.295 and
// 0.585 -> 0.540 ms).
//
// The streams are at different places of their code at any time, and what they fetch competes for the instruction cache
// (1.1 warps a scheduler wait for instructions per issue; 0.7 with short waits).  Short waits, 105 -> 83 KB of code: B=1, S=512, N=384,
// H=8, D=32 0.302 -> 0.277 ms; S=200, N=200, H=4 44 -> 40 us; S=256, N=1024, H=4, D=64 640 -> 575.  The producer's loop is
// unrolled over three streams, its masks requested ahead: one copy of it was 0.298 ms at the first shape (one warp is then too slow for
// three streams).  Over two streams, D = 64, one copy is the quicker: S=256, N=1024, H=4 597 -> 582 us, S=300, N=128 34.2 -> 32.7,
// B=4, S=1, N=1024, H=16 54.7 -> 53.6.  Rolling the loops over a tile's chunks: no gain.
//
// One maximum per 128 columns instead of one per 64 leaves one exact P a row and tile instead of two: O is 2 to 3 %
// further from 64 bits (relative error 2.11e-3 -> 2.16e-3 at N = 264, D = 64, of which 1.66e-3 is its own bf16).  Two
// maxima would take a second accumulator per stream, for which there is no tensor memory.
//
// The mask rides in an extra contraction block (evo_tiles.cuh, "EXTRA TILE"): the producer turns 128
// mask values into a [128][8] tile (m/scale in three bf16 parts, exact to fp32), columns past N get
// -inf.  The base of the exponentials: x in natural units, P = exp2(x log2e - m log2e).
// ---------------------------------------------------------------------------
template <int DH>
struct FwdCfg {
    static constexpr int G = (DH == 32) ? 3 : 2;               // item streams
    static constexpr bool HOLD = (G == 2);                     // x in registers, P in its own columns
    // every fourth column pair of the exp2 pass on the fused-multiply-add pipe: D = 32 (B=1, S=512, N=384,
    // H=8) 0.334 -> 0.323 ms; D = 64, whose warps have no issue slots to spare, 0.58 -> 0.63 ms
    static constexpr int POLY_EVERY = (DH == 32) ? 4 : 0;
    static constexpr int NSW = 4 * G;                          // softmax warps
    static constexpr int W_PROD = NSW;                         // producer, then G MMA warps (one warpgroup)
    static constexpr int THREADS = (NSW + 4) * 32;
    // setmaxnreg budgets: the CTA's register pool is the launch count (the cap ptxas derives from the
    // launch bound) times the threads; an increase that the pool cannot satisfy blocks for ever
    static constexpr int REGS_LAUNCH = (65536 / THREADS) & ~7;
    static constexpr int REGS_SOFTMAX = (G == 3) ? 152 : 216;
    static constexpr int REGS_OTHER = (G == 3) ? 56 : 72;
    static_assert((REGS_SOFTMAX * NSW + REGS_OTHER * 4) * 32 <= REGS_LAUNCH * THREADS, "register pool");
    static constexpr uint32_t ROWT = RowTile<DH>::BYTES;       // one [128][DH] bf16 tile
    static constexpr int NQ = (DH == 32) ? 2 : 1;              // Q buffers per stream
    static constexpr int NK = HOLD ? 2 : 1;                    // K (and mask tile) buffers per stream
    static constexpr int NR = G;                               // bias tiles in the ring
    static constexpr uint32_t ST_Q = 0, ST_K = NQ * ROWT, ST_V = ST_K + NK * ROWT, ST_XK = ST_V + ROWT;
    static constexpr uint32_t STREAM_BYTES = ST_XK + NK * XT_BYTES;
    static constexpr uint32_t OFF_BIAS = 0;                    // ring of bias tiles: two [128][64] halves each
    static constexpr uint32_t OFF_STREAM = NR * SQ_BYTES;
    // constant extra tiles, above every tile that refers to the zero tile
    static constexpr uint32_t OFF_XQ = OFF_STREAM + G * STREAM_BYTES;       // rows (1, 1, 1, 0, ...)
    static constexpr uint32_t OFF_ZERO = OFF_XQ + XT_BYTES;
    static constexpr uint32_t OFF_BARS = OFF_ZERO + XT_BYTES;
    static constexpr int BARS = 22;                            // barriers of a stream (FwdBars)
    static constexpr uint32_t OFF_MISC = OFF_BARS + (G * BARS + 2 * NR) * 8;
    static constexpr uint32_t SMEM_BYTES = OFF_MISC + 16 + 1024;   // + alignment slack
    static constexpr uint32_t TMEM_S = 0;                      // + 128 s
    static constexpr uint32_t TMEM_PV = 128 * G;               // + DH s
    static constexpr uint32_t TMEM_P = HOLD ? TMEM_PV + DH * G : TMEM_S;   // + 64 s, or the S columns of stream s
    static constexpr uint32_t TMEM_COLS = 512;
    static_assert((HOLD ? TMEM_P + 64 * G : TMEM_PV + DH * G) <= TMEM_COLS, "tensor memory budget");
    __device__ static __forceinline__ uint32_t p_col(int s) { return TMEM_P + s * (HOLD ? 64 : 128); }
    static_assert(SMEM_BYTES <= 232448, "shared memory budget");
    static_assert(STREAM_BYTES % 1024 == 0, "tile alignment");
};

// The barriers of one stream.
struct FwdBars {
    uint64_t *q_full, *q_empty;      // [NQ]
    uint64_t *k_full, *k_empty;      // [NK]: K and mask tile
    uint64_t *v_full;
    uint64_t *s_full, *s_free;       // S' complete / read (HOLD)
    uint64_t *p_ready, *pv_done;     // P written / PV complete
    uint64_t *o_staged;              // an item's results are in shared memory
    uint64_t *turn;                 // [2][4] by tile parity: warp w of the stream has left its exp2 pass
    __device__ __forceinline__ FwdBars(uint64_t* b)
        : q_full(b), q_empty(b + 2), k_full(b + 4), k_empty(b + 6), v_full(b + 8), s_full(b + 9), s_free(b + 10),
          p_ready(b + 11), pv_done(b + 12), o_staged(b + 13), turn(b + 14) {}
};

// A stream's walk over its items: coordinates in mixed radix (head, q tile, row or group of rows, batch),
// advanced by p.step without a division (a division costs a warp about a hundred clocks, on the stream's chain).
struct FwdItem {
    int h, qt, row, b;       // row of S: with groups, G apart
    __device__ __forceinline__ void next(int rows, int rstep, const FwdParams& p) {
        h += p.step.h;
        int c = h >= p.H;
        h -= c ? p.H : 0;
        qt += p.step.qt + c;
        c = qt >= p.QT;
        qt -= c ? p.QT : 0;
        row += (p.step.g + c) * rstep;
        c = row >= rows;
        row -= c ? rows : 0;
        b += p.step.b + c;
    }
    __device__ __forceinline__ bool valid(const FwdParams& p) const { return b < p.B && row < p.S; }
    __device__ __forceinline__ int bs(const FwdParams& p) const { return b * p.S + row; }
};

// Mask value m, divided by the scale, as three bf16 parts (24 significant bits), in the layout of words 0 and 1 of an
// extra-tile row.  A finite one stays finite, so that every mask that a type can hold ranks above the -inf of the columns
// past N (a row of which nothing else is left is then the mean of its N values); infinities and NaN go through.
__device__ __forceinline__ uint2 mask_term(float m, float inv_scale) {
    const float v = fmaxf(m * inv_scale, -3e38f);
    const float a = __bfloat162float(__float2bfloat16_rn(v));
    const float b = __bfloat162float(__float2bfloat16_rn(v - a));
    // (2^-60 m is nothing beside the third part of a finite m, and all of an infinite one)
    const uint32_t c = __bfloat16_as_ushort(__float2bfloat16_rn(fmaf(m, 8.67361738e-19f, (v - a) - b)));
    return make_uint2(pack_bf16(a, b), c);
}

// From this |m| of a row on (one, or the tiles of it so far, all masked by terms like -1e9 or -1e30) m log2e, rounded, is
// off by 32 and more, and 2^(x log2e - m log2e) no exponential of x - m any longer.  But there the logits are multiples
// of 32, so that all below m get nothing, whatever the base: with 2 instead of e, x - m is exact.
// (Kernel alone, without any of it / this: B=1, S=256, N=1024, H=4, D=64 0.600 / 0.602 ms; S=512, N=384, H=8, D=32
// 0.293 / 0.299; x - m formed first, in a branch for such rows, cost the first 17 %.)
constexpr float FWD_FAR = 536870912.f;         // 2^29

// GATED: the epilogue also writes sigmoid(gate) * O.  tm_2: the rounding residual (GATED: the gated output).
template <int DH, bool GATED>
__global__ void __launch_bounds__(FwdCfg<DH>::THREADS, 1)
evo_fwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
               const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_bias,
               const __grid_constant__ CUtensorMap tm_o, const __grid_constant__ CUtensorMap tm_2, const FwdParams p) {
    using C = FwdCfg<DH>;
    using RT = RowTile<DH>;
    using RD = RowDesc<DH>;
    constexpr int G = C::G, NSW = C::NSW, NQ = C::NQ, NK = C::NK, NR = C::NR;

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::OFF_BARS);
    uint64_t* bias_full = bars + G * C::BARS;            // [NR]
    uint64_t* bias_empty = bias_full + NR;               // [NR]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + C::OFF_MISC);
    volatile uint32_t* abort_flag = tmem_slot + 1;

    const int tid = threadIdx.x;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);      // uniform: what derives from it stays in uniform registers
    const int lane = tid & 31;
    const int NT = p.QT;
    const bool shared_bias = p.shared_bias != 0;
    WaitCtx wc{abort_flag, p.status};

    if (tid == 0) {
        *abort_flag = 0;
        tmem_slot[3] = 0;                   // the abort word of the waits before exit
        for (int s = 0; s < G; ++s) {
            const FwdBars b(bars + s * C::BARS);
            for (int i = 0; i < NQ; ++i) { mbar_init(&b.q_full[i], 1); mbar_init(&b.q_empty[i], 1); }
            for (int i = 0; i < NK; ++i) { mbar_init(&b.k_full[i], 1); mbar_init(&b.k_empty[i], 1); }
            mbar_init(b.v_full, 1);
            mbar_init(b.s_full, 1); mbar_init(b.s_free, 4);
            mbar_init(b.p_ready, 4); mbar_init(b.pv_done, 1);
            mbar_init(b.o_staged, 4);
            for (int i = 0; i < 8; ++i) mbar_init(&b.turn[i], 1);
        }
        for (int i = 0; i < NR; ++i) { mbar_init(&bias_full[i], 1); mbar_init(&bias_empty[i], shared_bias ? NSW : 4); }
        fence_mbar_init();
    }
    if (warp == C::W_PROD) {
        tmem_alloc(tmem_slot, C::TMEM_COLS);
        tmem_relinquish();
        if (lane == 0) { prefetch_tmap(&tm_q); prefetch_tmap(&tm_k); prefetch_tmap(&tm_v); prefetch_tmap(&tm_bias); prefetch_tmap(&tm_o); prefetch_tmap(&tm_2); }
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

    // Items.  h fastest, then q tile, then row (or group of G rows), so that CTAs side by side touch the
    // same 128-byte lines of q/k/v.  Every stream counts the same number of items; the last ones of a
    // stream, or rows of a group past S, may be missing.
    const int first = blockIdx.x, stride = gridDim.x;
    const int per_cta = stride * (shared_bias ? 1 : G);
    const int n_items = (p.total_items > first) ? (p.total_items - first + per_cta - 1) / per_cta : 0;
    // rows count in steps of G within a batch if they are taken in groups: row r of the group sits at g * G + r
    const int rstep = shared_bias ? G : 1;
    auto items_of = [&](int s) -> FwdItem {
        const FwdStep w = FwdStep::of(first + (shared_bias ? 0 : s * stride), p.H, p.QT, p.NG);
        return FwdItem{w.h, w.qt, w.g * rstep + (shared_bias ? s : 0), w.b};
    };
    auto advance = [&](FwdItem& x, int s) {
        const int shift = shared_bias ? s : 0;
        x.row -= shift;
        x.next(p.NG * rstep, rstep, p);
        x.row += shift;
    };
    // ring slot and phase parity of the bias tile of tile r of stream s
    auto bias_slot = [&](int s, int r, int& slot, uint32_t& ph) {
        slot = shared_bias ? r % NR : s;
        ph = static_cast<uint32_t>(shared_bias ? r / NR : r) & 1u;
    };

    if (warp >= C::W_PROD) {
        reg_dec<C::REGS_OTHER>();
        if (warp == C::W_PROD) {
            // ------------------------------ producer ------------------------------
            // Round r holds tile r of every stream (item r / NT, kv tile r % NT): the bias tile, then Q per
            // item, K and the mask tile.  (V is fetched by the stream's MMA warp, the first to know that its
            // buffer is free.)  The warp runs with all lanes and elects one to issue.
            int used[G], qn[G];      // tiles and items of the stream so far
            FwdItem item[3] = {items_of(0), items_of(1), items_of(2)};      // the first G of them are walked
#pragma unroll
            for (int s = 0; s < G; ++s) used[s] = qn[s] = 0;
            bool ok = true;
            int r = 0;
            // one copy of the code per stream, or (D = 64) for both (see above)
            auto each_stream = [&](auto&& f) {
                if constexpr (G == 3) {
#pragma unroll
                    for (int s = 0; s < G; ++s) f(s);
                } else {
#pragma unroll 1
                    for (int s = 0; s < G; ++s) f(s);
                }
            };
            auto load_tile = [&](int s, int j, int r) {
                if (!ok || !item[s].valid(p)) return;
                const int bs = item[s].bs(p), qt = item[s].qt, h = item[s].h;
                const FwdBars b(bars + s * C::BARS);
                uint8_t* sb = smem + C::OFF_STREAM + s * C::STREAM_BYTES;
                // four mask values per lane, requested before the waits
                const int c = j * TILE + 4 * lane;
                uint2 mw = make_uint2(0u, 0u);
                if (c < p.N) mw = __ldg(reinterpret_cast<const uint2*>(p.mask + static_cast<size_t>(bs) * p.N + c));
                if (j == 0) {
                    const int qb = qn[s] % NQ, use = qn[s] / NQ;
                    if (qn[s]++ >= NQ) ok = warp_all(mbar_wait(&b.q_empty[qb], (use - 1) & 1, wc, 0x10));
                    if (ok && elect_one()) {
                        mbar_arrive_expect_tx(&b.q_full[qb], C::ROWT);
                        tma_load_row_tile<DH>(sb + C::ST_Q + qb * C::ROWT, &tm_q, &b.q_full[qb], h, qt * TILE, bs);
                    }
                    __syncwarp();
                }
                if (!ok) return;
                const int n = used[s]++, kb = n % NK;
                if (n >= NK) ok = warp_all(mbar_wait(&b.k_empty[kb], ((n / NK) - 1) & 1, wc, 0x11));
                if (!ok) return;
                if (elect_one()) {
                    mbar_expect_tx(&b.k_full[kb], C::ROWT);
                    tma_load_row_tile<DH>(sb + C::ST_K + kb * C::ROWT, &tm_k, &b.k_full[kb], h, j * TILE, bs);
                }
                __syncwarp();
                const float mv[4] = {bf16_lo(mw.x), bf16_hi(mw.x), bf16_lo(mw.y), bf16_hi(mw.y)};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const uint2 w = mask_term(c < p.N ? mv[e] : -INFINITY, p.inv_scale);
                    *reinterpret_cast<uint4*>(sb + C::ST_XK + kb * XT_BYTES + (4 * lane + e) * 16) = make_uint4(w.x, w.y, 0u, 0u);
                }
                fence_async_smem();
                __syncwarp();
                if (elect_one()) mbar_arrive(&b.k_full[kb]);
                __syncwarp();
                // the bias tile: once per round if the streams share it (stream 0 always has the item)
                if (!shared_bias || s == 0) {
                    int slot; uint32_t ph;
                    bias_slot(s, r, slot, ph);
                    if (r >= (shared_bias ? NR : 1)) ok = warp_all(mbar_wait(&bias_empty[slot], ph ^ 1u, wc, 0x14));
                    if (ok && elect_one()) {
                        uint8_t* bt = smem + C::OFF_BIAS + slot * SQ_BYTES;
                        mbar_arrive_expect_tx(&bias_full[slot], SQ_BYTES);
                        tma_load_4d(bt, &tm_bias, &bias_full[slot], j * TILE, qt * TILE, h, item[s].b);
                        tma_load_4d(bt + SQ_SUB_BYTES, &tm_bias, &bias_full[slot], j * TILE + 64, qt * TILE, h, item[s].b);
                    }
                    __syncwarp();
                }
            };
            for (int it = 0; it < n_items && ok; ++it) {
                for (int j = 0; j < NT && ok; ++j, ++r) {
                    each_stream([&](int s) { load_tile(s, j, r); });
                }
                each_stream([&](int s) { advance(item[s], s); });
            }
            // the last loads have landed before the CTA exits (also if a wait gave up)
            const WaitCtx dc{tmem_slot + 3, p.status};
#pragma unroll
            for (int s = 0; s < G; ++s) {
                const FwdBars b(bars + s * C::BARS);
                for (int k = (used[s] > NK ? used[s] - NK : 0); k < used[s]; ++k) mbar_wait_landed(&b.k_full[k % NK], (k / NK) & 1, dc, 0x12);
                for (int k = (qn[s] > NQ ? qn[s] - NQ : 0); k < qn[s]; ++k) mbar_wait_landed(&b.q_full[k % NQ], (k / NQ) & 1, dc, 0x13);
            }
        } else if (warp - C::W_PROD - 1 < G) {
            // ------------------------------ MMA warp of one stream ------------------------------
            const int s = warp - C::W_PROD - 1;
            const FwdBars b(bars + s * C::BARS);
            constexpr uint32_t IDESC_S = make_idesc_bf16(128, 128, 0, 0);
            const uint32_t IDESC_PV = make_idesc_bf16(128, 16 * p.KB, 0, 1);   // N = the head-dim columns that hold data
            uint8_t* sb = smem + C::OFF_STREAM + s * C::STREAM_BYTES;
            const uint32_t aS = smem_u32(sb), aZero = smem_u32(smem + C::OFF_ZERO);
            const uint64_t d_xq = xt_desc(smem_u32(smem + C::OFF_XQ), aZero);
            const uint32_t v_lo = RD::mnmajor_lo(aS + C::ST_V);
            const uint32_t t_s = tmem + C::TMEM_S + 128 * s, t_pv = tmem + C::TMEM_PV + DH * s, t_p = tmem + C::p_col(s);
            bool ok = true;
            FwdItem cur = items_of(s);         // the item whose V tiles are being loaded
            int qn = 0;                        // items whose S' tiles have all been issued
            // S' of tile n (kv tile j of item qn): what it waits for, and the issue
            auto wait_s = [&](int n, int j) {
                if (j == 0) ok = warp_all(mbar_wait(&b.q_full[qn % NQ], (qn / NQ) & 1, wc, 0x20));
                if (ok) ok = warp_all(mbar_wait(&b.k_full[n % NK], (n / NK) & 1, wc, 0x21));
            };
            auto issue_s = [&](int n, int j) {
                const int kb = n % NK;
                tc_fence_after();
                if (elect_one()) {
                    const uint32_t q_lo = RD::kmajor_lo(aS + C::ST_Q + (qn % NQ) * C::ROWT), k_lo = RD::kmajor_lo(aS + C::ST_K + kb * C::ROWT);
#pragma unroll
                    for (int kk = 0; kk < RT::KBLOCKS; ++kk)
                        if (kk < p.KB)          // blocks past the true head dim are zero-filled: skipped
                            umma_ss(t_s, RD::kmajor(q_lo, kk), RD::kmajor(k_lo, kk), IDESC_S, kk > 0);
                    umma_ss(t_s, d_xq, xt_desc(aS + C::ST_XK + kb * XT_BYTES, aZero), IDESC_S, 1u);
                    umma_commit(b.s_full);
                    // (of an item's last tile, one of the two is held back: see store_item)
                    if (!C::HOLD || j < NT - 1) umma_commit(&b.k_empty[kb]);
                    if (C::HOLD && j == NT - 1) umma_commit(&b.q_empty[qn % NQ]);
                }
                __syncwarp();
                if (j == NT - 1) ++qn;
            };
            auto load_v = [&](int j) {         // of the item `cur`
                if (elect_one()) {
                    mbar_arrive_expect_tx(b.v_full, C::ROWT);
                    tma_load_row_tile<DH>(sb + C::ST_V, &tm_v, b.v_full, cur.h, j * TILE, cur.bs(p));
                }
                __syncwarp();
            };
            auto issue_pv = [&](int n, int j) {
                ok = warp_all(mbar_wait(b.v_full, n & 1, wc, 0x24));
                if (ok) ok = warp_all(mbar_wait(b.p_ready, n & 1, wc, 0x23));
                if (!ok) return;
                tc_fence_after();
                if (elect_one()) {
#pragma unroll
                    for (int kk = 0; kk < 8; ++kk)
                        umma_ts(t_pv, t_p + kk * 8, RD::mnmajor(v_lo, kk), IDESC_PV, (kk > 0 || j > 0) ? 1u : 0u);
                    umma_commit(b.pv_done);
                }
                __syncwarp();
            };
            // The results of item x (the stream's e-th, its last tile n) go out from V's buffer and from one that
            // the item's last S' has left: Q's, of two (D = 32), or K's, of two.
            const bool two = GATED || p.o_resid != nullptr;
            auto store_item = [&](const FwdItem& x, int e, int n) {
                ok = warp_all(mbar_wait(b.o_staged, e & 1, wc, 0x27));
                if (!ok) return;
                if (elect_one()) {
                    uint8_t* second = sb + (C::HOLD ? C::ST_K + (n % NK) * C::ROWT : C::ST_Q + (e % NQ) * C::ROWT);
                    tma_store_4d(&tm_o, sb + C::ST_V, 0, x.h, x.qt * TILE, x.bs(p));
                    if (two) tma_store_4d(&tm_2, second, 0, x.h, x.qt * TILE, x.bs(p));
                    tma_commit_group();
                    tma_wait_group_read<0>();
                    mbar_arrive(C::HOLD ? &b.k_empty[n % NK] : &b.q_empty[e % NQ]);
                }
                __syncwarp();
            };
            // with rows in groups, the last group of a batch may lack this stream's row: skipped
            int it = 0;
            auto skip_missing = [&]() -> bool {
                bool any = false;
                for (; it < n_items && !cur.valid(p); ++it, any = true) advance(cur, s);
                return any;
            };
            (void)skip_missing();
            int j = 0, loaded = 0, e = 0;
            if (it < n_items) { load_v(0); loaded = 1; wait_s(0, 0); if (ok) issue_s(0, 0); }
            bool more = it < n_items;
            for (int n = 0; more && ok; ++n) {
                const bool last = j == NT - 1;
                const FwdItem mine = cur;
                int j1 = j + 1;                // the tile after this one
                bool gap = false;              // items are missing before it
                if (last) { j1 = 0; ++it; advance(cur, s); gap = skip_missing(); }
                more = it < n_items;
                // S' of the next tile: its columns are free once the softmax has read them (HOLD), or once
                // PV of this tile, which reads P from them, is complete.  Behind a gap Q and K do not come
                // before the softmax has finished this item and passed the missing one's bias tiles on.
                const bool early = C::HOLD && more && !gap;
                auto s_free = [&]() { if (C::HOLD && ok) ok = warp_all(mbar_wait(b.s_free, n & 1, wc, 0x22)); };
                if (early) {
                    wait_s(n + 1, j1);
                    s_free();
                    if (!ok) break;
                    issue_s(n + 1, j1);
                }
                issue_pv(n, j);
                if (!ok) break;
                if (more) {
                    if (!early) wait_s(n + 1, j1);            // while PV runs
                    if (ok) ok = warp_all(mbar_wait(b.pv_done, n & 1, wc, 0x25));
                    if (!early) s_free();
                    if (!ok) break;
                    if (!early) issue_s(n + 1, j1);
                }
                if (last) store_item(mine, e++, n);
                if (!ok) break;
                if (more) {
                    load_v(j1);
                    ++loaded;
                }
                j = j1;
            }
            if (elect_one()) tma_wait_group<0>();
            __syncwarp();
            if (loaded > 0) mbar_wait_landed(b.v_full, (loaded - 1) & 1, WaitCtx{tmem_slot + 3, p.status}, 0x26);
        }
    } else {
        reg_inc<C::REGS_SOFTMAX>();
        // ------------------------------ softmax warps of one stream ------------------------------
        const int s = warp >> 2;
        const FwdBars b(bars + s * C::BARS);
        const int row = tid & 127;           // q row within the tile == TMEM lane
        const uint32_t lane_base = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16);
        const uint32_t tS = lane_base + C::TMEM_S + 128 * s, tPV = lane_base + C::TMEM_PV + DH * s, tP = lane_base + C::p_col(s);
        const uint32_t scratch_w = smem_u32(tmem_slot + 2);           // a word nobody reads
        const float2 sc2 = make_float2(p.scale, p.scale);
        // The exp2 pass loads the special-function unit, the passes around it the other pipes.  Left alone
        // the warps of a scheduler fall into step, all in the same pass at the same time; so the streams
        // take turns on it, scheduler by scheduler, and a warp hands its turn on halfway through the pass (a
        // single warp leaves the unit idle while its own multiplies and loads are in the way).
        uint64_t* turn_mine = &b.turn[warp & 3];
        uint64_t* turn_prev = &FwdBars(bars + (s > 0 ? s - 1 : G - 1) * C::BARS).turn[warp & 3];
        bool ok = true;
        int n = 0, r = 0, e = 0;              // tiles of the stream so far, tiles counting missing items, items
        auto take_turn = [&]() {
            // a stream may leave its pass of tile t + 1 before the one that waits for it looks at tile t: two
            // barriers by tile parity keep the waiter within one phase
            const int t = s > 0 ? r : r - 1;
            if (t >= 0) ok = warp_all(mbar_wait(turn_prev + 4 * (t & 1), (t >> 1) & 1, wc, 0x38));
        };

        FwdItem cur = items_of(s);
        for (int it = 0; it < n_items && ok; ++it) {
            if (!cur.valid(p)) {
                // no such item: hand the bias tiles (if shared) and the turns on
                for (int j = 0; j < NT && ok; ++j, ++r) {
                    if (shared_bias) {
                        int slot; uint32_t ph;
                        bias_slot(s, r, slot, ph);
                        ok = warp_all(mbar_wait(&bias_full[slot], ph, wc, 0x36));
                        if (!ok) break;
                        if (lane == 0) mbar_arrive(&bias_empty[slot]);
                    }
                    take_turn();
                    if (!ok) break;
                    __syncwarp();
                    if (lane == 0) mbar_arrive(turn_mine + 4 * (r & 1));
                }
                advance(cur, s);
                continue;
            }
            float m = -INFINITY, l = 0.f;
            for (int j = 0; j < NT; ++j, ++n, ++r) {
                int slot; uint32_t ph;
                bias_slot(s, r, slot, ph);
                const uint32_t aBias = smem_u32(smem + C::OFF_BIAS) + slot * SQ_BYTES;
                ok = warp_all(mbar_wait_both(&bias_full[slot], ph, b.s_full, n & 1, wc, 0x31));
                if (!ok) break;
                tc_fence_after();
                // pass 1: x = S' * scale + bias and the row maximum, 32 columns at a time
                float2 xh[C::HOLD ? 64 : 1];
                float tmx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
                uint32_t sv[2][32];
                tmem_ld32(tS, sv[0]);
#pragma unroll
                for (int ch = 0; ch < 4; ++ch) {
                    uint32_t (&cv)[32] = sv[ch & 1];
                    uint4 bv[4];
#pragma unroll
                    for (int q4 = 0; q4 < 4; ++q4) bv[q4] = lds128(aBias + sq_chunk_off(row, ch * 4 + q4));
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
                            if constexpr (C::HOLD) {
                                xh[ch * 16 + k] = x;
                            } else {
                                cv[2 * k] = __float_as_uint(x.x);
                                cv[2 * k + 1] = __float_as_uint(x.y);
                            }
                        }
                    }
                    if constexpr (!C::HOLD) tmem_st32(tS + 32 * ch, cv);
                }
                const float tmax = fmax_nan(fmax3_nan(tmx[0], tmx[1], tmx[2]), tmx[3]);
                if constexpr (C::HOLD) {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(b.s_free);
                }
                // the maximum depends on every bias value read: the producer may refill the tile
                mbar_release_after_loads(&bias_empty[slot], __float_as_uint(tmax), scratch_w);

                // the exact online softmax: the largest P of a row is exp2(0) = 1, which bf16 represents
                // exactly.  When the maximum rises, accumulator and row sum are rescaled.
                const float m_new = fmax_nan(m, tmax);
                const bool need = (j > 0) && (m_new > m);
                const float m_old = m;
                m = m_new;
                const float ms = (m == -INFINITY) ? 0.f : m;
                // Exponentials are 2^(x le - m le), one multiply-add each.  le is log2e, or 1 where |m| is so large that the
                // logits lie 32 and more apart (FWD_FAR).
                // (NaN or +inf among the logits makes m so, and with le = 0 all exponentials NaN, whichever columns they are in: those
                // that the polynomial takes would drop a NaN of their own)
                const float le = fabsf(m) < FWD_FAR ? LOG2E : (C::POLY_EVERY == 0 || m < INFINITY ? 1.f : 0.f);
                const float nm = -ms * le;
                if constexpr (C::HOLD) {
                    // P's columns are free and the accumulator is at rest once the previous PV is complete
                    if (n > 0) {
                        ok = warp_all(mbar_wait(b.pv_done, (n - 1) & 1, wc, 0x33));
                        if (!ok) break;
                        tc_fence_after();
                    }
                }
                if (__any_sync(0xffffffffu, need)) {
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
                take_turn();
                if (!ok) break;
                // pass 2: P = exp2(x log2e - m log2e), row sum, bf16 pairs into tensor memory
                const float2 nm2 = make_float2(nm, nm), le2 = make_float2(le, le);
                float2 rs[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
                if constexpr (!C::HOLD) {
                    tmem_wait_st();                     // x is written
                    tmem_ld32(tS, sv[0]);
                }
#pragma unroll
                for (int ch = 0; ch < 4; ++ch) {
                    uint32_t pk[16];
                    if constexpr (!C::HOLD) {
                        tmem_wait_ld();
                        if (ch < 3) tmem_ld32(tS + 32 * (ch + 1), sv[(ch + 1) & 1]);
                    }
#pragma unroll
                    for (int k = 0; k < 16; ++k) {
                        const float2 x = C::HOLD ? xh[C::HOLD ? ch * 16 + k : 0]
                                                 : u2f2(sv[ch & 1][2 * k], sv[ch & 1][2 * k + 1]);
                        const float2 d2 = ffma2(x, le2, nm2);
                        const float2 p2 = use_poly<C::POLY_EVERY>(k) ? ex2_poly2<5>(d2) : make_float2(ex2(d2.x), ex2(d2.y));
                        rs[k & 1] = fadd2(rs[k & 1], p2);
                        pk[k] = pack_bf16(p2.x, p2.y);
                    }
                    tmem_st16(tP + 16 * ch, pk);        // behind the columns that pass 2 has read
                    if (ch == 1) {
                        // the turn goes on; the store orders the arrive behind the exp2 of this chunk
                        __syncwarp();
                        if (lane == 0) {
                            asm volatile("st.shared.u32 [%0], %1;" ::"r"(scratch_w), "r"(pk[15]) : "memory");
                            mbar_arrive(turn_mine + 4 * (r & 1));
                        }
                    }
                }
                l += (rs[0].x + rs[0].y) + (rs[1].x + rs[1].y);
                tmem_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(b.p_ready);
            }
            if (!ok) break;
            // epilogue of the item; what does not need the last PV comes before the wait for it
            const int bs = cur.bs(p), qt = cur.qt, h = cur.h;
            const int qrow = qt * TILE + row;
            if (qrow < p.N) p.lse[(static_cast<size_t>(bs) * p.H + h) * p.N + qrow] = (m == -INFINITY) ? m : m + __logf(l);
            // (a row of which every logit is -inf has no softmax: NaN, and a log-sum-exp of -inf)
            const float inv = (m == -INFINITY) ? __int_as_float(0x7fffffff) : __frcp_rn(l);
            advance(cur, s);
            // Results go through shared memory (row r of a tile: 16-byte chunks, swizzled as the tensor map says)
            // and out by TMA, issued by the MMA warp.
            uint8_t* sb = smem + C::OFF_STREAM + s * C::STREAM_BYTES;
            const uint32_t aO = smem_u32(sb + C::ST_V);
            const uint32_t a2 = smem_u32(sb + (C::HOLD ? C::ST_K + ((n - 1) % NK) * C::ROWT : C::ST_Q + (e % NQ) * C::ROWT));
            ++e;
            ok = warp_all(mbar_wait(b.pv_done, (n - 1) & 1, wc, 0x34));
            if (!ok) break;
            tc_fence_after();
#pragma unroll
            for (int c = 0; c < DH / 32; ++c) {
                float o[32];
                __syncwarp();
                tmem_ld_f32<32>(tPV + c * 32, o);
                uint4 vr[4];
#pragma unroll
                for (int c8 = 0; c8 < 4; ++c8) {
                    uint32_t vw[4], rw[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float o0 = o[c8 * 8 + 2 * e] *= inv, o1 = o[c8 * 8 + 2 * e + 1] *= inv;
                        vw[e] = pack_bf16(o0, o1);
                        rw[e] = pack_bf16(o0 - bf16_lo(vw[e]), o1 - bf16_hi(vw[e]));
                    }
                    const uint32_t off = swz_off<RT::ROW_BYTES>(row, c * 4 + c8);
                    sts128(aO + off, make_uint4(vw[0], vw[1], vw[2], vw[3]));
                    vr[c8] = make_uint4(rw[0], rw[1], rw[2], rw[3]);
                    // rounding residual of O
                    if (!GATED && p.o_resid != nullptr) sts128(a2 + off, vr[c8]);
                }
                if constexpr (GATED) {
                    // O * sigmoid(gate), from the unrounded O.  Lane t of a quad of rows loads chunk t of each of
                    // the four (64 contiguous bytes per row), and stores the residual like that.
                    const int col = c * 32 + (lane & 3) * 8, qrow0 = qt * TILE + (row & ~3);
                    const size_t off0 = bs * p.lay.row + qrow0 * p.lay.n + h * p.lay.h + col;
                    uint4 vg[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        vg[e] = make_uint4(0u, 0u, 0u, 0u);
                        if (qrow0 + e < p.N && col < p.Dt) vg[e] = __ldg(reinterpret_cast<const uint4*>(p.gate + off0 + e * p.lay.n));
                    }
                    __syncwarp();
                    if (p.o_resid != nullptr) {
                        quad_transpose(vr);
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            if (qrow0 + e < p.N && col < p.Dt) *reinterpret_cast<uint4*>(p.o_resid + off0 + e * p.lay.n) = vr[e];
                        __syncwarp();
                    }
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
                        sts128(a2 + swz_off<RT::ROW_BYTES>(row, c * 4 + c8), make_uint4(ow[0], ow[1], ow[2], ow[3]));
                    }
                }
            }
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(b.o_staged);
        }
    }

    tc_fence_before();
    __syncthreads();
    if (tid == 0) { report_abort(wc); report_abort(WaitCtx{tmem_slot + 3, p.status}); }
    if (warp == C::W_PROD) tmem_dealloc(tmem, C::TMEM_COLS);
}

}  // namespace evo
#include "evo_fwd_wide.cuh"
namespace evo {

// lay_in: q, k, v; lay: the output side (o, o_resid, gate, o_gated)
template <int DH>
static int launch_fwd(const EvoDims* d, const ActLayout& lay_in, const ActLayout& lay, const void* q, const void* k, const void* v,
                      const void* bias, const void* mask, const void* gate, void* o, void* o_gated, void* o_resid,
                      float* lse, float scale, cudaStream_t st) {
    constexpr bool WIDE = (DH == 128);
    const int BS = d->B * d->S;
    const int QT = (d->N + TILE - 1) / TILE;

    CUtensorMap tq, tk, tv, tb;
    int rc;
    const int Dt = d->D;          // 16 on the D = 32 kernel: boxes of 32 columns over tensors of 16
    if ((rc = make_tmap_qkv(&tq, q, BS, d->N, d->H, Dt, TILE, lay_in, RowTile<DH>::BOX_D))) return rc;
    if ((rc = make_tmap_qkv(&tk, k, BS, d->N, d->H, Dt, TILE, lay_in, RowTile<DH>::BOX_D))) return rc;
    if ((rc = make_tmap_qkv(&tv, v, BS, d->N, d->H, Dt, TILE, lay_in, RowTile<DH>::BOX_D))) return rc;
    if ((rc = make_tmap_bias(&tb, bias, d->B, d->H, d->N))) return rc;

    FwdParams p{};
    p.B = d->B; p.S = d->S; p.N = d->N; p.H = d->H;
    p.Dt = Dt;
    p.KB = (Dt + 15) / 16;
    p.QT = QT;
    p.total_items = BS * QT * d->H;
    p.scale = (scale > 0.f) ? scale : 1.0f / sqrtf(static_cast<float>(Dt));
    p.inv_scale = 1.0f / p.scale;
    p.mask = static_cast<const __nv_bfloat16*>(mask);
    p.lse = lse;
    p.o = static_cast<__nv_bfloat16*>(o);
    p.o_resid = static_cast<__nv_bfloat16*>(o_resid);
    p.gate = static_cast<const __nv_bfloat16*>(gate);
    p.o_gated = static_cast<__nv_bfloat16*>(o_gated);
    p.lay = lay;
    p.status = status_word();
    if (!p.status) return EVO_ERR_CUDA;

    int sms = 0;
    if ((rc = sm_count(&sms))) return rc;
    if constexpr (WIDE) {
        using C = FwdWideCfg;
        // pairs of q tiles; with one q tile per row, items dealt to the two streams of a CTA in turn
        p.NG = d->S;
        p.QT = (QT + 1) / 2;
        p.total_items = BS * p.QT * d->H;
        const int grid = p.total_items < sms ? p.total_items : sms;
        p.step = FwdStep::of(grid * (QT == 1 ? 2 : 1), p.H, p.QT, p.NG);
        auto kernel = gate ? evo_fwd_wide_kernel<true> : evo_fwd_wide_kernel<false>;
        if ((rc = set_max_smem_once(reinterpret_cast<const void*>(kernel), static_cast<int>(C::SMEM_BYTES)))) return rc;
        prof_begin(0, st);
        rc = launch_chained(true, kernel, grid, C::THREADS, C::SMEM_BYTES, st, tq, tk, tv, tb, p);
        prof_end(0, st);
    } else {
        using C = FwdCfg<DH>;
        // Streams share bias tiles (rows taken G at a time) when that leaves no SM with more than 1/16 more rounds of
        // work than separate items would: a shared tile is loaded once instead of G times.
        const int sg = (d->S + C::G - 1) / C::G;
        const long units = static_cast<long>(d->B) * sg * QT * d->H;
        const long apart = (static_cast<long>(p.total_items) + static_cast<long>(C::G) * sms - 1) / (static_cast<long>(C::G) * sms);
        p.shared_bias = 0;
        p.NG = d->S;
        if ((units + sms - 1) / sms * 16 <= apart * 17 && p.total_items > sms) {
            p.shared_bias = 1;
            p.NG = sg;
            p.total_items = static_cast<int>(units);
        }
        const int grid = p.total_items < sms ? p.total_items : sms;
        p.step = FwdStep::of(grid * (p.shared_bias ? 1 : C::G), p.H, p.QT, p.NG);
        CUtensorMap to, t2;
        if ((rc = make_tmap_qkv(&to, o, BS, d->N, d->H, Dt, TILE, lay, RowTile<DH>::BOX_D))) return rc;
        t2 = to;
        const void* second = gate ? o_gated : o_resid;
        if (second && (rc = make_tmap_qkv(&t2, second, BS, d->N, d->H, Dt, TILE, lay, RowTile<DH>::BOX_D))) return rc;
        auto kernel = gate ? evo_fwd_kernel<DH, true> : evo_fwd_kernel<DH, false>;
        if ((rc = set_max_smem_once(reinterpret_cast<const void*>(kernel), static_cast<int>(C::SMEM_BYTES)))) return rc;
        prof_begin(0, st);
        rc = launch_chained(true, kernel, grid, C::THREADS, C::SMEM_BYTES, st, tq, tk, tv, tb, to, t2, p);
        prof_end(0, st);
    }
    return rc;
}

}  // namespace evo

extern "C" int evo_fwd(const EvoDims* dims, const void* q, const void* k, const void* v,
                       const void* pair_bias, const void* res_mask, void* o, void* o_resid, float* lse,
                       float scale, void* stream) {
    return evo_fwd_gated(dims, nullptr, q, k, v, pair_bias, res_mask, nullptr, o, nullptr, o_resid, lse, scale, stream);
}

extern "C" int evo_fwd_strided(const EvoDims* dims, const EvoStrides* strides, const void* q, const void* k,
                               const void* v, const void* pair_bias, const void* res_mask, void* o,
                               void* o_resid, float* lse, float scale, void* stream) {
    return evo_fwd_gated(dims, strides, q, k, v, pair_bias, res_mask, nullptr, o, nullptr, o_resid, lse, scale, stream);
}

extern "C" int evo_fwd_gated(const EvoDims* dims, const EvoStrides* strides, const void* q, const void* k,
                             const void* v, const void* pair_bias, const void* res_mask, const void* gate,
                             void* o, void* o_gated, void* o_resid, float* lse, float scale, void* stream) {
    return evo_fwd_views(dims, strides, strides, q, k, v, pair_bias, res_mask, gate, o, o_gated, o_resid, lse, scale,
                         stream);
}

extern "C" int evo_fwd_views(const EvoDims* dims, const EvoStrides* s_qkv, const EvoStrides* s_out, const void* q,
                             const void* k, const void* v, const void* pair_bias, const void* res_mask,
                             const void* gate, void* o, void* o_gated, void* o_resid, float* lse, float scale,
                             void* stream) {
    int rc = evo::check_dims(dims);
    if (rc) return rc;
    evo::ActLayout lay, lay_in;
    if ((rc = evo::layout_from_strides(dims, s_qkv, &lay_in))) return rc;
    if ((rc = evo::layout_from_strides(dims, s_out, &lay))) return rc;
    if (!q || !k || !v || !pair_bias || !res_mask || !o || !lse) return EVO_ERR_NULL_PTR;
    if ((gate == nullptr) != (o_gated == nullptr)) return EVO_ERR_NULL_PTR;
    const uintptr_t all = reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) |
                          reinterpret_cast<uintptr_t>(v) | reinterpret_cast<uintptr_t>(pair_bias) |
                          reinterpret_cast<uintptr_t>(o) | reinterpret_cast<uintptr_t>(o_resid) |
                          reinterpret_cast<uintptr_t>(res_mask) | reinterpret_cast<uintptr_t>(gate) |
                          reinterpret_cast<uintptr_t>(o_gated);
    if (all & 15u) return EVO_ERR_ALIGNMENT;
    if ((rc = evo::ensure_context())) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (dims->D <= 32)
        return evo::launch_fwd<32>(dims, lay_in, lay, q, k, v, pair_bias, res_mask, gate, o, o_gated,
                                                 o_resid, lse, scale, st);
    if (dims->D <= 64)
        return evo::launch_fwd<64>(dims, lay_in, lay, q, k, v, pair_bias, res_mask, gate, o, o_gated, o_resid, lse,
                                      scale, st);
    return evo::launch_fwd<128>(dims, lay_in, lay, q, k, v, pair_bias, res_mask, gate, o, o_gated, o_resid, lse,
                                   scale, st);
}
