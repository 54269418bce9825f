// EvoAttention backward for sm_100a.
//
// Replaces evo_bwd_prep_ker / evo_bwd_ker (evo_h100/tk_evoattention.cu:352-416,
// :613-890) and their host launcher (tk_evoattention.cu:1051-1197):
//
//   P  = exp(q k^T * scale + pair_bias + res_mask - LSE)      (recomputed)
//   dP = dO v^T,  dS = P o (dP - delta),  delta = rowsum(dO o O)
//   dV = P^T dO,  dK = scale * dS^T q,  dQ = scale * dS k
//   dBias[b,h,q,kv] = sum over s of dS        (unscaled, tk_evoattention.cu:824-833)
//
// Four launches on one stream:
//   1. bwd_prep_kernel    delta and the extra tiles through which the main kernels add
//                         (mask - LSE) / scale to S and -delta to dP inside the tensor
//                         core (evo_tiles.cuh, "EXTRA TILE"), padded to whole tiles so
//                         the main kernels need no edge predicates; zeroes the accumulators
//   2. evo_dbias_kernel   dBias (evo_dbias.cu): one CTA per pair-bias tile keeps its
//                         sum over the S rows in registers, no reduction traffic
//   3. evo_bwd_kernel     dQ, dK, dV (below; D <= 32: evo_bwd_halves.cuh, D > 64: evo_bwd_wide.cuh)
//   4. bwd_finish_kernel  fp32 dQ accumulator -> bf16 dQ in the caller layout (and dBias,
//                         summed over slices of S in fp32, to bf16 if the caller wants that)
#include "evo_dbias.cuh"
#include "evo_host.cuh"
#include "evo_ptx.cuh"
#include "evo_tiles.cuh"

#include <algorithm>
#include <mutex>
#include <type_traits>


namespace evo {

constexpr uint32_t BWD_TMEM_COLS = 512;

struct BwdParams {
    int B, S, N, H;
    int Dt;          // true head dim (16 runs on the D = 32 kernel: loads zero-filled, stores clipped)
    int KB;          // contraction blocks of 16 head-dim columns that hold data: ceil(Dt / 16)
    int NT;          // tiles per row: ceil(N / 128)
    int NTP;         // NT * 128
    int pairs;       // B * S * H
    int n_whole;     // pairs taken whole; the others are dealt by segments
    float scale;     // softmax scale
    float c1;        // scale * log2(e)
    const __nv_bfloat16* xq;   // [B*S][H][NTP][8] extra tiles of the q rows  (bwd_prep_kernel)
    const __nv_bfloat16* xk;   // [B*S][NTP][8]    extra tiles of the kv rows
    const __nv_bfloat16* bias; // [B][H][N][N]
    void* dbias;               // [B][H][N][N], fp32 or bf16 (written by this kernel only when S = 1)
    float* dq_scratch;         // whole pairs: per CTA scratch_stride 16-byte words, partial sums of dQ
    size_t scratch_stride;
    float* dq_acc;             // the others: [B*S - acc_row0][N][H][DH], zeroed before the launch
    int acc_row0;              // their first S row
    int seg_dj, seg_dp;        // from a CTA's single segment to its next: kv tiles, pairs (grid % NT, grid / NT)
    __nv_bfloat16* dq;    // activation layout `lay` (dq: of the whole pairs only)
    __nv_bfloat16* dk;
    __nv_bfloat16* dv;
    ActLayout lay;        // element strides of the activation tensors
    unsigned int* status;
};

// DBIAS_HERE (S = 1 only): dBias is dS itself, no sum over rows, so the compute groups store their
// dS straight to d_pair_bias and the dBias kernel (which would recompute S and dP for one step
// per item) is not launched.
enum DbiasHere { DBIAS_NO = 0, DBIAS_F32 = 1, DBIAS_BF16 = 2 };

// What a CTA of the dQ/dK/dV kernels walks: the segments (kv tiles) of whole pairs (S row, head) one after another,
// single segments, or the one and then the other.  A template parameter: chosen at run time it costs the drain warps,
// and all of a D = 128 step, 5 %.
enum Walk { WALK_SEGMENTS, WALK_WHOLE, WALK_BOTH };
template <int WALK>
struct Segments {
    int first, stride, NT, H, n_whole, n_ws, n;     // n_ws: segments of whole pairs; n: all
    __device__ __forceinline__ explicit Segments(const BwdParams& p)
        : first(blockIdx.x), stride(gridDim.x), NT(p.NT), H(p.H), n_whole(WALK == WALK_SEGMENTS ? 0 : p.n_whole) {
        auto share = [&](int total) { return total > first ? (total - first + stride - 1) / stride : 0; };
        n_ws = WALK == WALK_SEGMENTS ? 0 : share(n_whole) * NT;
        n = WALK == WALK_WHOLE ? n_ws : n_ws + share((p.pairs - n_whole) * NT);
    }
    __device__ __forceinline__ bool whole(int sg) const {
        return WALK == WALK_WHOLE || (WALK == WALK_BOTH && sg < n_ws);
    }
    __device__ __forceinline__ void decode(int sg, int& bs, int& h, int& j) const {
        int pair;
        if (whole(sg)) {
            j = sg % NT;
            pair = first + sg / NT * stride;
        } else {
            const int w = first + (sg - n_ws) * stride;
            j = w % NT;
            pair = n_whole + w / NT;
        }
        h = pair % H;
        bs = pair / H;
    }
};

}  // namespace evo
#include "evo_bwd_halves.cuh"
#include "evo_bwd_wide.cuh"
namespace evo {

// ---------------------------------------------------------------------------
// dQ, dK, dV at D = 64, and what the dQ/dK/dV kernels share (D <= 32: evo_bwd_halves.cuh; D = 96, 128: evo_bwd_wide.cuh).
// One persistent CTA per SM walks segments (S row, head h, kv tile j of 128 residues); a segment walks steps (q tile i).
// Everything is formed TRANSPOSED, kv rows in the tensor-memory lanes, so that P^T and dS^T are in place as A operands of
// the products that contract over q, without a trip through shared memory:
//
//   S'^T = K Q^T + extra block,  dP'^T = V dO^T + extra block         (evo_tiles.cuh, "EXTRA TILE")
//   P^T = exp2(S'^T c1 + bias^T log2e),  dS^T = P^T o dP'^T           (thread = one kv row)
//   dV += P^T dO,  dK += dS^T Q      A from tensor memory: 16 clocks per K = 16 block at N = 32, where an
//                                    A tile in shared memory costs 40 (it is read at 128 bytes a clock)
//   dQ = dS K                        A = dS from shared memory (M = q: MN-major), the one tile written there
//
// What bounds a step is the work of the compute warps, about 1400 issue slots and 1024 clocks of
// exponentials per scheduler, and the chain of barriers and products around it.  Sixteen compute warps,
// because with eight the loads, multiplies and exponentials of a warp hardly overlapped (2000 clocks for
// the same work).
//
//   D = 64: no columns for P^T and dS^T: they overwrite the columns they were computed from.  Two phases, P (from
//     S') and dS (from dP'), each with its own barriers, so that the products of one are formed during the other: dV
//     and S' of the next step while dS is computed, dK, dQ and dP' of the next step while its P is (B=1, S=256,
//     N=1024, H=4: 1.30 -> 1.11 ms).  The halves of the D <= 32 kernel measure the same here (1.13 and 1.12 ms) and lose
//     where a pair has two q tiles or one S row (S=200, N=200, H=4 78 -> 84 us; B=4, S=1, N=1024, H=16 106 -> 121): one
//     dQ accumulator and one K/V buffer are all that fits.
//
//   warps 0-15 (compute)  group g = warp / 4 owns q columns 32g .. 32g+31 of the tile
//   warps 16-19 (drain)   after every step 32 rows of dQ each, after a segment dK and dV as bf16 stores
//   warp 20 (producer)    TMA: per step Q, dO, the extra tile of the q rows, the pair-bias tile; per
//                         segment K, V and the extra tile of the kv rows
//   warps 21, 22, 23      MMA issuers, one chain family each: S'^T and dP'^T; dV and dK; dQ
//
// dQ is a sum over kv tiles.  A CTA takes all NT segments of a pair (S row, head) where it can, and so sees
// the whole sum.  With few tiles (two here, four at D <= 32) it stays in tensor memory until the last segment; otherwise
// the drain warps keep partial sums in a scratch area of the CTA, in L2 (written and added to by bulk copies: loads
// and stores of their own held up the compute warps' shared-memory accesses), and the last segment's go out
// as bf16.  Whole pairs fill whole rounds of the SMs; the pairs that are left over are dealt by segments, and
// their partial sums meet in an fp32 accumulator in memory (TMA reduce-add), which costs a pass to zero it and
// a pass to convert it, of those pairs only (against all pairs whole, or none, the kernel alone: S=384, N=384, H=4,
// D=32 182 -> 176 us; S=200, N=200, H=4 47 -> 44; S=1024, N=768, H=8 3333 -> 3255).
//
// Measured against one kernel with P and dS in shared memory and two compute groups (whole backward):
// S=256, N=1024, H=4, D=64 1.93 -> 1.59 ms; B=4, S=1, N=1024, H=16, D=64 0.24 -> 0.15.
// ---------------------------------------------------------------------------
struct BwdCfg {
    static constexpr int DH = 64;
    static constexpr int NG = 4;                       // compute groups
    static constexpr int CW = TILE / NG;               // q columns per group
    static constexpr int NCW = 4 * NG;
    static constexpr int W_DRAIN = NCW, W_PROD = NCW + 4, W_MMA = NCW + 5;
    static constexpr int THREADS = (NCW + 8) * 32;
    static constexpr int QS = 2;                       // Q/dO stages
    static constexpr int NKV = 1;                      // K/V buffers
    static constexpr int NB = 2;                       // bias tiles
    static constexpr int DQ_BUFS = 2;
    static constexpr uint32_t ROWT = RowTile<DH>::BYTES;
    static constexpr uint32_t ST_Q = 0, ST_DO = ROWT, ST_XQ = 2 * ROWT;
    static constexpr uint32_t STAGE_BYTES = 2 * ROWT + XT_BYTES;
    static constexpr uint32_t KV_K = 0, KV_V = ROWT, KV_XK = 2 * ROWT, KV_BYTES = 2 * ROWT + XT_BYTES;
    static constexpr uint32_t OFF_STAGE = 0;
    static constexpr uint32_t OFF_KV = OFF_STAGE + QS * STAGE_BYTES;
    static constexpr uint32_t OFF_BIAS = OFF_KV + NKV * KV_BYTES;
    static constexpr uint32_t OFF_DS = OFF_BIAS + NB * SQ_BYTES;
    // per drain warp a slot of [32 rows][32 fp32], for bulk copies of dQ, dK and dV
    static constexpr uint32_t WQ_BYTES = 32 * 32 * 4;
    static constexpr uint32_t OFF_WSTG = OFF_DS + SQ_BYTES;
    // constant extra tiles, above every tile that refers to the zero tile
    static constexpr uint32_t OFF_XDP = OFF_WSTG + 4 * WQ_BYTES;            // row selector of -delta
    static constexpr uint32_t OFF_ZERO = OFF_XDP + XT_BYTES;
    static constexpr uint32_t OFF_BARS = OFF_ZERO + XT_BYTES;
    static constexpr uint32_t NUM_BARS = 2 * QS + 2 * NKV + 2 * NB + 2 * DQ_BUFS + 8;
    static constexpr uint32_t OFF_MISC = OFF_BARS + NUM_BARS * 8;
    static constexpr uint32_t SMEM_BYTES = OFF_MISC + 16 + 1024;            // + alignment slack
    static constexpr uint32_t TMEM_S = 0, TMEM_DP = 128;
    static constexpr uint32_t TMEM_DQ = 256;                                // DQ_BUFS accumulators
    static constexpr uint32_t TMEM_DK = TMEM_DQ + 2 * DH, TMEM_DV = TMEM_DK + DH;
    // column of contraction block kk (16 q) of P^T / dS^T, inside the columns of its own group
    __device__ static __forceinline__ uint32_t p_col(int kk) { return TMEM_S + 32 * (kk >> 1) + 8 * (kk & 1); }
    __device__ static __forceinline__ uint32_t ds_col(int kk) { return p_col(kk) + 128; }
    static_assert(TMEM_DV + DH <= BWD_TMEM_COLS, "tensor memory budget");
    static_assert(SMEM_BYTES <= 232448, "shared memory budget");
    static_assert(STAGE_BYTES % 1024 == 0 && KV_BYTES % 1024 == 0 && WQ_BYTES % 1024 == 0, "tile alignment");
};

template <int WALK, int DBIAS_HERE>
__global__ void __launch_bounds__(BwdCfg::THREADS, 1)
evo_bwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
               const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_do,
               const __grid_constant__ CUtensorMap tm_bias, const __grid_constant__ CUtensorMap tm_dq,
               const __grid_constant__ CUtensorMap tm_dk, const __grid_constant__ CUtensorMap tm_dv,
               const __grid_constant__ CUtensorMap tm_acc, const BwdParams p) {
    using C = BwdCfg;
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
    uint64_t* s_full = kv_empty + NKV;         // [NB]: S' complete and the bias tile landed
    uint64_t* bias_empty = s_full + NB;        // [NB]
    uint64_t* dq_full = bias_empty + NB;       // [DQB]
    uint64_t* dq_free = dq_full + DQB;         // [DQB]
    uint64_t* dp_full = dq_free + DQB;         // dP' complete
    uint64_t* p_ready = dp_full + 1;           // P^T is written
    uint64_t* ds_ready = p_ready + 1;          // dS^T and the dS tile are written
    uint64_t* dv_done = ds_ready + 1;          // dV of the step is complete
    uint64_t* dk_done = dv_done + 1;           // dK
    uint64_t* dq_done = dk_done + 1;           // dQ
    uint64_t* dkv_full = dq_done + 1;          // dK, dV of the segment are complete
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
        for (int i = 0; i < NB; ++i) { mbar_init(&s_full[i], 2); mbar_init(&bias_empty[i], C::NCW); }
        for (int i = 0; i < DQB; ++i) { mbar_init(&dq_full[i], 1); mbar_init(&dq_free[i], 4); }
        for (uint64_t* x : {p_ready, ds_ready}) mbar_init(x, C::NCW);
        for (uint64_t* x : {dp_full, dv_done, dk_done, dq_done, dkv_full}) mbar_init(x, 1);
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

    if (warp == C::W_PROD) {
        // ------------------------------ producer ------------------------------
        bool ok = true;
        int gs = 0, n_st = 0, n_bias = 0, n_kv = 0;      // steps; loads issued
        for (int sg = 0; sg < n_segs && ok; ++sg) {
            int bs, h, j;
            seg.decode(sg, bs, h, j);
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
            for (int i = 0; i < NT && ok; ++i, ++gs) {
                const int st = gs % QS, bb = gs % NB;
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
                if (gs >= NB) ok = warp_all(mbar_wait(&bias_empty[bb], ((gs / NB) - 1) & 1, wc, 0x41));
                if (!ok) break;
                if (elect_one()) {
                    uint8_t* bt = smem + C::OFF_BIAS + bb * SQ_BYTES;
                    mbar_arrive_expect_tx(&s_full[bb], SQ_BYTES);
                    tma_load_4d(bt, &tm_bias, &s_full[bb], j * TILE, i * TILE, h, b);
                    tma_load_4d(bt + SQ_SUB_BYTES, &tm_bias, &s_full[bb], j * TILE + 64, i * TILE, h, b);
                }
                __syncwarp();
                ++n_bias;
            }
        }
        // The last loads have landed before the CTA exits, also if a wait gave up (a bias load shares its
        // barrier with an MMA commit, which may then never come: a bounded pause instead).
        const WaitCtx dc{tmem_slot + 3, p.status};
        for (int k = (n_st > QS ? n_st - QS : 0); k < n_st; ++k) mbar_wait_landed(&st_full[k % QS], (k / QS) & 1, dc, 0x43);
        for (int k = (n_kv > NKV ? n_kv - NKV : 0); k < n_kv; ++k) mbar_wait_landed(&kv_full[k % NKV], (k / NKV) & 1, dc, 0x45);
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
        const uint32_t aSt = smem_u32(smem + C::OFF_STAGE), aKV = smem_u32(smem + C::OFF_KV);
        const uint32_t aZero = smem_u32(smem + C::OFF_ZERO);
        const int role = warp - C::W_MMA;          // 0: S/dP, 1: dV/dK, 2: dQ
        bool ok = true;
        int gs = 0;
        for (int sg = 0; sg < n_segs && ok; ++sg) {
            const int kb = sg % NKV;
            const uint32_t kvb = aKV + kb * C::KV_BYTES;
            for (int i = 0; i < NT && ok; ++i, ++gs) {
                const int st = gs % QS;
                const uint32_t sb = aSt + st * C::STAGE_BYTES;
                if (role == 0) {
                    ok = warp_all(mbar_wait(&st_full[st], (gs / QS) & 1, wc, 0x50));
                    if (ok && i == 0) ok = warp_all(mbar_wait(&kv_full[kb], (sg / NKV) & 1, wc, 0x51));
                    // P^T in the columns is consumed
                    if (ok && gs > 0) ok = warp_all(mbar_wait(dv_done, (gs - 1) & 1, wc, 0x52));
                    if (!ok) break;
                    tc_fence_after();
                    const uint64_t d_xq = xt_desc(sb + C::ST_XQ, aZero);
                    if (elect_one()) {
                        const uint32_t q_lo = RD::kmajor_lo(sb + C::ST_Q), k_lo = RD::kmajor_lo(kvb + C::KV_K);
#pragma unroll
                        for (int kk = 0; kk < RT::KBLOCKS; ++kk)
                            if (kk < p.KB)      // the others are zero-filled blocks past the true head dim
                                umma_ss(tmem + C::TMEM_S, RD::kmajor(k_lo, kk), RD::kmajor(q_lo, kk), IDESC_SDP, kk > 0);
                        // + (mask - LSE) / scale: the extra contraction block
                        umma_ss(tmem + C::TMEM_S, xt_desc(kvb + C::KV_XK, aZero), d_xq, IDESC_SDP, 1u);
                        umma_commit(&s_full[gs % NB]);
                    }
                    __syncwarp();
                    if (gs > 0) ok = warp_all(mbar_wait(dk_done, (gs - 1) & 1, wc, 0x59));
                    if (!ok) break;
                    tc_fence_after();
                    if (elect_one()) {
                        const uint32_t do_lo = RD::kmajor_lo(sb + C::ST_DO), v_lo = RD::kmajor_lo(kvb + C::KV_V);
#pragma unroll
                        for (int kk = 0; kk < RT::KBLOCKS; ++kk)
                            if (kk < p.KB)
                                umma_ss(tmem + C::TMEM_DP, RD::kmajor(v_lo, kk), RD::kmajor(do_lo, kk), IDESC_SDP, kk > 0);
                        // - delta
                        umma_ss(tmem + C::TMEM_DP, xt_desc(smem_u32(smem + C::OFF_XDP), aZero), d_xq, IDESC_SDP, 1u);
                        umma_commit(dp_full);
                    }
                    __syncwarp();
                } else if (role == 1) {
                    const uint32_t acc = (i > 0) ? 1u : 0u;
                    // the first MMA of a segment overwrites dK / dV: the previous one's must be out
                    if (i == 0 && sg > 0) ok = warp_all(mbar_wait(dkv_free, (sg - 1) & 1, wc, 0x55));
                    const uint32_t q_lo = RD::mnmajor_lo(sb + C::ST_Q), do_lo = RD::mnmajor_lo(sb + C::ST_DO);
                    auto dv = [&](int kk) {
                        umma_ts(tmem + C::TMEM_DV, tmem + C::p_col(kk), RD::mnmajor(do_lo, kk), IDESC_DKV, kk > 0 ? 1u : acc);
                    };
                    auto dk = [&](int kk) {
                        umma_ts(tmem + C::TMEM_DK, tmem + C::ds_col(kk), RD::mnmajor(q_lo, kk), IDESC_DKV, kk > 0 ? 1u : acc);
                    };
                    if (ok) ok = warp_all(mbar_wait(p_ready, gs & 1, wc, 0x53));
                    if (!ok) break;
                    tc_fence_after();
                    if (elect_one()) {
#pragma unroll
                        for (int kk = 0; kk < 8; ++kk) dv(kk);
                        umma_commit(dv_done);
                    }
                    __syncwarp();
                    ok = warp_all(mbar_wait(ds_ready, gs & 1, wc, 0x5a));
                    if (!ok) break;
                    tc_fence_after();
                    if (elect_one()) {
#pragma unroll
                        for (int kk = 0; kk < 8; ++kk) dk(kk);
                        umma_commit(dk_done);
                        umma_commit(&st_empty[st]);
                        if (i == NT - 1) {
                            umma_commit(dkv_full);
                            umma_commit(&kv_empty[kb]);
                        }
                    }
                    __syncwarp();
                } else {
                    const bool whole = seg.whole(sg), resident = whole && res_ok;
                    const int j = whole ? sg % NT : 0, ev = dq_event(resident, sg, j, i);
                    if (ev >= DQB && !(resident && j > 0)) ok = warp_all(mbar_wait(&dq_free[ev % DQB], ((ev / DQB) - 1) & 1, wc, 0x54));
                    if (ok) ok = warp_all(mbar_wait(ds_ready, gs & 1, wc, 0x5b));
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
                        umma_commit(dq_done);
                        if (!resident || j == NT - 1) umma_commit(&dq_full[ev % DQB]);
                        if (i == NT - 1) umma_commit(&kv_empty[kb]);
                    }
                    __syncwarp();
                }
            }
        }
    } else if (warp >= C::W_DRAIN) {
        // ------------------------------ drain warps ------------------------------
        const int w4 = warp & 3;
        const int wrow0 = w4 * 32;           // tensor-memory lanes (tile rows) of this warp
        const uint32_t lane_base = tmem + (static_cast<uint32_t>(wrow0) << 16);
        uint8_t* const wslot = smem + C::OFF_WSTG + w4 * C::WQ_BYTES;
        // Where the next bulk copy (one group each) is staged, once the copy that used the place last has read it: the
        // slot, or its halves in turn for copies of half its size.
        int pos = 0;
        bool last_half = false;
        auto next_slot = [&](bool half) -> uint8_t* {
            if (lane == 0) {
                if (half && last_half) tma_wait_group_read<1>();
                else tma_wait_group_read<0>();
            }
            __syncwarp();
            last_half = half;
            pos ^= 1;
            return wslot + (half ? pos * (C::WQ_BYTES / 2) : 0);
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
            for (int sg = sg0; sg < sg1 && ok; ++sg) {
                int bs, h, j;
                seg.decode(sg, bs, h, j);
                const bool resident = whole && res_ok;
                for (int i = 0; i < NT && ok; ++i) {
                    if (resident && j < NT - 1) continue;          // dQ is still being summed
                    const int ev = dq_event(resident, sg, j, i), b = ev % DQB;
                    const bool rows = i * TILE + wrow0 < p.N;     // warp-uniform: some row of this warp exists
                    const bool final_sum = whole && j == NT - 1, add = final_sum && j > 0 && !resident && rows;
                    float4* ps = part + static_cast<size_t>(i * 4 + w4) * (DH / 4) * 32;
                    float4 old[8];
                    // The bulk copy that last wrote this part of the scratch area, NT >= 3 steps ago, is complete
                    // before the sum is added to or read: at least two were issued after it.
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
                        uint8_t* wq = next_slot(false);
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
    #pragma unroll
                for (int t = 0; t < 2; ++t) {                   // dK, then dV
                    uint4 u[DH / 32][4];
    #pragma unroll
                    for (int c = 0; c < DH / 32; ++c) {
                        float v[32];
                        __syncwarp();
                        tmem_ld_f32<32>(lane_base + (t ? C::TMEM_DV : C::TMEM_DK) + c * 32, v);
                        pack_rows(u[c], v, t ? 1.0f : p.scale);
                    }
                    if (t == 1) {
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(dkv_free);
                    }
    #pragma unroll
                    for (int c = 0; c < DH / 32; ++c)
                        if (some && c * 32 < p.Dt) store_rows(t ? &tm_dv : &tm_dk, u[c], h, j * TILE + wrow0, c * 32, bs);
                }
            }
        };
        if (WALK != WALK_SEGMENTS) drain(std::true_type{}, 0, seg.n_ws);
        if (WALK != WALK_WHOLE) drain(std::false_type{}, seg.n_ws, n_segs);
        if (lane == 0) tma_wait_group<0>();
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
        bool ok = true;
        int gs = 0;
        const float2 c1x2 = make_float2(p.c1, p.c1), l2e2 = make_float2(LOG2E, LOG2E);

        // one S row: a step's dS tile is the dBias tile (q tile i, kv tile j); columns 16 ch .. of this group
        auto store_dbias = [&](int ch, int i, int j, int bs, int h, const uint32_t (&pkd)[8], const float2 (&dsv)[8]) {
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
        };

        for (int sg = 0; sg < n_segs && ok; ++sg) {
            int bs = 0, h = 0, j = 0;
            if constexpr (DBIAS_HERE != DBIAS_NO) seg.decode(sg, bs, h, j);
            for (int i = 0; i < NT && ok; ++i, ++gs) {
                const int bb = gs % NB;
                // ---- phase P: x = S' c1 + bias log2e (S' already carries mask and -LSE through the extra
                // contraction block), P = exp2(x), P^T (bf16) into tensor memory
                // (S' of this step waited for dV of the previous one: its columns are free)
                ok = warp_all(mbar_wait(&s_full[bb], (gs / NB) & 1, wc, 0x63));
                if (!ok) break;
                tc_fence_after();
                float2 p2[16];
                uint32_t dep = 0;
#pragma unroll
                for (int ch = 0; ch < 2; ++ch) {          // 16 columns at a time
                    uint32_t sv[16], bq[16];
                    tmem_ld16(tS + 16 * ch, sv);
#pragma unroll
                    for (int k = 0; k < 16; ++k)
                        bq[k] = lds_u16(aBias + bb * SQ_BYTES + (16 * ch + k) * 128 + ((bchunk ^ (k & 7)) << 4));
                    tmem_wait_ld();
                    uint32_t pk[8];
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        const float2 b2 = fmul2(make_float2(__uint_as_float(bq[2 * k] << 16), __uint_as_float(bq[2 * k + 1] << 16)), l2e2);
                        const float2 x2 = ffma2(u2f2(sv[2 * k], sv[2 * k + 1]), c1x2, b2);
                        const float2 e2 = make_float2(ex2(x2.x), ex2(x2.y));
                        p2[8 * ch + k] = e2;
                        pk[k] = pack_bf16(e2.x, e2.y);
                    }
#pragma unroll
                    for (int k = 0; k < 8; ++k) dep ^= pk[k];      // depends on every bias value read
                    tmem_st8(lane_base + C::p_col(2 * g + ch), pk);
                }
                mbar_release_after_loads(&bias_empty[bb], dep, scratch_w);
                tmem_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(p_ready);

                // ---- phase dS: dS = P dP' (dP' already carries -delta), dS^T into tensor memory and the tile.
                // Both are free once dK and dQ of the previous step are complete.
                if (gs == 0)
                    ok = warp_all(mbar_wait(dp_full, 0, wc, 0x66));
                else                           // (dP' of this step waited for dK)
                    ok = warp_all(mbar_wait_both(dp_full, gs & 1, dq_done, (gs - 1) & 1, wc, 0x66));
                if (!ok) break;
                tc_fence_after();
#pragma unroll
                for (int ch = 0; ch < 2; ++ch) {
                    uint32_t dv[16];
                    tmem_ld16(tDP + 16 * ch, dv);
                    tmem_wait_ld();
                    uint32_t pkd[8];
                    float2 dsv[8];
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        dsv[k] = fmul2(p2[8 * ch + k], u2f2(dv[2 * k], dv[2 * k + 1]));
                        pkd[k] = pack_bf16(dsv[k].x, dsv[k].y);
                    }
                    tmem_st8(lane_base + C::ds_col(2 * g + ch), pkd);
#pragma unroll
                    for (int c = 0; c < 2; ++c)
                        sts128(aDS + sq_chunk_off(row, 4 * g + 2 * ch + c),
                               make_uint4(pkd[4 * c], pkd[4 * c + 1], pkd[4 * c + 2], pkd[4 * c + 3]));
                    store_dbias(ch, i, j, bs, h, pkd, dsv);
                }
                tmem_wait_st();
                tc_fence_before();
                fence_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(ds_ready);
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (tid == 0) { report_abort(wc); report_abort(WaitCtx{tmem_slot + 3, p.status}); }
    if (warp == C::W_MMA) tmem_dealloc(tmem, BWD_TMEM_COLS);
}

// ---------------------------------------------------------------------------
// prep: delta = rowsum(dO o O) (replaces evo_bwd_prep_ker, tk_evoattention.cu:352-416),
// and the extra tiles through which the main kernels add every per-row and per-column
// term of the logits inside the tensor core (evo_tiles.cuh, "EXTRA TILE"):
//
//   xq [B*S][H][NTP][8] bf16, row q:  ( 1, 1, a_hi, a_lo, -d_hi, -d_lo, 0, 0 )   a = -LSE / scale
//   xk [B*S][NTP][8]    bf16, row kv: ( m_hi, m_lo, 1, 1, 0, 0, 0, 0 )           m = mask / scale
//
// so that  Q K^T + xq xk^T = Q K^T + (mask - LSE) / scale  (times scale*log2e: the base-2
// logit minus the base-2 LSE) and  dO V^T + xq (0,0,0,0,1,1,0,0)^T = dP - delta.
// Values are split into a bf16 head and a bf16 remainder (16 significant bits).  Rows
// past N (padding up to whole tiles, NTP = tiles * 128) get a = m = -1e30: finite, so
// that a product with a zero of the other tile stays zero, and far below any logit.
// With o_resid (the bf16 rounding residual of O written by the forward), delta
// uses O to about 16 bits instead of 8: the rounding of O otherwise puts an
// error of order 2^-9 |dO||O| on every dS, which adds up over the S rows of dBias.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t split_bf16(float v) {
    // (head, remainder) as a bf16 pair, head in the low half
    v = fminf(fmaxf(v, -1e30f), 1e30f);
    const __nv_bfloat16 hi = __float2bfloat16_rn(v);
    const __nv_bfloat16 lo = __float2bfloat16_rn(v - __bfloat162float(hi));
    return static_cast<uint32_t>(__bfloat16_as_ushort(hi)) | (static_cast<uint32_t>(__bfloat16_as_ushort(lo)) << 16);
}

// With a gate (evo_bwd_gated) d_o is the gradient of the GATED output: the kernel then also forms
// sig = sigmoid(gate), writes the gradient that enters the attention, bf16(d_o * sig), to do_att
// (contiguous [B*S][N][H][Dt], what the main kernels read as their dO) and the gate's gradient
// d_o * O * sig * (1 - sig) to d_gate, and takes delta from the rounded do_att.
//
// Bound by DRAM: it reads O, its residual and dO once and also zeroes the accumulators of the later
// kernels (`zero`, n_zero 16-byte words), which saves two memset launches.  Dt / 8 lanes share a row
// (one 16-byte chunk each) and rows are walked in the order they lie in memory, so that a warp's loads
// are contiguous.
struct PrepParams {
    const __nv_bfloat16 *o, *o_resid, *d_o, *mask, *gate;
    const float* lse;
    uint4 *xq, *xk;
    __nv_bfloat16 *do_att, *d_gate;
    uint4* zero[2];
    size_t n_zero[2];
    float inv_scale;
    int BS, N, H, NTP, Dt;
    ActLayout lay;
};
// LANES per row: the power of two at or above Dt / 8.  U rows per thread at a time, their loads in flight
// together.  All blocks are resident: with a grid that the registers cut into two waves, as it was, the
// second wave held half of the threads (B=1, S=512, N=384, H=8, D=32 82 -> 61 us, 50 at the rate of a copy).
template <int U>
constexpr int prep_blocks() { return U == 1 ? 5 : 3; }      // per SM: 48 and 80 registers
template <int LANES, bool GATED, int U>
__global__ void __launch_bounds__(256, prep_blocks<U>()) bwd_prep_kernel(const PrepParams p) {
    constexpr uint32_t ONES = 0x3f803f80u;     // bf16 (1, 1)
    const size_t gstride = static_cast<size_t>(gridDim.x) * blockDim.x;
    const size_t t0 = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const int N = p.N, H = p.H, NTP = p.NTP;
    const size_t rows = static_cast<size_t>(p.BS) * N * H;
    const int c = static_cast<int>(t0 % LANES);      // this lane's chunk of eight head-dim columns
    const bool have = c * 8 < p.Dt;
    // which of the two outer axes lies closer together in memory
    const bool n_inner = p.lay.n <= p.lay.row;
    const uint32_t inner = n_inner ? N : p.BS;
    const size_t rstride = gstride / LANES;
    struct At { size_t bs, n, h; };
    auto at = [&](size_t r) -> At {
        uint32_t h, in_, out_;
        if (rows < 0x80000000ull) {              // 32-bit divisions where they suffice
            const uint32_t r32 = static_cast<uint32_t>(r), b32 = r32 / H;
            h = r32 - b32 * H;
            out_ = b32 / inner;
            in_ = b32 - out_ * inner;
        } else {
            const size_t bn = r / H;
            h = static_cast<uint32_t>(r - bn * H);
            out_ = static_cast<uint32_t>(bn / inner);
            in_ = static_cast<uint32_t>(bn - static_cast<size_t>(out_) * inner);
        }
        return At{n_inner ? out_ : in_, n_inner ? in_ : out_, h};
    };
    // (whole warps run the same number of iterations: the shuffles need all lanes)
    for (size_t r0 = (t0 - (threadIdx.x & 31)) / LANES; r0 < rows; r0 += U * rstride) {
        uint4 a[U], b[U], rr[U], g4[GATED ? U : 1];
        float lse[U];
        size_t off[U], ro[U], att[GATED ? U : 1];
        bool live[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const size_t r = r0 + (threadIdx.x & 31) / LANES + u * rstride;
            live[u] = r < rows;
            a[u] = b[u] = rr[u] = make_uint4(0u, 0u, 0u, 0u);
            lse[u] = 0.f;
            if constexpr (GATED) g4[u] = make_uint4(0u, 0u, 0u, 0u);
            if (!live[u]) continue;
            const At x = at(r);
            off[u] = x.bs * p.lay.row + x.n * p.lay.n + x.h * p.lay.h + c * 8;
            ro[u] = (x.bs * H + x.h) * NTP + x.n;
            if constexpr (GATED) att[u] = ((x.bs * N + x.n) * H + x.h) * static_cast<size_t>(p.Dt) + c * 8;
            if (have) {
                a[u] = __ldg(reinterpret_cast<const uint4*>(p.o + off[u]));
                b[u] = __ldg(reinterpret_cast<const uint4*>(p.d_o + off[u]));
                if (p.o_resid) rr[u] = __ldg(reinterpret_cast<const uint4*>(p.o_resid + off[u]));
                if constexpr (GATED) g4[u] = __ldg(reinterpret_cast<const uint4*>(p.gate + off[u]));
            }
            if (c == 0) lse[u] = __ldg(p.lse + (x.bs * H + x.h) * N + x.n);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint32_t aw[4] = {a[u].x, a[u].y, a[u].z, a[u].w}, rw[4] = {rr[u].x, rr[u].y, rr[u].z, rr[u].w};
            if constexpr (GATED) {
                const uint32_t gw[4] = {g4[u].x, g4[u].y, g4[u].z, g4[u].w}, dw[4] = {b[u].x, b[u].y, b[u].z, b[u].w};
                uint32_t aw2[4], gg[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float s0 = 1.0f / (1.0f + ex2(-bf16_lo(gw[e]) * LOG2E));
                    const float s1 = 1.0f / (1.0f + ex2(-bf16_hi(gw[e]) * LOG2E));
                    const float d0 = bf16_lo(dw[e]), d1 = bf16_hi(dw[e]);
                    const float o0 = bf16_lo(aw[e]) + bf16_lo(rw[e]), o1 = bf16_hi(aw[e]) + bf16_hi(rw[e]);
                    aw2[e] = pack_bf16(d0 * s0, d1 * s1);
                    gg[e] = pack_bf16(d0 * o0 * s0 * (1.0f - s0), d1 * o1 * s1 * (1.0f - s1));
                }
                b[u] = make_uint4(aw2[0], aw2[1], aw2[2], aw2[3]);
                if (live[u] && have) {
                    *reinterpret_cast<uint4*>(p.do_att + att[u]) = b[u];
                    *reinterpret_cast<uint4*>(p.d_gate + off[u]) = make_uint4(gg[0], gg[1], gg[2], gg[3]);
                }
            }
            const uint32_t bw[4] = {b[u].x, b[u].y, b[u].z, b[u].w};
            float s = 0.f;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                s = fmaf(bf16_lo(aw[e]) + bf16_lo(rw[e]), bf16_lo(bw[e]), s);
                s = fmaf(bf16_hi(aw[e]) + bf16_hi(rw[e]), bf16_hi(bw[e]), s);
            }
#pragma unroll
            for (int d = 1; d < LANES; d *= 2) s += __shfl_xor_sync(0xffffffffu, s, d);
            if (live[u] && c == 0) p.xq[ro[u]] = make_uint4(ONES, split_bf16(-lse[u] * p.inv_scale), split_bf16(-s), 0u);
        }
    }
    // padding of the per-row tiles, and the per-column tiles
    const int pad = NTP - N;
    const size_t npad = static_cast<size_t>(p.BS) * H * pad;
    for (size_t idx = t0; idx < npad; idx += gstride) {
        const size_t bh = idx / pad;
        const int n = N + static_cast<int>(idx % pad);
        p.xq[bh * NTP + n] = make_uint4(ONES, split_bf16(-1e30f), 0u, 0u);
    }
    const size_t nmask = static_cast<size_t>(p.BS) * NTP;
    for (size_t idx = t0; idx < nmask; idx += gstride) {
        const size_t bs = idx / NTP;
        const int n = static_cast<int>(idx % NTP);
        const float m = (n < N) ? __bfloat162float(p.mask[bs * N + n]) * p.inv_scale : -1e30f;
        p.xk[idx] = make_uint4(split_bf16(m), ONES, 0u, 0u);
    }
#pragma unroll
    for (int z = 0; z < 2; ++z)
        for (size_t i = t0; i < p.n_zero[z]; i += gstride) p.zero[z][i] = make_uint4(0u, 0u, 0u, 0u);
}

// The results that were accumulated in fp32, in their final type: dQ of the pairs from pair0 on, which lie
// in rows row0 and up ([row][N][H][DH]) -> bf16 in the activation layout; and dBias -> bf16 if the caller wants it so.
// Eight elements per thread.
struct FinishParams {
    const float* dq_acc;
    __nv_bfloat16* dq;
    size_t n8;                 // groups of eight of dq_acc
    int pair0, row0;
    int N, H, Dt;
    ActLayout lay;
    const float* dbias_acc;    // nullptr: dBias is final already
    __nv_bfloat16* dbias;
    size_t nb8;
};
__device__ __forceinline__ uint4 cvt8(const float* src) {
    const float4 a = __ldcs(reinterpret_cast<const float4*>(src)), b = __ldcs(reinterpret_cast<const float4*>(src) + 1);
    return make_uint4(pack_bf16(a.x, a.y), pack_bf16(a.z, a.w), pack_bf16(b.x, b.y), pack_bf16(b.z, b.w));
}
template <int DH>
__global__ void __launch_bounds__(256) bwd_finish_kernel(const FinishParams p) {
    const size_t gstride = static_cast<size_t>(gridDim.x) * blockDim.x;
    const size_t t0 = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    for (size_t i = t0; i < p.n8; i += gstride) {
        const size_t rowi = i / (DH / 8);                 // (row, n, h) of this group of eight
        const int d8 = static_cast<int>(i % (DH / 8));
        size_t bs, n, h;
        if (p.n8 < 0x80000000ull) {
            const uint32_t r32 = static_cast<uint32_t>(rowi), b32 = r32 / p.H, s32 = b32 / p.N;
            h = r32 - b32 * p.H;
            n = b32 - s32 * p.N;
            bs = s32;
        } else {
            const size_t bn = rowi / p.H;
            h = rowi - bn * p.H;
            bs = bn / p.N;
            n = bn - bs * p.N;
        }
        bs += p.row0;
        if (d8 * 8 >= p.Dt || bs * p.H + h < static_cast<size_t>(p.pair0)) continue;
        const uint4 u = cvt8(p.dq_acc + 8 * i);
        *reinterpret_cast<uint4*>(p.dq + bs * p.lay.row + n * p.lay.n + h * p.lay.h + d8 * 8) = u;
    }
    if (p.dbias_acc)
        for (size_t i = t0; i < p.nb8; i += gstride) reinterpret_cast<uint4*>(p.dbias)[i] = cvt8(p.dbias_acc + 8 * i);
}

struct BwdWorkspace {
    size_t off_xq, off_xk, off_do, off_db, off_dq, least, total;
};

// The fp32 dQ area, kernel width, comes last: the accumulator of B * S * H pairs takes N rows of each (`least`), the
// scratch of as many CTAs that take pairs whole N rounded up to 32 (`total`, what the entry points ask for).
static BwdWorkspace bwd_workspace(const EvoDims* d, bool gated = false, bool dbias_bf16 = false) {
    const size_t BS = static_cast<size_t>(d->B) * d->S;
    const size_t NTP = static_cast<size_t>((d->N + TILE - 1) / TILE) * TILE;
    auto up = [](size_t x) { return (x + 255) & ~static_cast<size_t>(255); };
    BwdWorkspace w;
    w.off_xq = 0;
    w.off_xk = up(w.off_xq + BS * d->H * NTP * 16);
    w.off_do = up(w.off_xk + BS * NTP * 16);
    w.off_db = gated ? up(w.off_do + BS * d->N * d->H * d->D * 2) : w.off_do;    // bf16 d_out * sigmoid(gate)
    // fp32 dBias of a caller that wants bf16 (one S row needs none: dBias is not a sum)
    w.off_dq = (dbias_bf16 && d->S > 1) ? up(w.off_db + static_cast<size_t>(d->B) * d->H * d->N * d->N * 4) : w.off_db;
    const size_t dh = d->D <= 32 ? 32 : (d->D <= 64 ? 64 : 128);
    w.least = up(w.off_dq + BS * d->H * d->N * dh * 4);
    w.total = up(w.off_dq + BS * d->H * ((d->N + 31) / 32 * 32) * dh * 4);
    return w;
}

template <int DH>
// lay_in: q, k, v; lay_out: o, o_resid, d_o, gate, d_gate; lay_grad: dq, dk, dv
static int launch_bwd(const EvoDims* d, const ActLayout& lay_in, const ActLayout& lay_out, const ActLayout& lay_grad,
                      const void* q, const void* k, const void* v, const void* bias,
                      const void* mask, const void* o, const void* o_resid, const float* lse, const void* d_o_in,
                      void* dq, void* dk, void* dv, void* dbias_out, bool dbias_bf16, uint8_t* ws, size_t ws_bytes, float scale,
                      unsigned phases, int reserved_sms, cudaStream_t st, const void* gate, void* d_gate) {
    const int BS = d->B * d->S;
    const int NT = (d->N + TILE - 1) / TILE;
    const BwdWorkspace w = bwd_workspace(d, gate != nullptr, dbias_bf16);
    // with a gate the kernels read the gradient entering the attention from the workspace (contiguous)
    const void* d_o = gate ? static_cast<const void*>(ws + w.off_do) : d_o_in;
    const ActLayout lay_do = gate ? contiguous_layout(d->N, d->H, d->D) : lay_out;
    uint4* xq = reinterpret_cast<uint4*>(ws + w.off_xq);
    uint4* xk = reinterpret_cast<uint4*>(ws + w.off_xk);
    float* dq_ws = reinterpret_cast<float*>(ws + w.off_dq);

    CUtensorMap tq, tk, tv, tdo, tb, tdq, tdk, tdv, tacc;
    int rc;
    const int Dt = d->D;          // 16 on the D = 32 kernel: boxes of 32 columns over tensors of 16
    if ((rc = make_tmap_qkv(&tq, q, BS, d->N, d->H, Dt, TILE, lay_in, RowTile<DH>::BOX_D))) return rc;
    if ((rc = make_tmap_qkv(&tk, k, BS, d->N, d->H, Dt, TILE, lay_in, RowTile<DH>::BOX_D))) return rc;
    if ((rc = make_tmap_qkv(&tv, v, BS, d->N, d->H, Dt, TILE, lay_in, RowTile<DH>::BOX_D))) return rc;
    if ((rc = make_tmap_qkv(&tdo, d_o, BS, d->N, d->H, Dt, TILE, lay_do, RowTile<DH>::BOX_D))) return rc;
    if ((rc = make_tmap_bias(&tb, bias, d->B, d->H, d->N, DH == 32 ? TILE / 2 : TILE))) return rc;

    BwdParams p{};
    p.B = d->B; p.S = d->S; p.N = d->N; p.H = d->H;
    p.NT = NT;
    p.NTP = NT * TILE;
    p.scale = (scale > 0.f) ? scale : 1.0f / sqrtf(static_cast<float>(Dt));
    p.Dt = Dt;
    p.KB = (Dt + 15) / 16;
    p.c1 = p.scale * LOG2E;
    p.xq = reinterpret_cast<const __nv_bfloat16*>(xq);
    p.xk = reinterpret_cast<const __nv_bfloat16*>(xk);
    p.bias = static_cast<const __nv_bfloat16*>(bias);
    p.dq = static_cast<__nv_bfloat16*>(dq);
    p.dk = static_cast<__nv_bfloat16*>(dk); p.dv = static_cast<__nv_bfloat16*>(dv);
    p.lay = lay_grad;          // D = 128: thread-level stores (D <= 64 stores through tensor maps)
    p.status = status_word();
    if (!p.status) return EVO_ERR_CUDA;

    int sms = 0;
    if ((rc = sm_count(&sms))) return rc;
    // SMs left to other work (a collective on another stream) while the dQ/dK/dV kernel runs
    int use_sms = sms - (reserved_sms > 0 ? reserved_sms : 0);
    if (use_sms < 1) use_sms = 1;
    // D <= 64: pairs (S row, head) are taken whole as far as they fill whole rounds of the SMs, and so are those left
    // over if single segments of them would not end a round sooner.  (Rounds are the same as with segments alone,
    // the accumulator and its passes are those of less than one round of pairs.)
    // D = 128: all or none, whole where that costs no more time than segments: the rounds of the fullest SM, against
    // those of segments plus the two passes over the accumulator (about 1 / (2 NT) of the kernel).  Most of the pairs
    // whole is no gain there: 148 pairs' operands and partial sums at a time outgrow the L2, and the kernel has one
    // load stage (B=1, S=40, N=768, H=4: 193 -> 214 us, passes 42 -> 25).
    const int pairs = BS * d->H;
    const size_t n32 = static_cast<size_t>((d->N + 31) / 32) * 32;
    // rows of the dQ area; a caller with less than the entry points ask for gets fewer whole pairs
    const size_t room = static_cast<size_t>(pairs) * (ws_bytes >= w.total ? n32 : static_cast<size_t>(d->N));
    const long t_seg = (static_cast<long>(pairs) * NT + use_sms - 1) / use_sms;
    if constexpr (DH == 128) {
        const long t_whole = static_cast<long>((pairs + use_sms - 1) / use_sms) * NT;
        p.n_whole = (NT == 1 || t_whole * 2 * NT <= t_seg * (2 * NT + 1)) ? pairs : 0;
    } else {
        const int left = pairs % use_sms, full = pairs - left;
        p.n_whole = (left && t_seg < static_cast<long>(full / use_sms + 1) * NT) ? full : pairs;
        // the workspace holds the partial sums of every CTA and the accumulator from the row on that pair `full` is in
        const size_t acc_n = static_cast<size_t>(pairs - full / d->H * d->H) * d->N;
        if (p.n_whole < pairs && static_cast<size_t>(full ? use_sms : 0) * n32 + acc_n > room) p.n_whole = 0;
    }
    // all whole: partial sums of every CTA, unless they stay in tensor memory (one tile; two at D = 64, four at D <= 32)
    constexpr int TILES_HELD = DH == 128 ? 1 : (DH == 64 ? BwdCfg::DQ_BUFS : BwdHalvesCfg::DQ_BUFS);
    if (p.n_whole == pairs && NT > TILES_HELD && std::min(pairs, use_sms) * n32 > room) p.n_whole = 0;
    p.pairs = pairs;
    p.acc_row0 = p.n_whole / d->H;
    const int rest_rows = p.n_whole < pairs ? BS - p.acc_row0 : 0;
    const int grid = static_cast<int>(std::min<long>(p.n_whole ? pairs : static_cast<long>(pairs) * NT, use_sms));
    // workspace: the partial sums of every CTA with whole pairs, then the accumulator of the rest
    p.scratch_stride = n32 * DH / 4;
    p.seg_dj = grid % NT;
    p.seg_dp = grid / NT;
    p.dq_scratch = dq_ws;
    p.dq_acc = dq_ws + (p.n_whole ? grid : 0) * p.scratch_stride * 4;
    if constexpr (DH <= 64) {
        // what the drain warps write: boxes of 32 rows x 32 columns
        if ((rc = make_tmap_qkv(&tdq, dq, BS, d->N, d->H, Dt, 32, lay_grad, 32)) ||
            (rc = make_tmap_qkv(&tdk, dk, BS, d->N, d->H, Dt, 32, lay_grad, 32)) ||
            (rc = make_tmap_qkv(&tdv, dv, BS, d->N, d->H, Dt, 32, lay_grad, 32)) ||
            (rc = rest_rows ? make_tmap_rows_box(&tacc, p.dq_acc, 4, rest_rows, d->N, d->H, DH, 32, 32) : 0))
            return rc;
        if (!rest_rows) tacc = tdq;
    }

    const size_t acc_bytes = static_cast<size_t>(rest_rows) * d->N * d->H * DH * 4;
    const size_t db_elems = static_cast<size_t>(d->B) * d->H * d->N * d->N;

    // one S row and the whole backward in this call: the dQ/dK/dV kernel writes dBias (= dS) itself
    const bool both = (phases & EVO_BWD_PHASE_DBIAS) && (phases & EVO_BWD_PHASE_DQKV);
    const bool dbias_here = (d->S == 1) && both;
    p.dbias = dbias_out;
    // otherwise the dBias kernel does: in one piece, or as an fp32 sum of slices of S
    const int slices = dbias_slices(d, sms);
    float* dbias_acc = (dbias_bf16 && !dbias_here) ? reinterpret_cast<float*>(ws + w.off_db) : static_cast<float*>(dbias_out);
    const bool convert_dbias = dbias_bf16 && !dbias_here && slices > 1;
    if (phases & EVO_BWD_PHASE_DBIAS) {
        PrepParams r;
        r.o = static_cast<const __nv_bfloat16*>(o);
        r.o_resid = static_cast<const __nv_bfloat16*>(o_resid);
        r.d_o = static_cast<const __nv_bfloat16*>(d_o_in);
        r.mask = static_cast<const __nv_bfloat16*>(mask);
        r.gate = static_cast<const __nv_bfloat16*>(gate);
        r.lse = lse;
        r.xq = xq;
        r.xk = xk;
        r.do_att = reinterpret_cast<__nv_bfloat16*>(ws + w.off_do);
        r.d_gate = static_cast<__nv_bfloat16*>(d_gate);
        r.zero[0] = reinterpret_cast<uint4*>(dbias_acc);
        r.n_zero[0] = (!dbias_here && slices > 1) ? db_elems / 4 : 0;
        r.zero[1] = reinterpret_cast<uint4*>(p.dq_acc);
        r.n_zero[1] = both ? acc_bytes / 16 : 0;      // a separate second phase zeroes its own accumulator
        r.inv_scale = 1.0f / p.scale;
        r.BS = BS; r.N = d->N; r.H = d->H; r.NTP = p.NTP; r.Dt = Dt;
        r.lay = lay_out;
        constexpr int LANES = DH / 8;
        auto prep = [&](auto lanes_c, auto gated_c) -> int {
            constexpr int L = decltype(lanes_c)::value;
            constexpr bool G = decltype(gated_c)::value;
            constexpr int U = G ? 2 : 4;
            // one row per thread where a single pass takes all of them (B=1, S=32, N=64, H=4, D=32: 4 us less)
            if (static_cast<size_t>(BS) * d->N * d->H * L <= static_cast<size_t>(sms) * prep_blocks<1>() * 256)
                bwd_prep_kernel<L, G, 1><<<sms * prep_blocks<1>(), 256, 0, st>>>(r);
            else
                bwd_prep_kernel<L, G, U><<<sms * prep_blocks<U>(), 256, 0, st>>>(r);
            return cuda_err(cudaGetLastError());
        };
        auto prep_lanes = [&](auto lanes_c) -> int { return gate ? prep(lanes_c, std::true_type{}) : prep(lanes_c, std::false_type{}); };
        if ((rc = Dt <= 16 ? prep_lanes(std::integral_constant<int, 2>{}) : prep_lanes(std::integral_constant<int, LANES>{}))) return rc;
        if (!dbias_here && (rc = launch_dbias(d, tq, tk, tv, tdo, bias, xq, xk, dbias_acc,
                                              (dbias_bf16 && !convert_dbias) ? dbias_out : nullptr, slices, p.scale, sms, st)))
            return rc;
    }
    if (!(phases & EVO_BWD_PHASE_DQKV)) return EVO_OK;

    if (!both && rest_rows && (rc = cuda_err(cudaMemsetAsync(p.dq_acc, 0, acc_bytes, st)))) return rc;
    const int mode = !dbias_here ? DBIAS_NO : (dbias_bf16 ? DBIAS_BF16 : DBIAS_F32);
    auto run = [&](auto kernel, int threads, uint32_t smem, auto... maps) -> int {
        const int e = set_max_smem_once(reinterpret_cast<const void*>(kernel), static_cast<int>(smem));
        if (e) return e;
        prof_begin(1, st);
        kernel<<<grid, threads, smem, st>>>(maps..., p);
        prof_end(1, st);
        return cuda_err(cudaGetLastError());
    };
    auto launch = [&](auto walk_c) -> int {
        constexpr int W = decltype(walk_c)::value;
        if constexpr (DH == 128) {
            using C = BwdWideCfg<DH>;
            auto kernel = mode == DBIAS_NO ? evo_bwd_wide_kernel<DH, W, DBIAS_NO>
                                           : (mode == DBIAS_BF16 ? evo_bwd_wide_kernel<DH, W, DBIAS_BF16> : evo_bwd_wide_kernel<DH, W, DBIAS_F32>);
            return run(kernel, C::THREADS, C::SMEM_BYTES, tq, tk, tv, tdo, tb);
        } else if constexpr (DH == 32) {
            using C = BwdHalvesCfg;
            auto kernel = mode == DBIAS_NO ? evo_bwd_halves_kernel<W, DBIAS_NO>
                                           : (mode == DBIAS_BF16 ? evo_bwd_halves_kernel<W, DBIAS_BF16> : evo_bwd_halves_kernel<W, DBIAS_F32>);
            return run(kernel, C::THREADS, C::SMEM_BYTES, tq, tk, tv, tdo, tb, tdq, tdk, tdv, tacc);
        } else {
            using C = BwdCfg;
            auto kernel = mode == DBIAS_NO ? evo_bwd_kernel<W, DBIAS_NO>
                                           : (mode == DBIAS_BF16 ? evo_bwd_kernel<W, DBIAS_BF16> : evo_bwd_kernel<W, DBIAS_F32>);
            return run(kernel, C::THREADS, C::SMEM_BYTES, tq, tk, tv, tdo, tb, tdq, tdk, tdv, tacc);
        }
    };
    if (p.n_whole == pairs) rc = launch(std::integral_constant<int, WALK_WHOLE>{});
    else if (p.n_whole == 0) rc = launch(std::integral_constant<int, WALK_SEGMENTS>{});
    else if constexpr (DH != 128) rc = launch(std::integral_constant<int, WALK_BOTH>{});
    if (rc || (!rest_rows && !convert_dbias)) return rc;

    FinishParams f;
    f.dq_acc = p.dq_acc;
    f.dq = static_cast<__nv_bfloat16*>(dq);
    f.n8 = acc_bytes / 32;
    f.pair0 = p.n_whole;
    f.row0 = p.acc_row0;
    f.N = d->N; f.H = d->H; f.Dt = Dt;
    f.lay = lay_grad;
    f.dbias_acc = convert_dbias ? dbias_acc : nullptr;
    f.dbias = static_cast<__nv_bfloat16*>(dbias_out);
    f.nb8 = db_elems / 8;
    bwd_finish_kernel<DH><<<sms * 8, 256, 0, st>>>(f);
    return cuda_err(cudaGetLastError());
}

}  // namespace evo

// ---------------------------------------------------------------------------
// Backward with built-in scratch.  The workspace lives in a file-scope device
// array, so the call allocates nothing.  In host code the array's name is only a
// handle; its device address comes from cudaGetSymbolAddress, looked up once per
// device (with that device current) and kept.
// ---------------------------------------------------------------------------
#ifndef EVO_STATIC_SCRATCH_BYTES
#define EVO_STATIC_SCRATCH_BYTES (32u << 20)
#endif
static __device__ __align__(256) unsigned char g_bwd_scratch[EVO_STATIC_SCRATCH_BYTES];

namespace evo {
static int static_scratch(uint8_t** out) {
    static std::mutex mu;
    static uint8_t* cache[64] = {nullptr};
    int dev = 0;
    int rc = cuda_err(cudaGetDevice(&dev));
    if (rc) return rc;
    if (dev < 0 || dev >= 64) return EVO_ERR_CUDA;
    std::lock_guard<std::mutex> lock(mu);
    if (!cache[dev]) {
        void* ptr = nullptr;
        rc = cuda_err(cudaGetSymbolAddress(&ptr, g_bwd_scratch));
        if (rc) return rc;
        cache[dev] = static_cast<uint8_t*>(ptr);
    }
    *out = cache[dev];
    return EVO_OK;
}
}  // namespace evo

extern "C" size_t evo_bwd_static_scratch_capacity(void) { return EVO_STATIC_SCRATCH_BYTES; }

extern "C" int evo_bwd_static_scratch(const EvoDims* dims, const void* q, const void* k, const void* v,
                                      const void* pair_bias, const void* res_mask, const void* o,
                                      const void* o_resid, const float* lse, const void* d_o, void* dq, void* dk,
                                      void* dv, float* dbias, float scale, void* stream) {
    int rc = evo::check_dims(dims);
    if (rc) return rc;
    if (evo::bwd_workspace(dims).least > EVO_STATIC_SCRATCH_BYTES) return EVO_ERR_TOO_LARGE;
    if ((rc = evo::ensure_context())) return rc;
    uint8_t* scratch = nullptr;
    if ((rc = evo::static_scratch(&scratch))) return rc;
    return evo_bwd(dims, q, k, v, pair_bias, res_mask, o, o_resid, lse, d_o, dq, dk, dv, dbias, scratch,
                   EVO_STATIC_SCRATCH_BYTES, scale, stream);
}

extern "C" size_t evo_bwd_workspace_bytes(const EvoDims* dims) {
    if (evo::check_dims(dims) != EVO_OK) return 0;
    return evo::bwd_workspace(dims).total;
}

extern "C" int evo_bwd(const EvoDims* dims, const void* q, const void* k, const void* v,
                       const void* pair_bias, const void* res_mask, const void* o, const void* o_resid,
                       const float* lse, const void* d_o, void* dq, void* dk, void* dv, float* dbias,
                       void* workspace, size_t workspace_bytes, float scale, void* stream) {
    return evo_bwd_phased(dims, nullptr, q, k, v, pair_bias, res_mask, o, o_resid, lse, d_o, dq, dk, dv, dbias,
                          workspace, workspace_bytes, scale, EVO_BWD_PHASE_DBIAS | EVO_BWD_PHASE_DQKV, 0, stream);
}

extern "C" int evo_bwd_strided(const EvoDims* dims, const EvoStrides* strides, const void* q, const void* k,
                               const void* v, const void* pair_bias, const void* res_mask, const void* o,
                               const void* o_resid, const float* lse, const void* d_o, void* dq, void* dk,
                               void* dv, float* dbias, void* workspace, size_t workspace_bytes, float scale,
                               void* stream) {
    return evo_bwd_phased(dims, strides, q, k, v, pair_bias, res_mask, o, o_resid, lse, d_o, dq, dk, dv, dbias,
                          workspace, workspace_bytes, scale, EVO_BWD_PHASE_DBIAS | EVO_BWD_PHASE_DQKV, 0, stream);
}

extern "C" int evo_bwd_phased(const EvoDims* dims, const EvoStrides* strides, const void* q, const void* k,
                              const void* v, const void* pair_bias, const void* res_mask, const void* o,
                              const void* o_resid, const float* lse, const void* d_o, void* dq, void* dk,
                              void* dv, float* dbias, void* workspace, size_t workspace_bytes, float scale,
                              unsigned phases, int reserved_sms, void* stream) {
    return evo_bwd_gated(dims, strides, q, k, v, pair_bias, res_mask, nullptr, o, o_resid, lse, d_o, dq, dk, dv, nullptr,
                         dbias, workspace, workspace_bytes, scale, phases, reserved_sms, stream);
}

extern "C" size_t evo_bwd_gated_workspace_bytes(const EvoDims* dims) {
    if (evo::check_dims(dims) != EVO_OK) return 0;
    return evo::bwd_workspace(dims, true).total;
}

extern "C" int evo_bwd_gated(const EvoDims* dims, const EvoStrides* strides, const void* q, const void* k,
                             const void* v, const void* pair_bias, const void* res_mask, const void* gate,
                             const void* o, const void* o_resid, const float* lse, const void* d_o, void* dq,
                             void* dk, void* dv, void* d_gate, float* dbias, void* workspace,
                             size_t workspace_bytes, float scale, unsigned phases, int reserved_sms,
                             void* stream) {
    return evo_bwd_views(dims, strides, strides, strides, q, k, v, pair_bias, res_mask, gate, o, o_resid, lse, d_o, dq,
                         dk, dv, d_gate, dbias, workspace, workspace_bytes, scale, phases, reserved_sms, stream);
}

extern "C" int evo_bwd_views(const EvoDims* dims, const EvoStrides* s_qkv, const EvoStrides* s_out,
                             const EvoStrides* s_grad, const void* q, const void* k, const void* v,
                             const void* pair_bias, const void* res_mask, const void* gate, const void* o,
                             const void* o_resid, const float* lse, const void* d_o, void* dq, void* dk, void* dv,
                             void* d_gate, float* dbias, void* workspace, size_t workspace_bytes, float scale,
                             unsigned phases, int reserved_sms, void* stream) {
    if (!dims) return EVO_ERR_NULL_PTR;
    const EvoBwdArgs a{*dims, s_qkv, s_out, s_grad, q, k, v, pair_bias, res_mask, gate, o, o_resid, lse, d_o, dq, dk, dv,
                       d_gate, dbias, 0, workspace, workspace_bytes, scale, phases, reserved_sms, stream};
    return evo_bwd_ex(&a);
}

extern "C" size_t evo_bwd_ex_workspace_bytes(const EvoDims* dims, int gated, int dbias_bf16) {
    if (evo::check_dims(dims) != EVO_OK) return 0;
    return evo::bwd_workspace(dims, gated != 0, dbias_bf16 != 0).total;
}

extern "C" int evo_bwd_ex(const EvoBwdArgs* a) {
    if (!a) return EVO_ERR_NULL_PTR;
    const EvoDims* dims = &a->dims;
    int rc = evo::check_dims(dims);
    if (rc) return rc;
    const unsigned both = EVO_BWD_PHASE_DBIAS | EVO_BWD_PHASE_DQKV;
    if (!(a->phases & both)) return EVO_ERR_BAD_DIMS;
    if (a->dbias_bf16 && (a->phases & both) != both) return EVO_ERR_BAD_DIMS;
    evo::ActLayout lay, lay_out, lay_grad;
    if ((rc = evo::layout_from_strides(dims, a->s_qkv, &lay))) return rc;
    if ((rc = evo::layout_from_strides(dims, a->s_out, &lay_out))) return rc;
    if ((rc = evo::layout_from_strides(dims, a->s_grad, &lay_grad))) return rc;
    const void* need[] = {a->q, a->k, a->v, a->pair_bias, a->res_mask, a->o, a->lse, a->d_out, a->dq, a->dk, a->dv, a->dbias, a->workspace};
    uintptr_t all = reinterpret_cast<uintptr_t>(a->o_resid) | reinterpret_cast<uintptr_t>(a->gate) | reinterpret_cast<uintptr_t>(a->d_gate);
    for (const void* ptr : need) {
        if (!ptr) return EVO_ERR_NULL_PTR;
        if (ptr != a->workspace && ptr != a->res_mask) all |= reinterpret_cast<uintptr_t>(ptr);
    }
    if ((a->gate == nullptr) != (a->d_gate == nullptr)) return EVO_ERR_NULL_PTR;
    if (all & 15u) return EVO_ERR_ALIGNMENT;
    if ((reinterpret_cast<uintptr_t>(a->workspace) & 255u) ||
        a->workspace_bytes < evo::bwd_workspace(dims, a->gate != nullptr, a->dbias_bf16 != 0).least)
        return EVO_ERR_WORKSPACE;
    if ((rc = evo::ensure_context())) return rc;
    auto launch = dims->D <= 32 ? evo::launch_bwd<32> : (dims->D <= 64 ? evo::launch_bwd<64> : evo::launch_bwd<128>);
    return launch(dims, lay, lay_out, lay_grad, a->q, a->k, a->v, a->pair_bias, a->res_mask, a->o, a->o_resid, a->lse,
                  a->d_out, a->dq, a->dk, a->dv, a->dbias, a->dbias_bf16 != 0, static_cast<uint8_t*>(a->workspace), a->workspace_bytes, a->scale,
                  a->phases, a->reserved_sms, static_cast<cudaStream_t>(a->stream), a->gate, a->d_gate);
}
