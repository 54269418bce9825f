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
//                         sum over the S rows in registers, no reduction traffic.  Not with one
//                         S row or a small problem: kernel 3 then writes dBias (DbiasHere)
//   3. evo_bwd_halves_kernel, evo_bwd_wide_kernel   dQ, dK, dV (D <= 64: evo_bwd_halves.cuh, above: evo_bwd_wide.cuh)
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
    void* dbias;               // [B][H][N][N], fp32 or bf16 (written by this kernel only: S = 1, or DBIAS_ADD)
    float* dbias_acc;          // DBIAS_ADD: the fp32 sum, zeroed before the launch
    int* dbias_done;           // DBIAS_ADD: rows added so far to each [32 x 32] part of dBias, zeroed; nullptr: the sum is the result
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
    // own_prep: there is no prep kernel ahead, the drain warps form the extra tiles of the CTA's one step (D <= 64)
    int own_prep;
    const __nv_bfloat16 *o, *o_resid, *d_o, *mask;
    const float* lse;
    ActLayout lay_out;    // of o, o_resid, d_o
};

// DBIAS_F32, DBIAS_BF16 (S = 1 only): dBias is dS itself, no sum over rows, so the compute groups store their
// dS straight to d_pair_bias and the dBias kernel (which would recompute S and dP for one step
// per item) is not launched.
// DBIAS_ADD (small problems): the compute groups add their dS to an fp32 sum in memory, whole rows at a time.  That takes a CTA
// about 1.3 us per step of a full tile (D = 32: 2, with the dBias kernel's polynomials), and saves the dBias kernel, 5 us and more with its launch and the
// second computation of S and dP.
enum DbiasHere { DBIAS_NO = 0, DBIAS_F32 = 1, DBIAS_BF16 = 2, DBIAS_ADD = 3 };

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

// ---------------------------------------------------------------------------
// What the dQ/dK/dV kernels share (D <= 64: evo_bwd_halves.cuh; D = 96, 128: evo_bwd_wide.cuh).
// One persistent CTA per SM walks segments (S row, head h, kv tile j of 128 residues); a segment walks steps (q tile i).
// Everything is formed TRANSPOSED, kv rows in the tensor-memory lanes, so that P^T (and dS^T) are in place as A operands of
// the products that contract over q, without a trip through shared memory:
//
//   S'^T = K Q^T + extra block,  dP'^T = V dO^T + extra block         (evo_tiles.cuh, "EXTRA TILE")
//   P^T = exp2(S'^T c1 + bias^T log2e),  dS^T = P^T o dP'^T           (thread = one kv row)
//   dV += P^T dO,  dK += dS^T Q
//   dQ = dS K                        A = dS from shared memory (M = q: MN-major), the one tile written there
//
// Sixteen compute warps, because with eight the loads, multiplies and exponentials of a warp hardly overlapped (2000 clocks
// for the same work).
//
// dQ is a sum over kv tiles.  A CTA takes all NT segments of a pair (S row, head) where it can, and so sees
// the whole sum.  With few tiles (four at D <= 32) it stays in tensor memory until the last segment; otherwise
// partial sums go to a scratch area of the CTA, in L2, and the last segment's go out as bf16.  Whole pairs fill whole rounds
// of the SMs; the pairs that are left over are dealt by segments, and
// their partial sums meet in an fp32 accumulator in memory (TMA reduce-add), which costs a pass to zero it and
// a pass to convert it, of those pairs only (against all pairs whole, or none, the kernel alone: S=384, N=384, H=4,
// D=32 182 -> 176 us; S=200, N=200, H=4 47 -> 44; S=1024, N=768, H=8 3333 -> 3255).
// ---------------------------------------------------------------------------

__device__ __forceinline__ uint32_t split_bf16(float v) {
    // (head, remainder) as a bf16 pair, head in the low half
    v = fminf(fmaxf(v, -1e30f), 1e30f);
    const __nv_bfloat16 hi = __float2bfloat16_rn(v);
    const __nv_bfloat16 lo = __float2bfloat16_rn(v - __bfloat162float(hi));
    return static_cast<uint32_t>(__bfloat16_as_ushort(hi)) | (static_cast<uint32_t>(__bfloat16_as_ushort(lo)) << 16);
}

}  // namespace evo
#include "evo_bwd_halves.cuh"
#include "evo_bwd_wide.cuh"
namespace evo {

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
// LANES per row: the power of two at or above Dt / 8.  All blocks are resident, six to an SM (40 registers): with one row per thread
// at a time, more threads keep more loads in flight than more rows per thread do.  Three blocks of four rows a thread (gated: two)
// / five of one / six of one, us: B=1, S=512, N=384, H=8, D=32 60.1 / 59.8 / 57.9 (50 at the rate of a copy); S=256, N=1024, H=4, D=64 80.0 / 78.8 / 77.6;
// S=128, N=768, H=4, D=128 87.5 / 88.7 / 86.6; S=384, N=384, H=4, D=32, gated 46.3 / 41.4 / 40.3 (36).
constexpr int PREP_BLOCKS = 6;      // per SM
template <int LANES, bool GATED>
__global__ void __launch_bounds__(256, PREP_BLOCKS) bwd_prep_kernel(const PrepParams p) {
    chain_wait();
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
    for (size_t r0 = (t0 - (threadIdx.x & 31)) / LANES; r0 < rows; r0 += rstride) {
        const size_t r = r0 + (threadIdx.x & 31) / LANES;
        const bool live = r < rows;
        uint4 a = make_uint4(0u, 0u, 0u, 0u), b = a, rr = a, g4 = a;
        float lse = 0.f;
        size_t off = 0, ro = 0, att = 0;
        if (live) {
            const At x = at(r);
            off = x.bs * p.lay.row + x.n * p.lay.n + x.h * p.lay.h + c * 8;
            ro = (x.bs * H + x.h) * NTP + x.n;
            if constexpr (GATED) att = ((x.bs * N + x.n) * H + x.h) * static_cast<size_t>(p.Dt) + c * 8;
            if (have) {
                a = __ldg(reinterpret_cast<const uint4*>(p.o + off));
                b = __ldg(reinterpret_cast<const uint4*>(p.d_o + off));
                if (p.o_resid) rr = __ldg(reinterpret_cast<const uint4*>(p.o_resid + off));
                if constexpr (GATED) g4 = __ldg(reinterpret_cast<const uint4*>(p.gate + off));
            }
            if (c == 0) lse = __ldg(p.lse + (x.bs * H + x.h) * N + x.n);
        }
        const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, rw[4] = {rr.x, rr.y, rr.z, rr.w};
        if constexpr (GATED) {
            const uint32_t gw[4] = {g4.x, g4.y, g4.z, g4.w}, dw[4] = {b.x, b.y, b.z, b.w};
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
            b = make_uint4(aw2[0], aw2[1], aw2[2], aw2[3]);
            if (live && have) {
                *reinterpret_cast<uint4*>(p.do_att + att) = b;
                *reinterpret_cast<uint4*>(p.d_gate + off) = make_uint4(gg[0], gg[1], gg[2], gg[3]);
            }
        }
        const uint32_t bw[4] = {b.x, b.y, b.z, b.w};
        float s = 0.f;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            s = fmaf(bf16_lo(aw[e]) + bf16_lo(rw[e]), bf16_lo(bw[e]), s);
            s = fmaf(bf16_hi(aw[e]) + bf16_hi(rw[e]), bf16_hi(bw[e]), s);
        }
#pragma unroll
        for (int d = 1; d < LANES; d *= 2) s += __shfl_xor_sync(0xffffffffu, s, d);
        if (live && c == 0) p.xq[ro] = make_uint4(ONES, split_bf16(-lse * p.inv_scale), split_bf16(-s), 0u);
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
    chain_wait();
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

// dBias is added up in memory (DBIAS_ADD) if the fullest CTA has no more steps than this.  Forward and backward queued back to
// back, dBias kernel / added up, us, bf16 dBias, by steps of the fullest CTA.  D = 32, where the dBias kernel's polynomials come on top (and the second
// computation of S and dP is cheap): 1 (S=32, N=64, H=4) 23.6 / 20.0, (S=18, N=128, H=8) 27.4 / 22.2; 2 (S=30, N=128, H=8) 28.8 / 24.9; 3 (S=32, N=128, H=12)
// 32.8 / 30.0; 4 (S=32, N=128, H=16) 39.3 / 37.6, (S=16, N=256, H=8) 35.6 / 34.1; 5 (H=20) 43.2 / 42.4, (N=64) 39.6 / 39.6; 6 (H=24) 47.2 / 48.1; 7 (H=32) 55.9 / 58.7.
// D = 64: 1 (S=32, N=64, H=4) 25.6 / 20.0; 4 (S=32, N=128, H=16) 49.0 / 41.7; 6 (H=24) 65.6 / 57.3, by segments (S=3, N=768, H=1) 42.3 / 40.8; 7 (H=32) 82.4 / 72.0;
// at 8 (S=32, N=256, H=8) the gain is down to 64.1 / 61.7, and left.
template <int DH> constexpr int DBIAS_ADD_STEPS = (DH == 32) ? 4 : 7;
// ... and if no more rows meet in a sum than this.  Where the sum lies within a few KB of something that the kernel reads (an fp32 dBias between the
// pair bias and the mask, as the allocator places small tensors), an add now and then takes 0.2 us per row of the sum: over 200 to 700
// placements, dBias kernel / added up, median and worst: S=512, N=40, H=1, D=32 41 / 34 and 149; S=518, N=64, H=2, D=64 68 / 62 and 99; S=100, N=40, H=8, D=64
// 54 / 49 and 68; S=128, N=192, H=1, D=64 39 / 34 and 45; S=60, N=200 33 / 27 and 39; S=48 31 / 26 and 34; S=32 30 / 25 and 29, N=64, H=4 24.6 / 19.6 and 19.6,
// N=40, H=8 28 / 24 and (one of 240) 32.  Sums of whole tiles hardly show it: N=128, H=8, D=64 S=64 48.1 / 42.0 and 42.2, S=100 64.5 / 58.2 and 58.6, S=128 80.3 / 71.6
// and 72.2, H=4 48.1 / 41.8 and 42.5, D=32 38.6 / 37.4 and 37.6; N=256, H=1 40.0 / 34.8 and 35.6; S=1036, N=128, H=1 84 / 73 and 81.
constexpr int dbias_add_rows(int N) { return N % TILE == 0 ? 128 : 32; }

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
    if ((rc = make_tmap_bias(&tb, bias, d->B, d->H, d->N, DH <= 64 ? TILE / 2 : TILE))) return rc;

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
    // all whole: partial sums of every CTA, unless they stay in tensor memory (one tile; four at D <= 32)
    constexpr int TILES_HELD = DH == 128 ? 1 : BwdHalvesCfg<DH == 128 ? 64 : DH>::DQ_BUFS;
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
    // with few steps a CTA they add it up in memory, unless the dBias kernel has the sum in registers or in two slices: then it comes out
    // the same in every call, which a sum of three or more in any order does not; and without several slices that kernel needs neither zeros nor a conversion.
    // By segments D = 32, dBias kernel / added up: S=9, N=200, H=4 28.9 / 25.2 us, S=25, N=256, H=1 27.6 / 24.3, S=20, N=384, H=2 34.0 / 31.0, S=8, N=392, H=2 34.9 / 34.8.
    // (Not where a CTA walks whole pairs and segments: that is six steps and more, and an instantiation that spills at D = 64.)
    const long steps = p.n_whole == pairs ? static_cast<long>((pairs + use_sms - 1) / use_sms) * NT * NT : t_seg * NT;
    // otherwise the dBias kernel does: in one piece, or as an fp32 sum of slices of S
    const int slices = dbias_slices(d, sms);
    const bool dbias_add = DH <= 64 && both && !dbias_here && slices > 2 && (p.n_whole == pairs || p.n_whole == 0) &&
                           steps <= DBIAS_ADD_STEPS<DH> && d->S <= dbias_add_rows(d->N);
    float* dbias_acc = (dbias_bf16 && !dbias_here) ? reinterpret_cast<float*>(ws + w.off_db) : static_cast<float*>(dbias_out);
    // An fp32 sum for a bf16 result is converted by the finish kernel, or by the warps that add the last row to each part of it.
    // That needs counters, where whole pairs need no scratch, and a fence behind every step's adds: with one step a CTA, where the
    // launch costs a caller's host 3 us and the device little (finish kernel / last adder, S=32, N=64, H=4: D=32 19.5 / 20.0 us, D=64 20.7 / 20.2; S=18, N=128, H=8
    // 21.1 / 22.2, 22.7 / 23.2); from two steps on the finish kernel is the better (S=30, N=128, H=8: D=32 24.7 / 28.1, D=64 26.8 / 29.2; S=32, H=16 38.2 / 45.1, 42.3 / 46.4).
    const size_t parts = static_cast<size_t>(d->B) * d->H * NT * NT * 16;
    const bool count = dbias_add && dbias_bf16 && steps <= 1 && p.n_whole == pairs && NT <= TILES_HELD && parts <= room * DH;
    const bool convert_dbias = dbias_bf16 && !dbias_here && (dbias_add ? !count : slices > 1);
    p.dbias_acc = dbias_acc;
    p.dbias_done = count ? reinterpret_cast<int*>(dq_ws) : nullptr;
    // One S row of one tile, at most one pair a CTA: the dQ/dK/dV kernel is all of the backward.  (Forward and backward queued back to back,
    // with the prep kernel / without: B=4, N=128, H=16, D=64 17.7 / 17.1 us, D=32 15.8 / 14.1, B=1, N=64, H=4 16.2 / 14.5, 15.1 / 12.4; and a launch of host work.  A sum over S rows needs its zeros written first,
    // and with more tiles every segment would form all of its pair's terms again.)
    p.own_prep = DH <= 64 && dbias_here && !gate && NT == 1 && pairs <= use_sms;
    if (p.own_prep) {
        p.o = static_cast<const __nv_bfloat16*>(o);
        p.o_resid = static_cast<const __nv_bfloat16*>(o_resid);
        p.d_o = static_cast<const __nv_bfloat16*>(d_o);
        p.mask = static_cast<const __nv_bfloat16*>(mask);
        p.lse = lse;
        p.lay_out = lay_out;
    }
    if ((phases & EVO_BWD_PHASE_DBIAS) && !p.own_prep) {
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
        r.n_zero[0] = (!dbias_here && (dbias_add || slices > 1)) ? db_elems / 4 : 0;
        r.zero[1] = reinterpret_cast<uint4*>(count ? dq_ws : p.dq_acc);
        r.n_zero[1] = count ? parts / 4 : both ? acc_bytes / 16 : 0;      // a separate second phase zeroes its own accumulator
        r.inv_scale = 1.0f / p.scale;
        r.BS = BS; r.N = d->N; r.H = d->H; r.NTP = p.NTP; r.Dt = Dt;
        r.lay = lay_out;
        constexpr int LANES = DH / 8;
        auto prep = [&](auto lanes_c, auto gated_c) -> int {
            constexpr int L = decltype(lanes_c)::value;
            constexpr bool G = decltype(gated_c)::value;
            return launch_chained(both && !(phases & EVO_BWD_BESIDE_COPIES), bwd_prep_kernel<L, G>, sms * PREP_BLOCKS, 256, 0, st, r);
        };
        auto prep_lanes = [&](auto lanes_c) -> int { return gate ? prep(lanes_c, std::true_type{}) : prep(lanes_c, std::false_type{}); };
        if ((rc = Dt <= 16 ? prep_lanes(std::integral_constant<int, 2>{}) : prep_lanes(std::integral_constant<int, LANES>{}))) return rc;
        if (!dbias_here && !dbias_add && (rc = launch_dbias(d, tq, tk, tv, tdo, bias, xq, xk, dbias_acc,
                                              (dbias_bf16 && !convert_dbias) ? dbias_out : nullptr, slices, p.scale, sms, both, st)))
            return rc;
    }
    if (!(phases & EVO_BWD_PHASE_DQKV)) return EVO_OK;

    if (!both && rest_rows && (rc = cuda_err(cudaMemsetAsync(p.dq_acc, 0, acc_bytes, st)))) return rc;
    const int mode = dbias_add ? DBIAS_ADD : !dbias_here ? DBIAS_NO : (dbias_bf16 ? DBIAS_BF16 : DBIAS_F32);
    auto run = [&](auto kernel, int threads, uint32_t smem, auto... maps) -> int {
        const int e = set_max_smem_once(reinterpret_cast<const void*>(kernel), static_cast<int>(smem));
        if (e) return e;
        prof_begin(1, st);
        const int e2 = launch_chained(both, kernel, grid, threads, smem, st, maps..., p);
        prof_end(1, st);
        return e2;
    };
    auto launch = [&](auto walk_c) -> int {
        constexpr int W = decltype(walk_c)::value;
        if constexpr (DH == 128) {
            using C = BwdWideCfg<DH>;
            auto kernel = mode == DBIAS_NO ? evo_bwd_wide_kernel<DH, W, DBIAS_NO>
                                           : (mode == DBIAS_BF16 ? evo_bwd_wide_kernel<DH, W, DBIAS_BF16> : evo_bwd_wide_kernel<DH, W, DBIAS_F32>);
            return run(kernel, C::THREADS, C::SMEM_BYTES, tq, tk, tv, tdo, tb);
        } else {
            using C = BwdHalvesCfg<DH>;
            if constexpr (W != WALK_BOTH) {
                if (mode == DBIAS_ADD) return run(evo_bwd_halves_kernel<DH, W, DBIAS_ADD>, C::THREADS, C::SMEM_BYTES, tq, tk, tv, tdo, tb, tdq, tdk, tdv, tacc);
            }
            auto kernel = mode == DBIAS_NO ? evo_bwd_halves_kernel<DH, W, DBIAS_NO>
                                           : (mode == DBIAS_BF16 ? evo_bwd_halves_kernel<DH, W, DBIAS_BF16> : evo_bwd_halves_kernel<DH, W, DBIAS_F32>);
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
    return launch_chained(both, bwd_finish_kernel<DH>, sms * 8, 256, 0, st, f);
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
