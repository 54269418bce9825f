// Launcher of the pair-bias gradient kernel (evo_dbias.cu), called by the
// backward launcher between its prep kernel and the dQ/dK/dV kernel.
#pragma once
#include "evo_host.cuh"

namespace evo {

// D = 32, whose arithmetic is little more than the exp2: every fourth pair of kv columns takes its exp2 on the
// fused-multiply-add pipe (see ex2_poly2; 0.187 -> 0.180 ms at B=1, S=512, N=384, H=8).  Whatever else forms dBias as a sum over rows
// takes the same columns' there (evo_bwd_halves.cuh), so that dBias does not depend on which kernel a call gets.
template <int DH> constexpr int DBIAS_POLY_EVERY = (DH == 32) ? 4 : 0;

// Slices of S that the launcher cuts the sum into (1: every dBias tile is one CTA's whole sum).
int dbias_slices(const EvoDims* d, int sms);

// dbias [B][H][N][N] fp32 must be zeroed on `st` before the call if there are several slices; with
// one, dbias16 (bf16, may be nullptr) is written instead if given.  tq, tk, tv, tdo: row-tile maps of
// q, k, v, d_o.  xq and xk are the extra tiles the prep kernel writes (see evo_bwd.cu): bf16
// [B*S][H][NTP][8] with the per-row terms and bf16 [B*S][NTP][8] with the per-column terms.
int launch_dbias(const EvoDims* d, const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tdo,
                 const void* bias, const void* xq, const void* xk, float* dbias, void* dbias16, int slices, float scale, int sms,
                 bool chained, cudaStream_t st);

}  // namespace evo
