// Host-side helpers shared by the launchers: error codes, the driver entry
// point for tensor-map encoding (resolved at run time so the library has no
// link-time dependency on libcuda), and tensor-map builders for the layouts
// this library reads and writes.
#pragma once
#include <cstddef>
#include <cstdint>
#include <cuda.h>
#include <cuda_runtime.h>

#include "../../include/evoattn.h"

namespace evo {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// Returns nullptr when no CUDA driver is present.
EncodeTiledFn encode_tiled_fn();

struct TmapDim {
    uint64_t extent;       // elements
    uint64_t stride_bytes; // ignored for dim 0 (contiguous)
    uint32_t box;          // elements
};

// rank <= 5; dims[0] is the contiguous one.  Returns EVO_OK or an error code.
int make_tmap(CUtensorMap* out, const void* base, CUtensorMapDataType dt, int rank,
              const TmapDim* dims, CUtensorMapSwizzle swz);

inline CUtensorMapSwizzle row_swizzle(int D) {
    return D == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B;
}

// Element strides of an activation tensor over (flattened B*S row, residue, head); D is contiguous.
struct ActLayout {
    long long row, n, h;
};
inline ActLayout contiguous_layout(int N, int H, int D) {
    return ActLayout{static_cast<long long>(N) * H * D, static_cast<long long>(H) * D, static_cast<long long>(D)};
}
// Checks EvoStrides against the rules of the header and flattens (B, S); NULL = contiguous.
int layout_from_strides(const EvoDims* d, const EvoStrides* s, ActLayout* out);

// bf16 activation tensor viewed as (D, H, N, BS) with the strides of `lay`; box = one
// head's [rows x box_d] tile (box_d = 0: D), swizzled by box row.  A box wider than D (D = 16
// read by the D = 32 kernels) is zero-filled past D on loads and clipped on stores.
int make_tmap_qkv(CUtensorMap* out, const void* base, int BS, int N, int H, int D, int rows,
                  const ActLayout& lay, int box_d = 0);
// [BS][N][H][D] of `elem_bytes`-wide elements (2: bf16, 4: fp32) with a box of
// [rows x box_cols]; the swizzle matches the box row (32, 64 or 128 bytes).
int make_tmap_rows_box(CUtensorMap* out, const void* base, int elem_bytes, int BS, int N, int H, int D,
                       int box_cols, int rows);
// bf16 [B][H][N][N] viewed as (N, N, H, B); box [rows x 64 cols], 128B swizzle.
int make_tmap_bias(CUtensorMap* out, const void* base, int B, int H, int N, int rows = 128);

int check_dims(const EvoDims* d);
// Makes the device's primary context current on this thread (see evo_host.cu).
int ensure_context();
// Device address of this device's status word (nullptr on failure).
unsigned int* status_word();
int cuda_err(cudaError_t e);
// SM count of the current device (read once per device).
int sm_count(int* out);
// cudaFuncSetAttribute(MaxDynamicSharedMemorySize) once per (device, kernel, size).
int set_max_smem_once(const void* func, int bytes);

// Event pairs around the main kernels when profiling is enabled (no-ops otherwise).
void prof_begin(int kernel, cudaStream_t st);
void prof_end(int kernel, cudaStream_t st);

// Launches a kernel that calls chain_wait ahead of its first access to global memory (evo_ptx.cuh).  chained: its blocks may be placed,
// and wait there, wherever there is room, as soon as all of the kernel before it on the stream have called chain_release or ended.
// The forward, dBias and dQ/dK/dV kernels release (dQ/dK/dV not where SMs are kept free for other work); behind any other kernel that does
// not, the prep and finish kernels and those of other libraries included, only the launch itself is early.
// Not chained: the two phases of a backward with a collective beside it, whose SMs blocks that wait would take.  Nor the prep kernel: its
// blocks, three or five to an SM, then go to the SMs in the order in which these become free, and read a step's tensors slower: B=1,
// S=512, N=384, H=8, D=32 a step 862 -> 885 us.
// Steps queued back to back, not chained / released at the start of each kernel / when its last loads are asked for: that step
// 857 / 855 / 848 us, D=64 S=200, N=200, H=4 156.4 / 150.4 / 148.5, B=4, S=1, N=512, H=16 63.9 / 58.1 / 57.9, D=32 S=32, N=64, H=4 35.1 / 28.7 /
// 26.8, D=128 S=128, N=768, H=4 1091.1 / 1094.2 / 1090.7.  A 4 MB elementwise kernel of a second stream beside them: 35 / 148 / 35 us beside
// the first step, 33 / 116 / 34 at D=64, S=128, N=1024, H=4, 26 / 65 / 26 at D=128, S=64, N=768; beside short kernels, whose ends are much of them, it
// keeps some of the difference (D=32 S=200, N=200 11 / 22 / 14, D=64 B=4, S=1, N=1024 15 / 34 / 19: steps that are 6 and 5 us shorter).
template <typename... P, typename... A>
int launch_chained(bool chained, void (*kernel)(P...), int grid, int threads, size_t smem, cudaStream_t st, const A&... args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(static_cast<unsigned>(grid));
    cfg.blockDim = dim3(static_cast<unsigned>(threads));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = chained ? 1 : 0;
    return cuda_err(cudaLaunchKernelEx(&cfg, kernel, args...));
}

}  // namespace evo
