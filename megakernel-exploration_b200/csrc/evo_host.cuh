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
// A kernel has been launched (counted while profiling is enabled).
void prof_count();

// Launches a kernel that calls chain_wait ahead of its first access to global memory (evo_ptx.cuh).  chained: as a programmatic launch, whose
// blocks may be placed as soon as those of the kernel before it on the stream, whichever that is, have all ended, without the rest of a
// launch's latency.  No kernel releases the next one ahead of its end (griddepcontrol.launch_dependents): blocks that wait take every SM that
// becomes free, ahead of another stream's of the same priority, and steps are no shorter for it.
// Steps queued back to back, not chained / released at the start of each kernel / chained as it is: B=1, S=512, N=384, H=8, D=32
// 857 / 853 / 847 us; S=32, N=64, H=4 33.9 / 28.1 / 26.1; D=64: S=200, N=200, H=4 156 / 151 / 149, B=4, S=1, N=512, H=16 63.0 / 55.6 / 55.2; D=128:
// S=128, N=768, H=4 1092 / 1095 / 1084 (released when a block has asked for its last loads: 847, 26.2, 149, 55.5, 1091).  A 4 MB elementwise
// kernel of a second stream beside them: 35 / 148 / 35 us beside the first, 33 / 116 / 34 at D=64, S=128, N=1024, H=4, 26 / 65 / 26 at D=128, S=64,
// N=768; beside short kernels, of whose gaps it lived, 11 / 22 / 13 (D=32, S=200, N=200, a step 118 / 111 / 111) and 15 / 34 / 19 (D=64, B=4, S=1,
// N=1024, 162 / 156 / 157).
// Not chained: the two phases of a backward with a collective beside it.  The prep kernel read a step's tensors slower when its predecessor released it
// early (its blocks, then three or five to an SM, went to the SMs as these became free: the first step 862 -> 885 us); behind a predecessor that has ended it
// is chained like the others (not chained / chained: the first step 845.5 / 842.3 us, S=200, N=200, H=4, D=32 106.1 / 103.4, S=384, N=384 349.9 / 347.6).
// Not so beside copies between host and device (EVO_BWD_BESIDE_COPIES), which take longer with it, for a reason that is not known: steps of
// HostStreamedEvoAttention, three engines in turn, not chained / chained: S=128, N=384, H=8, D=32 2958-2975 / 2987-3050 us (with half of its blocks 3000-3017),
// S=64, N=384, H=4, D=128 2897-2908 / 2923-2967, S=300, N=200, H=4, D=64 3437-3446 / 3423-3426, S=48, N=256, H=4 551-555 / 551-556, S=16, N=128, H=4
// 157 / 157.  With no kernel chained 2977, 2925, 3507, 545 and 159.
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
    const int rc = cuda_err(cudaLaunchKernelEx(&cfg, kernel, args...));
    if (rc == EVO_OK) prof_count();
    return rc;
}

}  // namespace evo
