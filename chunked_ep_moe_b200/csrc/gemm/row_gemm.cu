// Row-wise GEMMs on rows in expert order (see row_gemm.cuh).
#include "row_gemm.cuh"

namespace cem {

namespace {

// 152 registers per thread: 320 threads x 152 leave room in the register file for a 256-thread, 64-register copy CTA (the
// dispatch put, the fp8 expansion), which has to become resident BESIDE this kernel for the overlap to happen.
template <int MODE, bool RANGED>
__global__ void __cluster_dims__(2, 1, 1) __maxnreg__(152)
row_gemm_kernel(const __grid_constant__ GemmParams p, const __grid_constant__ CUtensorMap map_a,
                const __grid_constant__ TokenMaps maps_b) {
  row_gemm_body<MODE, RANGED, kRowsMapped>(p, map_a, &maps_b);
}

}  // namespace

int row_gemm_smem_bytes() { return kRowSmemBytes; }

void launch_row_gemm(int mode, const GemmParams& params, const CUtensorMap& map_a, const TokenMaps& maps_b, int grid,
                     cudaStream_t stream, bool behind) {
  grid &= ~1;  // whole pairs only
  GemmParams p = params;
  if (p.last_expert == 0 && p.n_tiles * p.k_blocks >= kByExpert) p.last_expert = p.lay.L;  // all experts, their tiles by expert
#define CEM_LAUNCH_ROW(M, RANGED)                                                                                        \
  {                                                                                                                      \
    static const int resident = resident_pair_grid(row_gemm_kernel<M, RANGED>, kRowThreads, kRowSmemBytes);              \
    const int g = grid < resident ? grid : resident;                                                                     \
    g_pair_grid_used = g;                                                                                                \
    launch_maybe_behind(behind, row_gemm_kernel<M, RANGED>, g, kRowThreads, kRowSmemBytes, stream, p, map_a, maps_b);    \
  }
#define CEM_LAUNCH_ROW_MODE(M)                   \
  case M:                                        \
    if (p.last_expert > 0) CEM_LAUNCH_ROW(M, true)  \
    else CEM_LAUNCH_ROW(M, false)                \
    break;
  switch (mode) {
    CEM_LAUNCH_ROW_MODE(kModeSwiglu)
    CEM_LAUNCH_ROW_MODE(kModeDownFwd)
    CEM_LAUNCH_ROW_MODE(kModeDswiglu)
    CEM_LAUNCH_ROW_MODE(kModeDx)
    default:
      break;
  }
#undef CEM_LAUNCH_ROW_MODE
#undef CEM_LAUNCH_ROW
}

}  // namespace cem
