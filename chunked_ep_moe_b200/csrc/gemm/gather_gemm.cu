// The up-projection of calls of few tokens, which gathers its rows itself (see row_gemm.cuh). Beside `row_gemm_kernel`, so that its
// registers are its own.
#include "row_gemm.cuh"

namespace cem {

namespace {

constexpr int kGatherThreads = kRowThreads + 32 * kGatherWarps;

__global__ void __cluster_dims__(2, 1, 1) __maxnreg__(168)
gather_swiglu_kernel(const __grid_constant__ GemmParams p, const __grid_constant__ CUtensorMap map_a) {
  row_gemm_body<kModeSwiglu, false, true>(p, map_a, nullptr);
}

}  // namespace

void launch_gather_swiglu(const GemmParams& p, const CUtensorMap& map_a, int grid, cudaStream_t stream, bool behind) {
  static const int resident = resident_pair_grid(gather_swiglu_kernel, kGatherThreads, kRowSmemBytes);
  grid &= ~1;  // whole pairs only
  const int g = grid < resident ? grid : resident;
  g_pair_grid_used = g;
  launch_maybe_behind(behind, gather_swiglu_kernel, g, kGatherThreads, kRowSmemBytes, stream, p, map_a);
}

}  // namespace cem
