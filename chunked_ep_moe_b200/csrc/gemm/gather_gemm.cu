// The up-projection of calls of few tokens, which gathers its rows itself (see row_gemm.cuh). Beside `row_gemm_kernel`, so that its
// registers are its own.
//
// Up to 32 expert ids it is also the kernel that the pass starts with: every CTA sorts the ids by itself, a lane an id (0.3 us), and
// the last one stores what the plan kernel would leave for the kernels behind it and for the host. One token of top-6 at D=1024, from the
// first kernel's start to the last one's end: 35.6 us with plan and put (five kernels), 34.5 with the rows gathered, 22.1 this way
// (three); a call on its own 70 -> 57 us.
#include "row_gemm.cuh"

namespace cem {

namespace {

constexpr int kGatherThreads = kRowThreads + 32 * kGatherWarps;

__global__ void __cluster_dims__(2, 1, 1) __maxnreg__(168)
gather_swiglu_kernel(const __grid_constant__ GemmParams p, const __grid_constant__ CUtensorMap map_a) {
  row_gemm_body<kModeSwiglu, false, kRowsGathered>(p, map_a, nullptr);
}

constexpr int kFewSmemBytes = kRowSmemBytes + static_cast<int>(sizeof(FewRows));
static_assert(kFewSmemBytes + 1024 <= 233472, "more shared memory than an SM has");

__global__ void __cluster_dims__(2, 1, 1) __maxnreg__(168)
few_swiglu_kernel(const __grid_constant__ GemmParams p, const __grid_constant__ CUtensorMap map_a, const __grid_constant__ FewPlan plan) {
  row_gemm_body<kModeSwiglu, false, kRowsFew>(p, map_a, nullptr, &plan);
}

}  // namespace

void launch_gather_swiglu(const GemmParams& p, const CUtensorMap& map_a, int grid, cudaStream_t stream, bool behind) {
  static const int resident = resident_pair_grid(gather_swiglu_kernel, kGatherThreads, kRowSmemBytes);
  grid &= ~1;  // whole pairs only
  const int g = grid < resident ? grid : resident;
  g_pair_grid_used = g;
  launch_maybe_behind(behind, gather_swiglu_kernel, g, kGatherThreads, kRowSmemBytes, stream, p, map_a);
}

void launch_few_swiglu(const GemmParams& p, const CUtensorMap& map_a, const FewPlan& plan, int grid, cudaStream_t stream, bool behind) {
  static const int resident = resident_pair_grid(few_swiglu_kernel, kGatherThreads, kFewSmemBytes);
  grid &= ~1;  // whole pairs only
  const int g = grid < resident ? grid : resident;
  g_pair_grid_used = g;
  launch_maybe_behind(behind, few_swiglu_kernel, g, kGatherThreads, kFewSmemBytes, stream, p, map_a, plan);
}

}  // namespace cem
