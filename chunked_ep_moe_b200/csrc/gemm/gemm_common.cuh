// Pieces shared by the two GEMM kernels (row-wise modes: row_gemm.cu; weight gradients: grouped_gemm_pair.cu).
#pragma once

#include "grouped_gemm.cuh"

#include "../common/umma.cuh"

namespace cem {
namespace {

// Source rank and send-order position of slice row `grow` of expert `g` (combine target).
__device__ __forceinline__ void resolve_source(const GemmParams& p, int g, int grow, int* src, int* pos) {
  const int stream_row = p.slice * p.lay.S + grow;
  const int* in_start = p.plan + p.lay.off_in_start;
  const int* in_size = p.plan + p.lay.off_in_size;
  const int* sss = p.plan + p.lay.off_src_send_start;
  *src = -1;
  *pos = 0;
  for (int s = 0; s < p.lay.P; ++s) {
    const int i = s * p.lay.L + g;
    const int st = in_start[i];
    if (stream_row >= st && stream_row < st + in_size[i]) {
      *src = s;
      *pos = sss[i] + (stream_row - st);
    }
  }
}

// Dispatch consumer: waits until the rows of local expert `g` that belong to slices <= p.slice have arrived from every
// source rank (lane s watches source s), then orders the async proxy behind what was observed, because the rows were
// written through the generic proxy and TMA reads them next. Returns false on expiry (status recorded, abort set).
__device__ __forceinline__ bool wait_expert_rows(const GemmParams& p, int mode, int g, int lane, volatile int* abort_flag) {
  bool ok = true;
  if (p.ready != nullptr) {
    // fp8 wire: the expansion kernel releases an expert's rows (bf16, local) once they have arrived and been expanded.
    if (lane == 0) {
      const int through = plan_clip((p.slice + 1) * p.lay.S - p.plan[p.lay.off_expert_start + g], 0,
                                    p.plan[p.lay.off_expert_rows + g]);
      const uint32_t target = p.ready_base[g] + static_cast<uint32_t>(through);
      uint32_t seen = 0;
      ok = spin_until_reached(p.ready + g, target, p.spin_limit, &seen);
      if (!ok) {
        report_status(p.status, kStatusArrivalTimeout, kKernelGemm, mode, p.slice, 10000 + g, target, seen);
        *abort_flag = 1;
      }
    }
  } else if (lane < p.lay.P) {
    const int i = lane * p.lay.L + g;
    const int through = plan_clip((p.slice + 1) * p.lay.S - p.plan[p.lay.off_in_start + i], 0,
                                  p.plan[p.lay.off_in_size + i]);
    const uint32_t target = p.pass_base[i] + static_cast<uint32_t>(through);
    uint32_t seen = 0;
    ok = spin_until_reached(p.arrive + i, target, p.spin_limit, &seen);
    if (!ok) {
      report_status(p.status, kStatusArrivalTimeout, kKernelGemm, mode, p.slice, i, target, seen);
      *abort_flag = 1;
    }
  }
  ok = __all_sync(0xffffffffu, ok);
  if (ok) fence_proxy_async_all();
  return ok;
}

// Sigmoid from the approximate exponential and reciprocal (2 ulp). The IEEE division the plain `/` compiles to is a subroutine of a
// dozen instructions, and in the SwiGLU epilogues it was most of the work per element; the results are rounded to bf16 right after,
// which has 16 bits less precision than the error made here. The forms that flush subnormals: neither 1 + 2^-127 nor the reciprocal
// of 2^127 differs by them in a sigmoid that is rounded to bf16, and the others cost eight more instructions an element.
constexpr float kMinusLog2e = -1.4426950408889634f;
__device__ __forceinline__ float exp2_approx(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float reciprocal_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float sigmoid_f(float g) { return reciprocal_approx(1.0f + exp2_approx(g * kMinusLog2e)); }
__device__ __forceinline__ float silu_f(float g) { return g * sigmoid_f(g); }
__device__ __forceinline__ f32x2 sigmoid_f(f32x2 g) {
  float a, b;
  split_f32x2(mul2(g, make_f32x2(kMinusLog2e, kMinusLog2e)), &a, &b);
  split_f32x2(add2(make_f32x2(1.0f, 1.0f), make_f32x2(exp2_approx(a), exp2_approx(b))), &a, &b);
  return make_f32x2(reciprocal_approx(a), reciprocal_approx(b));
}


// Largest persistent grid whose clusters of two are all resident at once (sets the kernel's shared-memory limit first). A
// cluster needs both SMs of one TPC free, so this can be fewer than SM-count / 2 clusters; a cluster that does not fit
// would only start after the first wave has finished ALL of its (statically assigned) tiles and double the kernel's time.
template <typename Kernel>
int resident_pair_grid(Kernel kernel, int threads, int smem_bytes) {
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2, 1, 1);
  cfg.blockDim = dim3(static_cast<unsigned>(threads), 1, 1);
  cfg.dynamicSmemBytes = static_cast<size_t>(smem_bytes);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int clusters = 0;
  if (cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) != cudaSuccess || clusters <= 0) {
    cudaGetLastError();
    return 2;
  }
  return 2 * clusters;
}

}  // namespace
}  // namespace cem
