#include "kernel_runner.h"

#include <ATen/cuda/CUDAContext.h>

#include <algorithm>
#include <stdexcept>
#include <string>

#include "../common/aligned.h"
#include "fused_rank.h"
#include "tensor_map.h"

namespace cem {

namespace {

void need(bool cond, const std::string& msg) {
  if (!cond) throw std::runtime_error("KernelRunner: " + msg);
}

void need_bf16(const torch::Tensor& t, int64_t rows, int64_t cols, const char* name) {
  need(t.is_cuda() && t.scalar_type() == torch::kBFloat16 && t.dim() == 2 && t.is_contiguous() && t.size(0) == rows &&
           t.size(1) == cols,
       std::string(name) + " must be a contiguous CUDA bf16 [" + std::to_string(rows) + ", " + std::to_string(cols) +
           "] matrix");
  need(at_16_bytes(t), std::string(name) + " must be at an address of 16 bytes");
}

void need_weights(const torch::Tensor& w, int64_t L, const char* name) {
  need(w.is_cuda() && w.scalar_type() == torch::kBFloat16 && w.dim() == 3 && w.is_contiguous() && w.size(0) == L,
       std::string(name) + " must be a contiguous CUDA bf16 [L, rows, cols] tensor");
}

cudaStream_t stream() { return at::cuda::getCurrentCUDAStream().stream(); }

}  // namespace

KernelRunner::KernelRunner(int L, int S, int stripe, int num_sms)
    : L_(L), S_(S), stripe_(stripe), num_sms_(std::max(2, num_sms)) {
  need(L >= 1 && L <= 1024, "1 <= L <= 1024");
  need(S >= 8 && S % 8 == 0, "S must be a positive multiple of 8");
  need(stripe == 32 || stripe == 64 || stripe == 128, "stripe must be 32, 64 or 128");
  lay_ = make_plan_layout(1, L, S, 1);
  status_ = torch::zeros({8}, torch::TensorOptions().device(torch::kCUDA).dtype(torch::kInt32));
}

KernelRunner KernelRunner::with_groups(torch::Tensor group_rows) const {
  need(group_rows.is_cuda() && group_rows.scalar_type() == torch::kInt32 && group_rows.is_contiguous() &&
           group_rows.numel() == L_,
       "group_rows must be a contiguous CUDA int32 tensor of L elements");
  KernelRunner bound = *this;
  bound.plan_ = torch::empty({lay_.total}, group_rows.options());
  PlanKernelParams pp{};
  pp.lay = lay_;
  pp.me = 0;
  pp.plan = bound.plan_.data_ptr<int>();
  pp.counts = group_rows.data_ptr<int>();  // (read on this stream)
  pp.my_counts = group_rows.data_ptr<int>();
  pp.spin_limit = 1;
  pp.status = reinterpret_cast<StatusBlock*>(status_.data_ptr());
  launch_plan_build(pp, stream());
  return bound;
}

GemmParams KernelRunner::base() const {
  need(plan_.defined(), "no groups (with_groups)");
  GemmParams p{};
  p.plan = plan_.data_ptr<int>();
  p.lay = lay_;
  p.slice = 0;
  p.me = 0;
  p.stripe = stripe_;
  p.spin_limit = 1u << 20;
  p.mbar_limit = 20u * 1000u * 1000u;
  p.status = reinterpret_cast<StatusBlock*>(status_.data_ptr());
  return p;
}

void KernelRunner::gmm_swiglu(torch::Tensor x, torch::Tensor w_up, torch::Tensor act, c10::optional<torch::Tensor> h) {
  need_weights(w_up, L_, "w_up");
  const int64_t D = w_up.size(1), F2 = w_up.size(2);
  need(D % 64 == 0 && F2 % 256 == 0 && (F2 / 2) % stripe_ == 0, "needs D % 64 == 0, 2F % 256 == 0, F % stripe == 0");
  need_bf16(x, S_, D, "x");
  need_bf16(act, S_, F2 / 2, "act");
  if (h.has_value()) need_bf16(*h, S_, F2, "h");
  GemmParams p = base();
  p.n_tiles = static_cast<int>(F2 / kBlockN);
  p.k_blocks = static_cast<int>(D / kBlockK);
  p.b_group_rows = static_cast<int>(D);
  p.out0 = reinterpret_cast<__nv_bfloat16*>(act.data_ptr());
  p.ld0 = static_cast<int>(F2 / 2);
  p.out1 = h.has_value() ? reinterpret_cast<__nv_bfloat16*>(h->data_ptr()) : nullptr;
  p.ld1 = static_cast<int>(F2);
  p.tail[0] = p.out0;
  p.tail_cols[0] = p.ld0;
  p.tail[1] = p.out1;
  p.tail_cols[1] = p.ld1;
  const CUtensorMap w = make_bf16_map_chunked(w_up.data_ptr(), static_cast<uint64_t>(L_) * D, F2, 64, stripe_ == 128 ? 1 : 2);
  launch_row_gemm(kModeSwiglu, p, w, make_token_maps(x.data_ptr(), S_, D), num_sms_, stream());
}

void KernelRunner::gmm(torch::Tensor lhs, torch::Tensor rhs, torch::Tensor out, bool transpose_rhs) {
  need_weights(rhs, L_, "rhs");
  const int64_t K = transpose_rhs ? rhs.size(2) : rhs.size(1), N = transpose_rhs ? rhs.size(1) : rhs.size(2);
  need(K % 64 == 0 && N % 256 == 0, "needs K % 64 == 0 and N % 256 == 0");
  need_bf16(lhs, S_, K, "lhs");
  need_bf16(out, S_, N, "out");
  // Rows go back to where they came from, which is their own position in `out`.
  GemmParams p = base();
  p.n_tiles = static_cast<int>(N / kBlockN);
  p.k_blocks = static_cast<int>(K / kBlockK);
  p.ld0 = static_cast<int>(N);
  p.out0 = reinterpret_cast<__nv_bfloat16*>(out.data_ptr());
  p.tail[0] = p.out0;
  p.tail_cols[0] = p.ld0;
  const TokenMaps rows = make_token_maps(lhs.data_ptr(), S_, K);
  if (!transpose_rhs) {
    p.b_group_rows = static_cast<int>(K);
    const CUtensorMap w = make_bf16_map_chunked(rhs.data_ptr(), static_cast<uint64_t>(L_) * K, N, 64, 2);
    launch_row_gemm(kModeDownFwd, p, w, rows, num_sms_, stream());
  } else {
    p.b_group_rows = static_cast<int>(N);
    const CUtensorMap w = make_bf16_map_2d(rhs.data_ptr(), static_cast<uint64_t>(L_) * N, K, 128);
    launch_row_gemm(kModeDx, p, w, rows, num_sms_, stream());
  }
}

void KernelRunner::gmm_dswiglu(torch::Tensor dy, torch::Tensor w_down, torch::Tensor h, torch::Tensor dh) {
  need_weights(w_down, L_, "w_down");
  const int64_t F = w_down.size(1), D = w_down.size(2);
  need(D % 64 == 0 && F % 256 == 0 && F % stripe_ == 0, "needs D % 64 == 0, F % 256 == 0, F % stripe == 0");
  need_bf16(dy, S_, D, "dy");
  need_bf16(h, S_, 2 * F, "h");
  need_bf16(dh, S_, 2 * F, "dh");
  GemmParams p = base();
  p.n_tiles = static_cast<int>(F / kBlockN);
  p.k_blocks = static_cast<int>(D / kBlockK);
  p.b_group_rows = static_cast<int>(F);
  p.in0 = reinterpret_cast<const __nv_bfloat16*>(h.data_ptr());
  p.out0 = reinterpret_cast<__nv_bfloat16*>(dh.data_ptr());
  p.ld0 = static_cast<int>(2 * F);
  p.tail[0] = p.out0;
  p.tail_cols[0] = p.ld0;
  const CUtensorMap w = make_bf16_map_2d(w_down.data_ptr(), static_cast<uint64_t>(L_) * F, D, 128);
  launch_row_gemm(kModeDswiglu, p, w, make_token_maps(dy.data_ptr(), S_, D), num_sms_, stream());
}

void KernelRunner::tgmm(torch::Tensor lhs, torch::Tensor rhs, torch::Tensor out) {
  need(lhs.dim() == 2 && rhs.dim() == 2, "lhs and rhs must be matrices");
  const int64_t M = lhs.size(1), N = rhs.size(1);
  need(M % 256 == 0 && N % 256 == 0, "needs M % 256 == 0 and N % 256 == 0");
  need_bf16(lhs, S_, M, "lhs");
  need_bf16(rhs, S_, N, "rhs");
  need(out.is_cuda() && out.scalar_type() == torch::kBFloat16 && out.is_contiguous() && out.dim() == 3 &&
           out.size(0) == L_ && out.size(1) == M && out.size(2) == N,
       "out must be a contiguous CUDA bf16 [L, M, N] tensor");
  GemmParams p = base();
  p.m_tiles = static_cast<int>(M / kBlockM);
  p.n_tiles = static_cast<int>(N / kBlockN);
  p.carry_in = nullptr;   // one slice: every group begins and ends in it, the carry is never touched
  p.carry_out = nullptr;
  p.grad_out = reinterpret_cast<__nv_bfloat16*>(out.data_ptr());
  const CUtensorMap a = make_bf16_map_chunked(lhs.data_ptr(), S_, M, 64, 2);
  const CUtensorMap b = make_bf16_map_chunked(rhs.data_ptr(), S_, N, 64, 2);
  const CUtensorMap c = make_bf16_map_2d(out.data_ptr(), static_cast<uint64_t>(L_) * M, N, 32);
  launch_weight_grad(p, a, b, c, num_sms_, S_, stream());
}

void KernelRunner::check_status() {
  int32_t host[8];
  cudaStream_t st = stream();
  cudaMemcpyAsync(host, status_.data_ptr(), sizeof(host), cudaMemcpyDeviceToHost, st);
  cudaStreamSynchronize(st);
  if (host[0] != 0) {
    const std::string message = format_status(std::vector<int64_t>(host, host + 8), 0);
    cudaMemsetAsync(status_.data_ptr(), 0, sizeof(host), st);
    cudaStreamSynchronize(st);
    throw std::runtime_error(message);
  }
}

}  // namespace cem
