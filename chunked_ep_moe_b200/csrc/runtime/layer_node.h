// The MoE layer as one autograd node: `chunked_moe` on the fused path.
#pragma once

#include <torch/extension.h>

#include <memory>

#include "fused_rank.h"

namespace cem {

// x [T, D] and the weights bf16, expert_ids [T, K], router weights [T, K] of any floating type; whatever their layout. What `FusedRank`
// takes (contiguous, int32 ids, fp32 weights) is made here. Gradients of x, the router weights and both weight tensors.
torch::Tensor chunked_moe_layer(std::shared_ptr<FusedRank> rank, const torch::Tensor& x, const torch::Tensor& expert_ids,
                                const torch::Tensor& weights, const torch::Tensor& w_up, const torch::Tensor& w_down);

}  // namespace cem
