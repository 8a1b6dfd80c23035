#include "layer_node.h"

#include <stdexcept>

#include "../common/aligned.h"

namespace cem {

namespace {

// Keeps the rank alive as long as a pass's backward may come.
struct Held : torch::CustomClassHolder {
  explicit Held(std::shared_ptr<FusedRank> r) : rank(std::move(r)) {}
  std::shared_ptr<FusedRank> rank;
};

// In C++ because the host is what bounds small passes: a node written in Python, its checks and conversions took 145 of 215 us a step
// of forward + backward of 192 tokens at D=F=256, and 22 of 46 us a one-token forward, during which the device idles: the forward ends
// with the plan's header on the host.
struct Layer : public torch::autograd::Function<Layer> {
  static torch::Tensor router_weights(const torch::Tensor& weights) {
    return weights.detach().to(torch::kFloat32).reshape(-1).contiguous();
  }

  static torch::Tensor forward(torch::autograd::AutogradContext* ctx, const torch::Tensor& x, const torch::Tensor& expert_ids,
                               const torch::Tensor& weights, const torch::Tensor& w_up, const torch::Tensor& w_down,
                               const std::shared_ptr<FusedRank>& rank, bool training) {
    const torch::Tensor ids = expert_ids.to(torch::kInt32).contiguous(), w_flat = router_weights(weights);
    const torch::Tensor xc = aligned(x.detach()), up = w_up.detach().contiguous(), down = w_down.detach().contiguous();
    auto [made, slices, kept_slices] = rank->forward_pass(xc, ids, w_flat, up, down, training, /*plan_wanted=*/training);
    if (training) {
      torch::autograd::variable_list saved{xc, weights, up, down};
      saved.insert(saved.end(), made.begin() + 1, made.end());
      ctx->save_for_backward(saved);
      ctx->saved_data["rank"] = c10::IValue::make_capsule(c10::make_intrusive<Held>(rank));
      ctx->saved_data["slices"] = slices;
      ctx->saved_data["kept_slices"] = kept_slices;
    }
    return made[0];
  }

  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list grads) {
    const auto saved = ctx->get_saved_variables();  // (hooks run here, before anything is locked)
    const std::shared_ptr<FusedRank> rank = static_cast<Held*>(ctx->saved_data["rank"].toCapsule().get())->rank;
    // (x and the plan's tables too: hooks may have put them elsewhere)
    const torch::Tensor x = aligned(saved[0]), plan = aligned(saved[4]), &weights = saved[1];
    const torch::Tensor g = aligned(grads[0].to(x.scalar_type()));
    const std::vector<torch::Tensor> kept(saved.begin() + 7, saved.end());
    auto [dx, d_weights, dw_up, dw_down] =
        rank->backward_pass(x, g, router_weights(weights), saved[2], saved[3], plan, saved[5], saved[6],
                            ctx->saved_data["slices"].toInt(), kept, ctx->saved_data["kept_slices"].toInt());
    return {dx, torch::Tensor(), d_weights.reshape(weights.sizes()).to(weights.scalar_type()), dw_up, dw_down, torch::Tensor(),
            torch::Tensor()};
  }
};

}  // namespace

torch::Tensor chunked_moe_layer(std::shared_ptr<FusedRank> rank, const torch::Tensor& x, const torch::Tensor& expert_ids,
                                const torch::Tensor& weights, const torch::Tensor& w_up, const torch::Tensor& w_down) {
  // (Released between the caller's look-up and this call; what is released later is refused by the pass.)
  if (rank == nullptr) throw std::runtime_error("chunked_moe fused path: the workspace was released before the forward");
  bool training = false;
  if (at::GradMode::is_enabled())
    training = x.requires_grad() || weights.requires_grad() || w_up.requires_grad() || w_down.requires_grad();
  return Layer::apply(x, expert_ids, weights, w_up, w_down, rank, training);
}

}  // namespace cem
