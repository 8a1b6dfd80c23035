// Operands of kernels that read 16 bytes at a time without a tensor map (which would refuse other addresses).
#pragma once

#include <torch/extension.h>

#include <cstdint>

namespace cem {

inline bool at_16_bytes(const torch::Tensor& t) { return reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0; }

// `t` contiguous and beginning at an address of 16 bytes: itself, or a copy. (A contiguous view may begin anywhere.)
inline torch::Tensor aligned(const torch::Tensor& t) {
  const torch::Tensor c = t.contiguous();
  return at_16_bytes(c) ? c : c.clone();
}

}  // namespace cem
