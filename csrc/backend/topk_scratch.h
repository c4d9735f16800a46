// Device memory of a top-k selection, from torch's caching allocator.
#pragma once

#include <ATen/ATen.h>
#include <c10/util/Exception.h>

#include <algorithm>

#include "kernels/topk_api.h"

namespace mccl {

// What the fastest path for this problem wants or, on a device without room for that, what the path that needs least
// can do with: a selection never fails for want of the list.
inline at::Tensor topk_scratch(int64_t n, int64_t k, bool dense, const at::TensorOptions& like) {
  auto bytes = [&](size_t b) { return at::empty({static_cast<int64_t>(b)}, like.dtype(at::kByte)); };
  try {
    return bytes(kern::topk_scratch_bytes(n, k));
  } catch (const c10::OutOfMemoryError&) {
    return bytes(dense ? std::max<size_t>(kern::topk_dense_min_scratch_bytes(n), 1) : kern::topk_min_scratch_bytes());
  }
}

}  // namespace mccl
