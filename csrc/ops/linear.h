// torch.nn.functional.linear for fp32 matrices on the tensor cores (kernels/gemm_f32.cu), with its gradients.
#pragma once

#include <ATen/ATen.h>

namespace mccl {

// x w^T + bias.  Whatever the kernels do not take (see linear_native) goes to at::linear.
at::Tensor linear(const at::Tensor& x, const at::Tensor& w, const c10::optional<at::Tensor>& bias);
// Whether this call would run on this library's kernels, in forward.
bool linear_native(const at::Tensor& x, const at::Tensor& w, const c10::optional<at::Tensor>& bias);
// For tests: the products of such a call, forward or (with `grad`) backward, whose kernels give every wait up after
// `wait_limit` cycles.
std::vector<at::Tensor> linear_with_limit(const at::Tensor& x, const at::Tensor& w, const c10::optional<at::Tensor>& grad,
                                          int64_t wait_limit);

}  // namespace mccl
