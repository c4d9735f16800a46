// Which tensors, and when, a native autograd function may take past the dispatcher.
#pragma once

#include <ATen/ATen.h>

namespace mccl {

// A tensor as the kernels read it: memory on the device, nothing lazy, no wrapper (vmap, functorch, subclasses), no tangent.
inline bool ordinary(const at::Tensor& t) {
  using c10::DispatchKey;
  constexpr auto allowed = c10::DispatchKeySet({DispatchKey::CUDA, DispatchKey::AutogradCUDA, DispatchKey::ADInplaceOrView,
                                                DispatchKey::AutocastCUDA});
  return t.defined() && allowed.isSupersetOf(t.key_set()) && !t._fw_grad(0).defined();
}
// No mode that wants to see the operators (Python modes, functorch transforms, functionalization).
inline bool no_modes() { return (c10::impl::tls_local_dispatch_key_set().included_ - c10::default_included_set).empty(); }

}  // namespace mccl
