#include "ops/linear.h"

#include <ATen/autocast_mode.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/autograd/custom_function.h>

#include <algorithm>
#include <mutex>

#include "common/errors.h"
#include "kernels/gemm_api.h"
#include "ops/ordinary.h"

namespace mccl {

namespace {

#define LINEAR_CK(expr)                                                      \
  do {                                                                       \
    cudaError_t _e = (expr);                                                 \
    if (_e != cudaSuccess) {                                                 \
      cudaGetLastError();                                                    \
      throw DeviceError(std::string(#expr) + ": " + cudaGetErrorString(_e)); \
    }                                                                        \
  } while (0)

// Words of mapped host memory, one per device, in which a kernel notes that one of its bounded waits ran out.
constexpr int kDevices = 64;
uint32_t* wait_status(const at::Tensor& t) {
  static uint32_t* words = [] {
    void* p = nullptr;
    auto mode = cudaStreamCaptureModeRelaxed;  // the first call may be under capture
    LINEAR_CK(cudaThreadExchangeStreamCaptureMode(&mode));
    const cudaError_t e = cudaHostAlloc(&p, kDevices * sizeof(uint32_t), cudaHostAllocMapped | cudaHostAllocPortable);
    LINEAR_CK(cudaThreadExchangeStreamCaptureMode(&mode));
    LINEAR_CK(e);
    std::fill_n(static_cast<uint32_t*>(p), kDevices, 0u);
    return static_cast<uint32_t*>(p);
  }();
  return words + t.get_device() % kDevices;
}
// Reports what a kernel has noted on the device, once.  What it gave up is NaN.
void check_waits(const at::Tensor& t) {
  uint32_t* word = wait_status(t);
  if (*static_cast<volatile uint32_t*>(word) != 0 && __atomic_exchange_n(word, 0u, __ATOMIC_RELAXED) != 0)
    throw DeviceError("a wait inside an earlier matrix product kernel ran out; what it should have written is NaN");
}

bool rows_ok(const at::Tensor& t) {
  return t.scalar_type() == at::kFloat && t.dim() == 2 && t.numel() > 0 && t.stride(1) == 1 && (t.size(0) == 1 || t.stride(0) >= t.size(1));
}
bool blackwell(int device) {
  const auto* p = at::cuda::getDeviceProperties(static_cast<c10::DeviceIndex>(device));
  return p->major == 10 && p->minor == 0;
}

kern::MatrixF32 matrix(const at::Tensor& t) {
  return {t.const_data_ptr<float>(), t.size(0) == 1 ? std::max(t.stride(0), t.size(1)) : t.stride(0), t.size(0), t.size(1)};
}

int64_t align(int64_t bytes) { return (bytes + 255) / 256 * 256; }

// Scratch of one or two products that run one behind the other: tickets, partial sums (shared), images.
struct Scratch {
  at::Tensor buffer;
  char* at = nullptr;
  char* take(int64_t bytes) {
    char* p = at;
    at += align(bytes);
    return p;
  }
};
// No memory for it: an empty one, and the product is left to torch, which needs less.
Scratch scratch_for(std::initializer_list<const kern::GemmPlan*> plans, const at::TensorOptions& like) {
  int64_t bytes = 0, partial = 0;
  for (const auto* p : plans) {
    bytes += align(p->tickets * 4) + align(p->a_image) + align(p->b_image);
    partial = std::max(partial, p->partial);
  }
  Scratch s;
  try {
    s.buffer = at::empty({bytes + align(partial)}, like.dtype(at::kByte));
    s.at = static_cast<char*>(s.buffer.data_ptr());
  } catch (const c10::OutOfMemoryError&) {
  }
  return s;
}

at::Tensor forward_product(const at::Tensor& x, const at::Tensor& w, const at::Tensor& bias, int64_t wait_limit = -1) {
  check_waits(x);
  c10::cuda::CUDAGuard guard(x.device());
  const auto stream = at::cuda::getCurrentCUDAStream();
  const kern::GemmPlan plan = kern::gemm_plan(kern::Product::kForward, x.size(0), w.size(1), w.size(0));
  Scratch s = scratch_for({&plan}, x.options());
  if (s.at == nullptr) return at::linear(x, w, bias.defined() ? c10::optional<at::Tensor>(bias) : c10::nullopt);
  at::Tensor y = at::empty({x.size(0), w.size(0)}, x.options());
  auto* tickets = reinterpret_cast<uint32_t*>(s.take(plan.tickets * 4));
  char* image = s.take(plan.b_image);
  auto* partial = reinterpret_cast<float*>(s.take(plan.partial));
  const kern::SplitJob job{matrix(x), image, plan.cols, nullptr};
  LINEAR_CK(kern::launch_split_f32(&job, 1, nullptr, tickets, plan.tickets, stream));
  const kern::MatrixF32 wm = matrix(w);
  kern::GemmArgs g{};
  g.product = kern::Product::kForward;
  g.plan = plan;
  g.weight = wm.data;
  g.ldw = wm.ld;
  g.b_image = image;
  g.bias = bias.defined() ? bias.const_data_ptr<float>() : nullptr;
  g.c = y.data_ptr<float>();
  g.ldc = w.size(0);
  g.partial = partial;
  g.tickets = tickets;
  g.failed = wait_status(x);
  g.wait_limit = wait_limit;
  LINEAR_CK(kern::launch_gemm_f32(g, stream));
  return y;
}

struct Gradients {
  at::Tensor x, w, bias;
};
Gradients backward_products(const at::Tensor& grad, const at::Tensor& x, const at::Tensor& w, bool need_x, bool need_w,
                            bool need_bias, int64_t wait_limit = -1) {
  check_waits(x);
  const int64_t batch = x.size(0), in = w.size(1), out = w.size(0);
  c10::cuda::CUDAGuard guard(x.device());
  const auto stream = at::cuda::getCurrentCUDAStream();
  Gradients r;
  bool own_x = need_x && kern::gemm_pays(kern::Product::kInput, batch, in, out);
  bool own_w = need_w && kern::gemm_pays(kern::Product::kWeight, batch, in, out);
  kern::GemmPlan px{}, pw{};
  if (own_x) px = kern::gemm_plan(kern::Product::kInput, batch, in, out);
  if (own_w) pw = kern::gemm_plan(kern::Product::kWeight, batch, in, out);
  Scratch s;
  if (own_x || own_w) s = scratch_for({&px, &pw}, x.options());
  if (s.at == nullptr) own_x = own_w = false;
  if (need_x && !own_x) r.x = grad.mm(w);
  if (need_w && !own_w) r.w = grad.t().mm(x);
  if (!own_x && !own_w) {
    if (need_bias) r.bias = grad.sum(0);
    return r;
  }
  auto* tickets = reinterpret_cast<uint32_t*>(s.take((px.tickets + pw.tickets) * 4));
  char *gx = s.take(px.b_image), *gw = s.take(pw.b_image), *xw = s.take(pw.a_image);
  auto* partial = reinterpret_cast<float*>(s.take(std::max(px.partial, pw.partial)));
  if (need_bias) r.bias = at::empty({out}, x.options());
  const kern::SplitJob jobs[2] = {{matrix(grad), own_x ? gx : nullptr, px.cols, own_w ? gw : nullptr},
                                  {matrix(x), nullptr, 0, xw}};
  LINEAR_CK(kern::launch_split_f32(jobs, own_w ? 2 : 1, need_bias ? r.bias.data_ptr<float>() : nullptr, tickets,
                                   px.tickets + pw.tickets, stream));
  if (own_x) {
    r.x = at::empty({batch, in}, x.options());
    const kern::MatrixF32 wm = matrix(w);
    kern::GemmArgs g{};
    g.product = kern::Product::kInput;
    g.plan = px;
    g.weight = wm.data;
    g.ldw = wm.ld;
    g.b_image = gx;
    g.c = r.x.data_ptr<float>();
    g.ldc = in;
    g.partial = partial;
    g.tickets = tickets;
    g.failed = wait_status(x);
    g.wait_limit = wait_limit;
    LINEAR_CK(kern::launch_gemm_f32(g, stream));
  }
  if (own_w) {
    r.w = at::empty({out, in}, x.options());
    kern::GemmArgs g{};
    g.product = kern::Product::kWeight;
    g.plan = pw;
    g.a_image = xw;
    g.b_image = gw;
    g.c = r.w.data_ptr<float>();
    g.ldc = in;
    g.partial = partial;
    g.tickets = tickets + px.tickets;
    g.failed = wait_status(x);
    g.wait_limit = wait_limit;
    LINEAR_CK(kern::launch_gemm_f32(g, stream));
  }
  return r;
}

struct LinearFn : torch::autograd::Function<LinearFn> {
  static at::Tensor forward(torch::autograd::AutogradContext* ctx, const at::Tensor& x, const at::Tensor& w,
                            const c10::optional<at::Tensor>& bias) {
    ctx->save_for_backward({x, w});
    ctx->saved_data["bias"] = bias.has_value();
    return forward_product(x, w, bias ? *bias : at::Tensor());
  }
  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx,
                                                 torch::autograd::variable_list grads) {
    at::Tensor grad = grads[0];
    if (!grad.defined()) return {at::Tensor(), at::Tensor(), at::Tensor()};
    const auto saved = ctx->get_saved_variables();
    const at::Tensor &x = saved[0], &w = saved[1];
    const bool need_x = ctx->needs_input_grad(0), need_w = ctx->needs_input_grad(1), 
               need_bias = ctx->saved_data["bias"].toBool() && ctx->needs_input_grad(2);
    // a second derivative, or tensors that are no longer what forward saw (a hook, vmap over the backward pass): operators
    // that autograd knows
    if (at::GradMode::is_enabled() || !no_modes() || !ordinary(grad) || grad.scalar_type() != at::kFloat || !ordinary(x) || !ordinary(w) || !rows_ok(x) ||
        !rows_ok(w) || x.device() != grad.device() || w.device() != grad.device())
      return {need_x ? grad.mm(w) : at::Tensor(), need_w ? grad.t().mm(x) : at::Tensor(),
              need_bias ? grad.sum(0) : at::Tensor()};
    if (!rows_ok(grad)) grad = grad.contiguous();
    Gradients r = backward_products(grad, x, w, need_x, need_w, need_bias);
    return {r.x, r.w, r.bias};
  }
};

}  // namespace

bool linear_native(const at::Tensor& x, const at::Tensor& w, const c10::optional<at::Tensor>& bias) {
  if (!no_modes() || !ordinary(x) || !ordinary(w) || !rows_ok(x) || !rows_ok(w) || x.size(1) != w.size(1) ||
      x.device() != w.device())
    return false;
  if (bias && bias->defined() &&
      (!ordinary(*bias) || bias->scalar_type() != at::kFloat || bias->dim() != 1 || bias->size(0) != w.size(0) || bias->stride(0) != 1 || bias->device() != x.device()))
    return false;
  // a program that lets torch round its fp32 products has asked for something else (the getter that torch's products use: the
  // older one throws where the newer setting has been used)
  if (at::globalContext().float32Precision(at::Float32Backend::CUDA, at::Float32Op::MATMUL) == at::Float32Precision::TF32 || at::autocast::is_autocast_enabled(at::kCUDA)) return false;
  return blackwell(x.get_device()) && kern::gemm_pays(kern::Product::kForward, x.size(0), w.size(1), w.size(0));
}

std::vector<at::Tensor> linear_with_limit(const at::Tensor& x, const at::Tensor& w, const c10::optional<at::Tensor>& grad,
                                          int64_t wait_limit) {
  TORCH_CHECK(wait_limit >= 0 && linear_native(x, w, c10::nullopt), "not a call for the kernels");
  if (!grad) return {forward_product(x, w, at::Tensor(), wait_limit)};
  TORCH_CHECK(rows_ok(*grad) && grad->device() == x.device() && grad->size(0) == x.size(0) && grad->size(1) == w.size(0),
              "not a gradient for the kernels");
  const Gradients g = backward_products(*grad, x, w, true, true, false, wait_limit);
  return {g.x, g.w};
}

at::Tensor linear(const at::Tensor& x, const at::Tensor& w, const c10::optional<at::Tensor>& bias) {
  if (!linear_native(x, w, bias)) return at::linear(x, w, bias);
  const bool has_bias = bias && bias->defined();
  if (!at::GradMode::is_enabled() || !(x.requires_grad() || w.requires_grad() || (has_bias && bias->requires_grad())))
    return forward_product(x, w, has_bias ? *bias : at::Tensor());
  return LinearFn::apply(x, w, has_bias ? bias : c10::nullopt);
}

}  // namespace mccl
