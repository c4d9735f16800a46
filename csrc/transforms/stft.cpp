#include "transforms/stft.h"

#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/autograd/custom_function.h>

#include <algorithm>
#include <cmath>
#include <limits>

#include "common/errors.h"
#include "kernels/stft_api.h"
#include "ops/ordinary.h"

namespace mccl {

namespace {

#define STFT_CK(expr)                                                             \
  do {                                                                            \
    cudaError_t _e = (expr);                                                      \
    if (_e != cudaSuccess) {                                                      \
      cudaGetLastError();                                                         \
      throw DeviceError(std::string(#expr) + ": " + cudaGetErrorString(_e));      \
    }                                                                             \
  } while (0)

void check_common(int64_t n_fft, int64_t hop, int64_t win_length, const at::Tensor& window,
                  const std::string& backend) {
  MCCL_CHECK_TENSOR(stft_cuda_supported(n_fft),
                    "n_fft must be a power of two in [8, " << kern::kStftMaxNfft << "], got " << n_fft);
  MCCL_CHECK_TENSOR(hop >= 1, "hop_length must be >= 1");
  MCCL_CHECK_TENSOR(win_length >= 1 && win_length <= n_fft, "win_length must be in [1, n_fft]");
  MCCL_CHECK_TENSOR(window.dim() == 1 && window.numel() == win_length, "window must be 1-D of win_length elements");
  MCCL_CHECK_TENSOR(backend == "auto" || backend == "cuda" || backend == "metal",
                    "the native STFT serves the CUDA backend (got '" << backend << "')");
}

// The kernels read memory: a lazy conjugation or negation (`spec.conj()`, the gradient that autograd hands back
// through it) is carried out before they run.
at::Tensor plain(const at::Tensor& t) { return t.is_conj() || t.is_neg() ? t.resolve_conj().resolve_neg() : t; }

// fp32 and contiguous on `like`'s device; the kernels centre its win_length samples in n_fft zeros
at::Tensor prepare_window(const at::Tensor& window, const at::Tensor& like) {
  return plain(window.to(like.device(), at::kFloat).contiguous());
}
kern::StftWindow centred(const at::Tensor& w, int64_t n_fft) {
  const int64_t len = w.numel();
  return {w.data_ptr<float>(), static_cast<int>(len), static_cast<int>((n_fft - len) / 2)};
}

at::Tensor as_batch(const at::Tensor& t) {
  MCCL_CHECK_TENSOR(t.is_cuda() && t.scalar_type() == at::kFloat, "expected a float32 CUDA tensor");
  const at::Tensor x = plain(t);
  if (x.dim() == 1) return x.unsqueeze(0).contiguous();
  if (x.dim() == 3 && x.size(1) == 1) return x.squeeze(1).contiguous();
  MCCL_CHECK_TENSOR(x.dim() == 2, "expected [time], [batch, time] or [batch, 1, time]");
  return x.contiguous();
}

void spec_strides(const at::Tensor& spec, int64_t n_fft, int64_t& sb, int64_t& sf, int64_t& st) {
  MCCL_CHECK_TENSOR(spec.is_cuda() && spec.scalar_type() == at::kComplexFloat && spec.dim() == 3,
                    "expected a complex64 CUDA spectrum [batch, freq, frames]");
  MCCL_CHECK_TENSOR(spec.size(1) == n_fft / 2 + 1, "spectrum must have n_fft/2+1 frequency bins");
  sb = spec.stride(0);
  sf = spec.stride(1);
  st = spec.stride(2);
}

// The kernels take an int.  Where frame 1 starts behind all samples of the padded signal every frame but the first is
// empty, and any longer hop does the same.
int kernel_hop(int64_t hop, int64_t samples, int64_t n_fft) {
  hop = std::min(hop, samples + 2 * n_fft);
  MCCL_CHECK_TENSOR(hop <= std::numeric_limits<int>::max(), "hop_length is out of range");
  return static_cast<int>(hop);
}

void run_ifft_ola(const kern::IfftOlaArgs& a, const at::Tensor& out) {
  at::Tensor scratch;
  const int64_t floats = kern::ifft_ola_scratch(a);
  if (floats > 0) scratch = at::empty({floats}, out.options());
  STFT_CK(kern::launch_ifft_ola(a, floats > 0 ? scratch.data_ptr<float>() : nullptr,
                                at::cuda::getCurrentCUDAStream()));
}

}  // namespace

bool stft_cuda_supported(int64_t n_fft) {
  return n_fft >= 8 && n_fft <= kern::kStftMaxNfft && (n_fft & (n_fft - 1)) == 0;
}

int64_t stft_num_frames(int64_t signal_len, int64_t n_fft, int64_t hop, bool center) {
  if (center) return 1 + signal_len / hop;
  MCCL_CHECK_TENSOR(signal_len >= n_fft, "signal shorter than n_fft without centering");
  return 1 + (signal_len - n_fft) / hop;
}

at::Tensor stft_forward(const at::Tensor& waveform, const at::Tensor& window, int64_t n_fft, int64_t hop,
                        int64_t win_length, bool center, bool normalized, const std::string& backend) {
  check_common(n_fft, hop, win_length, window, backend);
  at::Tensor x = as_batch(waveform);
  const int64_t B = x.size(0), T = x.size(1);
  const int64_t pad = center ? n_fft / 2 : 0;
  MCCL_CHECK_TENSOR(!center || T > pad, "reflect padding needs a signal longer than n_fft/2");
  const int64_t frames = stft_num_frames(T, n_fft, hop, center);
  c10::cuda::CUDAGuard guard(x.device());
  at::Tensor w = prepare_window(window, x);
  at::Tensor out = at::empty({B, frames, n_fft / 2 + 1}, x.options().dtype(at::kComplexFloat));
  kern::FftFramesArgs a{};
  a.signal = x.data_ptr<float>();
  a.signal_len = T;
  a.window = centred(w, n_fft);
  a.out = reinterpret_cast<float*>(out.data_ptr());
  a.batch = static_cast<int>(B);
  a.n_frames = static_cast<int>(frames);
  a.n_fft = static_cast<int>(n_fft);
  a.hop = kernel_hop(hop, T, n_fft);
  a.pad = static_cast<int>(pad);
  a.reflect = center ? 1 : 0;
  a.divide_envelope = 0;
  a.scale = normalized ? 1.0f / std::sqrt(static_cast<float>(n_fft)) : 1.0f;
  STFT_CK(kern::launch_fft_frames(a, at::cuda::getCurrentCUDAStream()));
  return out.transpose(1, 2);  // [batch, freq, frames]; frames-major storage keeps the kernel's writes coalesced
}

at::Tensor stft_backward(const at::Tensor& grad_spec_in, const at::Tensor& window, int64_t n_fft, int64_t hop,
                         int64_t win_length, bool center, bool normalized, int64_t length,
                         const std::string& backend) {
  check_common(n_fft, hop, win_length, window, backend);
  const at::Tensor grad_spec = plain(grad_spec_in);
  int64_t sb, sf, st;
  spec_strides(grad_spec, n_fft, sb, sf, st);
  const int64_t B = grad_spec.size(0), frames = grad_spec.size(2);
  c10::cuda::CUDAGuard guard(grad_spec.device());
  at::Tensor w = prepare_window(window, grad_spec);
  at::Tensor out = at::empty({B, length}, grad_spec.options().dtype(at::kFloat));
  kern::IfftOlaArgs a{};
  a.spec = reinterpret_cast<const float*>(grad_spec.data_ptr());
  a.stride_b = sb;
  a.stride_f = sf;
  a.stride_t = st;
  a.window = centred(w, n_fft);
  a.out = out.data_ptr<float>();
  a.out_len = length;
  a.batch = static_cast<int>(B);
  a.n_frames = static_cast<int>(frames);
  a.n_fft = static_cast<int>(n_fft);
  a.hop = kernel_hop(hop, length, n_fft);
  a.hermitian = 0;  // adjoint of the one-sided forward transform: upper bins contribute nothing
  a.scale = normalized ? 1.0f / std::sqrt(static_cast<float>(n_fft)) : 1.0f;
  a.pad = center ? static_cast<int>(n_fft / 2) : 0;
  a.fold_reflect = center ? 1 : 0;
  a.normalize_envelope = 0;
  run_ifft_ola(a, out);
  return out;
}

at::Tensor istft_forward(const at::Tensor& spec_in, const at::Tensor& window, int64_t n_fft, int64_t hop,
                         int64_t win_length, bool center, bool normalized, int64_t length,
                         const std::string& backend) {
  check_common(n_fft, hop, win_length, window, backend);
  const at::Tensor spec = plain(spec_in);
  int64_t sb, sf, st;
  spec_strides(spec, n_fft, sb, sf, st);
  const int64_t B = spec.size(0), frames = spec.size(2);
  MCCL_CHECK_TENSOR(length >= 1, "length must be >= 1");
  c10::cuda::CUDAGuard guard(spec.device());
  at::Tensor w = prepare_window(window, spec);
  at::Tensor out = at::empty({B, length}, spec.options().dtype(at::kFloat));
  kern::IfftOlaArgs a{};
  a.spec = reinterpret_cast<const float*>(spec.data_ptr());
  a.stride_b = sb;
  a.stride_f = sf;
  a.stride_t = st;
  a.window = centred(w, n_fft);
  a.out = out.data_ptr<float>();
  a.out_len = length;
  a.batch = static_cast<int>(B);
  a.n_frames = static_cast<int>(frames);
  a.n_fft = static_cast<int>(n_fft);
  a.hop = kernel_hop(hop, length, n_fft);
  a.hermitian = 1;
  a.scale = (normalized ? std::sqrt(static_cast<float>(n_fft)) : 1.0f) / static_cast<float>(n_fft);
  a.pad = center ? static_cast<int>(n_fft / 2) : 0;
  a.fold_reflect = 0;
  a.normalize_envelope = 1;
  run_ifft_ola(a, out);
  return out;
}

at::Tensor istft_backward(const at::Tensor& grad_waveform, const at::Tensor& window, int64_t n_fft, int64_t hop,
                          int64_t win_length, bool center, bool normalized, int64_t n_frames,
                          const std::string& backend) {
  check_common(n_fft, hop, win_length, window, backend);
  at::Tensor g = as_batch(grad_waveform);
  const int64_t B = g.size(0), T = g.size(1);
  c10::cuda::CUDAGuard guard(g.device());
  at::Tensor w = prepare_window(window, g);
  at::Tensor out = at::empty({B, n_frames, n_fft / 2 + 1}, g.options().dtype(at::kComplexFloat));
  kern::FftFramesArgs a{};
  a.signal = g.data_ptr<float>();
  a.signal_len = T;
  a.window = centred(w, n_fft);
  a.out = reinterpret_cast<float*>(out.data_ptr());
  a.batch = static_cast<int>(B);
  a.n_frames = static_cast<int>(n_frames);
  a.n_fft = static_cast<int>(n_fft);
  a.hop = kernel_hop(hop, T, n_fft);
  a.pad = center ? static_cast<int>(n_fft / 2) : 0;
  a.reflect = 0;
  a.divide_envelope = 1;
  a.scale = (normalized ? std::sqrt(static_cast<float>(n_fft)) : 1.0f) / static_cast<float>(n_fft);
  STFT_CK(kern::launch_fft_frames(a, at::cuda::getCurrentCUDAStream()));
  return out.transpose(1, 2);
}

namespace {

// n_fft, hop, win_length, center, normalized, and what the gradient's shape needs
using Config = std::vector<int64_t>;

at::Tensor forward_of(const at::Tensor& waveform, const at::Tensor& window, const Config& c) {
  const at::Tensor x = waveform.dim() == 3 && waveform.size(1) == 1 ? waveform.squeeze(1) : waveform;
  return stft_forward(x.contiguous().to(at::kFloat), window, c[0], c[1], c[2], c[3] != 0, c[4] != 0, "cuda");
}
at::Tensor inverse_of(const at::Tensor& spec, const at::Tensor& window, const Config& c) {
  return istft_forward(spec, window, c[0], c[1], c[2], c[3] != 0, c[4] != 0, c[5], "cuda");
}

struct StftFn : torch::autograd::Function<StftFn> {
  static at::Tensor forward(torch::autograd::AutogradContext* ctx, const at::Tensor& waveform, const at::Tensor& window,
                            const Config& c) {
    ctx->save_for_backward({window});
    ctx->saved_data["config"] = c;
    ctx->saved_data["shape"] = waveform.sizes().vec();
    return forward_of(waveform, window, c);
  }
  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx,
                                                 torch::autograd::variable_list grads) {
    const Config c = ctx->saved_data["config"].toIntVector(), shape = ctx->saved_data["shape"].toIntVector();
    const at::Tensor g = stft_backward(grads[0], ctx->get_saved_variables()[0], c[0], c[1], c[2], c[3] != 0, c[4] != 0,
                                       shape.back(), "cuda");
    return {g.reshape(shape), at::Tensor(), at::Tensor()};
  }
};

struct IstftFn : torch::autograd::Function<IstftFn> {
  static at::Tensor forward(torch::autograd::AutogradContext* ctx, const at::Tensor& spec, const at::Tensor& window,
                            const Config& c) {
    ctx->save_for_backward({window});
    ctx->saved_data["config"] = c;
    ctx->saved_data["frames"] = spec.dim() > 0 ? spec.size(-1) : int64_t(0);
    return inverse_of(spec, window, c);
  }
  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx,
                                                 torch::autograd::variable_list grads) {
    const Config c = ctx->saved_data["config"].toIntVector();
    const at::Tensor g = istft_backward(grads[0].contiguous(), ctx->get_saved_variables()[0], c[0], c[1], c[2], c[3] != 0,
                                        c[4] != 0, ctx->saved_data["frames"].toInt(), "cuda");
    return {g, at::Tensor(), at::Tensor()};
  }
};

template <typename Fn, typename Run>
c10::optional<at::Tensor> direct(const at::Tensor& t, const at::Tensor& window, const Config& c, Run&& run) {
  if (!no_modes() || !ordinary(t) || !ordinary(window)) return c10::nullopt;
  if (!at::GradMode::is_enabled() || !(t.requires_grad() || window.requires_grad())) return run(t, window, c);
  return Fn::apply(t, window, c);
}

}  // namespace

c10::optional<at::Tensor> stft_direct(const at::Tensor& waveform, const at::Tensor& window, int64_t n_fft, int64_t hop,
                                      int64_t win_length, bool center, bool normalized) {
  return direct<StftFn>(waveform, window, {n_fft, hop, win_length, center, normalized}, forward_of);
}

c10::optional<at::Tensor> istft_direct(const at::Tensor& spec, const at::Tensor& window, int64_t n_fft, int64_t hop,
                                       int64_t win_length, int64_t length, bool center, bool normalized) {
  return direct<IstftFn>(spec, window, {n_fft, hop, win_length, center, normalized, length}, inverse_of);
}

}  // namespace mccl
