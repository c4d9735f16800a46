// STFT / iSTFT kernels (sm_100a): register FFTs of half the frame length by a group of lanes of one
// warp (fft_warp.cuh), with the padding, windowing and scaling fused into the loads and stores and
// the overlap-add fused behind the inverse transform.  See stft_api.h for the decomposition.
// Replaces the reference's one-thread-per-frame Metal FFT (reference
// csrc/metal/shaders.metal:735-861) and its CPU-side padding and overlap-add
// (reference csrc/transforms/StftMetalKernels.mm:158-393).
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>

#include "kernels/fft_warp.cuh"
#include "kernels/launch_count.h"
#include "kernels/stft_api.h"

namespace mccl {
namespace kern {

namespace {

constexpr int kSms = 148;
constexpr size_t kMaxSmem = 227 << 10;    // per CTA
constexpr size_t kSmemPerSm = 228 << 10;  // of which each CTA takes another 1 KB

__device__ __forceinline__ float window_at(const StftWindow& w, int64_t n) {
  const int64_t i = n - w.left;
  return i >= 0 && i < w.len ? w.data[i] : 0.f;
}

// sum of window^2 over the frames covering padded position p
__device__ __forceinline__ float envelope_at(const StftWindow& window, int64_t p, int n_fft, int hop, int n_frames) {
  int64_t f_hi = p / hop;
  if (f_hi > n_frames - 1) f_hi = n_frames - 1;
  int64_t f_lo = (p - n_fft + hop) / hop;  // ceil((p - n_fft + 1) / hop) for non-negative values
  if (p - n_fft + 1 <= 0) f_lo = 0;
  float e = 0.f;
  for (int64_t f = f_lo; f <= f_hi; ++f) {
    const int64_t n = p - f * hop;
    if (n >= 0 && n < n_fft) {
      const float w = window_at(window, n);
      e += w * w;
    }
  }
  return e;
}

template <int kBytes>
__device__ __forceinline__ void copy_async(void* smem, const void* gmem) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(
                   static_cast<unsigned>(__cvta_generic_to_shared(smem))),
               "l"(gmem), "n"(kBytes)
               : "memory");
}
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Samples, times the window, of a frame that reaches over the signal's ends, in `buf`.  Every lane prepares the pairs that it
// will read back; the copies are asynchronous, so that a small call waits for memory once and not once per pair.
template <int LH>
__device__ __forceinline__ void load_edge_frame(const FftFramesArgs& a, const float* sig, const float* win, float2* buf, int f,
                                                int t, float2 (&v)[WarpFft<LH>::V]) {
  using F = WarpFft<LH>;
  const int64_t start = static_cast<int64_t>(f) * a.hop - a.pad;
  for (int r = 0; r < 2 * F::V; ++r) {
    const int j = 2 * ((r / 2) * F::L + t) + (r & 1);
    int64_t q = start + j;
    if (a.reflect) {  // without repeating the edge sample; the signal is longer than the padding: one reflection
      if (q < 0) q = -q;
      if (q >= a.signal_len) q = 2 * a.signal_len - 2 - q;
    }
    float* dst = reinterpret_cast<float*>(buf) + j;
    if (q >= 0 && q < a.signal_len) copy_async<4>(dst, sig + q);
    else *dst = 0.f;
  }
  copy_async_wait();
#pragma unroll
  for (int r = 0; r < F::V; ++r) {
    const float2 w = reinterpret_cast<const float2*>(win)[r * F::L + t];
    v[r] = buf[r * F::L + t];
    v[r].x *= w.x;
    v[r].y *= w.y;
  }
}

// Samples, times window / envelope, of a frame that lacks neighbours or reaches over the signal's ends.  Only rows of `hop`
// samples that lack a frame get an envelope of their own, several pairs of every lane at a time so that their loads overlap;
// the others take it from the table.  Every lane prepares the weights that it will read back, in `buf`.
// (2 x 48000 samples, n_fft 2048, the inverse's backward: 19.6 us with an envelope for every sample one by one, 12.6 us so.)
template <int LH>
__device__ __forceinline__ void load_edge_frame_over_envelope(const FftFramesArgs& a, const float* sig, const float* win,
                                                              const float* win_env, float2* buf, int f, int t, int hop,
                                                              int reach, float2 (&v)[WarpFft<LH>::V]) {
  using F = WarpFft<LH>;
  const int64_t start = static_cast<int64_t>(f) * a.hop - a.pad, left = a.signal_len - start;
  const float* src = sig + start;
  const int lo = start < 0 ? static_cast<int>(-start) : 0;  // samples [lo, hi) lie in the signal
  const int hi = left >= F::n ? F::n : left > 0 ? static_cast<int>(left) : 0;
#pragma unroll
  for (int r = 0; r < F::V; ++r) {
    const int j = 2 * (r * F::L + t);
    v[r] = make_float2(j >= lo && j < hi ? src[j] : 0.f, j + 1 >= lo && j + 1 < hi ? src[j + 1] : 0.f);
  }
  // Frames f - before .. f + after reach into this one.  A row of the padded signal has a full set of them from row
  // reach - 1 to row n_frames - 1: samples [full_lo, full_hi) of this frame.
  const int before = min(reach - 1, f), after = min(reach - 1, a.n_frames - 1 - f);
  const int full_lo = (reach - 1 - before) * hop, full_hi = after == reach - 1 ? F::n : (after + 1) * hop;
  auto place = [&](int r) { return 2 * ((r / 2) * F::L + t) + (r & 1); };
  float* weights = reinterpret_cast<float*>(buf);
#pragma unroll 4
  for (int r = 0; r < 2 * F::V; ++r) {
    const int j = place(r);
    weights[j] = j >= full_lo && j < full_hi ? win_env[j] : 0.f;
  }
  constexpr int kMost = LH <= 6 ? 4 : LH <= 8 ? 8 : 16;  // (short frames have 64 or 80 registers: more would spill)
  constexpr int kAhead = 2 * F::V < kMost ? 2 * F::V : kMost, kSpan = kAhead * F::L;
#pragma unroll 1
  for (int side = 0; side < 2; ++side) {
    const int j0 = max(side == 0 ? 0 : max(full_lo, full_hi), lo), j1 = min(side == 0 ? full_lo : F::n, hi);
#pragma unroll 1
    for (int base = j0 / kSpan * kSpan; base < j1; base += kSpan) {
      const int i_hi = min(before, (F::n - 1 - base) / hop), i_lo = -min(after, (base + kSpan - 1) / hop);
      float e[kAhead];
#pragma unroll
      for (int u = 0; u < kAhead; ++u) e[u] = 0.f;
#pragma unroll 1
      for (int i = i_hi; i >= i_lo; --i) {  // frame f - i, in frame order
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
          const int o = base + place(u) + i * hop;
          if (o >= 0 && o < F::n) e[u] += win[o] * win[o];
        }
      }
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        const int j = base + place(u);
        if (j >= j0 && j < j1) weights[j] = e[u] > 1e-11f ? win[j] / e[u] : 0.f;
      }
    }
  }
#pragma unroll
  for (int r = 0; r < F::V; ++r) {  // (a sample that no frame covers takes no part, whatever it is)
    const float2 w = buf[r * F::L + t];
    v[r] = make_float2(w.x != 0.f ? v[r].x * w.x : 0.f, w.y != 0.f ? v[r].y * w.y : 0.f);
  }
}

// Frames -> spectrum.  Bound by HBM (signal in, spectrum out) and by instruction issue, about equally: the
// values stay in registers from the load to the store, and a persistent grid computes the twiddle and window
// tables once per CTA.
// 16 x 1 Mi samples, n_fft 2048, hop 512 (336 MB): 453 us with one CTA per
// frame and five shared-memory passes, 92 us so.
template <int LH, bool kEnvelope>
__global__ void __launch_bounds__(256, LH <= 6 ? 4 : LH <= 8 ? 3 : LH <= 10 ? 2 : 1)
    fft_frames_kernel(const FftFramesArgs a, int64_t total) {
  using F = WarpFft<LH>;
  extern __shared__ float2 smem[];
  float2* tw = smem;
  float2* split = tw + F::h;
  float* win = reinterpret_cast<float*>(split + F::h / 2);
  float* win_env = win + F::n;  // window / envelope, for frames with a full set of neighbours
  float2* slots = reinterpret_cast<float2*>(win_env + (kEnvelope ? F::n : 0));
  F::fill_tables(tw, split);
  for (int j = threadIdx.x; j < F::n; j += blockDim.x) win[j] = window_at(a.window, j);
  __syncthreads();
  const int hop = min(a.hop, F::n);              // no sums beyond the int range with a hop near its end
  const int reach = (F::n + hop - 1) / hop;      // frames that cover a sample
  if (kEnvelope) {
    for (int j = threadIdx.x; j < hop; j += blockDim.x) {
      float e = 0.f;
      for (int i = j + (F::n - 1 - j) / hop * hop; i >= 0; i -= hop) e += win[i] * win[i];  // in frame order
      for (int i = j; i < F::n; i += hop) win_env[i] = e > 1e-11f ? win[i] / e : 0.f;
    }
    __syncthreads();
  }

  const int warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int sub = (threadIdx.x & 31) / F::L, t = threadIdx.x % F::L;
  float2* buf = slots + (warp * F::kPerWarp + sub) * F::kSlot;
  const float2* win2 = reinterpret_cast<const float2*>(kEnvelope ? win_env : win);
  const int64_t stride = static_cast<int64_t>(gridDim.x) * warps * F::kPerWarp;
  for (int64_t i0 = (static_cast<int64_t>(blockIdx.x) * warps + warp) * F::kPerWarp; i0 < total; i0 += stride) {
    const int64_t i = i0 + sub;
    const bool live = i < total;
    const int64_t b = live ? i / a.n_frames : 0;
    const int f = live ? static_cast<int>(i - b * a.n_frames) : 0;
    const float* sig = a.signal + b * a.signal_len;
    const int64_t start = static_cast<int64_t>(f) * a.hop - a.pad;
    bool inside = start >= 0 && start + F::n <= a.signal_len;
    if (kEnvelope) inside = inside && f >= reach - 1 && f <= a.n_frames - reach;
    float2 v[F::V];
    if (inside) {
      const float* src = sig + start;
      if ((reinterpret_cast<uintptr_t>(src) & 7) == 0) {
#pragma unroll
        for (int r = 0; r < F::V; ++r) v[r] = reinterpret_cast<const float2*>(src)[r * F::L + t];
      } else {
#pragma unroll
        for (int r = 0; r < F::V; ++r) v[r] = make_float2(src[2 * (r * F::L + t)], src[2 * (r * F::L + t) + 1]);
      }
#pragma unroll
      for (int r = 0; r < F::V; ++r) {
        const float2 w = win2[r * F::L + t];
        v[r].x *= w.x;
        v[r].y *= w.y;
      }
    } else {
      if constexpr (kEnvelope) load_edge_frame_over_envelope<LH>(a, sig, win, win_env, buf, f, t, hop, reach, v);
      else load_edge_frame<LH>(a, sig, win, buf, f, t, v);
    }
    __syncwarp();
    F::transform(v, tw, buf, t);
    float2* out = reinterpret_cast<float2*>(a.out) + (b * a.n_frames + f) * (F::h + 1);
    const float half = 0.5f * a.scale;  // split_bins gives twice the bins
    F::split_bins(v, split, t, [&](int k, float2 x) {
      float sc = half;
      if (kEnvelope) {  // gradient of an inverse real FFT: both halves of the spectrum, and real DC and Nyquist
        sc = k == 0 || k == F::h ? half : a.scale;
        if (k == 0 || k == F::h) x.y = 0.f;
      }
      if (live) out[k] = make_float2(x.x * sc, x.y * sc);
    });
  }
}

// Bins of one frame -> its windowed samples y (h float2) in `slot`, by one group of lanes.  A null `spec`
// means that the slot already holds the bins.
template <int LH>
__device__ __forceinline__ void inverse_frame(const IfftOlaArgs& a, const float2* spec, int64_t stride_f,
                                              const float2* tw, const float2* split, const float2* win2, float2* slot,
                                              int t) {
  using F = WarpFft<LH, false>;
  // hermitian: inverse real FFT of the one-sided bins.  Otherwise the adjoint of the forward
  // transform, Re(sum_{k<=h} X[k] e^{+2 pi i k n / N}), which equals half the inverse real FFT of the
  // same bins with the real parts of DC and Nyquist doubled.
  const float edge = a.hermitian ? 1.0f : 2.0f;
  const float post = a.hermitian ? a.scale : 0.5f * a.scale;
  float2 x[F::V], nyquist;
  if (spec != nullptr) {
#pragma unroll
    for (int r = 0; r < F::V; ++r) x[r] = spec[(r * F::L + t) * stride_f];
    nyquist = spec[F::h * stride_f];
  } else {
#pragma unroll
    for (int r = 0; r < F::V; ++r) x[r] = slot[r * F::L + t];
    nyquist = slot[F::h];
  }
  __syncwarp();
  F::merge_bins(x, nyquist, split, t, edge);
  F::transform(x, tw, slot, t);
  static_for<0, F::V>([&](auto ic) {
    constexpr int g = decltype(ic)::value / F::L, k2 = decltype(ic)::value % F::L;
    const int m = t + F::L * g + F::V * k2;
    const float2 z = x[F::at(g, k2)], w = win2[m];
    slot[m] = make_float2(z.y * post * w.x, z.x * post * w.y);
  });
}

struct OlaPlan {
  int segments;       // CTAs per batch entry
  int ring;           // frames held in shared memory
  int reach;          // frames that cover a sample
  int64_t row_base;   // row r of the padded signal is [r * hop, (r + 1) * hop)
  int64_t rows;       // rows to emit, from row_base on
  int64_t edge;       // rows of the first and of the last segment; 0: as many as the others have
  // first row of segment s, from row_base on
  __host__ __device__ int64_t begin(int64_t s) const {
    if (edge == 0) return rows * s / segments;
    return s == 0 ? 0 : s == segments ? rows : edge + (rows - 2 * edge) * (s - 1) / (segments - 2);
  }
};

// The sum over the frames that cover them of N pairs of samples, 64 apart, of row `row`: pair u of a lane is
// samples j + 64 u and the next one.  kFull: every pair lies in the row and in the frames.
template <int N, bool kFull, bool kNorm>
__device__ __forceinline__ void sum_pairs(const float2* slots, int slot_floats, const float* win, int n_fft, int hop,
                                          int ring, int s, int i_hi, int i_lo, int j, float2 (&v)[N], float2 (&e)[N]) {
#pragma unroll
  for (int u = 0; u < N; ++u) v[u] = e[u] = make_float2(0.f, 0.f);
  s -= i_hi;  // ring slot of frame row - i_hi
  if (s < 0) s += ring;
  for (int i = i_hi; i >= i_lo; --i) {  // in frame order
    const float* y = reinterpret_cast<const float*>(slots) + static_cast<int64_t>(s) * slot_floats + i * hop + j;
    const float* w = win + i * hop + j;
#pragma unroll
    for (int u = 0; u < N; ++u) {
      if (kFull || (j + 64 * u < hop && j + 64 * u + i * hop < n_fft)) {
        const float2 q = *reinterpret_cast<const float2*>(y + 64 * u);
        v[u].x += q.x;
        v[u].y += q.y;
        if (kNorm) {
          const float2 c = *reinterpret_cast<const float2*>(w + 64 * u);
          e[u].x += c.x * c.x;
          e[u].y += c.y * c.y;
        }
      }
    }
    if (++s == ring) s = 0;
  }
}

// Stores the finished sample q of a segment whose edges are folded.  The padded samples left of the signal are
// stored where they will be added, before the row that adds them; those right of it are added to what an earlier
// row stored.  Pass 1 stores, pass 2 adds; both happen within the first or the last segment.
__device__ __forceinline__ void store_folded(const IfftOlaArgs& a, float* out, int64_t q, float v, int pass) {
  const int64_t T = a.out_len;
  const bool waits = q >= T - 1 - a.pad && q <= T - 2;
  if (pass == 1) {
    if (q < 0) out[-q] = v;
    else if (waits) out[q] = v;
  } else if (q >= T) {
    const int64_t m = 2 * T - 2 - q;  // the sample that q is the mirror image of
    if (m >= T - 1 - a.pad && m <= T - 2) out[m] += v;
  } else if (q >= 0 && !waits) {
    out[q] = q >= 1 && q <= a.pad ? v + out[q] : v;
  }
}

// One row of finished samples, by one warp, two samples per lane (hop is even), N pairs of each lane at a time (a
// short hop has fewer: with N = 4 throughout and larger CTAs, n_fft 256 and hop 64 took 226 us instead of 174).
// pass: 0 away from folded edges.
template <int N, bool kNorm>
__device__ __forceinline__ void emit_row_pairs(const IfftOlaArgs& a, const float2* slots, int slot_floats,
                                               const float* win, int ring, int s, int i_hi, int i_lo, int64_t q0,
                                               float* out, int lane, int pass, int part, int parts) {
  const bool paired = pass == 0 && q0 >= 0 && q0 + a.hop <= a.out_len && (reinterpret_cast<uintptr_t>(out + q0) & 7) == 0;
  for (int c = 64 * N * part; c < a.hop; c += 64 * N * parts) {
    const int j = c + 2 * lane;
    float2 v[N], e[N];
    if (c + 64 * N <= a.hop && (i_hi + 1) * a.hop <= a.n_fft)
      sum_pairs<N, true, kNorm>(slots, slot_floats, win, a.n_fft, a.hop, ring, s, i_hi, i_lo, j, v, e);
    else
      sum_pairs<N, false, kNorm>(slots, slot_floats, win, a.n_fft, a.hop, ring, s, i_hi, i_lo, j, v, e);
#pragma unroll
    for (int u = 0; u < N; ++u) {
      if (j + 64 * u >= a.hop) break;
      if (kNorm) {
        v[u].x = e[u].x > 1e-11f ? v[u].x / e[u].x : 0.f;
        v[u].y = e[u].y > 1e-11f ? v[u].y / e[u].y : 0.f;
      }
      const int64_t q = q0 + j + 64 * u;
      if (paired) {
        *reinterpret_cast<float2*>(out + q) = v[u];
      } else if (kNorm || pass == 0) {
        if (q >= 0 && q < a.out_len) out[q] = v[u].x;
        if (q + 1 >= 0 && q + 1 < a.out_len) out[q + 1] = v[u].y;
      } else {
        store_folded(a, out, q, v[u].x, pass);
        store_folded(a, out, q + 1, v[u].y, pass);
      }
    }
  }
}

// Spectrum -> signal.  A CTA owns a run of rows (of `hop` samples), walks the frames that cover it, a batch of
// one frame per lane group at a time, and adds each finished row up from the ring of the last frames in shared
// memory.  Neighbouring CTAs both transform the reach - 1 frames between them; in return the frames stay on
// the chip, which takes 8 * n_fft / hop bytes of traffic off every sample.  Bound by instruction issue, at the
// 16 warps per SM that the ring leaves room for; two CTAs of 8 overlap one's transforms with the other's
// barriers and loads.
// 16 x 1 Mi samples, n_fft 2048, hop 512 (336 MB): 591 us with the frames written to memory and gathered
// by a second kernel, 144 us so.
// 16 x 240007 samples, n_fft 1024, hop 256, bins-major spectrum (77 MB): 247 us, 55 us so.
template <int LH>
__device__ __forceinline__ void ola_rows(const IfftOlaArgs& a, const OlaPlan& pl, const float2* tw, const float2* split, const float* win,
                                         float2* slots, int b, int64_t row0, int64_t row1, int seg) {
  using F = WarpFft<LH, false>;
  const int warp = threadIdx.x >> 5, warps = blockDim.x >> 5, lane = threadIdx.x & 31;
  const int sub = lane / F::L, t = lane % F::L;
  const int batch = warps * F::kPerWarp;             // frames transformed together
  const int64_t f_begin = row0 > pl.reach - 1 ? row0 - (pl.reach - 1) : 0;
  const int64_t f_end = row1 < a.n_frames ? row1 : a.n_frames;
  const float2* spec = reinterpret_cast<const float2*>(a.spec) + b * a.stride_b;
  float* out = a.out + b * a.out_len;
  const int64_t T = a.out_len;
  const bool at_edge = a.fold_reflect && (seg == 0 || seg == pl.segments - 1);
  const bool direct = a.stride_f == 1;

  int64_t f0 = f_begin, e0 = row0;
  int slot0 = 0;                                     // ring slot of frame f0
  for (;;) {
    const int nf = f_end - f0 < batch ? static_cast<int>(f_end - f0) : batch;  // may be <= 0: rows without frames
    if (!direct) {
      // bins of neighbouring frames are (usually) neighbours in memory: lanes run over the frames.  The copies
      // are asynchronous: a batch of spectra is in flight at once without a register held for it.
      const int f = static_cast<int>(threadIdx.x) % batch, step = static_cast<int>(blockDim.x) / batch;
      if (f < nf) {
        const float2* src = spec + (f0 + f) * a.stride_t;
        const int s = slot0 + f;
        float2* slot = slots + (s >= pl.ring ? s - pl.ring : s) * F::kSlot;
        for (int k = static_cast<int>(threadIdx.x) / batch; k <= F::h; k += step) copy_async<8>(slot + k, src + k * a.stride_f);
      }
      copy_async_wait();
      __syncthreads();
    }
    if (warp * F::kPerWarp < nf) {
      const int mine = warp * F::kPerWarp + sub;
      const int s = slot0 + mine;
      float2* slot = slots + (s >= pl.ring ? s - pl.ring : s) * F::kSlot;
      // a group without a frame of its own repeats the last one into a slot that nothing reads
      const int64_t f = f0 + (mine < nf ? mine : nf - 1);
      if (LH >= 10 && direct && f + batch < f_end) {  // bring the next frame's bins as far as L2 meanwhile
        // (n_fft 2048: 164 us without, 157 us with; shorter frames gain nothing)
        const float2* next = spec + (f + batch) * a.stride_t;
        for (int k = 16 * t; k <= F::h; k += 16 * F::L) prefetch_l2(next + k);
      }
      inverse_frame<LH>(a, direct ? spec + f * a.stride_t : nullptr, 1, tw, split,
                        reinterpret_cast<const float2*>(win), slot, t);
    }
    __syncthreads();
    const bool last = f0 + batch >= f_end;
    const int64_t e1 = last ? row1 : f0 + batch;

    const bool folding = at_edge && (e0 * a.hop - a.pad <= a.pad || e1 * a.hop - a.pad >= T - a.pad);
    for (int pass = folding ? 1 : 2; pass <= 2; ++pass) {
      // A warp per row, or, where the passes of a folded edge have few long rows each, per part of a row (2 x 48000 samples,
      // n_fft 4096, backward: 20.8 us with whole rows, 17.3 us so; n_fft 512, hop 128: 0.6 us slower).
      const int log_parts = LH < 10 || !folding || a.hop < 512 ? 0 : a.hop < 1024 ? 1 : 2, parts = 1 << log_parts;
      for (int64_t item = (e0 << log_parts) + warp; item < e1 << log_parts; item += warps) {
        const int64_t row = item >> log_parts;
        const int part = static_cast<int>(item) & (parts - 1);
        const int64_t q0 = row * a.hop - a.pad, q1 = q0 + a.hop;  // its output samples
        const bool folds = folding && (q0 <= a.pad || q1 >= T - a.pad);
        if (pass == 1) {  // rows that hold samples to store for later
          if (q0 >= 0 && (q1 < T - a.pad || q0 > T - 2)) continue;
        } else if (folds && (q1 <= 0 || (q0 >= T - 1 - a.pad && q1 < T))) {
          continue;       // rows that held nothing else
        }
        const int i_lo = row < a.n_frames ? 0
                         : row - a.n_frames + 1 < pl.reach ? static_cast<int>(row - a.n_frames + 1) : pl.reach;
        const int i_hi = row < pl.reach - 1 ? static_cast<int>(row) : pl.reach - 1;
        int s = i_lo < pl.reach ? slot0 + static_cast<int>(row - f0) : 0;  // slot of frame `row`
        if (s >= pl.ring) s -= pl.ring;
        if ((a.hop & 1) == 0) {
          const int p = folds ? pass : 0;
          if (a.normalize_envelope) {
            if (LH <= 8 && a.hop <= 64) emit_row_pairs<1, true>(a, slots, 2 * F::kSlot, win, pl.ring, s, i_hi, i_lo, q0, out, lane, p, part, parts);
            else emit_row_pairs<LH <= 8 ? 2 : 4, true>(a, slots, 2 * F::kSlot, win, pl.ring, s, i_hi, i_lo, q0, out, lane, p, part, parts);
          } else {
            if (LH <= 8 && a.hop <= 64) emit_row_pairs<1, false>(a, slots, 2 * F::kSlot, win, pl.ring, s, i_hi, i_lo, q0, out, lane, p, part, parts);
            else emit_row_pairs<LH <= 8 ? 2 : 4, false>(a, slots, 2 * F::kSlot, win, pl.ring, s, i_hi, i_lo, q0, out, lane, p, part, parts);
          }
          continue;
        }
        for (int j = 32 * part + lane; j < a.hop; j += 32 * parts) {
          float v = 0.f, e = 0.f;
          for (int i = i_hi; i >= i_lo; --i) {       // frame row - i, in frame order
            const int si = s - i < 0 ? s - i + pl.ring : s - i, o = j + i * a.hop;
            if (o < F::n) {
              v += reinterpret_cast<const float*>(slots + si * F::kSlot)[o];
              if (a.normalize_envelope) e += win[o] * win[o];
            }
          }
          if (a.normalize_envelope) v = e > 1e-11f ? v / e : 0.f;
          if (folds) store_folded(a, out, q0 + j, v, pass);
          else if (q0 + j >= 0 && q0 + j < T) out[q0 + j] = v;
        }
      }
      if (pass == 1) __syncthreads();
    }
    if (last) break;
    f0 += batch;
    slot0 += batch;
    if (slot0 >= pl.ring) slot0 -= pl.ring;
    if (e1 > e0) e0 = e1;
    __syncthreads();
  }
}

template <int LH>
__global__ void __launch_bounds__(LH >= 11 ? 256 : 512, 1) ifft_ola_kernel(const IfftOlaArgs a, const OlaPlan pl) {
  using F = WarpFft<LH>;
  extern __shared__ float2 smem[];
  float2* tw = smem;
  float2* split = tw + F::h;
  float* win = reinterpret_cast<float*>(split + F::h / 2);
  float2* slots = reinterpret_cast<float2*>(win + F::n);
  F::fill_tables(tw, split);
  for (int j = threadIdx.x; j < F::n; j += blockDim.x) win[j] = window_at(a.window, j);
  __syncthreads();
  const int b = blockIdx.x / pl.segments, seg = blockIdx.x % pl.segments;
  ola_rows<LH>(a, pl, tw, split, win, slots, b, pl.row_base + pl.begin(seg), pl.row_base + pl.begin(seg + 1), seg);
}

// sum of window^2 over the frames that cover sample j of row `row`
__device__ __forceinline__ float row_envelope(const float* win, int n_fft, int hop, int n_frames, int64_t row, int j) {
  float e = 0.f;
  const int i_hi = row * hop + j < n_fft ? static_cast<int>(row) : (n_fft - 1 - j) / hop;
  for (int i = i_hi; i >= 0; --i)  // frame row - i, in frame order
    if (row - i < n_frames) e += win[j + i * hop] * win[j + i * hop];
  return e;
}

// Spectrum -> signal, frames-major spectra of long signals.  A lane's samples of one frame are its own samples of the next
// frame as well, hop / 2L registers further down (hop is a multiple of 2L).  So a lane group walks a run of frames by itself:
// what later frames will add to stays in its lanes' own places in shared memory, every frame finishes one row, and nothing
// waits for another warp until the end, when each group adds what it has left to the rows that the next one opened.  Only
// the first group of a CTA repeats the reach - 1 frames before its rows.
// pl.edge rows at a folded end are left to ola_rows in the first and the last CTA of a batch entry.
template <int LH, bool kNorm>
__global__ void __launch_bounds__(512, 1) ifft_stream_kernel(IfftOlaArgs a, const OlaPlan pl) {
  using F = WarpFft<LH>;
  extern __shared__ float2 smem[];
  float2* tw = smem;
  float2* split = tw + F::h;
  float* win = reinterpret_cast<float*>(split + F::h / 2);
  float* env = win + F::n;  // of a row that a full set of frames covers
  float2* slots = reinterpret_cast<float2*>(env + (kNorm ? a.hop : 0));
  F::fill_tables(tw, split);
  for (int j = threadIdx.x; j < F::n; j += blockDim.x) win[j] = window_at(a.window, j);
  __syncthreads();
  const float edge = a.hermitian ? 1.0f : 2.0f, post = a.hermitian ? a.scale : 0.5f * a.scale;
  if (!kNorm) {  // the window serves nothing else: it takes the scale
    for (int j = threadIdx.x; j < F::n; j += blockDim.x) win[j] *= post;
    a.scale = a.hermitian ? 1.0f : 2.0f;
    __syncthreads();
  }
  if (kNorm) {
    for (int j = threadIdx.x; j < a.hop; j += blockDim.x)
      env[j] = row_envelope(win, F::n, a.hop, a.n_frames, pl.reach - 1, j);
    __syncthreads();
  }
  const int b = blockIdx.x / pl.segments, seg = blockIdx.x % pl.segments;
  int64_t r0 = pl.row_base + pl.rows * seg / pl.segments, r1 = pl.row_base + pl.rows * (seg + 1) / pl.segments;
  if (pl.edge > 0 && seg == 0) {
    ola_rows<LH>(a, pl, tw, split, win, slots, b, r0, r0 + pl.edge, seg);
    r0 += pl.edge;
    __syncthreads();
  }
  if (pl.edge > 0 && seg == pl.segments - 1) r1 -= pl.edge;

  const int warp = threadIdx.x >> 5, warps = blockDim.x >> 5, lane = threadIdx.x & 31;
  const int t = lane % F::L, group = warp * F::kPerWarp + lane / F::L, groups = warps * F::kPerWarp;
  const int done = a.hop / (2 * F::L), kept = F::V - done;  // registers of a lane that a frame finishes, and leaves open
  float* buf = reinterpret_cast<float*>(slots) + group * F::kHalfSlot;
  float2* open = reinterpret_cast<float2*>(reinterpret_cast<float*>(slots) + groups * F::kHalfSlot) + group * kept * F::L + t;
  const int warm = r0 < pl.reach - 1 ? static_cast<int>(r0) : pl.reach - 1;
  const int steps = static_cast<int>(r1 - r0) + warm, each = (steps + groups - 1) / groups;
  const int64_t first = r0 - warm + static_cast<int64_t>(group) * each;
  const int count = max(0, min(each, steps - group * each));
  const float2* spec = reinterpret_cast<const float2*>(a.spec) + b * a.stride_b;
  float* out = a.out + b * a.out_len;
  const float2* win2 = reinterpret_cast<const float2*>(win) + t;
  // One pair of finished samples; `raw`: another group has more to add.
  auto put = [&](int64_t row, int64_t q0, int j, float2 v, bool raw) {
    if (kNorm && !raw) {
      const bool full = row >= pl.reach - 1 && row < a.n_frames;
      const float2 e = full ? *reinterpret_cast<const float2*>(env + j)
                            : make_float2(row_envelope(win, F::n, a.hop, a.n_frames, row, j),
                                          row_envelope(win, F::n, a.hop, a.n_frames, row, j + 1));
      v.x = e.x > 1e-11f ? v.x / e.x : 0.f;
      v.y = e.y > 1e-11f ? v.y / e.y : 0.f;
    }
    const int64_t q = q0 + j;
    if (q >= 0 && q + 1 < a.out_len && (reinterpret_cast<uintptr_t>(out + q) & 7) == 0) {
      *reinterpret_cast<float2*>(out + q) = v;
    } else {
      if (q >= 0 && q < a.out_len) out[q] = v.x;
      if (q + 1 >= 0 && q + 1 < a.out_len) out[q + 1] = v.y;
    }
  };
  for (int r = 0; r < kept; ++r) open[r * F::L] = make_float2(0.f, 0.f);
#pragma unroll 1
  for (int i = 0; i < each; ++i) {
    const int64_t row = first + i;
    const bool live = i < count, framed = live && row < a.n_frames;
    float2 x[F::V];
    if (__any_sync(0xFFFFFFFFu, framed)) {
      const float2* from = spec + (framed ? row : a.n_frames - 1) * a.stride_t;
#pragma unroll
      for (int r = 0; r < F::V; ++r) x[r] = from[r * F::L + t];
      const float2 nyquist = from[F::h];
      if (LH >= 10 && i + 1 < count && row + 1 < a.n_frames)
        for (int k = 16 * t; k <= F::h; k += 16 * F::L) prefetch_l2(from + a.stride_t + k);
      F::merge_bins(x, nyquist, split, t, edge);
      F::transform_halves(x, tw, buf, t);
    }
    const int64_t q0 = row * a.hop - a.pad;
    const bool emits = live && row >= r0;
    // a whole row of aligned pairs with nothing more to come and (kNorm) a full set of frames; others go through `put`
    const bool plain = emits && q0 >= 0 && q0 + a.hop <= a.out_len && (reinterpret_cast<uintptr_t>(out + q0) & 7) == 0 &&
                       (group == 0 || i * done >= kept) && (!kNorm || (row >= pl.reach - 1 && row < a.n_frames));
    float2* to = reinterpret_cast<float2*>(out + q0) + t;
    float2* later = reinterpret_cast<float2*>(buf) + t;
    const float2* before = open;
    if (!framed) {
#pragma unroll
      for (int r = 0; r < F::V; ++r) x[r] = make_float2(0.f, 0.f);
    }
    static_for<0, F::V>([&](auto rc) {
      constexpr int r = decltype(rc)::value, g = r % F::G, k2 = r / F::G;
      const float2 z = x[F::at(g, k2)], w = win2[r * F::L];
      float2 y = kNorm ? make_float2(z.y * post * w.x, z.x * post * w.y) : make_float2(z.y * w.x, z.x * w.y);
      if (r < F::V / 2 || r < kept) {  // at the first frame the open places hold zeros
        const float2 sum = before[r * F::L];
        y = add2<true>(sum, y);
      }
      if (r < F::V / 2 && r < done) {
        if (plain) {
          if (kNorm) {
            const float2 e = reinterpret_cast<const float2*>(env)[r * F::L + t];
            y = make_float2(e.x > 1e-11f ? y.x / e.x : 0.f, e.y > 1e-11f ? y.y / e.y : 0.f);
          }
          to[r * F::L] = y;
        } else {
          later[r * F::L] = y;
        }
      } else if (live) {
        open[(r - done) * F::L] = y;
      }
    });
    if (emits && !plain)
#pragma unroll 1
      for (int r = 0; r < done; ++r) put(row, q0, 2 * (r * F::L + t), later[r * F::L], group > 0 && i * done + r < kept);
  }
  __syncthreads();
  // what this group's frames add to the rows that the next group has opened
  if (count == each && first + each < r1) {
    int64_t row = first + each;
    int at = 0;
#pragma unroll 1
    for (int r = 0; r < kept && row < r1; ++r) {
      const int64_t q0 = row * a.hop - a.pad;
      const int j = 2 * (at * F::L + t);
      const int64_t q = q0 + j;
      float2 v = open[r * F::L];
      if (q >= 0 && q < a.out_len) v.x += out[q];
      if (q + 1 >= 0 && q + 1 < a.out_len) v.y += out[q + 1];
      put(row, q0, j, v, false);
      if (++at == done) at = 0, ++row;
    }
  }
  if (pl.edge > 0 && seg == pl.segments - 1) {
    __syncthreads();
    ola_rows<LH>(a, pl, tw, split, win, slots, b, r1, r1 + pl.edge, seg);
  }
}

// Spectrum -> windowed frames in global memory (only where ifft_ola_kernel cannot run).
template <int LH>
__global__ void __launch_bounds__(256, LH <= 8 ? 3 : LH <= 10 ? 2 : 1)
    ifft_frames_kernel(const IfftOlaArgs a, float* frames, int64_t total) {
  using F = WarpFft<LH>;
  extern __shared__ float2 smem[];
  float2* tw = smem;
  float2* split = tw + F::h;
  float* win = reinterpret_cast<float*>(split + F::h / 2);
  float2* slots = reinterpret_cast<float2*>(win + F::n);
  F::fill_tables(tw, split);
  for (int j = threadIdx.x; j < F::n; j += blockDim.x) win[j] = window_at(a.window, j);
  __syncthreads();
  const int warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int sub = (threadIdx.x & 31) / F::L, t = threadIdx.x % F::L;
  float2* slot = slots + (warp * F::kPerWarp + sub) * F::kSlot;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * warps * F::kPerWarp;
  for (int64_t i0 = (static_cast<int64_t>(blockIdx.x) * warps + warp) * F::kPerWarp; i0 < total; i0 += stride) {
    const int64_t i = i0 + sub < total ? i0 + sub : total - 1;
    const int64_t b = i / a.n_frames, f = i - b * a.n_frames;
    const float2* spec = reinterpret_cast<const float2*>(a.spec) + b * a.stride_b + f * a.stride_t;
    inverse_frame<LH>(a, spec, a.stride_f, tw, split, reinterpret_cast<const float2*>(win), slot, t);
    __syncwarp();
    if (i0 + sub < total) {
      float2* dst = reinterpret_cast<float2*>(frames + i * F::n);
      for (int m = t; m < F::h; m += F::L) dst[m] = slot[m];
    }
    __syncwarp();
  }
}

__device__ __forceinline__ float ola_at(const float* frames, int64_t p, int n_fft, int hop, int n_frames) {
  if (p < 0) return 0.f;
  int64_t f_hi = p / hop;
  if (f_hi > n_frames - 1) f_hi = n_frames - 1;
  int64_t f_lo = p - n_fft + 1 <= 0 ? 0 : (p - n_fft + hop) / hop;
  float acc = 0.f;
  for (int64_t f = f_lo; f <= f_hi; ++f) {
    const int64_t n = p - f * hop;
    if (n >= 0 && n < n_fft) acc += frames[f * n_fft + n];
  }
  return acc;
}

__global__ void __launch_bounds__(256) ola_gather_kernel(const IfftOlaArgs a, const float* all_frames) {
  const int b = blockIdx.y;
  const float* frames = all_frames + static_cast<int64_t>(b) * a.n_frames * a.n_fft;
  float* out = a.out + static_cast<int64_t>(b) * a.out_len;
  const int64_t T = a.out_len;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; t < T; t += stride) {
    const int64_t p = t + a.pad;
    float v = ola_at(frames, p, a.n_fft, a.hop, a.n_frames);
    if (a.fold_reflect && a.pad > 0) {
      // adjoint of reflect padding: padded[pad - i] and padded[pad + 2T - 2 - i] also came from x[i]
      if (t >= 1 && t <= a.pad) v += ola_at(frames, a.pad - t, a.n_fft, a.hop, a.n_frames);
      if (t <= T - 2 && t >= T - 1 - a.pad) v += ola_at(frames, a.pad + 2 * T - 2 - t, a.n_fft, a.hop, a.n_frames);
    }
    if (a.normalize_envelope) {
      const float e = envelope_at(a.window, p, a.n_fft, a.hop, a.n_frames);
      v = e > 1e-11f ? v / e : 0.f;
    }
    out[t] = v;
  }
}

int ilog2(int n) {
  int l = 0;
  while ((1 << l) < n) ++l;
  return l;
}

bool valid_nfft(int n) { return n >= 8 && n <= kStftMaxNfft && (n & (n - 1)) == 0; }

// Dynamic shared memory above 48 KB has to be asked for, once per kernel and device.
cudaError_t allow_smem(const void* kernel, std::atomic<uint64_t>& done) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const uint64_t bit = uint64_t(1) << (dev & 63);
  if (dev < 64 && (done.load(std::memory_order_acquire) & bit)) return cudaSuccess;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kMaxSmem));
  if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_release);
  return e;
}

template <int LH>
size_t table_bytes() { return WarpFft<LH>::kTables * sizeof(float2) + WarpFft<LH>::n * sizeof(float); }

// Warps per CTA and grid of the frame-parallel kernels: as many resident CTAs as fit, each looping over
// frames; calls too small for that spread over the SMs in CTAs of at least four warps, which share the work
// of filling the tables.
struct FrameGrid {
  unsigned ctas;
  int threads;
  size_t smem;
};
template <int LH>
FrameGrid frame_grid(int64_t total, size_t extra) {
  using F = WarpFft<LH>;
  const int64_t warps_wanted = (total + F::kPerWarp - 1) / F::kPerWarp;
  const int warps = static_cast<int>(std::min<int64_t>(8, std::max<int64_t>(4, (warps_wanted + kSms - 1) / kSms)));
  FrameGrid g;
  g.threads = 32 * warps;
  g.smem = table_bytes<LH>() + extra + static_cast<size_t>(warps) * F::kPerWarp * F::kSlot * sizeof(float2);
  const int by_regs = LH <= 6 ? 4 : LH <= 8 ? 3 : LH <= 10 ? 2 : 1;
  const int resident = static_cast<int>(std::min<size_t>(by_regs, kMaxSmem / (g.smem + 1024)));
  g.ctas = static_cast<unsigned>(std::min<int64_t>((warps_wanted + warps - 1) / warps, kSms * std::max(1, resident)));
  return g;
}

template <int LH, bool kEnvelope>
cudaError_t run_fft_frames(const FftFramesArgs& a, cudaStream_t s) {
  static std::atomic<uint64_t> smem_set{0};
  const void* fn = reinterpret_cast<const void*>(fft_frames_kernel<LH, kEnvelope>);
  cudaError_t e = allow_smem(fn, smem_set);
  if (e != cudaSuccess) return e;
  const int64_t total = static_cast<int64_t>(a.batch) * a.n_frames;
  const FrameGrid g = frame_grid<LH>(total, kEnvelope ? WarpFft<LH>::n * sizeof(float) : 0);
  fft_frames_kernel<LH, kEnvelope><<<g.ctas, g.threads, g.smem, s>>>(a, total);
  return cudaGetLastError();
}

template <int LH>
cudaError_t run_ifft_frames(const IfftOlaArgs& a, float* frames, cudaStream_t s) {
  static std::atomic<uint64_t> smem_set{0};
  const void* fn = reinterpret_cast<const void*>(ifft_frames_kernel<LH>);
  cudaError_t e = allow_smem(fn, smem_set);
  if (e != cudaSuccess) return e;
  const int64_t total = static_cast<int64_t>(a.batch) * a.n_frames;
  const FrameGrid g = frame_grid<LH>(total, 0);
  ifft_frames_kernel<LH><<<g.ctas, g.threads, g.smem, s>>>(a, frames, total);
  return cudaGetLastError();
}

// Geometry of the fused inverse: the first choice whose frames, with the reach - 1 frames before them, fit
// shared memory.  threads == 0: this problem takes the two-kernel path,
// because a batch would be shorter than the overlap (tiny hops: neighbours would mostly repeat each other's
// frames) or because the signal is so short that the two folded edges meet.
struct OlaGrid {
  OlaPlan plan;
  int batch = 0;      // frames transformed together
  int64_t most = 0;   // segments of one batch entry that are resident together
  int resident = 1;   // CTAs per SM
  int threads = 0;
  size_t smem = 0;
};
template <int LH>
OlaGrid ola_grid(const IfftOlaArgs& a) {
  using F = WarpFft<LH>;
  OlaGrid g;
  OlaPlan& pl = g.plan;
  const bool fold = a.fold_reflect != 0;
  const int64_t reach = (static_cast<int64_t>(F::n) + a.hop - 1) / a.hop;
  if ((fold && a.out_len < F::n + 2) || a.hop > (1 << 24)) return g;
  const int64_t end = a.out_len + a.pad + (fold ? a.pad : 0);
  pl.row_base = fold ? 0 : a.pad / a.hop;
  pl.rows = (end + a.hop - 1) / a.hop - pl.row_base;
  pl.reach = static_cast<int>(reach);
  // {warps, CTAs per SM}.  Several small CTAs before one of 16 warps, that before whatever fits: the phases of one
  // overlap with another's.  Frames of up to 512 samples (several per warp) do best with four of 4 warps; for 1024
  // three of 5 repeat too many frames at the segments' ends (160 us against 137 us for 16 x 1 Mi samples).
  static const int kChoices[][2] = {{LH <= 8 ? 4 : 8, LH <= 8 ? 4 : 2}, {8, 2}, {16, 1}, {8, 1}, {4, 1}};
  for (const auto& choice : kChoices) {
    const int warps = choice[0];
    int resident = choice[1];
    if (LH >= 11 && warps * resident > 8) continue;  // 255 registers
    const int64_t batch = warps * F::kPerWarp;
    const int64_t ring = batch + reach - 1;
    const size_t smem = table_bytes<LH>() + static_cast<size_t>(ring) * F::kSlot * sizeof(float2);
    if (batch < reach || resident * (smem + 1024) > kSmemPerSm) continue;
    // As many segments as are resident together; where one batch of frames is enough for each, no more than it takes, but none
    // with a second batch for a row or two too many.  (2 x 48000 samples, n_fft 2048: 18 segments of 5 and 6 rows, the longer
    // ones in two batches: backward 12.3, inverse 13.3 us; none above 5 rows: 10.9 and 8.8 us.  With more rounds the last,
    // short one costs less than segments of full batches would: 8 x 200000 samples, n_fft 1024: 18.5 and 20.6 us.)
    const int64_t most = std::max<int64_t>(1, static_cast<int64_t>(kSms) * resident / a.batch);
    const int64_t rounds = (((pl.rows + most - 1) / most) + (reach - 1) + batch - 1) / batch;
    const int64_t longest = rounds * batch - (reach - 1);
    int64_t segments = rounds == 1 ? (pl.rows + longest - 1) / longest : most;
    // a folded edge lies within one segment: reach + 1 rows are enough for either, and the first and the last segment have
    // no frames before or behind them to repeat
    const int64_t edge = reach + 1;
    pl.edge = 0;
    if (fold && segments > 1 && pl.rows / segments < edge) {
      if (pl.rows > 2 * edge) pl.edge = edge;
      segments = pl.edge > 0 ? 2 + (pl.rows - 2 * edge + longest - 1) / longest : 1;
    }
    if (segments * a.batch > 0x7FFFFFFF) continue;
    g.batch = static_cast<int>(batch);
    g.most = most;
    g.resident = resident;
    pl.segments = static_cast<int>(segments);
    pl.ring = static_cast<int>(ring);
    g.threads = 32 * warps;
    g.smem = smem;
    break;
  }
  return g;
}

// What the stream kernel takes for a frame of every lane group and around them, and what ola_rows takes for a batch of frames of up to
// two, four and more frames per sample, in tenths of a microsecond; [0] the adjoint, [1] the inverse with its division.  Fitted to 970
// pairs of times: hop n_fft / 8, / 4, 5 / 16 and / 2, 1 to 200 signals of 64 Ki to 1 Mi samples (B200).
struct StreamCosts {
  int frame[2], ends[2], batch[2][3];
};
constexpr int kBatchEnds = 140;
constexpr StreamCosts stream_costs(int lh) {
  return lh <= 6   ? StreamCosts{{18, 20}, {200, 170}, {{40, 48, 61}, {42, 50, 63}}}
         : lh == 7 ? StreamCosts{{33, 36}, {240, 240}, {{56, 53, 73}, {61, 55, 76}}}
         : lh == 8 ? StreamCosts{{29, 34}, {260, 240}, {{46, 40, 39}, {51, 43, 41}}}
                   : StreamCosts{{59, 77}, {470, 360}, {{86, 85, 87}, {98, 94, 94}}};
}

// The stream kernel's geometry; threads == 0: not for this problem.  It wants runs of frames that are long against what two
// neighbours share, and its CTAs, one per SM and in whole numbers per signal, to fill the device about as well as the batch kernel's.
template <int LH>
OlaGrid stream_grid(const IfftOlaArgs& a) {
  using F = WarpFft<LH>;
  OlaGrid g;
  if (LH < 6 || a.stride_f != 1 || a.hop % (2 * F::L) != 0 || a.hop > F::n / 2) return g;
  const OlaGrid rows = ola_grid<LH>(a);
  if (rows.threads == 0) return g;
  const bool fold = a.fold_reflect != 0;
  // 16 x 1 Mi samples, hop n_fft / 4, backward, batches and streams: n_fft 256 166 and 121 us, 512 131 and 110, 2048 144 and
  // 136 (inverse 156 and 152); but 1024 133 and 145, 4096 185 and 218: two frames per warp in 128 registers, and half the warps
  if (LH == 9 || LH == 11) return g;
  constexpr int warps = 16, groups = warps * F::kPerWarp;
  g.plan = rows.plan;
  OlaPlan& pl = g.plan;
  pl.edge = fold ? pl.reach + 1 : 0;
  pl.ring = groups + pl.reach - 1;
  const int64_t most = std::max<int64_t>(1, kSms / a.batch);
  const int64_t least = 3ll * (pl.reach - 1) * groups + 2 * pl.edge;  // rows of a CTA
  pl.segments = static_cast<int>(std::min<int64_t>(most, pl.rows / std::max<int64_t>(1, least)));
  if (pl.segments < 1 || (pl.segments < most && static_cast<int64_t>(pl.segments) * a.batch < kSms * 3 / 4)) return g;
  // Frames of the busiest lane group against batches of the busiest CTA, each as often as its CTAs need turns on the device.  Of those
  // 970 pairs the streams, wherever signals were long, were 4 % or more behind in 186; so in none, and left out where they are as
  // much ahead in 17.  Us in batches and streams, 80 x 1 Mi samples, 512, hop 128, backward: 612 and 748, on 80 SMs; 32 x 256 Ki, 2048,
  // 1024: 52 and 65; but 32 x 1 Mi, 512, 128: 250 and 211; 120 x 1 Mi, 2048, 512: 1110 and 788; 80 x 1 Mi, 128, 16: 3591 and 1731.
  constexpr StreamCosts costs = stream_costs(LH);
  const int kind = a.normalize_envelope ? 1 : 0;
  auto ceil_div = [](int64_t x, int64_t y) { return (x + y - 1) / y; };
  auto longest = [&](int64_t segments, int64_t together) { return ceil_div(ceil_div(pl.rows, segments) + pl.reach - 1, together); };
  const int64_t turns = ceil_div(static_cast<int64_t>(pl.segments) * a.batch, kSms);
  const int64_t row_turns = ceil_div(static_cast<int64_t>(rows.plan.segments) * a.batch, static_cast<int64_t>(kSms) * rows.resident);
  int batch_cost = costs.batch[kind][pl.reach <= 2 ? 0 : pl.reach <= 4 ? 1 : 2];
  if (F::n % a.hop != 0) batch_cost = batch_cost * 9 / 8;
  if (turns * (longest(pl.segments, groups) * costs.frame[kind] + costs.ends[kind]) >
      row_turns * (longest(rows.plan.segments, rows.batch) * batch_cost + kBatchEnds))
    return g;
  const size_t kept = F::V - a.hop / (2 * F::L);
  const size_t stream = groups * (F::kHalfSlot * sizeof(float) + kept * F::L * sizeof(float2)) +
                        (a.normalize_envelope ? a.hop * sizeof(float) : 0);
  const size_t edges = fold ? static_cast<size_t>(pl.ring) * F::kSlot * sizeof(float2) : 0;
  g.smem = table_bytes<LH>() + std::max(stream, edges);
  if (g.smem > kMaxSmem) return g;
  g.threads = 32 * warps;
  return g;
}

template <int LH>
cudaError_t run_ifft_stream(const IfftOlaArgs& a, const OlaGrid& g, cudaStream_t s) {
  static std::atomic<uint64_t> smem_set[2] = {};
  const int norm = a.normalize_envelope ? 1 : 0;
  const auto kernel = norm ? ifft_stream_kernel<LH, true> : ifft_stream_kernel<LH, false>;
  cudaError_t e = allow_smem(reinterpret_cast<const void*>(kernel), smem_set[norm]);
  if (e != cudaSuccess) return e;
  kernel<<<static_cast<unsigned>(g.plan.segments) * a.batch, g.threads, g.smem, s>>>(a, g.plan);
  return cudaGetLastError();
}

template <int LH>
cudaError_t run_ifft_ola(const IfftOlaArgs& a, const OlaGrid& g, cudaStream_t s) {
  static std::atomic<uint64_t> smem_set{0};
  const void* fn = reinterpret_cast<const void*>(ifft_ola_kernel<LH>);
  cudaError_t e = allow_smem(fn, smem_set);
  if (e != cudaSuccess) return e;
  ifft_ola_kernel<LH><<<static_cast<unsigned>(g.plan.segments) * a.batch, g.threads, g.smem, s>>>(a, g.plan);
  return cudaGetLastError();
}

// Calls f(std::integral_constant<int, log2(n_fft / 2)>).
template <typename R, typename Fn>
R for_size(int n_fft, Fn&& f) {
  switch (ilog2(n_fft / 2)) {
    case 2: return f(std::integral_constant<int, 2>{});
    case 3: return f(std::integral_constant<int, 3>{});
    case 4: return f(std::integral_constant<int, 4>{});
    case 5: return f(std::integral_constant<int, 5>{});
    case 6: return f(std::integral_constant<int, 6>{});
    case 7: return f(std::integral_constant<int, 7>{});
    case 8: return f(std::integral_constant<int, 8>{});
    case 9: return f(std::integral_constant<int, 9>{});
    case 10: return f(std::integral_constant<int, 10>{});
    default: return f(std::integral_constant<int, 11>{});
  }
}

OlaGrid ola_grid_for(const IfftOlaArgs& a) {
  return for_size<OlaGrid>(a.n_fft, [&](auto lh) { return ola_grid<decltype(lh)::value>(a); });
}
OlaGrid stream_grid_for(const IfftOlaArgs& a) {
  return for_size<OlaGrid>(a.n_fft, [&](auto lh) { return stream_grid<decltype(lh)::value>(a); });
}

bool valid(const IfftOlaArgs& a) {
  return valid_nfft(a.n_fft) && a.batch > 0 && a.n_frames > 0 && a.hop > 0 && a.out_len > 0;
}

}  // namespace

cudaError_t launch_fft_frames(const FftFramesArgs& a, cudaStream_t s) {
  if (!valid_nfft(a.n_fft) || a.batch <= 0 || a.n_frames <= 0) return cudaErrorInvalidValue;
  note_launch();
  return for_size<cudaError_t>(a.n_fft, [&](auto lh) {
    return a.divide_envelope ? run_fft_frames<decltype(lh)::value, true>(a, s)
                             : run_fft_frames<decltype(lh)::value, false>(a, s);
  });
}

OlaShape ifft_ola_shape(const IfftOlaArgs& a) {
  OlaShape shape{};
  if (!valid(a)) return shape;
  const OlaGrid g = ola_grid_for(a);
  if (g.threads == 0) return shape;
  shape.reach = g.plan.reach;
  shape.batch = g.batch;
  shape.most = g.most;
  for (int s = 0; s <= g.plan.segments; ++s) shape.begins.push_back(g.plan.row_base + g.plan.begin(s));
  return shape;
}

int64_t ifft_ola_scratch(const IfftOlaArgs& a) {
  if (!valid(a) || ola_grid_for(a).threads > 0) return 0;
  return static_cast<int64_t>(a.batch) * a.n_frames * a.n_fft;
}

bool ifft_ola_streams(const IfftOlaArgs& a) { return valid(a) && stream_grid_for(a).threads > 0; }

cudaError_t launch_ifft_ola(const IfftOlaArgs& a, float* scratch, cudaStream_t s) {
  if (!valid(a)) return cudaErrorInvalidValue;
  const OlaGrid stream = stream_grid_for(a);
  if (stream.threads > 0) {
    note_launch();
    return for_size<cudaError_t>(a.n_fft, [&](auto lh) -> cudaError_t {
      if constexpr (decltype(lh)::value >= 6 && decltype(lh)::value != 9 && decltype(lh)::value != 11) return run_ifft_stream<decltype(lh)::value>(a, stream, s);
      return cudaErrorInvalidValue;
    });
  }
  const OlaGrid g = ola_grid_for(a);
  if (g.threads > 0) {
    note_launch();
    return for_size<cudaError_t>(a.n_fft, [&](auto lh) { return run_ifft_ola<decltype(lh)::value>(a, g, s); });
  }
  note_launch(2);
  cudaError_t e =
      for_size<cudaError_t>(a.n_fft, [&](auto lh) { return run_ifft_frames<decltype(lh)::value>(a, scratch, s); });
  if (e != cudaSuccess) return e;
  const int64_t blocks = std::min<int64_t>((a.out_len + 255) / 256, kSms * 8);
  ola_gather_kernel<<<dim3(static_cast<unsigned>(blocks), a.batch), 256, 0, s>>>(a, scratch);
  return cudaGetLastError();
}

}  // namespace kern
}  // namespace mccl
