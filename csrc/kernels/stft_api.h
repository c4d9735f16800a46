// Launchers of the STFT / iSTFT kernels (plain C++ header).
//
// Frames -> spectrum (fft_frames): a group of lanes per (batch, frame) loads n_fft samples (reflect
//     padding or an envelope division fused into the load), multiplies by the window, transforms in
//     registers and writes the n_fft/2+1 one-sided bins.
// Spectrum -> signal (ifft_ola): a CTA owns a run of output samples, inverse-transforms every frame
//     that covers it into shared memory and adds the overlapping frames up from there, in frame
//     order: the frames never travel to global memory.  It either folds the reflect padding back
//     (STFT backward) or divides by the window envelope and trims (iSTFT forward).
// Where the overlapping frames of a sample do not fit shared memory (very small hops) or the signal
// is so short that both folded edges meet, ifft_frames writes the windowed frames to a buffer and
// ola_gather adds them up without atomics.
#pragma once

#include <cuda_runtime_api.h>

#include <cstdint>
#include <vector>

namespace mccl {
namespace kern {

constexpr int kStftMaxNfft = 4096;

// A window of `len` samples centred (from `left` on) in n_fft zeros.
struct StftWindow {
  const float* data;
  int len, left;
};

struct FftFramesArgs {
  const float* signal;   // [batch, signal_len]
  int64_t signal_len;
  StftWindow window;
  float* out;            // [batch, n_frames, n_fft/2+1] interleaved complex
  int batch, n_frames, n_fft, hop;
  int pad;               // frame f starts at f*hop - pad in signal coordinates
  int reflect;           // 1: indices outside [0, signal_len) are reflected once; 0: they read as zero
  int divide_envelope;   // 1 (iSTFT backward): each sample is divided by the window-square envelope first, and
                         // bins 1..n_fft/2-1 are doubled, DC and Nyquist made real
  float scale;           // multiplied into every bin
};

struct IfftOlaArgs {
  const float* spec;     // complex, addressed with the strides below (in complex elements)
  int64_t stride_b, stride_f, stride_t;
  StftWindow window;
  float* out;            // [batch, out_len]
  int64_t out_len;
  int batch, n_frames, n_fft, hop;
  int hermitian;         // 1: inverse real FFT (mirror bins); 0: upper bins are zero (adjoint of forward)
  float scale;
  int pad;               // output sample t corresponds to padded position t + pad
  int fold_reflect;      // 1: add the mirrored padded regions back (adjoint of reflect padding)
  int normalize_envelope;// 1: divide by sum of window^2 over the covering frames
};

cudaError_t launch_fft_frames(const FftFramesArgs& a, cudaStream_t s);
// Floats of scratch that launch_ifft_ola needs for this problem (0: it runs as one fused kernel).
int64_t ifft_ola_scratch(const IfftOlaArgs& a);
// How the fused kernel cuts one batch entry into rows of `hop` samples (host arithmetic only; for the tests).
struct OlaShape {
  int reach, batch;             // frames that cover a sample; frames that a CTA transforms together
  int64_t most;                 // segments that are resident together
  std::vector<int64_t> begins;  // first row of every segment, and the end; empty where it cannot run
};
OlaShape ifft_ola_shape(const IfftOlaArgs& a);
// Whether launch_ifft_ola walks the frames in streams (host arithmetic only).
bool ifft_ola_streams(const IfftOlaArgs& a);
cudaError_t launch_ifft_ola(const IfftOlaArgs& a, float* scratch, cudaStream_t s);

}  // namespace kern
}  // namespace mccl
