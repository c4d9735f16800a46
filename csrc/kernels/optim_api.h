// Launcher of the fused multi-tensor AdamW kernel (plain C++ header).
#pragma once

#include <cuda_runtime_api.h>
#include <vector_types.h>

#include <cstdint>

namespace mccl {
namespace kern {

// Elements handled by one CTA: 256 threads, four 16-byte vectors of each array, two of them in flight together.
// (Chunks of 16384 with one vector in flight: 85 M parameters 385 us, 6.17 TB/s; so: 362 us, 6.56 TB/s, and a
// small model spreads over four times as many SMs.)
constexpr int kAdamWChunk = 4096;

// All pointers are device pointers; arrays are indexed by tensor id.
struct AdamWTable {
  const uint64_t* params;      // float* per tensor
  const uint64_t* grads;       // const float* per tensor
  const uint64_t* exp_avg;     // float* per tensor
  const uint64_t* exp_avg_sq;  // float* per tensor
  const int64_t* sizes;        // elements per tensor
  const int2* chunks;          // per CTA: {tensor id, chunk index}
  int num_chunks;
};

struct AdamWHyper {
  float lr;
  float beta1, beta2;
  float eps;
  float weight_decay;
  float step_size;       // lr / (1 - beta1^t)
  float inv_sqrt_bias2;  // 1 / sqrt(1 - beta2^t)
  float grad_scale;      // multiplied into every gradient first
};

// `max_ctas` > 0 caps the grid (each CTA then walks several chunks): a step that runs beside other
// kernels (a bucket's update during backward) can be kept to a share of the SMs and of HBM bandwidth.
cudaError_t launch_adamw_multi(const AdamWTable& tab, const AdamWHyper& h, cudaStream_t s, int max_ctas = 0);

}  // namespace kern
}  // namespace mccl
