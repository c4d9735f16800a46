// Launchers of the fp32 matrix products on the tensor cores (plain C++ header).
//
// A product is two launches on one stream: split_f32 cuts its smaller operand (or both) into the bf16 parts that the tensor
// cores read, laid out as the product's stages, and gemm_f32 multiplies.  The images and the partial sums live in one
// scratch that the caller provides.
#pragma once

#include <cuda_runtime_api.h>

#include <cstdint>

namespace mccl {
namespace kern {

// A row-major matrix of fp32 numbers, `ld` numbers from one row to the next.
struct MatrixF32 {
  const float* data;
  int64_t ld, rows, cols;
};

// How one product c[j, i] = sum over k of a(i, k) b(j, k) is cut: tiles of 128 by `cols`, the reduction in stages of 32, a
// tile's stages over `splits` CTAs.
struct GemmPlan {
  int64_t rows_i, rows_j, depth;
  int cols;
  int tiles_i, tiles_j;
  int stages, per_split, splits;
  int64_t a_image, b_image;  // bytes; a_image 0: a is read as it is
  int64_t partial;           // bytes of partial sums, and of tickets
  int64_t tickets;
};
// kForward: c = x w^T (+ bias): i, j, k = out features, rows of x, in features.  kInput: c = g w.  kWeight: c = g^T x.
enum class Product { kForward, kInput, kWeight };
GemmPlan gemm_plan(Product p, int64_t batch, int64_t in, int64_t out);
// Whether the product is worth its launches, against the library's fp32 kernels.
bool gemm_pays(Product p, int64_t batch, int64_t in, int64_t out);

// Cuts `m` into an image whose k is m's columns (`by_cols`, tiles of `tile` rows) and/or one whose k is m's rows
// (`by_rows`, tiles of 128 columns); either may be null.
struct SplitJob {
  MatrixF32 m;
  void* by_cols;
  int tile;
  void* by_rows;
};
// Up to two matrices in one launch: the first is the products' `b` (cut at half its value), the second an `a`; column sums of
// the first to `sums` unless null; `zeroed` 32-bit words set to zero.
cudaError_t launch_split_f32(const SplitJob* jobs, int n, float* sums, uint32_t* zero, int64_t zeroed, cudaStream_t s);

// `weight`: fp32, of kForward and kInput; kWeight reads a_image in its place.  `c`: rows of ldc numbers.
struct GemmArgs {
  Product product;
  GemmPlan plan;
  const float* weight;
  int64_t ldw;
  const void *a_image, *b_image;
  const float* bias;
  float* c;
  int64_t ldc;
  float* partial;
  uint32_t* tickets;
  uint32_t* failed;     // set to 1 where a wait runs out, whose tiles then are NaN; or null
  int64_t wait_limit;   // cycles of a quarter of a wait; negative: about a second in all
};
cudaError_t launch_gemm_f32(const GemmArgs& g, cudaStream_t s);

}  // namespace kern
}  // namespace mccl
