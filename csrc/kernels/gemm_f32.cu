// fp32 matrix products on the fifth-generation tensor cores (sm_100a).
//
// A float is the sum of three bf16 numbers: hi its upper 8 significant bits (rounded to nearest, or cut off where that would
// overflow), mid the next 8 (rounded), lo what is left, exactly.  A product of two floats is six bf16 products (hi hi; hi mid +
// mid hi; hi lo + mid mid + lo hi); what is left out is below 2^-24 of it.  mid and lo are stored 2^7 and 2^14 times as large, so
// that they keep all their bits from 2^-123 on, and every order of magnitude has an accumulator of its own in tensor memory:
//     c = 2 (acc0 + 2^-7 (acc1 + 2^-7 acc2))
// The tensor cores cut off their sums, which a long chain shows: acc0 is taken out and added in registers, rounded to
// nearest, every kGroup stages of the reduction.  Infinities and NaN come out of acc0 as they would out of a
// multiplication; where it holds one the other two, which may hold inf - inf, are left out.  Finite results never overflow on
// the way: `b` takes part with half its value, so that hi hi, which may be 2^-7 above its product, has room, and mid as
// stored is at most half of hi, so the terms of acc1 are no larger than those of acc0.
// (With hi cut off everywhere mid was up to all of hi: what was left out came to 2^-22, and acc1 overflowed at half of FLT_MAX.)
#include <cuda_bf16.h>

#include <algorithm>
#include <atomic>

#include "kernels/gemm_api.h"
#include "kernels/launch_count.h"

namespace mccl {
namespace kern {
namespace {

constexpr int kSms = 148;
constexpr int kRows = 128;                // tile rows of `a`: the lanes of tensor memory
constexpr int kDepth = 32;                // k per stage
// Stages between two turns of acc0.  Error of 8 x 512 x 256, forward, against 64 bits with 1, 2, 4 stages: 0.80, 0.92,
// 1.31e-7 (cuBLAS 1.07e-7); 256 x 3072 x 3072 takes 28.2, 27.3, 26.8 us.
constexpr int kGroup = 2;
constexpr int kAhead = 3;                 // stages of `a` that a producer holds in registers
// warps 0 .. 7 take the accumulators out, warp 8 issues the products, the others fill the stages
constexpr int kAdders = 256, kIssuer = kAdders / 32, kProducer0 = kAdders + 32;
constexpr int kProducers = 256;           // where `a` is read as it is; one warp otherwise
constexpr float kUnscale = 1.0f / 128.0f;
constexpr int kPartA = kRows * kDepth * 2;

// ---- PTX ----------------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void bar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool bar_try(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
  return done != 0;
}
// Waits for the phase of that parity, for four times `limit` cycles at most.  A pause of the whole device (another process has it, a
// debugger stopped it) uses up one of the four.
constexpr long long kWaitLimit = 500000000ll, kLanding = 2000000ll;  // about a quarter of a second and a millisecond
__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity, long long limit) {
  if (bar_try(bar, parity)) return true;
#pragma unroll 1
  for (int left = 4; left > 0; --left) {
    const long long begin = clock64();
    do {
      if (bar_try(bar, parity)) return true;
    } while (clock64() - begin <= limit);
  }
  return false;
}
// Shared-memory matrix descriptors.  k innermost: rows of 64 bytes (32 k), 64-byte swizzle, 512 bytes per eight rows.
// Own index innermost: rows of 128 bytes (64 rows of the operand, one k), 128-byte swizzle, 1024 bytes per eight k, 4096
// from 64 rows to the next.
template <bool kInner>
__device__ __forceinline__ uint64_t make_desc(uint32_t addr) {
  return static_cast<uint64_t>((addr & 0x3FFFFu) >> 4) | (static_cast<uint64_t>(kInner ? 1 : 4096 >> 4) << 16) |
         (static_cast<uint64_t>((kInner ? 512 : 1024) >> 4) << 32) | (1ull << 46) | ((kInner ? 4ull : 2ull) << 61);
}
// from 16 k to the next, in descriptor units
template <bool kInner>
constexpr uint32_t kStep = (kInner ? 32 : 2048) >> 4;
// bf16 x bf16 into fp32; `cols` columns, 128 rows
__host__ __device__ constexpr uint32_t make_idesc(bool a_inner, bool b_inner, int cols) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (a_inner ? 0u : 1u << 15) | (b_inner ? 0u : 1u << 16) |
         (static_cast<uint32_t>(cols >> 3) << 17) | ((kRows >> 4) << 24);
}
__device__ __forceinline__ void mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(static_cast<uint32_t>(accumulate))
      : "memory");
}
__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// 16 consecutive columns of the calling thread's lane
__device__ __forceinline__ void tmem_load16(uint32_t addr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(addr));
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ bool elect() {
  uint32_t one;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xFFFFFFFF;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(one));
  return one != 0;
}

// A float to be cut off where its bf16 neighbours' middle would round away from zero: half a step further from zero.  At the largest
// numbers the sum stops, so they don't become infinite as rounding to nearest would make them; infinities and NaN stay.
// (Rounded to nearest by the conversion, with a look for what that made infinite, 256 x 3072 x 3072 took 41.8 us forward and 41.4 for the
// input gradient, 40.2 and 39.3 so; the half step itself costs 0.8 us.)
__device__ __forceinline__ float half_step(float x) {
  return __fmaf_rz(__uint_as_float(__float_as_uint(x) & 0xFF800000u), 0x1p-8f, x);
}
// Two floats into three bf16 pairs.
__device__ __forceinline__ void split2(float x0, float x1, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  asm("cvt.rz.bf16x2.f32 %0, %1, %2;" : "=r"(hi) : "f"(half_step(x1)), "f"(half_step(x0)));
  const float r0 = (x0 - __uint_as_float(hi << 16)) * 128.0f;
  const float r1 = (x1 - __uint_as_float(hi & 0xFFFF0000u)) * 128.0f;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(mid) : "f"(r1), "f"(r0));
  const float s0 = (r0 - __uint_as_float(mid << 16)) * 128.0f;
  const float s1 = (r1 - __uint_as_float(mid & 0xFFFF0000u)) * 128.0f;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(lo) : "f"(s1), "f"(s0));
}

// Where 16 bytes (eight bf16) of a stage lie within their part: row r, eight numbers from `at` on.
template <bool kInner>
__device__ __forceinline__ int place(int r, int at) {
  return kInner ? r * 64 + (((at >> 3) ^ ((r >> 1) & 3)) << 4) : r * 128 + (((at >> 3) ^ (r & 7)) << 4);
}

// Eight floats of a row, zero outside of the matrix.
__device__ __forceinline__ void load8(const float* data, int64_t ld, int64_t rows, int64_t cols, bool vec, int64_t row, int64_t col,
                                      float (&v)[8]) {
  const float* p = data + row * ld + col;
  if (vec && row < rows && col + 8 <= cols) {
    const float4 x = *reinterpret_cast<const float4*>(p), y = *reinterpret_cast<const float4*>(p + 4);
    v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
    v[4] = y.x; v[5] = y.y; v[6] = y.z; v[7] = y.w;
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = row < rows && col + i < cols ? p[i] : 0.f;
  }
}

struct Split8 {
  uint4 part[3];
};
__device__ __forceinline__ Split8 split8(const float (&v)[8]) {
  Split8 s;
  split2(v[0], v[1], s.part[0].x, s.part[1].x, s.part[2].x);
  split2(v[2], v[3], s.part[0].y, s.part[1].y, s.part[2].y);
  split2(v[4], v[5], s.part[0].z, s.part[1].z, s.part[2].z);
  split2(v[6], v[7], s.part[0].w, s.part[1].w, s.part[2].w);
  return s;
}
__device__ __forceinline__ void store8(char* to, int part, const Split8& s) {
#pragma unroll
  for (int p = 0; p < 3; ++p) *reinterpret_cast<uint4*>(to + p * part) = s.part[p];
}

// ---- images -------------------------------------------------------------------------------------------------
struct SplitWork {
  const float* data;
  int64_t ld, rows, cols;
  bool vec;
  char *by_cols, *by_rows;
  int tile;
  int64_t col_stages, row_stages;    // of by_cols: stages along the columns; of by_rows: along the rows
  int64_t rows_cols, rows_rows;      // rows that each image has
  int64_t blocks_r, blocks_c, warps; // units of eight rows and 32 columns
};
struct SplitAll {
  SplitWork job[2];
  int64_t warps;
  int split_blocks, sum_blocks;
  float* sums;
  uint32_t* zero;
  int64_t zeroed;
};

// Bound by launch and latency: 2.0 us for 32 x 3072, 2.7 for 256 x 3072 numbers, 3.6 with three images and the column sums,
// which take torch's reduction 5.4 by themselves.  The sums are carried in 64 bits.
__global__ void __launch_bounds__(256) split_f32_kernel(const SplitAll w) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (static_cast<int>(blockIdx.x) >= w.split_blocks) {
    // column sums: 32 columns per block, its warps share the rows
    __shared__ double part[8][32];
    const SplitWork& m = w.job[0];
    const int64_t col = (static_cast<int64_t>(blockIdx.x) - w.split_blocks) * 32 + lane;
    double sum[4] = {0.0, 0.0, 0.0, 0.0};
    if (col < m.cols) {
      int64_t r = warp;
      for (; r + 24 < m.rows; r += 32)
#pragma unroll
        for (int i = 0; i < 4; ++i) sum[i] += m.data[(r + 8 * i) * m.ld + col];
      for (; r < m.rows; r += 8) sum[0] += m.data[r * m.ld + col];
    }
    part[warp][lane] = (sum[0] + sum[1]) + (sum[2] + sum[3]);
    __syncthreads();
    if (warp == 0 && col < m.cols) {
      double total = part[0][lane];
#pragma unroll
      for (int i = 1; i < 8; ++i) total += part[i][lane];
      w.sums[col] = static_cast<float>(total);
    }
    return;
  }
  for (int64_t i = blockIdx.x * 256ll + threadIdx.x; i < w.zeroed; i += w.split_blocks * 256ll) w.zero[i] = 0u;
  for (int64_t u = blockIdx.x * 8ll + warp; u < w.warps; u += w.split_blocks * 8ll) {
    const SplitWork& m = u < w.job[0].warps ? w.job[0] : w.job[1];
    const int64_t unit = u < w.job[0].warps ? u : u - w.job[0].warps;
    const int64_t row = unit % m.blocks_r * 8 + (lane >> 2), col = unit / m.blocks_r * 32 + (lane & 3) * 8;
    float v[8];
    load8(m.data, m.ld, m.rows, m.cols, m.vec, row, col, v);
    if (u < w.job[0].warps)  // `b`
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] *= 0.5f;
    const Split8 s = split8(v);
    if (m.by_cols && row < m.rows_cols && col < m.col_stages * kDepth) {
      const int part = m.tile * kDepth * 2;
      store8(m.by_cols + ((row / m.tile) * m.col_stages + col / kDepth) * 3 * part +
                 place<true>(static_cast<int>(row % m.tile), static_cast<int>(col % kDepth)),
             part, s);
    }
    if (m.by_rows && row < m.row_stages * kDepth)
      store8(m.by_rows + ((col / kRows) * m.row_stages + row / kDepth) * 3 * kPartA + ((col % kRows) / 64) * 4096 +
                 place<false>(static_cast<int>(row % kDepth), static_cast<int>(col % 64)),
             kPartA, s);
  }
}

// ---- product ------------------------------------------------------------------------------------------------
// Where the stages of `a` come from: weights read as they are, k innermost or not, or an image (k not innermost).
enum Source { kWeightRows, kWeightCols, kImage };

struct Work {
  const float* weight;
  int64_t ldw;
  bool vec;
  const char *a_image, *b_image;
  const float* bias;
  float* c;
  int64_t ldc, rows_i, rows_j, depth;
  int tiles_i, tiles;               // tile t: i from t % tiles_i, j from t / tiles_i
  int stages, per_split, splits;
  float* partial;
  uint32_t* tickets;
  uint32_t* failed;
  long long limit;                  // of each wait
};

template <int kSource>
constexpr int kThreads = kProducer0 + (kSource == kImage ? 32 : kProducers);
template <int NT>
struct Shape {
  static constexpr int part_b = NT * kDepth * 2;
  static constexpr int stage = 3 * (kPartA + part_b);  // bytes
  static constexpr int stages = 4;
  static constexpr int smem = stages * stage + 1024;
  static constexpr int columns = NT == 128 ? 512 : NT == 64 ? 256 : 128;  // of tensor memory: 3 NT, a power of two
};

__device__ __forceinline__ void bulk_load(uint32_t to, const void* from, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(to),
               "l"(from), "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void bar_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

// One tile of 128 by NT per CTA and, where the tiles do not fill the device, a share of its reduction; tiles in turn where
// there are more than SMs.  One warp issues all products, eight take acc0 out while the other products of a stage run,
// the rest cut the weights (once per tile: no pass over them before) or copy images in, four stages ahead (six or seven for the
// narrow tiles took 20.0 us where four took 19.3, 32 x 3072 x 3072 forward: what the stages leave is the weights' cache).
// Bound by shared memory: a stage of NT = 128 moves 128 KB through it, 1024 cycles, where its products take 768; measured
// 870 without the weights' share, 1300 with it.  256 x 3072 x 3072 with weights that come from memory, us, with the images'
// launch (B200): forward 125.9 with cuBLAS's fp32 kernel, 37.8 so; input gradient 122.8 and 37.9; weight gradient, whose
// images take the second-level cache 9 TB/s, 99.5 and 32.7: 130 to 150 TFLOP/s of fp32 products, 0.8 to 0.9 PFLOP/s of bf16.
// Tried and left: pairs of CTAs on one tile (92 KB per stage, but each turn waits for both: 47.5 us), weights cut straight
// into tensor memory (72 KB; a lane's 32 loads per stage cost what that saves: 36.0 and 48.4 us).
template <int NT, int kSource>
__global__ void __launch_bounds__(kThreads<kSource>, 1) gemm_f32_kernel(const Work w) {
  constexpr bool kAInner = kSource == kWeightRows, kBInner = kSource != kImage;
  constexpr int kStages = Shape<NT>::stages, kStage = Shape<NT>::stage, kPartB = Shape<NT>::part_b;
  static_assert(kBInner || NT == 128, "an operand with its own index innermost comes in runs of 64 rows");
  extern __shared__ char raw[];
  __shared__ alignas(8) uint64_t bars[2 * kStages + 5];
  __shared__ uint32_t tmem_base, last_here;
  char* smem = raw + ((1024u - (smem_addr(raw) & 1023u)) & 1023u);
  const uint32_t smem0 = smem_addr(smem);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t bar0 = smem_addr(bars);
  auto full = [&](int s) { return bar0 + 8u * s; };
  auto empty = [&](int s) { return bar0 + 8u * (kStages + s); };
  const uint32_t acc0_full = bar0 + 8u * (2 * kStages), acc0_free = acc0_full + 8, all_full = acc0_full + 16,
                 all_free = acc0_full + 24, drained = acc0_full + 32;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) {
      bar_init(full(s), kSource == kImage ? 1 : kProducers / 32 + 1);
      bar_init(empty(s), 1);
    }
    bar_init(acc0_full, 1);
    bar_init(acc0_free, kAdders / 32);
    bar_init(all_full, 1);
    bar_init(all_free, kAdders / 32);
    bar_init(drained, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kIssuer) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_base)),
                 "n"(Shape<NT>::columns)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = tmem_base;
  const int rank = static_cast<int>(blockIdx.x) % w.splits;
  const int first_tile = static_cast<int>(blockIdx.x) / w.splits, tile_step = static_cast<int>(gridDim.x) / w.splits;
  const int c0 = rank * w.per_split, c1 = min(w.stages, c0 + w.per_split);  // host: c0 < stages
  bool ok = true;  // alike in a warp's lanes, but for the lanes that load images and issue products on their own
  bool issues = false;

  if (warp > kIssuer) {
    const int ptid = tid - kProducer0;
    auto load_images = [&](int tile, int c, int s) {
      const int64_t at = static_cast<int64_t>(tile / w.tiles_i) * w.stages + c;
      const uint32_t to = smem0 + s * kStage;
      bar_expect(full(s), (kSource == kImage ? 3 * kPartA : 0) + 3 * kPartB);
      if (kSource == kImage)
        bulk_load(to, w.a_image + (static_cast<int64_t>(tile % w.tiles_i) * w.stages + c) * (3 * kPartA), 3 * kPartA, full(s));
      bulk_load(to + 3 * kPartA, w.b_image + at * (3 * kPartB), 3 * kPartB, full(s));
    };
    int s = 0, turn = 0;
    if constexpr (kSource == kImage) {
      if (elect()) {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        for (int tile = first_tile; ok && tile < w.tiles; tile += tile_step)
          for (int c = c0; ok && c < c1; ++c) {
            ok = bar_wait(empty(s), (turn & 1) ^ 1, w.limit);
            if (!ok) break;
            load_images(tile, c, s);
            if (++s == kStages) s = 0, ++turn;
          }
      }
      __syncwarp();
    } else {
      // rows of a stage: 32 k of one weight row, or one k of 64 weight columns
      const int row = kAInner ? ptid >> 2 : ptid >> 3, at = (kAInner ? ptid & 3 : ptid & 7) * 8;
      char* mine = smem + place<kAInner>(row, at);
      float v[kAhead][2][8];
      // where the next stage's numbers lie, two groups of eight per thread: rows 64 apart, or one row's columns
      const int64_t step = kAInner ? kDepth : kDepth * w.ldw, apart = kAInner ? 64 * w.ldw : 64;
      const float* from = nullptr;
      int ft = first_tile, fc = c1, left = 0;  // left: of the reduction, from this thread's numbers on
      int own[2] = {0, 0};                     // of the own index
      auto fetch = [&](float (&x)[2][8]) {
        if (fc == c1) {
          if (ft >= w.tiles) return;
          const int64_t i0 = static_cast<int64_t>(ft % w.tiles_i) * kRows, k0 = static_cast<int64_t>(c0) * kDepth;
          const int64_t i = i0 + (kAInner ? row : at), k = k0 + (kAInner ? at : row);
          from = w.weight + (kAInner ? i * w.ldw + k : k * w.ldw + i);
          left = static_cast<int>(min(w.depth - k, static_cast<int64_t>(1 << 30)));
#pragma unroll
          for (int j = 0; j < 2; ++j) own[j] = static_cast<int>(max(min(w.rows_i - i - 64 * j, static_cast<int64_t>(8)), static_cast<int64_t>(0)));
          fc = c0;
          ft += tile_step;
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const float* p = from + j * apart;
          const int n = kAInner ? (own[j] > 0 ? left : 0) : (left > 0 ? own[j] : 0);
          if (w.vec && n >= 8) {
            const float4 lo = *reinterpret_cast<const float4*>(p), hi = *reinterpret_cast<const float4*>(p + 4);
            x[j][0] = lo.x; x[j][1] = lo.y; x[j][2] = lo.z; x[j][3] = lo.w;
            x[j][4] = hi.x; x[j][5] = hi.y; x[j][6] = hi.z; x[j][7] = hi.w;
          } else {
#pragma unroll
            for (int e = 0; e < 8; ++e) x[j][e] = e < n ? p[e] : 0.f;
          }
        }
        from += step;
        left -= kDepth;
        ++fc;
      };
#pragma unroll
      for (int b = 0; b < kAhead; ++b) fetch(v[b]);
      const bool loads = warp == kIssuer + 1 && elect();
      if (loads) asm volatile("griddepcontrol.wait;" ::: "memory");
      int tile = first_tile, c = c0, missed = 0;
      while (ok && tile < w.tiles) {
#pragma unroll
        for (int b = 0; b < kAhead; ++b) {
          if (tile >= w.tiles) break;
          // no branch before the numbers are cut, which needs no stage: warps agree on having given up after a few
          const bool got = bar_wait(empty(s), (turn & 1) ^ 1, w.limit);
          if (got && loads) load_images(tile, c, s);
          char* to = mine + s * kStage;
#pragma unroll
          for (int j = 0; j < 2; ++j) store8(to + j * 4096, kPartA, split8(v[b][j]));
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          if (!got) missed = 1;
          if (lane == 0 && missed == 0) bar_arrive(full(s));
          fetch(v[b]);
          if (++s == kStages) s = 0, ++turn;
          if (++c == c1) c = c0, tile += tile_step;
        }
        ok = __all_sync(0xFFFFFFFFu, missed == 0);
      }
    }
  } else if (warp == kIssuer) {
    issues = elect();
    if (issues) {
      ok = w.limit > 0;  // a limit of zero, of tests: no product is issued, and all others wait in vain
      constexpr uint32_t one = make_idesc(kAInner, kBInner, NT), two = make_idesc(kAInner, kBInner, 2 * NT);
      constexpr uint32_t step_a = kStep<kAInner>, step_b = kStep<kBInner>;
      const uint32_t acc0 = tmem, acc1 = tmem + NT, acc2 = tmem + 2 * NT;
      const uint64_t a0 = make_desc<kAInner>(smem0), b0 = make_desc<kBInner>(smem0 + 3 * kPartA);
      int groups = 0, done = 0, s = 0, turn = 0;
      for (int tile = first_tile; ok && tile < w.tiles; tile += tile_step, ++done) {
        if (done > 0) ok = bar_wait(all_free, (done - 1) & 1, w.limit);
        for (int c = c0; ok && c < c1; ++c) {
          const bool opens = (c - c0) % kGroup == 0, closes = (c - c0) % kGroup == kGroup - 1 || c == c1 - 1;
          if (opens && groups > 0) ok = bar_wait(acc0_free, (groups - 1) & 1, w.limit);
          ok = ok && bar_wait(full(s), turn & 1, w.limit);
          if (!ok) break;
          fence_after();
          const uint64_t ah = a0 + s * (kStage >> 4), am = ah + (kPartA >> 4), al = am + (kPartA >> 4);
          const uint64_t bh = b0 + s * (kStage >> 4), bm = bh + (kPartB >> 4);
#pragma unroll
          for (int k = 0; k < kDepth / 16; ++k) mma(acc0, ah + k * step_a, bh + k * step_b, one, !opens || k > 0);
          if (closes) {
            mma_commit(acc0_full);
            ++groups;
          }
          // the parts of b lie one behind the other, and so do acc1 and acc2: two products in one
#pragma unroll
          for (int k = 0; k < kDepth / 16; ++k) mma(acc1, ah + k * step_a, bm + k * step_b, two, c > c0 || k > 0);
#pragma unroll
          for (int k = 0; k < kDepth / 16; ++k) mma(acc1, am + k * step_a, bh + k * step_b, two, true);
#pragma unroll
          for (int k = 0; k < kDepth / 16; ++k) mma(acc2, al + k * step_a, bh + k * step_b, one, true);
          mma_commit(empty(s));
          if (++s == kStages) s = 0, ++turn;
        }
        mma_commit(all_full);
      }
    }
    __syncwarp();
  } else {
    // lanes 32 q .. 32 q + 31 of tensor memory are open to the warps with warp % 4 == q; two of them share the columns
    constexpr int kCols = NT / 2;
    const int q = warp & 3, half = warp >> 2;
    const uint32_t lanes = tmem + (static_cast<uint32_t>(32 * q) << 16) + half * kCols;
    int groups = 0, done = 0;
    for (int tile = first_tile; ok && tile < w.tiles; tile += tile_step, ++done) {
      float sum[kCols];
#pragma unroll
      for (int i = 0; i < kCols; ++i) sum[i] = 0.f;
      for (int c = c0; ok && c < c1; c += kGroup) {
        // the other five products of the group's last stage run while acc0 is taken out
        const bool got = bar_wait(acc0_full, groups++ & 1, w.limit);
        fence_after();
#pragma unroll
        for (int i = 0; i < kCols; i += 16) {
          float v[16];
          tmem_load16(lanes + i, v);
          tmem_wait();
#pragma unroll
          for (int e = 0; e < 16; ++e) sum[i + e] += v[e];
        }
        fence_before();
        __syncwarp();
        if (lane == 0) bar_arrive(acc0_free);
        ok = __all_sync(0xFFFFFFFFu, got);
      }
      const bool got = ok && bar_wait(all_full, done & 1, w.limit);
      fence_after();
#pragma unroll
      for (int i = 0; i < kCols; i += 16) {
        float v1[16], v2[16];
        tmem_load16(lanes + NT + i, v1);
        tmem_load16(lanes + 2 * NT + i, v2);
        tmem_wait();
#pragma unroll
        for (int e = 0; e < 16; ++e)
          sum[i + e] = fabsf(sum[i + e]) < INFINITY ? sum[i + e] + kUnscale * (v1[e] + kUnscale * v2[e]) : sum[i + e];
      }
      fence_before();
      __syncwarp();
      ok = __all_sync(0xFFFFFFFFu, got);
      if (!ok) break;
      if (lane == 0) bar_arrive(all_free);
      if (w.splits > 1) {
        float* part = w.partial + (static_cast<int64_t>(tile) * w.splits + rank) * (NT * kRows) + half * kCols * kRows + 32 * q + lane;
#pragma unroll
        for (int e = 0; e < kCols; ++e) __stcg(part + e * kRows, sum[e]);
        __threadfence();
        continue;
      }
      const int64_t i = static_cast<int64_t>(tile % w.tiles_i) * kRows + 32 * q + lane;
      const int64_t j0 = static_cast<int64_t>(tile / w.tiles_i) * NT + half * kCols;
      if (i < w.rows_i) {
        const float add = w.bias ? w.bias[i] : 0.f;
        float* out = w.c + j0 * w.ldc + i;
        const int cols = static_cast<int>(min(static_cast<int64_t>(kCols), w.rows_j - j0));
#pragma unroll
        for (int e = 0; e < kCols; ++e)
          if (e < cols) out[e * w.ldc] = w.bias ? fmaf(2.f, sum[e], add) : 2.f * sum[e];
      }
    }
  }
  fence_before();
  const bool failed = __syncthreads_or(!ok);
  fence_after();
  if (failed) {
    if (tid == 0) {
      if (w.failed) *w.failed = 1u;
      // The copies in flight, microseconds, end before this CTA's shared memory is another's.
      for (const long long begin = clock64(); clock64() - begin < kLanding;) {
      }
    }
    if (issues) {  // and the products, before tensor memory is
      mma_commit(drained);
      bar_wait(drained, 0, kWaitLimit);
    }
    __syncwarp();
    // no number that looks like a result
    for (int tile = first_tile; tile < w.tiles; tile += tile_step) {
      const int64_t i0 = static_cast<int64_t>(tile % w.tiles_i) * kRows, j0 = static_cast<int64_t>(tile / w.tiles_i) * NT;
      for (int v = tid; v < NT * kRows; v += kThreads<kSource>) {
        const int64_t i = i0 + v % kRows, j = j0 + v / kRows;
        if (w.splits > 1) __stcg(w.partial + (static_cast<int64_t>(tile) * w.splits + rank) * (NT * kRows) + v, NAN);
        else if (i < w.rows_i && j < w.rows_j) w.c[j * w.ldc + i] = NAN;
      }
    }
    __threadfence();
    __syncthreads();
  }
  if (w.splits > 1) {
    // The CTA that is the last of its tile adds up all parts, in order.  Eight loads of four numbers per thread in flight:
    // with one part after the other, and the bias only then, the three parts of a forward product took 2 us longer.
    const int tile = first_tile;
    if (tid == 0) last_here = atomicAdd(w.tickets + tile, 1u) == static_cast<uint32_t>(w.splits - 1);
    __syncthreads();
    if (last_here) {
      __threadfence();
      constexpr int kStride = kThreads<kSource>, kVecs = NT * kRows / 4;
      const float4* from = reinterpret_cast<const float4*>(w.partial) + static_cast<int64_t>(tile) * w.splits * kVecs;
      const int64_t i = static_cast<int64_t>(tile % w.tiles_i) * kRows + tid % (kRows / 4) * 4;
      static_assert(kStride % (kRows / 4) == 0, "all numbers of a thread belong to the same four i");
      float add[4];
#pragma unroll
      for (int n = 0; n < 4; ++n) add[n] = w.bias && i + n < w.rows_i ? w.bias[i + n] : 0.f;
      constexpr int kBatch = 4;
      for (int v0 = tid; v0 < kVecs; v0 += kBatch * kStride) {
        float4 sum[kBatch];
        for (int r = 0; r < w.splits; r += 2) {  // two parts of four vectors in flight
          float4 x[2][kBatch];
#pragma unroll
          for (int p = 0; p < 2; ++p)
#pragma unroll
            for (int e = 0; e < kBatch; ++e)
              x[p][e] = r + p < w.splits && v0 + e * kStride < kVecs ? __ldcg(from + (r + p) * kVecs + v0 + e * kStride)
                                                                     : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
          for (int e = 0; e < kBatch; ++e) {
            if (r == 0) sum[e] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int p = 0; p < 2; ++p) {
              sum[e].x += x[p][e].x; sum[e].y += x[p][e].y; sum[e].z += x[p][e].z; sum[e].w += x[p][e].w;
            }
          }
        }
#pragma unroll
        for (int e = 0; e < kBatch; ++e) {
          const int v = v0 + e * kStride;
          const int64_t j = static_cast<int64_t>(tile / w.tiles_i) * NT + v / (kRows / 4);
          if (v >= kVecs || j >= w.rows_j) continue;
          const float out[4] = {sum[e].x, sum[e].y, sum[e].z, sum[e].w};
#pragma unroll
          for (int n = 0; n < 4; ++n)
            if (i + n < w.rows_i) w.c[j * w.ldc + i + n] = w.bias ? fmaf(2.f, out[n], add[n]) : 2.f * out[n];
        }
      }
    }
  }
  if (warp == kIssuer)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(Shape<NT>::columns));
}

template <int NT, int kSource>
cudaError_t run(const Work& w, cudaStream_t s) {
  const auto kernel = gemm_f32_kernel<NT, kSource>;
  static std::atomic<uint64_t> smem_set{0};
  int device = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return e;
  const uint64_t bit = 1ull << (device & 63);
  if (!(smem_set.load(std::memory_order_acquire) & bit)) {
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Shape<NT>::smem);
    if (e != cudaSuccess) return e;
    smem_set.fetch_or(bit, std::memory_order_release);
  }
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(w.splits > 1 ? w.tiles * w.splits : std::min(w.tiles, kSms)));
  cfg.blockDim = dim3(kThreads<kSource>);
  cfg.dynamicSmemBytes = Shape<NT>::smem;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  note_launch();
  return cudaLaunchKernelEx(&cfg, kernel, w);
}

int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }
bool aligned(const float* p, int64_t ld) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0 && ld % 4 == 0; }

}  // namespace

GemmPlan gemm_plan(Product p, int64_t batch, int64_t in, int64_t out) {
  GemmPlan g{};
  g.rows_i = p == Product::kForward ? out : in;
  g.rows_j = p == Product::kWeight ? out : batch;
  g.depth = p == Product::kForward ? in : p == Product::kInput ? out : batch;
  g.cols = p == Product::kWeight || g.rows_j > 64 ? 128 : g.rows_j > 32 ? 64 : 32;
  g.tiles_i = static_cast<int>(ceil_div(g.rows_i, kRows));
  g.tiles_j = static_cast<int>(ceil_div(g.rows_j, g.cols));
  g.stages = static_cast<int>(ceil_div(g.depth, kDepth));
  const int tiles = g.tiles_i * g.tiles_j;
  int splits = 1;
  while (splits < 8 && tiles * (splits + 1) <= kSms && g.stages / (splits + 1) >= 4) ++splits;
  g.per_split = static_cast<int>(ceil_div(g.stages, splits));
  g.splits = static_cast<int>(ceil_div(g.stages, g.per_split));
  const int64_t b_tile = static_cast<int64_t>(g.cols) * kDepth * 6;
  g.a_image = p == Product::kWeight ? static_cast<int64_t>(g.tiles_i) * g.stages * 3 * kPartA : 0;
  g.b_image = static_cast<int64_t>(g.tiles_j) * g.stages * b_tile;
  g.partial = g.splits > 1 ? static_cast<int64_t>(tiles) * g.splits * g.cols * kRows * 4 : 0;
  g.tickets = g.splits > 1 ? tiles : 0;
  return g;
}

// From sweeps of 1 to 4096 rows over 26 layers, 65536 to 16 features and the reverse among them, and of 8 to 255 rows over 81 of
// 256 to 3000 (B200, both sides from CUDA graphs; here with the launch that makes the images; weights from memory and, up to 40 MB
// of them, from the second-level cache).  What is left to the library, us there and here, rows and features in -> out:
//  - little to do, less than the two launches cost: 64, 256 -> 512 forward 11.7 and 12.0;
//  - short sums: tiles of 128 rows (of 65 and more) take 15 to 17 us at least, narrower ones 10 to 12, the library 8 to 13: 96,
//    256 -> 3000 forward 9.3 and 14.6, 33 9.4 and 11.2;
//  - rows of a tile that the layer does not have: 64, 65536 -> 16 forward 117 and 215; weight gradient of 64, 100000 -> 64 25 and 34;
//  - few CTAs with long shares of the reduction: 64, 100000 -> 64 forward 180 and 327, 16, 16384 -> 128 21 and 59;
//  - next to no rows, for which the library reads the weights at 5 TB/s and this kernel at 2.3: 1, 8192 -> 8192 forward 49 and 115.
// Of the 1380 products that size alone let through 138 were slower than the library's by 5 % or more, 81 by 20 %; of the 1241 now, 33
// and 5.  Those are of 65 rows and more, 300 to 850 deep, most of them within 2 us, and two to four times closer to the exact sums;
// lines that left them to the library would take that from a model's other gradients too.
// Images are one and a half times their matrix: none above 1 GB.
bool gemm_pays(Product p, int64_t batch, int64_t in, int64_t out) {
  constexpr double kImageLimit = 1 << 30;
  const double macs = static_cast<double>(batch) * in * out, layer = static_cast<double>(in) * out;
  if (6.0 * batch * (static_cast<double>(in) + 2.0 * out) > kImageLimit || layer > 1e10) return false;
  const bool fwd = p == Product::kForward;
  if (p == Product::kWeight ? batch < 32 || macs < 1e8 : layer < 7e5 || macs < (fwd ? 2e7 : 3e7)) return false;
  const GemmPlan g = gemm_plan(p, batch, in, out);
  const int64_t tiles = static_cast<int64_t>(g.tiles_i) * g.tiles_j;
  if (p == Product::kWeight) return 4.0 * layer >= 3.0 * kRows * kRows * static_cast<double>(tiles);
  if (4 * g.rows_i < 3 * kRows * static_cast<int64_t>(g.tiles_i) || g.depth < 64) return false;
  const bool deep = layer < 3e7 || g.depth >= (fwd ? 2 : 1) * g.rows_i;
  if (batch < (deep ? 2 : fwd ? 16 : 8)) return false;
  if (tiles * g.splits < 24 && (batch < 32 || g.per_split > 64)) return false;
  return g.depth >= (fwd ? 512 : 288) || macs >= 2.5e8;
}

cudaError_t launch_split_f32(const SplitJob* jobs, int n, float* sums, uint32_t* zero, int64_t zeroed, cudaStream_t s) {
  if (n < 1 || n > 2) return cudaErrorInvalidValue;
  SplitAll w{};
  for (int i = 0; i < n; ++i) {
    const SplitJob& j = jobs[i];
    SplitWork& t = w.job[i];
    t.data = j.m.data;
    t.ld = j.m.ld;
    t.rows = j.m.rows;
    t.cols = j.m.cols;
    t.vec = aligned(j.m.data, j.m.ld);
    t.by_cols = static_cast<char*>(j.by_cols);
    t.by_rows = static_cast<char*>(j.by_rows);
    t.tile = j.tile;
    t.col_stages = ceil_div(t.cols, kDepth);
    t.row_stages = ceil_div(t.rows, kDepth);
    t.rows_cols = j.by_cols ? ceil_div(t.rows, j.tile) * j.tile : 0;
    t.rows_rows = j.by_rows ? t.row_stages * kDepth : 0;
    t.blocks_r = std::max(t.rows_cols, t.rows_rows) / 8;
    t.blocks_c = j.by_rows ? ceil_div(t.cols, kRows) * (kRows / 32) : t.col_stages;
    t.warps = t.blocks_r * t.blocks_c;
    w.warps += t.warps;
  }
  w.split_blocks = static_cast<int>(std::min<int64_t>(ceil_div(w.warps, 8), 8 * kSms));
  w.sum_blocks = sums ? static_cast<int>(ceil_div(jobs[0].m.cols, 32)) : 0;
  w.sums = sums;
  w.zero = zero;
  w.zeroed = zeroed;
  note_launch();
  split_f32_kernel<<<w.split_blocks + w.sum_blocks, 256, 0, s>>>(w);
  return cudaGetLastError();
}

cudaError_t launch_gemm_f32(const GemmArgs& g, cudaStream_t s) {
  const GemmPlan& p = g.plan;
  if (p.rows_i <= 0 || p.rows_j <= 0 || p.depth <= 0) return cudaErrorInvalidValue;
  Work w{};
  w.weight = g.weight;
  w.ldw = g.ldw;
  w.vec = aligned(g.weight, g.ldw);
  w.a_image = static_cast<const char*>(g.a_image);
  w.b_image = static_cast<const char*>(g.b_image);
  w.bias = g.bias;
  w.c = g.c;
  w.ldc = g.ldc;
  w.rows_i = p.rows_i;
  w.rows_j = p.rows_j;
  w.depth = p.depth;
  w.tiles_i = p.tiles_i;
  w.tiles = p.tiles_i * p.tiles_j;
  w.stages = p.stages;
  w.per_split = p.per_split;
  w.splits = p.splits;
  w.partial = g.partial;
  w.tickets = g.tickets;
  w.failed = g.failed;
  w.limit = g.wait_limit >= 0 ? g.wait_limit : kWaitLimit;
  if (g.product == Product::kWeight) return run<128, kImage>(w, s);
  const bool fwd = g.product == Product::kForward;
  switch (p.cols) {
    case 128: return fwd ? run<128, kWeightRows>(w, s) : run<128, kWeightCols>(w, s);
    case 64: return fwd ? run<64, kWeightRows>(w, s) : run<64, kWeightCols>(w, s);
    default: return fwd ? run<32, kWeightRows>(w, s) : run<32, kWeightCols>(w, s);
  }
}

}  // namespace kern
}  // namespace mccl
