// Top-k selection with a single pass over the data (sm_100a).
//
// A gradient that fits the shared memory of one thread-block cluster is selected from there by one launch: exact
// radix select, ordered output or dense result, one read and one write of every element.  A larger one takes five:
//   sample   a cluster reads 64 Ki evenly spread elements of g + e and takes, from their exact selection, a
//            magnitude that clearly more than k elements reach and one that clearly fewer do
//   adjust   all SMs: a = g + e, e = a (and g = 0 where the result is dense); the few elements that reach the
//            sampled magnitude go to a candidate list, tile by tile in index order, and into a histogram of 1/1024
//            octave per bin, from which the last block takes the bin of the k-th element; where the result is dense,
//            those above the second magnitude are sent at once
//   select   candidates above the bin are selected, those inside it are gathered, and the last block finds the
//            exact threshold (and the index limit among ties) on them; what was sent too early is taken back
//   output   a count per run of tiles, then the ordered output: pairs sorted by index; a dense result only gets the
//            entries of the k-th element's bin
// Each comes up while the one before ends (a dependent launch: 8 of 44 us at 700 000 elements).
//
// The sample decides speed, never results.  Heavily tied data (more elements than the list holds, or a crowded bin):
// the select launch takes the exact threshold from the whole adjusted vector and the last two rank the ties in index
// order.  Fewer non-zeros than k, or all elements sent: the same two take all of them and the first zeros.  A k-th element
// below the sampled magnitude (by five standard deviations, or a ratio above 0.98, at which nothing is listed) or two octaves
// and more above it (hardly more non-zeros than k; layers of very different scale in one bucket; small ratios of heavy-tailed data): the select launch
// first finds its bin, from the whole vector or from the list, its blocks meeting between two counts, and goes on from there.
#include <cooperative_groups.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <atomic>
#include <cmath>

#include "kernels/launch_count.h"
#include "kernels/topk_api.h"

namespace cg = cooperative_groups;

namespace mccl {
namespace kern {

bool topk_fits_cluster(int64_t n) { return n <= 8 * 48 * 1024; }

namespace {

constexpr int kThreads = 1024;
constexpr int kWarps = kThreads / 32;
constexpr int kMaxCluster = 16;
constexpr int kBins = 2048;              // 11 bits per radix level
constexpr int kItemCap = 48 * 1024;      // floats a CTA keeps in shared memory (192 KB beside 17 KB of state)
constexpr int kSample = 64 * 1024;       // elements of the sample
constexpr int kTile = 1024;              // elements a warp adjusts at a time
// Candidates a warp stages before it appends them to the list.  Small: what shared memory takes is taken from the
// L1 that holds the loads in flight (1024, 72 KB per CTA, cost a quarter of the adjust kernel's bandwidth).
constexpr int kStage = 256;

__device__ __forceinline__ uint32_t key_of(float a) { return __float_as_uint(a) & 0x7FFFFFFFu; }

template <bool kBf16>
__device__ __forceinline__ float load_grad(const void* grad, int64_t i) {
  return kBf16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(grad)[i]) : static_cast<const float*>(grad)[i];
}
template <bool kBf16>
__device__ __forceinline__ void store_dense(void* grad, int64_t i, float v) {
  if (kBf16) static_cast<__nv_bfloat16*>(grad)[i] = __float2bfloat16_rn(v);
  else static_cast<float*>(grad)[i] = v;
}
// zero + value * scale: the entry of a list added to a zero-filled vector
__device__ __forceinline__ float scaled(float v, float scale) { return fmaf(v, scale, 0.f); }

__device__ __forceinline__ int64_t at_most(int64_t a, int64_t b) { return a < b ? a : b; }

constexpr int kBinShift = 13;            // keys per histogram bin: 1/1024 octave
constexpr int kSubBins = 1 << kBinShift;
constexpr int kCoarseShift = 20;         // kWide, kWhole: 11 bits, then 7; 13 are left
constexpr int kFineBins = 1 << (kCoarseShift - kBinShift);
constexpr int kRun = 4;                  // tiles whose pairs one warp puts out
// Entries of the k-th element's bin that one block resolves; more (ties) are left to the whole grid.  51.5 M bf16
// elements, dense result: 255 levels at 1 %, about 50 thousand entries, 222 us with one block and 441 us with the grid;
// 40 levels at 1 %, 190 thousand, 480 and 450 us; 40 levels at 10 %, over a million, 1709 and 509 us (that block then also
// sent them).
constexpr uint32_t kOneBlock = 128 * 1024;
// kList: from the candidates.  kWide: from the candidates, among those of the open-ended last bin.  kTies: the bin is known,
// threshold and ties come from the vector.  kWhole: the bin comes from the vector as well.  kZeros: all non-zeros and the
// first zeros.  kAll: all non-zeros are listed, and a dense result needs no more.
enum Mode : uint32_t { kList, kWide, kWhole, kTies, kZeros, kAll };

// The exact rule: an element is sent if key > threshold, or key == threshold and index <= last_index (kList) or it is
// one of the first `need` (kTies, kZeros).
struct ListState {
  uint32_t hist[kBins];  // candidates by (key - base) >> kBinShift, the last bin open-ended
  uint32_t base;         // smallest magnitude key that is a candidate
  uint32_t sure;         // dense result: candidates above it were sent by the adjust launch
  uint32_t count;        // entries in the list
  uint32_t overflow;     // the list did not hold them all
  uint32_t mode;         // how the selection is decided: Mode
  uint32_t bin, need;    // the k-th element's bin, and how many of that bin are selected
  uint32_t in_bin;       // entries gathered from the bin
  uint32_t threshold, last_index;
  uint32_t ticket[3];    // blocks done: adjust, select, counts
  uint32_t sub[kSubBins];  // kTies: elements of the bin by key
  uint32_t coarse[kBins];    // kWide, kWhole: keys by key >> kCoarseShift
  uint32_t fine[kFineBins];  // and of the chosen coarse bin
  uint32_t pad[3];
  uint32_t gate[4][2];   // kWide, kWhole: blocks that came to a meeting, and how it ended
};
static_assert(sizeof(ListState) % sizeof(uint4) == 0, "8-byte entries follow it in the scratch");
// scratch: ListState, {start, count} per tile, counts per run, the list of {index, value}, its entries inside the bin
struct ListView {
  ListState* state;
  uint2* tiles;
  uint2* runs;
  uint2* list;
  uint2* bin_list;
  uint32_t cap;
};

__host__ __device__ inline int64_t tile_count(int64_t n) { return (n + kTile - 1) / kTile; }
__host__ __device__ inline int64_t run_count(int64_t n) { return (tile_count(n) + kRun - 1) / kRun; }
// How many of the sampled elements reach the magnitude that is taken: five standard deviations more than are
// expected to belong to the selection, so that the list all but never misses one of it.
inline uint32_t sample_rank(int64_t n, int64_t k) {
  const double hits = static_cast<double>(kSample) * static_cast<double>(k) / static_cast<double>(n);
  return static_cast<uint32_t>(std::min<double>(kSample, hits + 5.0 * std::sqrt(hits) + 8.0));
}
// The other bound: so few sampled elements lie above the magnitude of this rank that fewer than k of all do (five standard
// deviations again).  0: the selection is too small for one.
inline uint32_t sure_rank(int64_t n, int64_t k) {
  const double hits = static_cast<double>(kSample) * static_cast<double>(k) / static_cast<double>(n);
  return sample_rank(n, k) == kSample ? 0u : static_cast<uint32_t>(std::max(0.0, hits - 5.0 * std::sqrt(hits) - 8.0));
}
// Room for the elements that reach it: six standard deviations above their expected number, and some for ties.
// None where the whole sample would be needed, at ratios above 0.98: its smallest element bounds nothing, and the list would
// hold twice the vector's bytes (6.5 M fp32 elements, ratio 0.99: 359 us dense, 372 us pairs with it, 144 and 146 us without).
inline int64_t list_capacity(int64_t n, int64_t k) {
  if (sample_rank(n, k) == kSample) return 0;
  const double rank = sample_rank(n, k), expected = rank / kSample * static_cast<double>(n);
  return std::min<int64_t>(n, static_cast<int64_t>(expected * (1.06 + 6.0 / std::sqrt(rank))) + 4096);
}
inline int64_t table_bytes(int64_t n) {
  return static_cast<int64_t>(sizeof(ListState)) + (tile_count(n) + run_count(n)) * static_cast<int64_t>(sizeof(uint2));
}
// The entries of one bin: at most as many as the list has, or one block resolves.
inline int64_t bin_capacity(int64_t cap) { return std::min<int64_t>(cap, kOneBlock); }
// The list takes what there is room for; one that is too short overflows, which is as good as heavily tied data.
inline ListView list_view(void* scratch, size_t bytes, int64_t n, int64_t k) {
  const int64_t room = (static_cast<int64_t>(bytes) - table_bytes(n)) / static_cast<int64_t>(sizeof(uint2));
  ListView v;
  v.state = static_cast<ListState*>(scratch);
  v.tiles = reinterpret_cast<uint2*>(v.state + 1);
  v.runs = v.tiles + tile_count(n);
  v.list = v.runs + run_count(n);
  v.cap = static_cast<uint32_t>(std::min(list_capacity(n, k), std::max(room / 2, room - static_cast<int64_t>(kOneBlock))));
  v.bin_list = v.list + v.cap;
  return v;
}

// ---- launches that follow one another ----------------------------------------------------------------------
// The next launch's blocks may come up now; they wait, before they touch anything, until this one is complete.
__device__ __forceinline__ void start_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// ---- selection by a cluster ---------------------------------------------------------------------------------
// True in exactly one block of the grid: the one that finishes last.  What the others wrote before their call is
// visible to it.
__device__ __forceinline__ bool last_block_done(uint32_t* ticket) {
  __shared__ bool s_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (s_last) __threadfence();
  return s_last;
}

template <int kRanks>
struct Counts {
  uint32_t hist[kRanks * kBins];   // this CTA's counts
  uint32_t total[kRanks * kBins];  // the cluster's
  uint32_t wsum[33];
  uint32_t digit[kRanks], above[kRanks], inside[kRanks];
};
struct ClusterShared : Counts<1> {
  uint2 counts_of[kMaxCluster];
  uint2 warp_counts[kWarps];
};

__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t* warp_sums) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t inc = v;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, inc, o);
    if (lane >= o) inc += t;
  }
  if (lane == 31) warp_sums[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    const uint32_t w = lane < (blockDim.x >> 5) ? warp_sums[lane] : 0u;
    uint32_t winc = w;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, winc, o);
      if (lane >= o) winc += t;
    }
    warp_sums[lane] = winc - w;
  }
  __syncthreads();
  return warp_sums[warp] + inc - v;
}

// The keys of the need[r]-th largest items of the cluster and how many items equal to each belong to the selection.
// each(f) calls f(key) for every item of the calling thread; every thread of the cluster calls this together, and
// there are at least `need` items.  With two levels instead of three the lowest 9 of the 31 bits stay open (zero).  Where
// everything equal or larger down to some bits is selected, the key just below, and none of its equals.
// No CTA's shared memory is touched by another after the return.
template <int kLevels, int kRanks, typename Each>
__device__ void cluster_thresholds(Counts<kRanks>& sh, uint32_t (&need)[kRanks], Each&& each, uint32_t (&threshold)[kRanks]) {
  cg::cluster_group cluster = cg::this_cluster();
  const int ctas = static_cast<int>(cluster.num_blocks()), me = static_cast<int>(cluster.block_rank());
  const int tid = threadIdx.x, lane = tid & 31;
  int width = 11, shift = 20;  // 31 bits of magnitude
  uint32_t prefix[kRanks] = {};
  for (int level = 0;; ++level) {
    const int ranks = level == 0 ? 1 : kRanks;  // the first level's counts serve all
    for (int i = tid; i < ranks * kBins; i += kThreads) sh.hist[i] = 0;
    __syncthreads();
    uint32_t lowest = 0;  // the lowest bin's items (zeros, where there are many) are counted in a register
    const uint32_t mask = (1u << width) - 1u;
    each([&](uint32_t key) {
#pragma unroll
      for (int r = 0; r < kRanks; ++r) {
        if (r >= ranks || (key >> shift) >> width != prefix[r]) continue;
        const uint32_t d = (key >> shift) & mask;
        if (r == 0 && d == 0) ++lowest;
        else atomicAdd(&sh.hist[r * kBins + d], 1u);
      }
    });
    lowest = __reduce_add_sync(0xFFFFFFFFu, lowest);
    if (lane == 0 && lowest) atomicAdd(&sh.hist[0], lowest);
    cluster.sync();
    // Every CTA adds up its share of the bins over the cluster and hands the sums to all.  A thread per bin, its
    // loads independent (spreading a bin over several threads, or warps over CTAs, measured 15 to 30 % slower).
    const int share = ranks * kBins / ctas;
    if (tid < share) {
      uint32_t sum = 0;
#pragma unroll
      for (int c = 0; c < kMaxCluster; ++c)
        if (c < ctas) sum += *cluster.map_shared_rank(&sh.hist[me * share + tid], (me + c) & (ctas - 1));
#pragma unroll
      for (int c = 0; c < kMaxCluster; ++c)
        if (c < ctas) *cluster.map_shared_rank(&sh.total[me * share + tid], (me + c) & (ctas - 1)) = sum;
    }
    cluster.sync();
    // from the top bin down: the bin at which the running count reaches `need`
    const int top = kBins - 1 - 2 * tid;
#pragma unroll
    for (int r = 0; r < kRanks; ++r) {
      const uint32_t* total = sh.total + (level == 0 ? 0 : r * kBins);
      const uint32_t c0 = total[top], c1 = total[top - 1];
      const uint32_t above = block_excl_scan(c0 + c1, sh.wsum);
      if (above < need[r] && above + c0 >= need[r]) {
        sh.digit[r] = top;
        sh.above[r] = above;
        sh.inside[r] = c0;
      } else if (above + c0 < need[r] && above + c0 + c1 >= need[r]) {
        sh.digit[r] = top - 1;
        sh.above[r] = above + c0;
        sh.inside[r] = c1;
      }
      __syncthreads();
      need[r] -= sh.above[r];
      prefix[r] = (prefix[r] << width) | sh.digit[r];
    }
    if (level == kLevels - 1) break;
    if (kRanks == 1 && sh.inside[0] == need[0] && prefix[0] != 0) {
      // All of the bin is wanted, so where in it the last one lies does not matter.  After two levels a bin is 2^-14 of its
      // values wide: of 262144 normal elements, 1 %, it holds one or two (dense result: 20.5 us with three levels, 16.4 so).
      threshold[0] = (prefix[0] << shift) - 1u;
      need[0] = 0;
      return;
    }
    width = shift < 11 ? shift : 11;
    shift -= width;
  }
#pragma unroll
  for (int r = 0; r < kRanks; ++r) threshold[r] = prefix[r] << shift;
}
template <int kLevels, typename Each>
__device__ void cluster_threshold(Counts<1>& sh, uint32_t need, Each&& each, uint32_t* threshold, uint32_t* need_eq) {
  uint32_t left[1] = {need}, found[1];
  cluster_thresholds<kLevels, 1>(sh, left, each, found);
  *threshold = found[0];
  *need_eq = left[0];
}

// Emits the selection in index order.  walk(f) calls f(index, value, valid) with all lanes of the calling warp, for
// the warp's run of items in index order; emit(index, value, position, selected) sees every valid item.
template <typename Walk, typename Emit>
__device__ void cluster_emit(ClusterShared& sh, uint32_t threshold, uint32_t need_eq, Walk&& walk, Emit&& emit) {
  cg::cluster_group cluster = cg::this_cluster();
  const int ctas = static_cast<int>(cluster.num_blocks()), me = static_cast<int>(cluster.block_rank());
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint32_t gt = 0, eq = 0;
  walk([&](uint32_t, float v, bool valid) {
    gt += valid && key_of(v) > threshold;
    eq += valid && key_of(v) == threshold;
  });
  gt = __reduce_add_sync(0xFFFFFFFFu, gt);
  eq = __reduce_add_sync(0xFFFFFFFFu, eq);
  if (lane == 0) sh.warp_counts[warp] = make_uint2(gt, eq);
  __syncthreads();
  uint2 w = sh.warp_counts[lane];
  if (warp == 0) {
    const uint32_t g = __reduce_add_sync(0xFFFFFFFFu, w.x), e = __reduce_add_sync(0xFFFFFFFFu, w.y);
    if (lane < ctas) *cluster.map_shared_rank(&sh.counts_of[me], lane) = make_uint2(g, e);
  }
  if (lane >= warp) w = make_uint2(0u, 0u);
  cluster.sync();  // the last access to another CTA's shared memory
  if (lane < me) {
    w.x += sh.counts_of[lane].x;
    w.y += sh.counts_of[lane].y;
  }
  uint32_t before_gt = __reduce_add_sync(0xFFFFFFFFu, w.x), before_eq = __reduce_add_sync(0xFFFFFFFFu, w.y);
  walk([&](uint32_t i, float v, bool valid) {
    const uint32_t key = key_of(v);
    const bool is_gt = valid && key > threshold, is_eq = valid && key == threshold;
    const uint32_t m_gt = __ballot_sync(0xFFFFFFFFu, is_gt), m_eq = __ballot_sync(0xFFFFFFFFu, is_eq);
    const uint32_t lower = (1u << lane) - 1u;
    const uint32_t r_gt = before_gt + __popc(m_gt & lower), r_eq = before_eq + __popc(m_eq & lower);
    const bool selected = is_gt || (is_eq && r_eq < need_eq);
    if (valid) emit(i, v, r_gt + (r_eq < need_eq ? r_eq : need_eq), selected);
    before_gt += __popc(m_gt);
    before_eq += __popc(m_eq);
  });
}

struct SelectArgs {
  void* grad;
  float* residual;
  uint2* pairs;
  int64_t n;
  uint32_t k;
  float scale;
  ListView list;
};

// The whole selection of a gradient that fits the cluster's shared memory: read once, written once.
// Bound by latency: two cluster barriers per radix level, three levels, two for the rest.
// 262144 fp32 elements, 1 %, dense result: 65 us in eight launches of all SMs, 16 to 20 us so; from about twice that size
// on the launches below take over (700000 elements: 38 us from one cluster).
template <bool kBf16, bool kDense>
__global__ void __launch_bounds__(kThreads, 1) topk_cluster_kernel(const SelectArgs a, int per) {
  extern __shared__ __align__(16) float items[];
  __shared__ ClusterShared sh;
  const int me = static_cast<int>(cg::this_cluster().block_rank());
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t lo = at_most(a.n, static_cast<int64_t>(me) * per);
  const int m = static_cast<int>(at_most(a.n - lo, per));
  // `per` is a multiple of 8: with aligned arrays every CTA's run is aligned as well
  const bool vec = ((reinterpret_cast<uintptr_t>(a.grad) | reinterpret_cast<uintptr_t>(a.residual)) & 15) == 0;
  const int whole = vec ? m / 4 * 4 : 0;
#pragma unroll 4
  for (int i = 4 * tid; i < whole; i += 4 * kThreads) {
    float4 v = *reinterpret_cast<const float4*>(a.residual + lo + i);
    if (kBf16) {
      const uint2 raw = *reinterpret_cast<const uint2*>(static_cast<const __nv_bfloat16*>(a.grad) + lo + i);
      const __nv_bfloat162 g0 = *reinterpret_cast<const __nv_bfloat162*>(&raw.x);
      const __nv_bfloat162 g1 = *reinterpret_cast<const __nv_bfloat162*>(&raw.y);
      v.x += __low2float(g0); v.y += __high2float(g0); v.z += __low2float(g1); v.w += __high2float(g1);
    } else {
      const float4 g = *reinterpret_cast<const float4*>(static_cast<const float*>(a.grad) + lo + i);
      v.x += g.x; v.y += g.y; v.z += g.z; v.w += g.w;
    }
    *reinterpret_cast<float4*>(items + i) = v;
  }
  for (int i = whole + tid; i < m; i += kThreads) items[i] = load_grad<kBf16>(a.grad, lo + i) + a.residual[lo + i];
  __syncthreads();
  uint32_t threshold, need_eq;
  cluster_threshold<3>(sh, a.k, [&](auto&& f) {
    for (int i = tid; i < m; i += kThreads) f(key_of(items[i]));
  }, &threshold, &need_eq);
  const int per_warp = (m + kWarps - 1) / kWarps;
  const int w0 = min(m, warp * per_warp), w1 = min(m, w0 + per_warp);
  cluster_emit(sh, threshold, need_eq,
               [&](auto&& f) {
                 for (int i = w0; i < w1; i += 32)
                   f(static_cast<uint32_t>(lo + i + lane), i + lane < w1 ? items[i + lane] : 0.f, i + lane < w1);
               },
               [&](uint32_t i, float v, uint32_t pos, bool selected) {
                 a.residual[i] = selected ? 0.f : v;  // sent: nothing left to feed back
                 if (kDense) store_dense<kBf16>(a.grad, i, selected ? scaled(v, a.scale) : 0.f);
                 else if (selected) a.pairs[pos] = make_uint2(i, __float_as_uint(v));
               });
}

// The magnitude that `rank` of the kSample sampled elements reach, as the list's smallest key, and the one that `sure` of
// them reach, rounded up (0: none).
template <bool kBf16>
__global__ void __launch_bounds__(kThreads, 1) topk_sample_kernel(const SelectArgs a, uint32_t rank, uint32_t sure) {
  constexpr int kMost = kSample / 8 / kThreads;  // per thread, in a cluster of eight CTAs
  __shared__ Counts<2> sh;
  start_dependents();
  cg::cluster_group cluster = cg::this_cluster();
  const int per = kSample / static_cast<int>(cluster.num_blocks()), mine = per / kThreads;
  const int64_t stride = a.n / kSample;
  uint32_t key[kMost];
#pragma unroll
  for (int j = 0; j < kMost; ++j) {
    if (j >= mine) break;
    // evenly spread, at a different place of each stride (no fixed column of a row-major matrix)
    const uint32_t s = cluster.block_rank() * per + j * kThreads + threadIdx.x;
    const int64_t i = s * stride + (static_cast<uint64_t>((s * 2654435761u) >> 8) * stride >> 24);
    key[j] = key_of(load_grad<kBf16>(a.grad, i) + a.residual[i]);
  }
  uint32_t need[2] = {rank, sure > 0 ? sure : 1u}, found[2];
  cluster_thresholds<2, 2>(sh, need, [&](auto&& f) {
#pragma unroll
    for (int j = 0; j < kMost; ++j)
      if (j < mine) f(key[j]);
  }, found);
  if (cluster.block_rank() == 0) {
    uint32_t* words = reinterpret_cast<uint32_t*>(a.list.state);
    for (int i = threadIdx.x; i < static_cast<int>(sizeof(ListState) / 4); i += kThreads) words[i] = 0u;
    __syncthreads();
    if (threadIdx.x == 0) {
      a.list.state->base = rank == kSample ? 0xFFFFFFFFu : found[0] > 0 ? found[0] : 1u;  // zeros are never worth listing
      a.list.state->sure = sure > 0 ? found[1] | 0x1FFu : 0xFFFFFFFFu;
    }
  }
}

// Sends one entry: nothing is left to feed back, and (kDense) its scaled value is the result.
template <bool kBf16, bool kDense>
__device__ __forceinline__ void send(const SelectArgs& a, uint32_t i, float v) {
  a.residual[i] = 0.f;
  if (kDense) store_dense<kBf16>(a.grad, i, scaled(v, a.scale));
}
// Takes one back that was sent.
template <bool kBf16, bool kDense>
__device__ __forceinline__ void unsend(const SelectArgs& a, uint32_t i, float v) {
  a.residual[i] = v;
  if (kDense) store_dense<kBf16>(a.grad, i, 0.f);
}

__device__ __forceinline__ uint32_t bin_of(uint32_t key_above_base) {
  const uint32_t b = key_above_base >> kBinShift;
  return b < kBins ? b : kBins - 1;
}

// a = g + e, e = a, candidates to the list.  A warp owns `group` consecutive tiles at a time and appends their
// candidates in index order: one global atomic per group, entries of a group contiguous.
// A dense result gets its surely selected entries here, while the lines just written are in the cache: sent by the next
// launch, half a million scattered pairs of stores fetched and wrote a sector each (select 64 us, all 211 us a pass among
// others; so 165); kept back until a warp's stage was full they did no better (207), and worked into the vector stores they
// cost registers (218).
// Bound by HBM: 12 bytes per bf16 element with a dense result.
// 50257 x 1024 bf16 elements (618 MB): 122 us among others, 5.1 TB/s, 112 without the entries.
template <bool kBf16, bool kVec, bool kDense>
__global__ void __launch_bounds__(256, 3) topk_adjust_kernel(const SelectArgs a, int group) {
  extern __shared__ __align__(16) uint2 staging[];
  __shared__ uint32_t hist[kBins];
  for (int i = threadIdx.x; i < kBins; i += blockDim.x) hist[i] = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint2* stage = staging + warp * kStage;
  const ListView list = a.list;
  start_dependents();
  wait_for_previous();
  const uint32_t base = list.state->base, sure = kDense ? list.state->sure : 0xFFFFFFFFu;
  const int64_t tiles = tile_count(a.n);
  const uint32_t lower = (1u << lane) - 1u;
  const int64_t step = static_cast<int64_t>(gridDim.x) * (blockDim.x / 32) * group;
  for (int64_t g0 = (static_cast<int64_t>(blockIdx.x) * (blockDim.x / 32) + warp) * group; g0 < tiles; g0 += step) {
    const int64_t g1 = g0 + group < tiles ? g0 + group : tiles;
    int64_t first = g0;   // the tile under which the staged candidates will be found
    uint32_t staged = 0;
    // room for `cnt` entries in the list, to be found under tile `t`; false if there is none
    auto reserve = [&](int64_t t, uint32_t cnt, uint32_t* at) {
      uint32_t start = 0;
      if (lane == 0) {
        if (cnt) start = atomicAdd(&list.state->count, cnt);
        list.tiles[t] = make_uint2(start, cnt);
      }
      *at = start = __shfl_sync(0xFFFFFFFFu, start, 0);
      if (start <= list.cap && cnt <= list.cap - start) return true;
      if (lane == 0) list.state->overflow = 1u;
      for (uint32_t i = start + lane; i < list.cap; i += 32) list.list[i] = make_uint2(0u, 0u);  // the list's end: no entries
      return false;
    };
    auto flush = [&]() {
      uint32_t start;
      __syncwarp();
      const bool fits = reserve(first, staged, &start);
      for (uint32_t i = lane; i < staged; i += 32) {
        const uint2 e = stage[i];
        const uint32_t key = e.y & 0x7FFFFFFFu;
        if (fits) list.list[start + i] = e;
        else if (key > sure) unsend<kBf16, kDense>(a, e.x, __uint_as_float(e.y));  // what is sent is listed
        atomicAdd(&hist[bin_of(key - base)], 1u);
      }
      __syncwarp();
      staged = 0;
    };
    for (int64_t tile = g0; tile < g1; ++tile) {
      const int64_t t0 = tile * kTile + 4 * lane;
      float v[8][4];
      const bool whole = kVec && tile * kTile + kTile <= a.n;
      if (whole) {
        float4 r[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) r[q] = __ldcs(reinterpret_cast<const float4*>(a.residual + t0 + 128 * q));
        if (kBf16) {
          uint2 raw[8];
#pragma unroll
          for (int q = 0; q < 8; ++q)
            raw[q] = __ldcs(reinterpret_cast<const uint2*>(static_cast<const __nv_bfloat16*>(a.grad) + t0 + 128 * q));
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const __nv_bfloat162 x = *reinterpret_cast<const __nv_bfloat162*>(&raw[q].x);
            const __nv_bfloat162 y = *reinterpret_cast<const __nv_bfloat162*>(&raw[q].y);
            v[q][0] = __low2float(x) + r[q].x; v[q][1] = __high2float(x) + r[q].y;
            v[q][2] = __low2float(y) + r[q].z; v[q][3] = __high2float(y) + r[q].w;
          }
        } else {
          float4 g[8];
#pragma unroll
          for (int q = 0; q < 8; ++q) g[q] = __ldcs(reinterpret_cast<const float4*>(static_cast<const float*>(a.grad) + t0 + 128 * q));
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            v[q][0] = g[q].x + r[q].x; v[q][1] = g[q].y + r[q].y;
            v[q][2] = g[q].z + r[q].z; v[q][3] = g[q].w + r[q].w;
          }
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          *reinterpret_cast<float4*>(a.residual + t0 + 128 * q) = make_float4(v[q][0], v[q][1], v[q][2], v[q][3]);
          if (kDense) {
            if (kBf16) *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(a.grad) + t0 + 128 * q) = make_uint2(0u, 0u);
            else *reinterpret_cast<float4*>(static_cast<float*>(a.grad) + t0 + 128 * q) = make_float4(0.f, 0.f, 0.f, 0.f);
          }
        }
      } else {
#pragma unroll
        for (int q = 0; q < 8; ++q)
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int64_t i = t0 + 128 * q + j;
            v[q][j] = i < a.n ? load_grad<kBf16>(a.grad, i) + a.residual[i] : 0.f;
          }
#pragma unroll
        for (int q = 0; q < 8; ++q)
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int64_t i = t0 + 128 * q + j;
            if (i < a.n) {
              a.residual[i] = v[q][j];
              if (kDense) store_dense<kBf16>(a.grad, i, 0.f);
            }
          }
      }
      uint32_t mine = 0;  // bit 4 q + j: element (q, j) is a candidate (elements past the end are zero: never)
#pragma unroll
      for (int q = 0; q < 8; ++q)
#pragma unroll
        for (int j = 0; j < 4; ++j) mine |= static_cast<uint32_t>(key_of(v[q][j]) >= base) << (4 * q + j);
      const uint32_t here = __reduce_add_sync(0xFFFFFFFFu, __popc(mine));
      uint32_t direct = 0;  // a tile with more candidates than the stage holds goes to the list by itself
      bool fits = true;
      if (staged + here > kStage) {
        if (first < tile) flush();
        if (here > kStage) {
          fits = reserve(tile, here, &direct);
          first = tile + 1;
        } else {
          first = tile;
        }
      } else if (tile != first && lane == 0) {
        list.tiles[tile] = make_uint2(0u, 0u);  // found under `first`
      }
      uint2* to = here > kStage ? list.list + direct : stage + staged;
      if (here) {
        uint32_t put = 0;
#pragma unroll
        for (int q = 0; q < 8; ++q) {  // 128 consecutive elements, four per lane
          const uint32_t nib = (mine >> (4 * q)) & 15u;
          if (__ballot_sync(0xFFFFFFFFu, nib != 0) == 0) continue;
          uint32_t before = 0, all = 0;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const uint32_t m = __ballot_sync(0xFFFFFFFFu, (nib >> j) & 1u);
            before += __popc(m & lower);
            all += __popc(m);
          }
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if ((nib >> j) & 1u) {
              if (fits) {
                to[put + before + __popc(nib & ((1u << j) - 1u))] =
                    make_uint2(static_cast<uint32_t>(t0 + 128 * q + j), __float_as_uint(v[q][j]));
                // while the lines just written are in the cache
                if (key_of(v[q][j]) > sure) send<kBf16, kDense>(a, static_cast<uint32_t>(t0 + 128 * q + j), v[q][j]);
              }
              if (here > kStage) atomicAdd(&hist[bin_of(key_of(v[q][j]) - base)], 1u);
            }
          put += all;
        }
        if (here <= kStage) staged += here;
      }
    }
    if (first < g1) flush();
  }
  __syncthreads();
  for (int i = threadIdx.x; i < kBins; i += blockDim.x)
    if (hist[i]) atomicAdd(&list.state->hist[i], hist[i]);
  if (!last_block_done(&list.state->ticket[0])) return;

  // from the top bin down, eight bins per thread: the bin at which the running count reaches k
  __shared__ uint32_t wsum[33];
  constexpr int kPer = kBins / 256;
  const int top = kBins - 1 - kPer * static_cast<int>(threadIdx.x);
  const uint32_t count = __ldcg(&list.state->count), missing = __ldcg(&list.state->overflow);
  uint32_t c[kPer], run = 0;
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    c[i] = __ldcg(&list.state->hist[top - i]);
    run += c[i];
  }
  uint32_t above = block_excl_scan(run, wsum);
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    if (above < a.k && above + c[i] >= a.k) {
      list.state->bin = static_cast<uint32_t>(top - i);
      list.state->need = a.k - above;
      if (top - i == kBins - 1) list.state->mode = missing ? kWhole : kWide;
      else list.state->mode = missing || c[i] > kOneBlock ? kTies : kList;
    }
    above += c[i];
  }
  if (threadIdx.x == 0 && count < a.k) {
    // every non-zero is a candidate, everything is sent, or the sample missed (or none was taken)
    list.state->mode = kDense && base == 1u && missing == 0u ? kAll : base == 1u || a.k == a.n ? kZeros : kWhole;
    list.state->threshold = 0u;
    list.state->need = a.k == a.n ? a.k : a.k - count;
  }
}

// The need-th largest (kDown) or smallest of the m entries' words of `bits` bits, found by one block 11 bits at a
// time; `need` becomes the number of entries still wanted among the `equal` ones that share it.  word(i) is an entry's word, or
// kNone to leave the entry out.
constexpr uint64_t kNone = ~uint64_t(0);
template <bool kDown, typename Word>
__device__ uint32_t block_nth(uint32_t* hist, uint32_t* wsum, uint32_t* s_pick, uint32_t m, uint32_t* need,
                              uint32_t* equal, int bits, Word&& word) {
  const int tid = threadIdx.x;
  int width = bits < 11 ? bits : 11, shift = bits - width;
  uint32_t prefix = 0, left = *need;
  for (;;) {
    for (int i = tid; i < kBins; i += kThreads) hist[i] = 0;
    __syncthreads();
    const uint32_t mask = (1u << width) - 1u;
#pragma unroll 4
    for (uint32_t i = tid; i < m; i += kThreads) {
      const uint64_t w = word(i);
      if (w != kNone && (static_cast<uint32_t>(w) >> shift) >> width == prefix)
        atomicAdd(&hist[(static_cast<uint32_t>(w) >> shift) & mask], 1u);
    }
    __syncthreads();
    const int b0 = kDown ? kBins - 1 - 2 * tid : 2 * tid, b1 = kDown ? b0 - 1 : b0 + 1;
    const uint32_t c0 = hist[b0], c1 = hist[b1];
    const uint32_t before = block_excl_scan(c0 + c1, wsum);
    if (before < left && before + c0 >= left) {
      s_pick[0] = b0;
      s_pick[1] = before;
    } else if (before + c0 < left && before + c0 + c1 >= left) {
      s_pick[0] = b1;
      s_pick[1] = before + c0;
    }
    __syncthreads();
    left -= s_pick[1];
    prefix = (prefix << width) | s_pick[0];
    __syncthreads();
    if (shift == 0) break;
    width = shift < 11 ? shift : 11;
    shift -= width;
  }
  *need = left;
  *equal = hist[s_pick[0]];
  __syncthreads();
  return prefix;
}

// Adds n keys to this block's counts by digit(key); those whose digit is `bins` or more are left out.  What comes here is
// mostly tied: the digits of two lanes of a warp are counted for all that share them, and only the rest one by one.  One
// source of keys at a time: a choice between two within `key` keeps the loads from going out together (51.5 M equal bf16
// elements: 527 and 670 us).
template <typename Key, typename Digit>
__device__ __forceinline__ void count_digits(uint32_t* counts, uint32_t bins, int64_t n, Key&& key, Digit&& digit) {
  const int tid = threadIdx.x, lane = tid & 31;
  constexpr int kAhead = 8;
  const int64_t step = static_cast<int64_t>(gridDim.x) * kThreads * kAhead;
  for (int64_t i0 = static_cast<int64_t>(blockIdx.x) * kThreads * kAhead; i0 < n; i0 += step) {
    uint32_t d[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const int64_t i = i0 + u * kThreads + tid;
      d[u] = i < n ? key(i) : 0u;
    }
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      d[u] = digit(d[u]);
      bool in = i0 + u * kThreads + tid < n && d[u] < bins;
#pragma unroll
      for (int round = 0; round < 2; ++round) {
        const uint32_t left = __ballot_sync(0xFFFFFFFFu, in);
        if (left == 0u) break;
        const int leader = __ffs(left) - 1;
        const uint32_t first = __shfl_sync(0xFFFFFFFFu, d[u], leader);  // by all lanes, whether counted or not
        const bool same = in && d[u] == first;
        const uint32_t all = __ballot_sync(0xFFFFFFFFu, same);
        if (lane == leader) atomicAdd(&counts[first], static_cast<uint32_t>(__popc(all)));
        in = in && !same;
      }
      if (in) atomicAdd(&counts[d[u]], 1u);
    }
  }
  __syncthreads();
}

__device__ __forceinline__ void clear_counts(uint32_t* counts, int bins) {
  for (int i = threadIdx.x; i < bins; i += kThreads) counts[i] = 0;
  __syncthreads();
}

// Waits for all blocks of the grid, with a limit: true in every block (what the others wrote before is then visible) or,
// if one did not come in time because another grid holds its SM, false in every block.  One word decides.
__device__ __forceinline__ bool grid_meets(uint32_t* gate, int tries) {
  constexpr uint32_t kMet = 1u, kMissed = 2u;
  __shared__ uint32_t s_end;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t end = 0u;
    const bool last = atomicAdd(&gate[0], 1u) == gridDim.x - 1;
    for (int i = 0; !last && end == 0u && i < tries; ++i) {
      __nanosleep(100);
      end = *reinterpret_cast<volatile uint32_t*>(&gate[1]);
    }
    if (end == 0u) {
      const uint32_t mine = last ? kMet : kMissed, was = atomicCAS(&gate[1], 0u, mine);
      end = was == 0u ? mine : was;
    }
    __threadfence();
    s_end = end;
  }
  __syncthreads();
  return s_end == kMet;
}

// A listed key above the given one; another is no key at all.
__device__ __forceinline__ uint32_t listed_key(const uint2* list, int64_t i, uint32_t above) {
  const uint32_t key = list[i].y & 0x7FFFFFFFu;
  return key > above ? key : 0xFFFFFFFFu;
}

// The kBinShift-wide bin that holds the need-th largest of the vector's n keys and the listed ones above `above_key`, from two
// counts by the whole grid; *need becomes how many of its entries are selected, *entries how many it has.  False if the grid
// could not meet.  Not inlined: the ordinary selection does not come here.
__device__ __noinline__ bool find_bin(ListState* st, uint32_t* counts, uint32_t* wsum, uint32_t* s_pick, int64_t n,
                                      int64_t listed, const uint2* list, uint32_t above_key, const float* vector,
                                      uint32_t* floor_key, uint32_t* need, uint32_t* entries) {
  const int tid = threadIdx.x;
  uint32_t prefix = 0;
  // All blocks start as soon as the launch before is done; once they have met they only wait for the slowest count.
  if (!grid_meets(st->gate[0], 500)) return false;
#pragma unroll 1
  for (int level = 0; level < 2; ++level) {
    const int bins = level == 0 ? kBins : kFineBins;
    uint32_t* total = level == 0 ? st->coarse : st->fine;
    auto digit = [&](uint32_t k) {
      if (level == 0) return k >> kCoarseShift;
      return k >> kCoarseShift == prefix ? (k >> kBinShift) & (kFineBins - 1u) : 0xFFFFFFFFu;
    };
    clear_counts(counts, bins);
    count_digits(counts, bins, n, [&](int64_t i) { return key_of(__ldcs(vector + i)); }, digit);
    count_digits(counts, bins, listed, [&](int64_t i) { return listed_key(list, i, above_key); }, digit);
    for (int i = tid; i < bins; i += kThreads)
      if (counts[i]) atomicAdd(&total[i], counts[i]);
    if (!grid_meets(st->gate[level + 1], 1000000)) return false;
    const int top = bins - 1 - 2 * tid;  // from the top bin down, two per thread
    const uint32_t c0 = top > 0 ? __ldcg(&total[top]) : 0u, c1 = top > 0 ? __ldcg(&total[top - 1]) : 0u;
    const uint32_t above = block_excl_scan(c0 + c1, wsum), left = *need;
    if (above < left && above + c0 >= left) {
      s_pick[0] = top;
      s_pick[1] = above;
      s_pick[2] = c0;
    } else if (above + c0 < left && above + c0 + c1 >= left) {
      s_pick[0] = top - 1;
      s_pick[1] = above + c0;
      s_pick[2] = c1;
    }
    __syncthreads();
    *need = left - s_pick[1];
    *entries = s_pick[2];
    prefix = level == 0 ? s_pick[0] : prefix * kFineBins + s_pick[0];
    __syncthreads();
  }
  *floor_key = prefix << kBinShift;
  return true;
}

// Selection among the candidates, a grid of whole clusters; for kTies and kWhole only the threshold, from the whole vector.
// e and (kDense) g hold the values of elements that are not selected.
// 51.5 M fp32 elements, k = 0.1 % of two populations, the larger 1.1 k (kWide), pairs: the three passes of topk.cu 345 us, one
// cluster over the vector 2287 us, so 181 us.  All of them sent (ratio 1, kZeros): 519, 2755 and 366 us.
template <bool kBf16, bool kDense>
__global__ void __launch_bounds__(kThreads, 1) topk_select_kernel(const SelectArgs a) {
  __shared__ ClusterShared sh;
  __shared__ uint32_t s_count, s_base, s_pick[3];
  extern __shared__ __align__(16) uint32_t sub[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  ListState* st = a.list.state;
  start_dependents();
  wait_for_previous();
  uint32_t mode = st->mode;
  if (mode == kZeros) return;
  // What the adjust launch has sent is zero in the vector and is counted from the list.  All of it belongs to the selection;
  // where the sample was wrong about that, it is taken back.
  const uint32_t sure = kDense ? st->sure : 0xFFFFFFFFu;
  const int64_t listed = st->count < a.list.cap ? st->count : a.list.cap;
  auto sent_early = [&](int64_t i) { return kDense && (a.list.list[i].y & 0x7FFFFFFFu) > sure; };
  if (mode == kAll) {
    for (int64_t i = blockIdx.x * kThreads + tid; i < listed; i += gridDim.x * kThreads) {
      const uint2 e = a.list.list[i];
      if (!sent_early(i)) send<kBf16, kDense>(a, e.x, __uint_as_float(e.y));
    }
    return;
  }
  uint32_t floor_key = st->base + (st->bin << kBinShift), need = st->need;  // the k-th element's bin
  if (mode == kWide || mode == kWhole) {
    const bool wide = mode == kWide;
    uint32_t floor_found, need_found = a.k, entries;
    if (find_bin(st, sub, sh.wsum, s_pick, wide ? 0 : a.n, wide || kDense ? listed : 0, a.list.list, wide ? 0u : sure, a.residual,
                 &floor_found, &need_found, &entries)) {
      floor_key = floor_found;
      need = need_found;
      mode = wide && entries <= kOneBlock ? kList : kTies;
    }
  }
  if (mode == kTies) {
    auto digit = [&](uint32_t key) { return key - floor_key; };
    clear_counts(sub, kSubBins);
    count_digits(sub, kSubBins, a.n, [&](int64_t i) { return key_of(__ldcs(a.residual + i)); }, digit);
    if (kDense) count_digits(sub, kSubBins, listed, [&](int64_t i) { return listed_key(a.list.list, i, sure); }, digit);
    for (int i = tid; i < kSubBins; i += kThreads)
      if (sub[i]) atomicAdd(&st->sub[i], sub[i]);
    if (!last_block_done(&st->ticket[1])) return;
    constexpr int kPer = kSubBins / kThreads;
    const int top = kSubBins - 1 - kPer * tid;
    uint32_t c[kPer], run = 0;
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      c[i] = __ldcg(&st->sub[top - i]);
      run += c[i];
    }
    uint32_t above = block_excl_scan(run, sh.wsum);
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      if (above < need && above + c[i] >= need) {
        st->threshold = s_base = floor_key + static_cast<uint32_t>(top - i);
        st->need = need - above;
      }
      above += c[i];
    }
    if (tid == 0) st->mode = kTies;
    __syncthreads();
    if (kDense && s_base > sure)
      for (int64_t i = tid; i < listed; i += kThreads) {
        const uint2 e = a.list.list[i];
        if (sent_early(i) && (e.y & 0x7FFFFFFFu) <= s_base) unsend<kBf16, kDense>(a, e.x, __uint_as_float(e.y));
      }
    return;
  }
  if (mode == kList) {
    const uint32_t count = st->count;
    uint2* bin_list = a.list.bin_list;
    constexpr int kAhead = 8;
    const uint32_t step = gridDim.x * kThreads * kAhead;
    for (uint32_t i0 = blockIdx.x * kThreads * kAhead; i0 < count; i0 += step) {
      uint2 e[kAhead];
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        const uint32_t i = i0 + u * kThreads + tid;
        e[u] = i < count ? a.list.list[i] : make_uint2(0u, 0u);
      }
      if (tid == 0) s_count = 0;
      __syncthreads();
      uint32_t at[kAhead];
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        const bool valid = i0 + u * kThreads + tid < count;
        const float v = __uint_as_float(e[u].y);
        const uint32_t key = key_of(v), from_floor = key - floor_key;  // wraps below the bin
        if (kDense && valid && key >= floor_key && from_floor >= kSubBins && key <= sure) send<kBf16, kDense>(a, e[u].x, v);
        if (kDense && valid && key < floor_key && key > sure) unsend<kBf16, kDense>(a, e[u].x, v);
        const bool inside = valid && from_floor < kSubBins;
        at[u] = inside ? atomicAdd(&s_count, 1u) : 0xFFFFFFFFu;
      }
      __syncthreads();
      if (tid == 0 && s_count) s_base = atomicAdd(&st->in_bin, s_count);
      __syncthreads();
#pragma unroll
      for (int u = 0; u < kAhead; ++u)
        if (at[u] != 0xFFFFFFFFu) bin_list[s_base + at[u]] = e[u];  // kList: no more than bin_capacity()
      __syncthreads();
    }
    if (!last_block_done(&st->ticket[1])) return;
    // the bin's entries: the exact key, then the index limit among the entries that share it
    const uint32_t m = __ldcg(&st->in_bin);
    uint32_t equal = 0;
    if (tid == 0) st->mode = kList;
    const uint32_t low = block_nth<true>(sh.hist, sh.wsum, s_pick, m, &need, &equal, kBinShift, [&](uint32_t i) {
      return static_cast<uint64_t>((__ldcg(&bin_list[i].y) & 0x7FFFFFFFu) - floor_key);
    });
    const uint32_t threshold = floor_key + low;
    uint32_t last_index = 0xFFFFFFFFu;
    if (need < equal)
      last_index = block_nth<false>(sh.hist, sh.wsum, s_pick, m, &need, &equal, 32, [&](uint32_t i) {
        const uint2 e = __ldcg(&bin_list[i]);
        return (e.y & 0x7FFFFFFFu) == threshold ? static_cast<uint64_t>(e.x) : kNone;
      });
    if (tid == 0) {
      st->threshold = threshold;
      st->last_index = last_index;
    }
    return;
  }
  // the grid is not resident as a whole: the first cluster selects from the vector, the others leave
  cg::cluster_group cluster = cg::this_cluster();
  const int ctas = static_cast<int>(cluster.num_blocks()), me = static_cast<int>(cluster.block_rank());
  if (static_cast<int>(blockIdx.x) >= ctas) return;
  uint32_t threshold, need_eq;
  const int64_t per = (a.n + ctas - 1) / ctas;
  const int64_t lo = at_most(a.n, per * me), hi = at_most(a.n, lo + per);
  constexpr int kAhead = 16;
  cluster_threshold<3>(sh, a.k, [&](auto&& f) {
    for (int64_t i = lo + tid; i < hi; i += kAhead * kThreads) {
      float v[kAhead];
#pragma unroll
      for (int u = 0; u < kAhead; ++u) v[u] = i + u * kThreads < hi ? __ldcg(a.residual + i + u * kThreads) : 0.f;
#pragma unroll
      for (int u = 0; u < kAhead; ++u)
        if (i + u * kThreads < hi) f(key_of(v[u]));
    }
    for (int64_t i = me * kThreads + tid; kDense && i < listed; i += ctas * kThreads)
      if (sent_early(i)) f(a.list.list[i].y & 0x7FFFFFFFu);
  }, &threshold, &need_eq);
  if (kDense && threshold > sure) {
    for (int64_t i = me * kThreads + tid; i < listed; i += ctas * kThreads) {
      const uint2 e = a.list.list[i];
      if (sent_early(i) && (e.y & 0x7FFFFFFFu) <= threshold) unsend<kBf16, kDense>(a, e.x, __uint_as_float(e.y));
    }
    __threadfence();
    cluster.sync();
  }
  const int64_t per_warp = (hi - lo + kWarps - 1) / kWarps;
  const int64_t w0 = at_most(hi, lo + per_warp * warp), w1 = at_most(hi, w0 + per_warp);
  cluster_emit(sh, threshold, need_eq,
               [&](auto&& f) {
                 for (int64_t i = w0; i < w1; i += 32 * kAhead) {
                   float v[kAhead];
#pragma unroll
                   for (int u = 0; u < kAhead; ++u)
                     v[u] = i + 32 * u + lane < w1 ? __ldcg(a.residual + i + 32 * u + lane) : 0.f;
#pragma unroll
                   for (int u = 0; u < kAhead; ++u) {
                     if (i + 32 * u >= w1) break;
                     f(static_cast<uint32_t>(i + 32 * u + lane), v[u], i + 32 * u + lane < w1);
                   }
                 }
               },
               [&](uint32_t i, float v, uint32_t pos, bool selected) {
                 if (!selected || (kDense && key_of(v) == 0u)) return;  // a zero, or sent already
                 send<kBf16, kDense>(a, i, v);
                 if (!kDense) a.pairs[pos] = make_uint2(i, __float_as_uint(v));
               });
}

// What is left to put out, in index order.  A warp owns a run of tiles; kCount: how many of its elements lie above the
// threshold and at it, and the last block turns the counts into offsets; otherwise they are put out.  kList: pairs
// from the candidates (a dense result is complete already).  kTies, kZeros: from the vector.
template <bool kCount, bool kBf16, bool kDense>
__global__ void __launch_bounds__(kThreads, 1) topk_output_kernel(const SelectArgs a) {
  const int lane = threadIdx.x & 31;
  ListState* st = a.list.state;
  start_dependents();
  wait_for_previous();
  const uint32_t mode = st->mode;
  if (mode == kWhole || mode == kWide || mode == kAll) return;
  const uint32_t threshold = st->threshold, last_index = st->last_index, need = st->need;
  const bool early = kDense && st->sure != 0xFFFFFFFFu;
  if (mode == kList && kDense) {
    // the entries of the k-th element's bin: by one block, where they were gathered, 14 thousand took 24 us
    if (!kCount) return;
    const uint32_t sure = st->sure, m = st->in_bin;
    for (uint32_t i = blockIdx.x * kThreads + threadIdx.x; i < m; i += gridDim.x * kThreads) {
      const uint2 e = __ldcg(&a.list.bin_list[i]);
      const uint32_t key = e.y & 0x7FFFFFFFu;
      const bool selected = key > threshold || (key == threshold && e.x <= last_index);
      if (selected && key <= sure) send<kBf16, kDense>(a, e.x, __uint_as_float(e.y));
      if (!selected && key > sure) unsend<kBf16, kDense>(a, e.x, __uint_as_float(e.y));
    }
    return;
  }
  const uint32_t lower = (1u << lane) - 1u;
  const int64_t tiles = tile_count(a.n), runs = run_count(a.n);
  for (int64_t run = static_cast<int64_t>(blockIdx.x) * kWarps + (threadIdx.x >> 5); run < runs; run += gridDim.x * kWarps) {
    const int64_t t0 = run * kRun;
    uint2 done = kCount ? make_uint2(0u, 0u) : a.list.runs[run];
    if (mode == kList) {
      const uint2 place = lane < kRun && t0 + lane < tiles ? a.list.tiles[t0 + lane] : make_uint2(0u, 0u);
      for (int l = 0; l < kRun; ++l) {
        const uint32_t start = __shfl_sync(0xFFFFFFFFu, place.x, l), cnt = __shfl_sync(0xFFFFFFFFu, place.y, l);
#pragma unroll 4
        for (uint32_t i = 0; i < cnt; i += 32) {
          const uint2 e = i + lane < cnt ? a.list.list[start + i + lane] : make_uint2(0u, 0u);
          const uint32_t key = e.y & 0x7FFFFFFFu;
          const bool sent = i + lane < cnt && (key > threshold || (key == threshold && e.x <= last_index));
          const uint32_t m = __ballot_sync(0xFFFFFFFFu, sent);
          if (!kCount && sent) {
            a.pairs[done.x + __popc(m & lower)] = e;
            a.residual[e.x] = 0.f;  // nothing left to feed back
          }
          done.x += __popc(m);
        }
      }
    } else {
      const int64_t lo = t0 * kTile, hi = at_most(a.n, lo + kRun * kTile);
      constexpr int kAhead = 8;
      for (int64_t i0 = lo; i0 < hi; i0 += 32 * kAhead) {
        float v[kAhead];
#pragma unroll
        for (int u = 0; u < kAhead; ++u) v[u] = i0 + 32 * u + lane < hi ? __ldcg(a.residual + i0 + 32 * u + lane) : 0.f;
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
          const int64_t i = i0 + 32 * u + lane;
          const uint32_t key = key_of(v[u]);
          const bool gt = i < hi && key > threshold, eq = i < hi && key == threshold;
          const uint32_t m_gt = __ballot_sync(0xFFFFFFFFu, gt), m_eq = __ballot_sync(0xFFFFFFFFu, eq);
          if (!kCount) {
            const uint32_t r_gt = done.x + __popc(m_gt & lower), r_eq = done.y + __popc(m_eq & lower);
            if (gt || (eq && r_eq < need && !(early && key == 0u))) {  // a zero may be one that was sent, and sends nothing
              send<kBf16, kDense>(a, static_cast<uint32_t>(i), v[u]);
              if (!kDense) a.pairs[r_gt + (r_eq < need ? r_eq : need)] = make_uint2(static_cast<uint32_t>(i), __float_as_uint(v[u]));
            }
          }
          done.x += __popc(m_gt);
          done.y += __popc(m_eq);
        }
      }
    }
    if (kCount && lane == 0) a.list.runs[run] = done;
  }
  if (!kCount || !last_block_done(&st->ticket[2])) return;
  __shared__ uint32_t wsum[33];
  const int64_t per = (runs + kThreads - 1) / kThreads;
  const int64_t r0 = at_most(runs, threadIdx.x * per), r1 = at_most(runs, r0 + per);
  uint2 sum = make_uint2(0u, 0u);
  for (int64_t r = r0; r < r1; ++r) {
    const uint2 c = __ldcg(&a.list.runs[r]);
    sum.x += c.x;
    sum.y += c.y;
  }
  uint2 before;
  before.x = block_excl_scan(sum.x, wsum);
  __syncthreads();
  before.y = block_excl_scan(sum.y, wsum);
  for (int64_t r = r0; r < r1; ++r) {
    const uint2 c = __ldcg(&a.list.runs[r]);
    a.list.runs[r] = before;
    before.x += c.x;
    before.y += c.y;
  }
}

// Sixteen CTAs where a cluster of that size can be resident (it needs a GPC with as many free SMs), else the
// portable eight; `resident`: how many such clusters the device holds at once.  Asked once per kernel and device.
struct ClusterSize {
  std::atomic<int> of[64] = {};  // size + 64 * resident
};
cudaError_t cluster_size(const void* kernel, ClusterSize& cache, size_t most_smem, int* out, int* resident = nullptr) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  int size = dev < 64 ? cache.of[dev].load(std::memory_order_acquire) : 0;
  if (size == 0) {
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(most_smem));
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = kMaxCluster;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.gridDim = dim3(kMaxCluster);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = most_smem;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) != cudaSuccess || clusters <= 0) {
      attr.val.clusterDim.x = 8;
      cfg.gridDim = dim3(8);
      if (cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) != cudaSuccess || clusters <= 0) clusters = 1;
    }
    cudaGetLastError();  // a failed query only means the portable size
    size = static_cast<int>(cfg.gridDim.x) + 64 * clusters;
    if (dev < 64) cache.of[dev].store(size, std::memory_order_release);
  }
  *out = size % 64;
  if (resident != nullptr) *resident = size / 64;
  return cudaSuccess;
}

// `ctas`: of a cluster; `follows`: the blocks come up while the launch before ends, and wait for it.
template <typename... Params, typename... Args>
cudaError_t launch(void (*kernel)(Params...), unsigned grid, int threads, int ctas, size_t smem, bool follows, cudaStream_t s,
                   Args... args) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = attr;
  if (ctas > 1) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attr[cfg.numAttrs].val.clusterDim.x = ctas;
    attr[cfg.numAttrs].val.clusterDim.y = attr[cfg.numAttrs].val.clusterDim.z = 1;
    ++cfg.numAttrs;
  }
  if (follows) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[cfg.numAttrs].val.programmaticStreamSerializationAllowed = 1;
    ++cfg.numAttrs;
  }
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

template <bool kBf16, bool kDense>
cudaError_t run(const TopkArgs& t, const SelectArgs& a, cudaStream_t s) {
  static ClusterSize small_size, sample_size, select_size;
  constexpr size_t kItemBytes = kItemCap * sizeof(float);
  int ctas = 0;
  if (topk_fits_cluster(a.n)) {
    auto small = topk_cluster_kernel<kBf16, kDense>;
    cudaError_t e = cluster_size(reinterpret_cast<const void*>(small), small_size, kItemBytes, &ctas);
    if (e != cudaSuccess) return e;
    const int per = static_cast<int>(((a.n + ctas - 1) / ctas + 7) / 8 * 8);
    note_launch();
    return launch(small, ctas, kThreads, ctas, per * sizeof(float), false, s, a, per);
  }
  auto sample = topk_sample_kernel<kBf16>;
  cudaError_t e = cluster_size(reinterpret_cast<const void*>(sample), sample_size, 0, &ctas);
  if (e != cudaSuccess) return e;
  const uint32_t rank = sample_rank(a.n, a.k);
  note_launch(5);
  e = launch(sample, ctas, kThreads, ctas, 0, false, s, a, rank, sure_rank(a.n, a.k));
  if (e != cudaSuccess) return e;

  // tiles per group: about half a stage of candidates, and every warp of the grid busy
  const int64_t tiles = tile_count(a.n);
  const int resident = 148 * 3 * 8;
  const int64_t by_ratio = static_cast<int64_t>(0.5 * kStage * kSample / (static_cast<double>(rank) * kTile));
  const int group = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>({8, by_ratio, tiles / resident})));
  const int64_t blocks = (tiles + 8 * group - 1) / (8 * group);
  const unsigned grid = static_cast<unsigned>(std::min<int64_t>(148 * 3, blocks));
  constexpr size_t smem = 8 * kStage * sizeof(uint2);
  static_assert(smem + (kBins + 64) * sizeof(uint32_t) <= 48 << 10, "more would have to be asked for");
  const bool vec = ((reinterpret_cast<uintptr_t>(t.grad) | reinterpret_cast<uintptr_t>(t.residual)) & 15) == 0;
  auto adjust = vec ? topk_adjust_kernel<kBf16, true, kDense> : topk_adjust_kernel<kBf16, false, kDense>;
  e = launch(adjust, grid, 256, 1, smem, true, s, a, group);
  if (e != cudaSuccess) return e;

  auto select = topk_select_kernel<kBf16, kDense>;
  int resident_clusters = 0;
  e = cluster_size(reinterpret_cast<const void*>(select), select_size, kSubBins * sizeof(uint32_t), &ctas, &resident_clusters);
  if (e != cudaSuccess) return e;
  // no more than can meet (kWhole)
  const int clusters = static_cast<int>(std::min<int64_t>({128 / ctas, resident_clusters, (a.n + (1 << 20) - 1) >> 20}));
  e = launch(select, clusters * ctas, kThreads, ctas, kSubBins * sizeof(uint32_t), true, s, a);
  if (e != cudaSuccess) return e;
  const unsigned pgrid = static_cast<unsigned>(std::min<int64_t>(148, (run_count(a.n) + kWarps - 1) / kWarps));
  e = launch(topk_output_kernel<true, kBf16, kDense>, pgrid, kThreads, 1, 0, true, s, a);
  if (e != cudaSuccess) return e;
  return launch(topk_output_kernel<false, kBf16, kDense>, pgrid, kThreads, 1, 0, true, s, a);
}

}  // namespace

size_t topk_list_min_scratch_bytes(int64_t n) { return static_cast<size_t>(table_bytes(n)) + 2 * kTile * sizeof(uint2); }
size_t topk_list_scratch_bytes(int64_t n, int64_t k) {
  const int64_t cap = list_capacity(n, k);
  return std::max(topk_list_min_scratch_bytes(n),
                  static_cast<size_t>(table_bytes(n) + (cap + bin_capacity(cap)) * static_cast<int64_t>(sizeof(uint2))));
}

cudaError_t launch_topk_cluster(const TopkArgs& t, bool dense, cudaStream_t s) {
  SelectArgs a{};
  a.grad = const_cast<void*>(t.grad);
  a.residual = t.residual;
  a.pairs = static_cast<uint2*>(t.pairs);
  a.n = t.n;
  a.k = static_cast<uint32_t>(t.k);
  a.scale = t.scale;
  if (!topk_fits_cluster(t.n)) a.list = list_view(t.scratch, t.scratch_bytes, t.n, t.k);
  if (t.grad_is_bf16) return dense ? run<true, true>(t, a, s) : run<true, false>(t, a, s);
  return dense ? run<false, true>(t, a, s) : run<false, false>(t, a, s);
}

}  // namespace kern
}  // namespace mccl
