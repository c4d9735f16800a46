// Real FFT of 2^(LH+1) points by a group of lanes of one warp, with the values in registers.
//
// A real frame of N = 2h samples is a complex FFT of half the length, z[m] = x[2m] + i x[2m+1], and one pass
// that separates the even and odd halves.  The h values are a V x L matrix (V >= L, both powers of two): L lanes
// hold V values each, transform the columns in registers (radix V), exchange once through shared memory and
// transform the rows (radix L).  One exchange and two rounds of twiddles replace the log4(h) passes over shared
// memory of a Stockham FFT, and nothing wider than a warp ever has to wait: short frames share a warp.
//
//   h     4   8  16  32  64 128 256 512 1024 2048
//   V     2   4   4   8   8  16  16  32   32   64     values per lane
//   L     2   2   4   4   8   8  16  16   32   32     lanes per frame
#pragma once

#include <cuda_runtime.h>

#include <type_traits>

namespace mccl {
namespace kern {
namespace {

template <int I, int N, typename F>
__device__ __forceinline__ void static_for(F&& f) {
  if constexpr (I < N) {
    f(std::integral_constant<int, I>{});
    static_for<I + 1, N>(f);
  }
}

// cos and sin of 2 pi k / r, 0 <= k < r, by their power series on [0, pi/4]
constexpr double kTwoPi = 6.283185307179586476925286766559;
__host__ __device__ constexpr double series_cos(double x) {
  double term = 1.0, sum = 1.0;
  for (int i = 1; i < 12; ++i) {
    term *= -x * x / ((2.0 * i - 1.0) * (2.0 * i));
    sum += term;
  }
  return sum;
}
__host__ __device__ constexpr double series_sin(double x) {
  double term = x, sum = x;
  for (int i = 1; i < 12; ++i) {
    term *= -x * x / ((2.0 * i) * (2.0 * i + 1.0));
    sum += term;
  }
  return sum;
}
__host__ __device__ constexpr double root_cos(int k, int r) {
  return 2 * k >= r ? -root_cos(k - r / 2, r) : 4 * k > r ? -root_cos(r / 2 - k, r)
                   : (8 * k > r ? series_sin(kTwoPi * (r - 4 * k) / (4.0 * r)) : series_cos(kTwoPi * k / r));
}
__host__ __device__ constexpr double root_sin(int k, int r) {
  return 2 * k >= r ? -root_sin(k - r / 2, r) : 4 * k > r ? root_sin(r / 2 - k, r)
                   : (8 * k > r ? series_cos(kTwoPi * (r - 4 * k) / (4.0 * r)) : series_sin(kTwoPi * k / r));
}

// The 4096th roots of unity of the first octant, correctly rounded: every twiddle of every size is one of these
// with its parts swapped or negated.  (Computing the tables with sincospif cost a small call several
// microseconds before its first butterfly.)
constexpr int kRootOrder = 4096, kRootOctant = kRootOrder / 8;
struct RootTable {
  float c[kRootOctant + 1], s[kRootOctant + 1];
};
constexpr RootTable make_roots() {
  RootTable t{};
  for (int k = 0; k <= kRootOctant; ++k) {
    t.c[k] = static_cast<float>(series_cos(kTwoPi * k / kRootOrder));
    t.s[k] = static_cast<float>(series_sin(kTwoPi * k / kRootOrder));
  }
  return t;
}
__device__ constexpr RootTable kRoots = make_roots();

// exp(-2 pi i k / 4096), 0 <= k < 4096
__device__ __forceinline__ float2 root4096(int k) {
  const int octant = k / kRootOctant, i = k % kRootOctant;
  const int at = octant & 1 ? kRootOctant - i : i;
  const float c = kRoots.c[at], s = kRoots.s[at];
  const bool swapped = (octant + 1) & 2;  // octants 1, 2, 5, 6
  const float x = swapped ? s : c, y = swapped ? c : s;
  return make_float2(octant >= 2 && octant <= 5 ? -x : x, octant < 4 ? -y : y);
}

__host__ __device__ constexpr int bit_reverse(int v, int n) {
  int r = 0;
  for (int m = 1; m < n; m *= 2) {
    r = 2 * r + (v & 1);
    v >>= 1;
  }
  return r;
}

// Sums and differences of complex numbers.  kPacked: both parts in one instruction, which rounds as two do and takes one issue
// slot, but wants its numbers in pairs of registers.  Forward, 16 x 1 Mi samples, hop n_fft / 4, n_fft 512 .. 4096: 81, 88, 89,
// 133 us without, 76, 82, 82, 118 with it; for the window, the split and the scale as well: 78, 84, 88, 119.
template <bool kPacked>
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  if constexpr (kPacked) return __fadd2_rn(a, b);
  else return make_float2(a.x + b.x, a.y + b.y);
}
template <bool kPacked>
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
  if constexpr (kPacked) return __ffma2_rn(b, make_float2(-1.f, -1.f), a);
  else return make_float2(a.x - b.x, a.y - b.y);
}
// d * exp(-2 pi i K / R); kOpen: at an odd multiple of an eighth turn without the factor sqrt(1/2), which whoever adds the
// number up next multiplies in (`add_open`): one rounding less, as the compiler has it where sums are not packed.
constexpr float kHalfRoot = static_cast<float>(root_cos(1, 8));
template <int K, int R, bool kOpen>
__device__ __forceinline__ float2 mul_root(float2 d) {
  constexpr float c = static_cast<float>(root_cos(K, R)), s = static_cast<float>(root_sin(K, R));
  if constexpr (K == 0) return d;
  else if constexpr (4 * K == R) return make_float2(d.y, -d.x);
  else if constexpr (8 * K == R && kOpen) return make_float2(d.x + d.y, d.y - d.x);
  else if constexpr (8 * K == 3 * R && kOpen) return make_float2(d.y - d.x, -d.x - d.y);
  else if constexpr (8 * K == R) return make_float2(c * (d.x + d.y), c * (d.y - d.x));
  else if constexpr (8 * K == 3 * R) return make_float2(s * (d.y - d.x), -s * (d.x + d.y));
  else return make_float2(d.x * c + d.y * s, d.y * c - d.x * s);
}
// a + or - sqrt(1/2) b
template <int kSign>
__device__ __forceinline__ float2 add_open(float2 a, float2 b) {
  return __ffma2_rn(b, make_float2(kSign * kHalfRoot, kSign * kHalfRoot), a);
}

// Forward FFT of v[O .. O + R), in place, decimation in frequency: X[k] ends up in v[O + bit_reverse(k, R)].
// Radix 4 (a value meets one twiddle where two radix-2 stages would have two: fewer roundings and fewer
// instructions), with a last radix-2 stage for odd powers of two.
// kTurn: the values come from a stage that has turned number j by kTurn * j / 4R (0: from elsewhere).  Packed, those at an odd
// multiple of an eighth are open: j = R / 2 for 1 and 3, j = R / 4 and 3R / 4 for 2.
template <bool kPacked, int R, int O, int kTurn = 0, int N>
__device__ __forceinline__ void fft_registers(float2 (&v)[N]) {
  constexpr bool kOpenHalf = kPacked && (kTurn == 1 || kTurn == 3), kOpenQuarters = kPacked && kTurn == 2 && R >= 4;
  if constexpr (R == 2) {
    const float2 p = v[O], q = v[O + 1];
    v[O] = kOpenHalf ? add_open<1>(p, q) : add2<kPacked>(p, q);
    v[O + 1] = kOpenHalf ? add_open<-1>(p, q) : sub2<kPacked>(p, q);
  } else if constexpr (R >= 4) {
    constexpr int Q = R / 4;
    static_for<0, Q>([&](auto jc) {
      constexpr int j = decltype(jc)::value;
      constexpr bool half = kOpenHalf && j == 0, quarters = kOpenQuarters && j == 0;
      const float2 v0 = v[O + j], v2 = v[O + j + 2 * Q], v3 = v[O + j + 3 * Q];
      const float2 v1 = quarters ? make_float2(kHalfRoot * v[O + j + Q].x, kHalfRoot * v[O + j + Q].y) : v[O + j + Q];
      const float2 a0 = half ? add_open<1>(v0, v2) : add2<kPacked>(v0, v2), a1 = half ? add_open<-1>(v0, v2) : sub2<kPacked>(v0, v2);
      const float2 a2 = quarters ? add_open<1>(v1, v3) : add2<kPacked>(v1, v3);
      const float2 a3 = quarters ? add_open<-1>(v1, v3) : sub2<kPacked>(v1, v3);
      v[O + j] = add2<kPacked>(a0, a2);
      v[O + j + Q] = mul_root<2 * j, R, kPacked>(sub2<kPacked>(a0, a2));
      v[O + j + 2 * Q] = mul_root<j, R, kPacked>(make_float2(a1.x + a3.y, a1.y - a3.x));
      v[O + j + 3 * Q] = mul_root<3 * j, R, kPacked>(make_float2(a1.x - a3.y, a1.y + a3.x));
    });
    fft_registers<kPacked, Q, O>(v);
    fft_registers<kPacked, Q, O + Q, 2>(v);
    fft_registers<kPacked, Q, O + 2 * Q, 1>(v);
    fft_registers<kPacked, Q, O + 3 * Q, 3>(v);
  }
}

// kPacked: forward transforms and the stream kernel (see stft.cu); the kernel that shares its registers with an overlap-add
// by the whole CTA loses more to the pairs than it gains (16 x 1 Mi samples, n_fft 2048, bins-major: 229 and 238 us).
template <int LH, bool kPacked = true>
struct WarpFft {
  static constexpr int h = 1 << LH, n = 2 * h;
  static constexpr int V = 1 << ((LH + 1) / 2);  // values per lane
  static constexpr int L = 1 << (LH / 2);        // lanes per frame
  static constexpr int G = V / L;                // rows per lane (1 or 2)
  static constexpr int kPerWarp = 32 / L;        // frames per warp
  // float2 slots of one frame in shared memory: V rows of L + 1 (no bank conflict when a lane reads its row);
  // an odd total keeps different frames' values of one bin on different banks
  static constexpr int kSlot = (V * (L + 1) + (L == 8 ? 8 : 0)) | 1;
  static_assert(kSlot > h, "a slot also holds the h + 1 bins of a spectrum");

  // tw[r * L + c] = exp(-2 pi i r c / h): between the two radices;
  // split[k] = exp(-2 pi i k / n), k < h / 2: separates (or joins) the even and odd samples
  static constexpr int kTables = h + h / 2;
  static __device__ __forceinline__ void fill_tables(float2* tw, float2* split) {
    for (int i = threadIdx.x; i < h; i += blockDim.x) tw[i] = root4096((i / L) * (i % L) * (kRootOrder / h));
    for (int i = threadIdx.x; i < h / 2; i += blockDim.x) split[i] = root4096(i * (kRootOrder / n));
  }

  // In: v[r] = z[r * L + t].  Out: Z[t + L * g + V * k] in v[at(g, k)].  `buf`: the frame's slot.
  __host__ __device__ static constexpr int at(int g, int k) { return g * L + bit_reverse(k, L); }
  static __device__ __forceinline__ void transform(float2 (&v)[V], const float2* tw, float2* buf, int t) {
    fft_registers<kPacked, V, 0>(v);
    static_for<0, V>([&](auto rc) {
      constexpr int r = decltype(rc)::value;
      float2 z = v[bit_reverse(r, V)];
      if constexpr (r > 0) {
        const float2 w = tw[r * L + t];
        z = make_float2(z.x * w.x - z.y * w.y, z.x * w.y + z.y * w.x);
      }
      buf[r * (L + 1) + t] = z;
    });
    __syncwarp();
    static_for<0, V>([&](auto ic) {
      constexpr int i = decltype(ic)::value;
      v[i] = buf[(t + L * (i / L)) * (L + 1) + i % L];
    });
    __syncwarp();
    fft_registers<kPacked, L, 0>(v);
    if constexpr (G == 2) fft_registers<kPacked, L, L>(v);
  }

  // The same with half the shared memory: real parts first, then imaginary ones, in a slot of kHalfSlot floats.  (Where several
  // frames share a warp their slots start on different banks.)
  static constexpr int kHalfSlot = V * (L + 1) + (L == 16 && V == 32 ? 16 : L == 8 && V == 16 ? 8 : 0);
  static __device__ __forceinline__ void transform_halves(float2 (&v)[V], const float2* tw, float* buf, int t) {
    fft_registers<kPacked, V, 0>(v);
    static_for<1, V>([&](auto rc) {
      constexpr int r = decltype(rc)::value, at = bit_reverse(r, V);
      const float2 z = v[at], w = tw[r * L + t];
      v[at] = make_float2(z.x * w.x - z.y * w.y, z.x * w.y + z.y * w.x);
    });
    static_for<0, V>([&](auto rc) { buf[decltype(rc)::value * (L + 1) + t] = v[bit_reverse(decltype(rc)::value, V)].x; });
    __syncwarp();
    static_for<0, V>([&](auto ic) {
      constexpr int i = decltype(ic)::value;
      v[i].x = buf[(t + L * (i / L)) * (L + 1) + i % L];
    });
    __syncwarp();
    static_for<0, V>([&](auto rc) { buf[decltype(rc)::value * (L + 1) + t] = v[bit_reverse(decltype(rc)::value, V)].y; });
    __syncwarp();
    static_for<0, V>([&](auto ic) {
      constexpr int i = decltype(ic)::value;
      v[i].y = buf[(t + L * (i / L)) * (L + 1) + i % L];
    });
    __syncwarp();
    fft_registers<kPacked, L, 0>(v);
    if constexpr (G == 2) fft_registers<kPacked, L, L>(v);
  }

  static __device__ __forceinline__ float2 from_mirror_lane(float2 v, int t) {
    return make_float2(__shfl_sync(0xFFFFFFFFu, v.x, (L - t) & (L - 1), L),
                       __shfl_sync(0xFFFFFFFFu, v.y, (L - t) & (L - 1), L));
  }

  // Calls emit(k, 2 X[k]) for every bin k = 0 .. h, in pairs (k, h - k) that share their sums and their product:
  //   2E = Z[k] + conj Z[h-k],  2O = (Z[k] - conj Z[h-k]) / i,  X[k] = E + W_n^k O,  X[h-k] = conj(E - W_n^k O).
  // Z[h-k] sits in the mirrored lane at a register index fixed at compile time; lane 0 mirrors onto itself.
  template <typename Emit>
  static __device__ __forceinline__ void split_bins(const float2 (&v)[V], const float2* split, int t, Emit&& emit) {
    static_for<0, V / 2>([&](auto ic) {
      constexpr int g = decltype(ic)::value % G, k2 = decltype(ic)::value / G;
      const int k = t + L * g + V * k2;  // < h / 2
      const float2 zk = v[at(g, k2)];
      float2 zm = from_mirror_lane(v[at(G - 1 - g, L - 1 - k2)], t);
      const float2 own = g == 0 ? v[at(0, (L - k2) % L)] : v[at((G - g) % G, L - 1 - k2)];
      if (t == 0) zm = own;
      const float2 e = make_float2(zk.x + zm.x, zk.y - zm.y), o = make_float2(zk.y + zm.y, zm.x - zk.x);
      const float2 w = split[k];
      const float2 p = make_float2(w.x * o.x - w.y * o.y, w.x * o.y + w.y * o.x);
      emit(k, make_float2(e.x + p.x, e.y + p.y));
      emit(h - k, make_float2(e.x - p.x, p.y - e.y));
    });
    const float2 mid = v[at(0, L / 2)];  // lane 0: Z[h / 2], its own mirror image
    if (t == 0) emit(h / 2, make_float2(2.0f * mid.x, -2.0f * mid.y));
  }

  // The inverse of the split, in place, on x[r] = X[r * L + t] (and X[h] in `nyquist` on lane 0):
  //   P = X[k] + conj X[h-k],  Q = W_n^{-k} (X[k] - conj X[h-k]),  Z[k] = P + iQ,  Z[h-k] = conj(P - iQ)
  // with the parts swapped, so that the forward transform of the result is the swapped inverse transform.
  // Each lane forms the pairs of its lower half and hands Z[h-k] to the mirrored lane.  Lane 0 keeps its own
  // pairs, whose upper partner sits one register higher than in the other lanes.
  // `edge` scales the real parts of DC and Nyquist; their imaginary parts do not take part.
  static __device__ __forceinline__ void merge_bins(float2 (&x)[V], float2 nyquist, const float2* split, int t,
                                                    float edge) {
    if (t == 0) {
      x[0] = make_float2(edge * x[0].x, 0.f);
      nyquist = make_float2(edge * nyquist.x, 0.f);
    }
    static_for<0, V / 2>([&](auto rc) {
      constexpr int r = decltype(rc)::value, s = V - 1 - r;
      const float2 xk = x[r];
      float2 xm = from_mirror_lane(x[s], t);
      if (t == 0) xm = r == 0 ? nyquist : x[(s + 1) % V];
      const float2 p = make_float2(xk.x + xm.x, xk.y - xm.y), d = make_float2(xk.x - xm.x, xk.y + xm.y);
      const float2 w = split[r * L + t];
      const float2 q = make_float2(d.x * w.x + d.y * w.y, d.y * w.x - d.x * w.y);  // d * conj(w)
      x[r] = make_float2(p.y + q.x, p.x - q.y);
      const float2 upper = make_float2(q.x - p.y, p.x + q.y);
      const float2 got = from_mirror_lane(upper, t);
      if (t != 0) x[s] = got;
      if (r > 0 && t == 0) x[(s + 1) % V] = upper;
    });
    if (t == 0) x[V / 2] = make_float2(-2.0f * x[V / 2].y, 2.0f * x[V / 2].x);  // Z[h/2] = 2 conj X[h/2]
  }
};

}  // namespace
}  // namespace kern
}  // namespace mccl
