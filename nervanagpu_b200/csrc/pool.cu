// Max pooling over (feature map, depth, height, width) windows J,T,R,S on CDHWN tensors.
// Replaces hpool_max / spool_max (kernels/sass/hpool_max.sass) launched by
// NervanaGPU.fprop_pool / bprop_pool (nervanagpu/nervanagpu.py:773-818); output dimensions as
// PoolLayer (nervanagpu/layers.py:565-569).
//
// Numerics follow the reference kernel: taps are scanned in j,t,r,s order with a strict '>'
// compare so the first maximum wins (hpool_max.sass:264-281), taps outside the tensor are
// skipped, and the backward pass adds E[k,m,p,q,n] to dI at the argmax of window (k,m,p,q).
// Here the backward pass is a gather in two stages: the first records the argmax of every window
// (a scratch array in the library's workspace), the second lets each dI element visit the
// windows that contain it in increasing (k,m,p,q) order and sum, in fp32, the errors of those
// whose argmax it is. Overlapping windows so need neither atomics nor a zero-fill pass and the
// result is deterministic. Windows that do not overlap take one pass. The common 2-D shapes
// (2x2/2, 3x3/3, 3x3/2 and 3x3/1) have compile-time specialisations. The innermost
// dimension N is contiguous: each thread owns 8 images (one 16-byte lane) when N % 8 == 0, else 1.
#include <algorithm>
#include <cfloat>
#include <cuda_fp16.h>

#include "../../include/nervana_b200.h"
#include "host.h"

namespace ngb {
namespace {

struct PoolGeo {
  int N, C, D, H, W, J, T, R, S, K, M, P, Q;
  int pad_j, pad_d, pad_h, pad_w, str_j, str_d, str_h, str_w;
};

int pool_out_dim(int x, int f, int pad, int str) { return (x - f + 1 + 2 * pad + str - 1) / str; }

int make_pool_geo(const ng_pool_desc* d, PoolGeo& g) {
  if (!d) return fail(NG_ERR_INVALID_ARG, "pool descriptor is null");
  g.N = d->N; g.C = d->C; g.D = d->D; g.H = d->H; g.W = d->W;
  g.J = d->J; g.T = d->T; g.R = d->R; g.S = d->S;
  g.pad_j = d->pad_j; g.pad_d = d->pad_d; g.pad_h = d->pad_h; g.pad_w = d->pad_w;
  g.str_j = d->str_j; g.str_d = d->str_d; g.str_h = d->str_h; g.str_w = d->str_w;
  if (g.N < 1 || g.C < 1 || g.D < 1 || g.H < 1 || g.W < 1 || g.J < 1 || g.T < 1 || g.R < 1 || g.S < 1 ||
      g.str_j < 1 || g.str_d < 1 || g.str_h < 1 || g.str_w < 1 || g.pad_j < 0 || g.pad_d < 0 || g.pad_h < 0 ||
      g.pad_w < 0)
    return fail(NG_ERR_INVALID_ARG, "pool descriptor has a non-positive dimension");
  g.K = pool_out_dim(g.C, g.J, g.pad_j, g.str_j);
  g.M = pool_out_dim(g.D, g.T, g.pad_d, g.str_d);
  g.P = pool_out_dim(g.H, g.R, g.pad_h, g.str_h);
  g.Q = pool_out_dim(g.W, g.S, g.pad_w, g.str_w);
  if (g.K < 1 || g.M < 1 || g.P < 1 || g.Q < 1) return fail(NG_ERR_INVALID_ARG, "window larger than padded input");
  return NG_OK;
}

template <typename T, int V>
struct Vec;
template <>
struct Vec<__half, 8> {
  uint4 raw;
  __device__ float get(int i) const { return __half2float(reinterpret_cast<const __half*>(&raw)[i]); }
  __device__ void set(int i, float v) { reinterpret_cast<__half*>(&raw)[i] = __float2half_rn(v); }
};
template <>
struct Vec<__half, 1> {
  __half raw;
  __device__ float get(int) const { return __half2float(raw); }
  __device__ void set(int, float v) { raw = __float2half_rn(v); }
};
template <>
struct Vec<float, 4> {
  float4 raw;
  __device__ float get(int i) const { return reinterpret_cast<const float*>(&raw)[i]; }
  __device__ void set(int i, float v) { reinterpret_cast<float*>(&raw)[i] = v; }
};
template <>
struct Vec<float, 1> {
  float raw;
  __device__ float get(int) const { return raw; }
  __device__ void set(int, float v) { raw = v; }
};

// Scan window (k,m,p,q): per image lane the max and the flat (c,z,y,x) index of its first occurrence.
template <typename T, int V>
__device__ __forceinline__ void window_max(const PoolGeo& g, const T* __restrict__ I, int k, int m, int p, int q,
                                           int nv, float (&best)[V], int (&arg)[V]) {
#pragma unroll
  for (int i = 0; i < V; ++i) { best[i] = -FLT_MAX; arg[i] = 0; }
  const int c0 = k * g.str_j - g.pad_j, z0 = m * g.str_d - g.pad_d, y0 = p * g.str_h - g.pad_h,
            x0 = q * g.str_w - g.pad_w;
  for (int j = 0; j < g.J; ++j) {
    const int c = c0 + j;
    if (c < 0 || c >= g.C) continue;
    for (int t = 0; t < g.T; ++t) {
      const int z = z0 + t;
      if (z < 0 || z >= g.D) continue;
      for (int r = 0; r < g.R; ++r) {
        const int y = y0 + r;
        if (y < 0 || y >= g.H) continue;
        for (int s = 0; s < g.S; ++s) {
          const int x = x0 + s;
          if (x < 0 || x >= g.W) continue;
          const int flat = ((c * g.D + z) * g.H + y) * g.W + x;
          const Vec<T, V> v = *reinterpret_cast<const Vec<T, V>*>(I + (1ll * flat * g.N + nv * V));
#pragma unroll
          for (int i = 0; i < V; ++i) {
            const float f = v.get(i);
            if (f > best[i]) { best[i] = f; arg[i] = flat; }
          }
        }
      }
    }
  }
}

// first window index along one axis that can contain coordinate x, and the last
__device__ __forceinline__ void window_range(int x, int pad, int f, int str, int nout, int& lo, int& hi) {
  // windows w with w*str - pad <= x <= w*str - pad + f - 1
  const int a = x + pad - f + 1;
  lo = a <= 0 ? 0 : (a + str - 1) / str;
  hi = min(nout - 1, (x + pad) / str);
}

// O and/or arg_out may be null: the forward pass stores the maxima, the first stage of the
// backward pass stores the flat (c,z,y,x) index of each window's first maximum.
template <typename T, int V>
__global__ void pool_fprop_kernel(PoolGeo g, const T* __restrict__ I, T* __restrict__ O, int* __restrict__ arg_out,
                                  int mask_pos) {
  const int nvec = g.N / V;
  const long long total = 1ll * g.K * g.M * g.P * g.Q * nvec;
  for (long long i = blockIdx.x * 1ll * blockDim.x + threadIdx.x; i < total; i += 1ll * gridDim.x * blockDim.x) {
    long long r = i;
    const int nv = r % nvec; r /= nvec;
    const int q = r % g.Q; r /= g.Q;
    const int p = r % g.P; r /= g.P;
    const int m = r % g.M; r /= g.M;
    const int k = static_cast<int>(r);
    float best[V];
    int arg[V];
    window_max<T, V>(g, I, k, m, p, q, nv, best, arg);
    if (O) {
      Vec<T, V> out;
#pragma unroll
      for (int j = 0; j < V; ++j) out.set(j, best[j]);
      *reinterpret_cast<Vec<T, V>*>(O + i * V) = out;
    }
    if (arg_out) {
#pragma unroll
      for (int j = 0; j < V; ++j) arg_out[i * V + j] = (mask_pos && !(best[j] > 0.0f)) ? -1 : arg[j];
    }
  }
}

// Second stage of the backward pass: every input element sums the errors of the windows whose
// recorded argmax it is, visiting them in increasing (k,m,p,q) order.
template <typename T, int V>
__global__ void pool_gather_kernel(PoolGeo g, const int* __restrict__ arg, const T* __restrict__ E,
                                   T* __restrict__ dI) {
  const int nvec = g.N / V;
  const long long total = 1ll * g.C * g.D * g.H * g.W * nvec;
  for (long long i = blockIdx.x * 1ll * blockDim.x + threadIdx.x; i < total; i += 1ll * gridDim.x * blockDim.x) {
    long long r = i;
    const int nv = r % nvec; r /= nvec;
    const int flat = static_cast<int>(r);
    const int x = r % g.W; r /= g.W;
    const int y = r % g.H; r /= g.H;
    const int z = r % g.D; r /= g.D;
    const int c = static_cast<int>(r);
    int k0, k1, m0, m1, p0, p1, q0, q1;
    window_range(c, g.pad_j, g.J, g.str_j, g.K, k0, k1);
    window_range(z, g.pad_d, g.T, g.str_d, g.M, m0, m1);
    window_range(y, g.pad_h, g.R, g.str_h, g.P, p0, p1);
    window_range(x, g.pad_w, g.S, g.str_w, g.Q, q0, q1);
    float acc[V];
#pragma unroll
    for (int j = 0; j < V; ++j) acc[j] = 0.0f;
    for (int k = k0; k <= k1; ++k)
      for (int m = m0; m <= m1; ++m)
        for (int p = p0; p <= p1; ++p)
          for (int q = q0; q <= q1; ++q) {
            const long long o = ((((1ll * k * g.M + m) * g.P + p) * g.Q + q) * g.N) + nv * V;
            const Vec<T, V> e = *reinterpret_cast<const Vec<T, V>*>(E + o);
#pragma unroll
            for (int j = 0; j < V; ++j)
              if (arg[o + j] == flat) acc[j] += e.get(j);
          }
    Vec<T, V> out;
#pragma unroll
    for (int j = 0; j < V; ++j) out.set(j, acc[j]);
    *reinterpret_cast<Vec<T, V>*>(dI + i * V) = out;
  }
}

// ------------------------------------------------------------------------------------------
// Common 2-D windows (J = T = 1, rows of whole 16-byte vectors): window, strides and padding are
// compile-time constants. A thread owns one 16-byte vector of images and walks a strip of L rows
// of outputs (inputs, on the way back) of one pixel column, so that an input row that several of
// its windows share is read and reduced along x once: with one output per thread a 3x3 stride-1
// window fetches every input nine times through L1, with strips of four rows 4.5 times, and takes
// nine compares per output instead of six. Measured (fp16, forward / backward, before -> now):
// 3x3/1 pad 1 on 192 x 28 x 28 x 128: 63.7 -> 22.7 us (3.4 TB/s) / 236 -> 85 us; 3x3/2 on
// 64 x 55 x 55 x 128: 16.9 -> 10.4 us (5.9 TB/s); 2x2/2 on 64 x 224 x 224 x 64 backward without a
// record: 164 -> 136 us (6.8 TB/s, HBM bound); 2x2/2 fp32 on 50 x 107 x 107 x 112: 78 -> 47 us /
// 363 -> 87 us (6.7 TB/s). The 3x3/1 backward pass is bound by its compares: every input is tested
// against the records of nine windows (strips of 1, 2, 3, 4 rows: 90, 85, 92, 88 us).
// ------------------------------------------------------------------------------------------
template <typename T>
struct Vec16;

// Eight fp16 images. Maxima stay in fp16, in packed pairs: a mask per pair says which of the two
// running maxima a candidate beats, and maxima and tap numbers (16 bits each) are merged under it.
template <>
struct Vec16<__half> {
  static constexpr int kLanes = 8;
  uint32_t w[4];
  __device__ void load(const __half* p) {
    const uint4 r = __ldg(reinterpret_cast<const uint4*>(p));
    w[0] = r.x; w[1] = r.y; w[2] = r.z; w[3] = r.w;
  }
  __device__ void store(__half* p) const { *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]); }
  __device__ void to_float(float (&f)[8]) const {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 v = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
      f[2 * i] = v.x; f[2 * i + 1] = v.y;
    }
  }
  __device__ void from_float(const float (&f)[8]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const __half2 h = __floats2half2_rn(f[2 * i], f[2 * i + 1]);
      w[i] = *reinterpret_cast<const uint32_t*>(&h);
    }
  }
};
template <>
struct Vec16<float> {
  static constexpr int kLanes = 4;
  float w[4];
  __device__ void load(const float* p) {
    const float4 r = __ldg(reinterpret_cast<const float4*>(p));
    w[0] = r.x; w[1] = r.y; w[2] = r.z; w[3] = r.w;
  }
  __device__ void store(float* p) const { *reinterpret_cast<float4*>(p) = make_float4(w[0], w[1], w[2], w[3]); }
  __device__ void to_float(float (&f)[4]) const {
#pragma unroll
    for (int i = 0; i < 4; ++i) f[i] = w[i];
  }
  __device__ void from_float(const float (&f)[4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = f[i];
  }
};

// One byte per image: the tap that holds a window's first maximum.
template <typename T>
struct ArgBytes;
template <>
struct ArgBytes<__half> { uint32_t w[2]; };
template <>
struct ArgBytes<float> { uint32_t w[1]; };
template <typename T>
__device__ __forceinline__ ArgBytes<T> load_args(const uint8_t* p) {
  ArgBytes<T> a;
  if (sizeof(T) == 2) {
    const uint2 r = __ldg(reinterpret_cast<const uint2*>(p));
    a.w[0] = r.x; a.w[sizeof(T) == 2 ? 1 : 0] = r.y;
  } else {
    a.w[0] = __ldg(reinterpret_cast<const uint32_t*>(p));
  }
  return a;
}

// The tap that a window keeps when none of its values is above the initial maximum (NaN, minus infinity, in
// fp32 the lowest number). The general kernels keep input pixel 0, whether it lies in the window or not:
// `none` says so, and no_tap is the tap that no gradient goes to. The unpadded fp16 windows of 2-D data keep
// their own first tap.
constexpr uint32_t no_tap = 255u;

// Running maximum and tap of its first occurrence, per image.
template <typename T>
struct Best;
template <>
struct Best<__half> {
  uint32_t best[4], arg[4];
  __device__ void init(uint32_t tap = 0u) {   // `tap` stays where no value is above the first
#pragma unroll
    for (int i = 0; i < 4; ++i) { best[i] = 0xfc00fc00u; arg[i] = tap * 0x00010001u; }   // -inf
  }
  __device__ void merge(int i, uint32_t v, uint32_t a) {
    const uint32_t m = __hgt2_mask(*reinterpret_cast<const __half2*>(&v), *reinterpret_cast<const __half2*>(&best[i]));
    best[i] = (v & m) | (best[i] & ~m);
    arg[i] = (a & m) | (arg[i] & ~m);
  }
  __device__ void take(const Vec16<__half>& v, int tap) {
#pragma unroll
    for (int i = 0; i < 4; ++i) merge(i, v.w[i], static_cast<uint32_t>(tap) * 0x00010001u);
  }
  // The maximum without its tap. (__hmax2 ranks -0 below +0, of which the first is wanted; with it the padded 3x3
  // windows took 18.7 us at stride 1 and 10.5 at stride 2, on 192 x 28 x 28 x 128, instead of 22.7 and 12.5.)
  __device__ void raise(const Vec16<__half>& v) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t m = __hgt2_mask(*reinterpret_cast<const __half2*>(&v.w[i]), *reinterpret_cast<const __half2*>(&best[i]));
      best[i] = (v.w[i] & m) | (best[i] & ~m);
    }
  }
  __device__ void take(const Best<__half>& row, int tap) {   // the row's taps start at `tap`
#pragma unroll
    for (int i = 0; i < 4; ++i) merge(i, row.best[i], row.arg[i] + static_cast<uint32_t>(tap) * 0x00010001u);
  }
  __device__ Vec16<__half> value() const {
    Vec16<__half> v;
#pragma unroll
    for (int i = 0; i < 4; ++i) v.w[i] = best[i];
    return v;
  }
  // mask_pos 1: a window whose maximum is not positive names no tap (its error is dropped);
  // mask_pos 2: such windows are flagged in bit 7 and the backward pass decides
  __device__ ArgBytes<__half> bytes(int mask_pos) const {
    uint32_t a[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      a[i] = arg[i];
      if (mask_pos) {
        const uint32_t zero2 = 0u;
        const uint32_t pos = __hgt2_mask(*reinterpret_cast<const __half2*>(&best[i]), *reinterpret_cast<const __half2*>(&zero2));
        a[i] = mask_pos == 1 ? ((a[i] & pos) | (0x00ff00ffu & ~pos)) : (a[i] | (0x00800080u & ~pos));
      }
    }
    ArgBytes<__half> o;
    o.w[0] = __byte_perm(a[0], a[1], 0x6420);   // low byte of each 16-bit tap number
    o.w[1] = __byte_perm(a[2], a[3], 0x6420);
    return o;
  }
  // `e` where the maximum is tap `tap`, zero elsewhere
  __device__ Vec16<__half> credit(const Vec16<__half>& e, int tap) const {
    Vec16<__half> v;
#pragma unroll
    for (int i = 0; i < 4; ++i) v.w[i] = e.w[i] & __vcmpeq2(arg[i], static_cast<uint32_t>(tap) * 0x00010001u);
    return v;
  }
  __device__ void drop_not_positive() {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t zero2 = 0u;
      arg[i] |= ~__hgt2_mask(*reinterpret_cast<const __half2*>(&best[i]), *reinterpret_cast<const __half2*>(&zero2));
    }
  }
};
template <>
struct Best<float> {
  float best[4];
  uint32_t arg[4];
  __device__ void init(uint32_t tap = 0u) {
#pragma unroll
    for (int i = 0; i < 4; ++i) { best[i] = -FLT_MAX; arg[i] = tap; }
  }
  __device__ void take(const Vec16<float>& v, int tap) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (v.w[i] > best[i]) { best[i] = v.w[i]; arg[i] = static_cast<uint32_t>(tap); }
  }
  __device__ void raise(const Vec16<float>& v) {
#pragma unroll
    for (int i = 0; i < 4; ++i) best[i] = v.w[i] > best[i] ? v.w[i] : best[i];
  }
  __device__ void take(const Best<float>& row, int tap) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (row.best[i] > best[i]) { best[i] = row.best[i]; arg[i] = row.arg[i] + static_cast<uint32_t>(tap); }
  }
  __device__ Vec16<float> value() const {
    Vec16<float> v;
#pragma unroll
    for (int i = 0; i < 4; ++i) v.w[i] = best[i];
    return v;
  }
  __device__ ArgBytes<float> bytes(int mask_pos) const {
    ArgBytes<float> o;
    o.w[0] = 0u;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      uint32_t a = arg[i];
      if (mask_pos && !(best[i] > 0.0f)) a = mask_pos == 1 ? 255u : (a | 128u);
      o.w[0] |= a << (8 * i);
    }
    return o;
  }
  __device__ Vec16<float> credit(const Vec16<float>& e, int tap) const {
    Vec16<float> v;
#pragma unroll
    for (int i = 0; i < 4; ++i) v.w[i] = arg[i] == static_cast<uint32_t>(tap) ? e.w[i] : 0.0f;
    return v;
  }
  __device__ void drop_not_positive() {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (!(best[i] > 0.0f)) arg[i] = 0xffffffffu;
  }
};

struct Plane2d {
  int H, W, N, P, Q, strips;
  int none;    // see no_tap
};
// thread -> (strip, pixel column, first image of its vector); false past the end
__device__ __forceinline__ bool strip_pos(const Plane2d& g, int columns, int lanes, int& strip, int& x, int& n0) {
  const uint32_t nvec = static_cast<uint32_t>(g.N / lanes), t = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t px = t / nvec;
  n0 = static_cast<int>(t - px * nvec) * lanes;
  strip = static_cast<int>(px / static_cast<uint32_t>(columns));
  x = static_cast<int>(px) - strip * columns;
  return strip < g.strips;
}

// Forward pass. Rows are reduced along x first (first maximum of the
// row), then along y: the order in which ties are broken stays (r, s).
// kKind: the maximum alone, the maximum (O, may be null) and its tap (arg_out), or the mean.
enum Pool2dKind : int { P2_MAX = 0, P2_MAX_ARG = 1, P2_AVG = 2 };
template <typename T, int R, int S, int SH, int SW, int PH, int PW, int L, int kKind>
__global__ void __launch_bounds__(256) pool2d_fprop_kernel(Plane2d g, const T* __restrict__ I, T* __restrict__ O,
                                                          uint8_t* __restrict__ arg_out, int mask_pos) {
  constexpr bool kAvg = kKind == P2_AVG;
  constexpr int V = Vec16<T>::kLanes, NR = (L - 1) * SH + R;
  int strip, q, n0;
  if (!strip_pos(g, g.Q, V, strip, q, n0)) return;
  const int p0 = strip * L, y0 = p0 * SH - PH, x0 = q * SW - PW;
  const T* plane = I + static_cast<long long>(blockIdx.y) * g.H * g.W * g.N + n0;
  const long long out0 = ((static_cast<long long>(blockIdx.y) * g.P + p0) * g.Q + q) * g.N + n0;
  // (a window without padding lies inside the tensor; a strip may run past the last window)
  auto inside = [&](int j, int s) {
    const int y = y0 + j, x = x0 + s;
    return (PH == 0 || y >= 0) && ((PH == 0 && L == 1) || y < g.H) && (PW == 0 || (x >= 0 && x < g.W));
  };
  Vec16<T> raw[2][S];
  auto fetch = [&](int j, Vec16<T> (&row)[S]) {
#pragma unroll
    for (int s = 0; s < S; ++s)
      if (inside(j, s)) row[s].load(plane + (static_cast<long long>(y0 + j) * g.W + x0 + s) * g.N);
  };
  fetch(0, raw[0]);
  Best<T> win[L];
  float acc[kAvg ? L : 1][V];
#pragma unroll
  for (int j = 0; j < NR; ++j) {
    if (j + 1 < NR) fetch(j + 1, raw[(j + 1) & 1]);   // one row ahead of the reduction
    Best<T> row;
    float sum[V];
    if (kAvg) {
#pragma unroll
      for (int i = 0; i < V; ++i) sum[i] = 0.0f;
    } else {
      row.init();
    }
#pragma unroll
    for (int s = 0; s < S; ++s) {
      if (!inside(j, s)) continue;
      if (kAvg) {
        float f[V];
        raw[j & 1][s].to_float(f);
#pragma unroll
        for (int i = 0; i < V; ++i) sum[i] += f[i];
      } else {
        if (kKind == P2_MAX) row.raise(raw[j & 1][s]);
        else row.take(raw[j & 1][s], s);
      }
    }
#pragma unroll
    for (int l = 0; l < L; ++l) {
      const int r = j - l * SH;
      if (r < 0 || r >= R) continue;
      if (kAvg) {
#pragma unroll
        for (int i = 0; i < V; ++i) acc[kAvg ? l : 0][i] = r == 0 ? sum[i] : acc[kAvg ? l : 0][i] + sum[i];
      } else {
        if (r == 0) {
          const int top = y0 + l * SH;
          const bool has0 = blockIdx.y == 0 && top <= 0 && top + R > 0 && x0 <= 0 && x0 + S > 0;
          win[l].init(!g.none ? 0u : (has0 ? static_cast<uint32_t>(-top * S - x0) : no_tap));
        }
        if (kKind == P2_MAX) win[l].raise(row.value());
        else win[l].take(row, r * S);
      }
      if (r == R - 1 && p0 + l < g.P) {
        const long long o = out0 + static_cast<long long>(l) * g.Q * g.N;
        if (kAvg) {
          Vec16<T> v;
#pragma unroll
          for (int i = 0; i < V; ++i) acc[kAvg ? l : 0][i] *= 1.0f / static_cast<float>(R * S);
          v.from_float(acc[kAvg ? l : 0]);
          v.store(O + o);
        } else {
          if (kKind == P2_MAX || O) win[l].value().store(O + o);
          if (kKind == P2_MAX_ARG) {
            const ArgBytes<T> a = win[l].bytes(mask_pos);
            if (sizeof(T) == 2) *reinterpret_cast<uint2*>(arg_out + o) = make_uint2(a.w[0], a.w[sizeof(T) == 2 ? 1 : 0]);
            else *reinterpret_cast<uint32_t*>(arg_out + o) = a.w[0];
          }
        }
      }
    }
  }
}

// Backward pass from the recorded argmax bytes (maximum) or of the mean. A thread owns a column of
// L blocks of SH x SW inputs; it reads the error of every window that overlaps them once, in
// increasing (p, q) order, and adds it, in fp32, to the input that the record names.
// byte_and 0x7f7f7f7f drops the "maximum not positive" flag of the records (no ReLU mask wanted);
// with 0xffffffff a flagged byte is >= 128 and matches no tap.
template <typename T, int R, int S, int SH, int SW, int PH, int PW, int L, bool kAvg>
__global__ void __launch_bounds__(256) pool2d_gather_kernel(Plane2d g, int BW, const uint8_t* __restrict__ arg,
                                                           const T* __restrict__ E, T* __restrict__ dI,
                                                           uint32_t byte_and) {
  constexpr int V = Vec16<T>::kLanes, WP = (R + SH - 1) / SH, WQ = (S + SW - 1) / SW, NP = L + WP - 1;
  int strip, b, n0;
  if (!strip_pos(g, BW, V, strip, b, n0)) return;
  const int a0 = strip * L;
  const long long win0 = static_cast<long long>(blockIdx.y) * g.P * g.Q * g.N + n0;
  float acc[L][SH][SW][V];
#pragma unroll
  for (int l = 0; l < L; ++l)
#pragma unroll
    for (int dy = 0; dy < SH; ++dy)
#pragma unroll
      for (int dx = 0; dx < SW; ++dx)
#pragma unroll
        for (int i = 0; i < V; ++i) acc[l][dy][dx][i] = 0.0f;
  auto live = [&](int j, int wq) {
    const int p = a0 - (WP - 1) + j, q = b - (WQ - 1) + wq;
    return p >= 0 && p < g.P && q >= 0 && q < g.Q;
  };
  ArgBytes<T> rec[2][WQ];
  Vec16<T> err[2][WQ];
  auto fetch = [&](int j, int slot) {
#pragma unroll
    for (int wq = 0; wq < WQ; ++wq)
      if (live(j, wq)) {
        const long long o = win0 + (static_cast<long long>(a0 - (WP - 1) + j) * g.Q + b - (WQ - 1) + wq) * g.N;
        if (!kAvg) rec[slot][wq] = load_args<T>(arg + o);
        err[slot][wq].load(E + o);
      }
  };
  fetch(0, 0);
#pragma unroll
  for (int j = 0; j < NP; ++j) {
    if (j + 1 < NP) fetch(j + 1, (j + 1) & 1);
#pragma unroll
    for (int wq = 0; wq < WQ; ++wq) {
      if (!live(j, wq)) continue;
      float e[V];
      err[j & 1][wq].to_float(e);
      uint32_t idx[V];
      if (!kAvg) {
#pragma unroll
        for (int i = 0; i < V; ++i) idx[i] = ((rec[j & 1][wq].w[i >> 2] & byte_and) >> (8 * (i & 3))) & 255u;
      }
#pragma unroll
      for (int l = 0; l < L; ++l)
#pragma unroll
        for (int dy = 0; dy < SH; ++dy) {
          const int r = (l + WP - 1 - j) * SH + dy;      // tap row of this input inside window row j
          if (r < 0 || r >= R) continue;
#pragma unroll
          for (int dx = 0; dx < SW; ++dx) {
            const int s = (WQ - 1 - wq) * SW + dx;
            if (s >= S) continue;
#pragma unroll
            for (int i = 0; i < V; ++i) {
              // (the mean's shares one by one, as in the general kernel: their sum may exceed fp32 where none of them does)
              if (kAvg) acc[l][dy][dx][i] = fmaf(e[i], 1.0f / static_cast<float>(R * S), acc[l][dy][dx][i]);
              else if (idx[i] == static_cast<uint32_t>(r * S + s)) acc[l][dy][dx][i] += e[i];
            }
          }
        }
    }
  }
#pragma unroll
  for (int l = 0; l < L; ++l)
#pragma unroll
    for (int dy = 0; dy < SH; ++dy) {
      const int y = (a0 + l) * SH + dy - PH;
      if (y < 0 || y >= g.H) continue;
#pragma unroll
      for (int dx = 0; dx < SW; ++dx) {
        const int x = b * SW + dx - PW;
        if (x < 0 || x >= g.W) continue;
        Vec16<T> v;
        v.from_float(acc[l][dy][dx]);
        v.store(dI + ((static_cast<long long>(blockIdx.y) * g.H + y) * g.W + x) * g.N + n0);
      }
    }
}

// Backward pass when windows do not overlap, without a record: the thread of block (a, b) reads its
// window, finds the first maximum and writes the whole block.
template <typename T, int R, int S, int SH, int SW>
__global__ void __launch_bounds__(256) pool2d_bprop_kernel(Plane2d g, int BW, const T* __restrict__ I,
                                                          const T* __restrict__ E, T* __restrict__ dI, int mask_pos) {
  constexpr int V = Vec16<T>::kLanes;
  int a, b, n0;
  if (!strip_pos(g, BW, V, a, b, n0)) return;
  const long long base = (static_cast<long long>(blockIdx.y) * g.H + a * SH) * g.W + b * SW;
  Best<T> best;
  Vec16<T> e;
  best.init(g.none && !(blockIdx.y == 0 && a == 0 && b == 0) ? no_tap : 0u);
  const bool live = a < g.P && b < g.Q;     // (a ragged border belongs to no window)
  if (live) {
    Vec16<T> raw[R * S];
#pragma unroll
    for (int k = 0; k < R * S; ++k)
      raw[k].load(I + (base + static_cast<long long>(k / S) * g.W + k % S) * g.N + n0);
    e.load(E + ((static_cast<long long>(blockIdx.y) * g.P + a) * g.Q + b) * g.N + n0);
#pragma unroll
    for (int k = 0; k < R * S; ++k) best.take(raw[k], k);
    if (mask_pos) best.drop_not_positive();
  }
#pragma unroll
  for (int dy = 0; dy < SH; ++dy) {
    if (a * SH + dy >= g.H) break;
#pragma unroll
    for (int dx = 0; dx < SW; ++dx) {
      if (b * SW + dx >= g.W) break;
      Vec16<T> v;
      if (live && dy < R && dx < S) {
        v = best.credit(e, dy * S + dx);
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) v.w[i] = 0;
      }
      v.store(dI + (base + static_cast<long long>(dy) * g.W + dx) * g.N + n0);
    }
  }
}

// mode: 0 forward, 1 backward, 2 backward + ReLU mask, 3 forward that records the argmax in `arg`
// (bit 7: maximum not positive), 4 / 5 backward from such a record without / with the ReLU mask.
template <typename T, int R, int S, int SH, int SW, int PH, int PW, int LF, int LB, bool kAvg>
int launch_pool2d_strips(const PoolGeo& g, const T* I, T* EO, T* out, int mode, uint8_t* arg, cudaStream_t stream) {
  const int nvec = g.N / Vec16<T>::kLanes, planes = g.C * g.D;
  const int none = !(sizeof(T) == 2 && g.D == 1 && PH == 0 && PW == 0);
  Plane2d f = {g.H, g.W, g.N, g.P, g.Q, (g.P + LF - 1) / LF, none};
  const int BH = (g.H + PH + SH - 1) / SH, BW = (g.W + PW + SW - 1) / SW;
  Plane2d b = {g.H, g.W, g.N, g.P, g.Q, (BH + LB - 1) / LB, none};
  auto grid = [&](int strips, int columns) {
    return dim3(static_cast<unsigned>((1ll * strips * columns * nvec + 255) / 256), planes);
  };
  if (mode == 0) {
    pool2d_fprop_kernel<T, R, S, SH, SW, PH, PW, LF, kAvg ? P2_AVG : P2_MAX><<<grid(f.strips, g.Q), 256, 0, stream>>>(
        f, I, EO, nullptr, 0);
    NG_CHECK_LAUNCH();
    return NG_OK;
  }
  if (!kAvg && mode == 3) {
    pool2d_fprop_kernel<T, R, S, SH, SW, PH, PW, LF, P2_MAX_ARG><<<grid(f.strips, g.Q), 256, 0, stream>>>(f, I, EO, arg, 2);
    NG_CHECK_LAUNCH();
    return NG_OK;
  }
  if (!kAvg && mode < 3) {
    if constexpr (R <= SH && S <= SW) {
      b.strips = BH;
      pool2d_bprop_kernel<T, R, S, SH, SW><<<grid(BH, BW), 256, 0, stream>>>(b, BW, I, EO, out, mode == 2);
      NG_CHECK_LAUNCH();
      return NG_OK;
    } else {
      pool2d_fprop_kernel<T, R, S, SH, SW, PH, PW, LF, P2_MAX_ARG><<<grid(f.strips, g.Q), 256, 0, stream>>>(
          f, I, nullptr, arg, mode == 2);
      NG_CHECK_LAUNCH();
    }
  }
  pool2d_gather_kernel<T, R, S, SH, SW, PH, PW, LB, kAvg><<<grid(b.strips, BW), 256, 0, stream>>>(
      b, BW, arg, EO, out, mode == 4 ? 0x7f7f7f7fu : 0xffffffffu);
  NG_CHECK_LAUNCH();
  return NG_OK;
}

// Strips where they leave enough threads for the device, single rows elsewhere.
template <typename T, int R, int S, int SH, int SW, int PH, int PW, int LF, int LB, bool kAvg>
int launch_pool2d(const DeviceCtx* c, const PoolGeo& g, const void* I, const void* EO, void* out, int mode, void* arg,
                  cudaStream_t stream) {
  const T* in = static_cast<const T*>(I);
  T* eo = static_cast<T*>(const_cast<void*>(EO));
  const long long threads = 1ll * g.C * g.D * g.P * g.Q * (g.N / Vec16<T>::kLanes);
  if (threads >= 4ll * 1024 * c->sm_count)
    return launch_pool2d_strips<T, R, S, SH, SW, PH, PW, LF, LB, kAvg>(g, in, eo, static_cast<T*>(out), mode,
                                                                      static_cast<uint8_t*>(arg), stream);
  return launch_pool2d_strips<T, R, S, SH, SW, PH, PW, 1, 1, kAvg>(g, in, eo, static_cast<T*>(out), mode,
                                                                  static_cast<uint8_t*>(arg), stream);
}

// The window shapes that have kernels of their own: NG_OK when one ran, 1 when the general path must.
template <typename T, bool kAvg>
int try_pool2d(const DeviceCtx* c, const PoolGeo& g, const void* I, const void* EO, void* out, int mode, void* arg,
               cudaStream_t stream) {
  auto al = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
  const bool plain = g.J == 1 && g.T == 1 && g.str_j == 1 && g.str_d == 1 && g.pad_j == 0 && g.pad_d == 0 &&
                     g.N % Vec16<T>::kLanes == 0 && 1ll * g.C * g.D <= 65535 && al(I) && al(EO) && al(out) &&
                     1ll * (g.H + g.R) * (g.W + g.S) * (g.N / Vec16<T>::kLanes) < 0x7fffffffll;
  if (!plain || g.R != g.S || g.str_h != g.str_w || g.pad_h != g.pad_w) return 1;
#define NG_POOL2D(r, st, pd, lf, lb) \
  if (g.R == r && g.str_h == st && g.pad_h == pd) return launch_pool2d<T, r, r, st, st, pd, pd, lf, lb, kAvg>(c, g, I, EO, out, mode, arg, stream)
  NG_POOL2D(3, 2, 0, 3, 1);
  NG_POOL2D(2, 2, 0, 1, 1);
  NG_POOL2D(3, 3, 0, 1, 1);
  NG_POOL2D(3, 1, 1, 4, 2);
  NG_POOL2D(3, 2, 1, 3, 1);
#undef NG_POOL2D
  return 1;
}

// ------------------------------------------------------------------------------------------
// Windows without padding in any number of dimensions: every tap of every window exists, at the
// same distance from the window's first element. A thread owns one window and vector of images
// and requests eight taps at a time; HBM bound. 2x2x2x2 on 64 x 16 x 56 x 56 x 32, fp16: forward
// 54.9 -> 35.1 us (6.2 TB/s), backward 88 -> 65.8 us (6.4 TB/s).
// ------------------------------------------------------------------------------------------
constexpr int kTapTable = 64;
struct TapTable {
  int n;
  int off[kTapTable];   // elements, in (j, t, r, s) order
};
bool make_tap_table(const PoolGeo& g, TapTable& t) {
  if (g.pad_j || g.pad_d || g.pad_h || g.pad_w) return false;
  const long long n = 1ll * g.J * g.T * g.R * g.S;
  if (n > kTapTable || 1ll * g.J * g.D * g.H * g.W * g.N > 0x7fffffffll || 1ll * g.K * g.M * g.P * g.Q * g.N > 0x7fffffffll)
    return false;
  t.n = 0;
  for (int j = 0; j < g.J; ++j)
    for (int d = 0; d < g.T; ++d)
      for (int r = 0; r < g.R; ++r)
        for (int s = 0; s < g.S; ++s) t.off[t.n++] = (((j * g.D + d) * g.H + r) * g.W + s) * g.N;
  return true;
}
template <typename T>
__device__ __forceinline__ const T* window_base(const PoolGeo& g, const T* I, uint32_t t) {
  const uint32_t nvec = static_cast<uint32_t>(g.N / Vec16<T>::kLanes);
  uint32_t r = t / nvec;
  const int n0 = static_cast<int>(t - r * nvec) * Vec16<T>::kLanes;
  uint32_t d = r / g.Q;
  const int q = static_cast<int>(r - d * g.Q);
  r = d / g.P;
  const int p = static_cast<int>(d - r * g.P);
  d = r / g.M;
  const int m = static_cast<int>(r - d * g.M);
  return I + (((1ll * d * g.str_j * g.D + m * g.str_d) * g.H + p * g.str_h) * g.W + q * g.str_w) * g.N + n0;
}
template <typename T, bool kArg>
__device__ __forceinline__ void table_max(const TapTable& taps, const T* base, uint32_t first, Best<T>& best) {
  best.init(first);
  for (int k = 0; k < taps.n; k += 8) {
    Vec16<T> raw[8];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (k + u < taps.n) raw[u].load(base + taps.off[k + u]);
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (k + u < taps.n) {
        if (kArg) best.take(raw[u], k + u);
        else best.raise(raw[u]);
      }
  }
}
template <typename T>
__global__ void __launch_bounds__(256) pool_table_fprop_kernel(PoolGeo g, const __grid_constant__ TapTable taps,
                                                              uint32_t total, const T* __restrict__ I, T* __restrict__ O) {
  const uint32_t t = blockIdx.x * 256u + threadIdx.x;
  if (t >= total) return;
  Best<T> best;
  table_max<T, false>(taps, window_base(g, I, t), 0u, best);
  best.value().store(O + static_cast<size_t>(t) * Vec16<T>::kLanes);
}
// Backward pass when the windows tile the input exactly: the window's inputs are written where it
// was read, the error at the first maximum and zero elsewhere.
template <typename T>
__global__ void __launch_bounds__(256) pool_table_bprop_kernel(PoolGeo g, const __grid_constant__ TapTable taps,
                                                              uint32_t total, const T* __restrict__ I,
                                                              const T* __restrict__ E, T* __restrict__ dI, int mask_pos) {
  const uint32_t t = blockIdx.x * 256u + threadIdx.x;
  if (t >= total) return;
  Vec16<T> e;
  e.load(E + static_cast<size_t>(t) * Vec16<T>::kLanes);
  const T* base = window_base(g, I, t);
  Best<T> best;
  table_max<T, true>(taps, base, base - I < g.N ? 0u : no_tap, best);
  if (mask_pos) best.drop_not_positive();
  T* out = dI + (base - I);
#pragma unroll 4
  for (int k = 0; k < taps.n; ++k) best.credit(e, k).store(out + taps.off[k]);
}

int grid_for(long long total, const DeviceCtx* c) {
  const long long blocks = (total + 255) / 256;
  return static_cast<int>(std::max<long long>(1, std::min<long long>(blocks, c->sm_count * 32ll)));
}

// Backward pass when the windows tile the input exactly (no padding, stride == window and the
// extents divisible, in all four pooled dimensions): one thread per window and vector of images
// reads the window once, finds its first maximum and writes every input of the window (the error
// at the maximum, zero elsewhere). One pass, no scratch, each byte moved once.
template <typename T, int V>
__global__ void pool_bprop_tiled_kernel(PoolGeo g, const T* __restrict__ I, const T* __restrict__ E,
                                        T* __restrict__ dI, int mask_pos) {
  const int nvec = g.N / V;
  const long long total = 1ll * g.K * g.M * g.P * g.Q * nvec;
  for (long long i = blockIdx.x * 1ll * blockDim.x + threadIdx.x; i < total; i += 1ll * gridDim.x * blockDim.x) {
    long long r = i;
    const int nv = r % nvec; r /= nvec;
    const int q = r % g.Q; r /= g.Q;
    const int p = r % g.P; r /= g.P;
    const int m = r % g.M; r /= g.M;
    const int k = static_cast<int>(r);
    float best[V];
    int arg[V];
    window_max<T, V>(g, I, k, m, p, q, nv, best, arg);
    const Vec<T, V> e = *reinterpret_cast<const Vec<T, V>*>(E + i * V);
    for (int j = 0; j < g.J; ++j)
      for (int t = 0; t < g.T; ++t)
        for (int rr = 0; rr < g.R; ++rr)
          for (int s = 0; s < g.S; ++s) {
            const int flat = (((k * g.J + j) * g.D + m * g.T + t) * g.H + p * g.R + rr) * g.W + q * g.S + s;
            Vec<T, V> out;
#pragma unroll
            for (int l = 0; l < V; ++l)
              out.set(l, (arg[l] == flat && !(mask_pos && !(best[l] > 0.0f))) ? e.get(l) : 0.0f);
            *reinterpret_cast<Vec<T, V>*>(dI + (1ll * flat * g.N + nv * V)) = out;
          }
  }
}

// ------------------------------------------------------------------------------------------
// Average and L2 pooling. The reference declares both ops and defines them in numpy
// (benchmarks/pool_test.py:141-146: the mean, and the root of the sum of squares, over all
// J*T*R*S window positions, positions outside the tensor counting as zeros), but its device path
// runs the max kernel whatever the op (nervanagpu/nervanagpu.py:797). The backward passes are
// the derivatives of those definitions: dI += E / (J*T*R*S), and dI += E * I / O (0 where O is 0).
// ------------------------------------------------------------------------------------------
enum PoolOp : int { POOL_MAX = 0, POOL_AVG = 1, POOL_L2 = 2 };

// sum (avg) or sum of squares (l2) of window (k,m,p,q), per image lane
template <typename T, int V>
__device__ __forceinline__ void window_sum(const PoolGeo& g, const T* __restrict__ I, int k, int m, int p, int q,
                                           int nv, bool squares, float (&acc)[V]) {
#pragma unroll
  for (int i = 0; i < V; ++i) acc[i] = 0.0f;
  const int c0 = k * g.str_j - g.pad_j, z0 = m * g.str_d - g.pad_d, y0 = p * g.str_h - g.pad_h,
            x0 = q * g.str_w - g.pad_w;
  for (int j = 0; j < g.J; ++j) {
    const int c = c0 + j;
    if (c < 0 || c >= g.C) continue;
    for (int t = 0; t < g.T; ++t) {
      const int z = z0 + t;
      if (z < 0 || z >= g.D) continue;
      for (int r = 0; r < g.R; ++r) {
        const int y = y0 + r;
        if (y < 0 || y >= g.H) continue;
        for (int s = 0; s < g.S; ++s) {
          const int x = x0 + s;
          if (x < 0 || x >= g.W) continue;
          const long long flat = ((1ll * c * g.D + z) * g.H + y) * g.W + x;
          const Vec<T, V> v = *reinterpret_cast<const Vec<T, V>*>(I + (flat * g.N + nv * V));
#pragma unroll
          for (int i = 0; i < V; ++i) {
            const float f = v.get(i);
            acc[i] += squares ? f * f : f;
          }
        }
      }
    }
  }
}

template <typename T, int V>
__global__ void pool_fprop_op_kernel(PoolGeo g, int op, const T* __restrict__ I, T* __restrict__ O) {
  const int nvec = g.N / V;
  const long long total = 1ll * g.K * g.M * g.P * g.Q * nvec;
  const float inv = 1.0f / static_cast<float>(g.J * g.T * g.R * g.S);
  for (long long i = blockIdx.x * 1ll * blockDim.x + threadIdx.x; i < total; i += 1ll * gridDim.x * blockDim.x) {
    long long r = i;
    const int nv = r % nvec; r /= nvec;
    const int q = r % g.Q; r /= g.Q;
    const int p = r % g.P; r /= g.P;
    const int m = r % g.M; r /= g.M;
    const int k = static_cast<int>(r);
    float acc[V];
    window_sum<T, V>(g, I, k, m, p, q, nv, op == POOL_L2, acc);
    Vec<T, V> out;
#pragma unroll
    for (int j = 0; j < V; ++j) out.set(j, op == POOL_L2 ? sqrtf(acc[j]) : acc[j] * inv);
    *reinterpret_cast<Vec<T, V>*>(O + i * V) = out;
  }
}

// One thread per input element (and image lane group): sums over the windows that contain it, in
// increasing (k,m,p,q) order. The L2 pass recomputes each such window's norm.
template <typename T, int V>
__global__ void pool_bprop_op_kernel(PoolGeo g, int op, const T* __restrict__ I, const T* __restrict__ E,
                                     T* __restrict__ dI) {
  const int nvec = g.N / V;
  const long long total = 1ll * g.C * g.D * g.H * g.W * nvec;
  const float inv = 1.0f / static_cast<float>(g.J * g.T * g.R * g.S);
  for (long long i = blockIdx.x * 1ll * blockDim.x + threadIdx.x; i < total; i += 1ll * gridDim.x * blockDim.x) {
    long long r = i;
    const int nv = r % nvec; r /= nvec;
    const int x = r % g.W; r /= g.W;
    const int y = r % g.H; r /= g.H;
    const int z = r % g.D; r /= g.D;
    const int c = static_cast<int>(r);
    int k0, k1, m0, m1, p0, p1, q0, q1;
    window_range(c, g.pad_j, g.J, g.str_j, g.K, k0, k1);
    window_range(z, g.pad_d, g.T, g.str_d, g.M, m0, m1);
    window_range(y, g.pad_h, g.R, g.str_h, g.P, p0, p1);
    window_range(x, g.pad_w, g.S, g.str_w, g.Q, q0, q1);
    const Vec<T, V> own = *reinterpret_cast<const Vec<T, V>*>(I + i * V);
    float acc[V];
#pragma unroll
    for (int j = 0; j < V; ++j) acc[j] = 0.0f;
    for (int k = k0; k <= k1; ++k)
      for (int m = m0; m <= m1; ++m)
        for (int p = p0; p <= p1; ++p)
          for (int q = q0; q <= q1; ++q) {
            const long long o = ((((1ll * k * g.M + m) * g.P + p) * g.Q + q) * g.N) + nv * V;
            const Vec<T, V> e = *reinterpret_cast<const Vec<T, V>*>(E + o);
            if (op == POOL_AVG) {
#pragma unroll
              for (int j = 0; j < V; ++j) acc[j] += e.get(j) * inv;
            } else {
              float sq[V];
              window_sum<T, V>(g, I, k, m, p, q, nv, true, sq);
#pragma unroll
              for (int j = 0; j < V; ++j) {
                // the forward pass stored the norm rounded to T: divide by that value
                Vec<T, 1> o1;
                o1.set(0, sqrtf(sq[j]));
                const float norm = o1.get(0);
                if (norm > 0.0f) acc[j] += e.get(j) * own.get(j) / norm;
              }
            }
          }
    Vec<T, V> out;
#pragma unroll
    for (int j = 0; j < V; ++j) out.set(j, acc[j]);
    *reinterpret_cast<Vec<T, V>*>(dI + i * V) = out;
  }
}

template <typename T, int VW>
int run_pool_op(const PoolGeo& g, int op, const void* I, const void* E, void* out, bool backward, DeviceCtx* c,
                cudaStream_t stream) {
  if (op == POOL_AVG) {
    const int rc = try_pool2d<T, true>(c, g, I, backward ? E : out, out, backward, nullptr, stream);
    if (rc <= 0) return rc;
  }
  const bool vec = g.N % VW == 0 && (reinterpret_cast<uintptr_t>(I) & 15u) == 0 &&
                   (reinterpret_cast<uintptr_t>(E) & 15u) == 0 && (reinterpret_cast<uintptr_t>(out) & 15u) == 0;
  const long long out_elems = 1ll * g.K * g.M * g.P * g.Q * g.N;
  const long long in_elems = 1ll * g.C * g.D * g.H * g.W * g.N;
  const T* in = static_cast<const T*>(I);
  if (!backward) {
    if (vec) pool_fprop_op_kernel<T, VW><<<grid_for(out_elems / VW, c), 256, 0, stream>>>(g, op, in, static_cast<T*>(out));
    else pool_fprop_op_kernel<T, 1><<<grid_for(out_elems, c), 256, 0, stream>>>(g, op, in, static_cast<T*>(out));
  } else {
    const T* err = static_cast<const T*>(E);
    if (vec) pool_bprop_op_kernel<T, VW><<<grid_for(in_elems / VW, c), 256, 0, stream>>>(g, op, in, err, static_cast<T*>(out));
    else pool_bprop_op_kernel<T, 1><<<grid_for(in_elems, c), 256, 0, stream>>>(g, op, in, err, static_cast<T*>(out));
  }
  NG_CHECK_LAUNCH();
  return NG_OK;
}

bool tiles_exactly(const PoolGeo& g) {
  return g.pad_j == 0 && g.pad_d == 0 && g.pad_h == 0 && g.pad_w == 0 && g.str_j == g.J && g.str_d == g.T &&
         g.str_h == g.R && g.str_w == g.S && g.C % g.J == 0 && g.D % g.T == 0 && g.H % g.R == 0 && g.W % g.S == 0;
}

template <typename T, int VW>
int run_pool(const PoolGeo& g, const void* I, const void* EO, void* out, int mode, DeviceCtx* c,
             cudaStream_t stream) {
  const bool vec = g.N % VW == 0 && (reinterpret_cast<uintptr_t>(I) & 15u) == 0 &&
                   (reinterpret_cast<uintptr_t>(EO) & 15u) == 0 && (reinterpret_cast<uintptr_t>(out) & 15u) == 0;
  const long long out_elems = 1ll * g.K * g.M * g.P * g.Q * g.N;
  const long long in_elems = 1ll * g.C * g.D * g.H * g.W * g.N;
  // backward = record each window's argmax (scratch: one int per output element, in the
  // library workspace), then gather
  int* arg_ws = nullptr;
  if (mode != 0) {
    int rc = ensure_workspace(c, stream, static_cast<size_t>(out_elems) * sizeof(int));
    if (rc != NG_OK) return rc;
    arg_ws = reinterpret_cast<int*>(c->ws);
  }
  {
    const int rc = try_pool2d<T, false>(c, g, I, EO, out, mode, arg_ws, stream);
    if (rc <= 0) return rc;
  }
  TapTable taps;
  const bool table = vec && make_tap_table(g, taps);
  if (mode != 0 && tiles_exactly(g)) {
    if (table)
      pool_table_bprop_kernel<T><<<static_cast<unsigned>((out_elems / VW + 255) / 256), 256, 0, stream>>>(
          g, taps, static_cast<uint32_t>(out_elems / VW), static_cast<const T*>(I), static_cast<const T*>(EO),
          static_cast<T*>(out), mode == 2);
    else if (vec)
      pool_bprop_tiled_kernel<T, VW><<<grid_for(out_elems / VW, c), 256, 0, stream>>>(
          g, static_cast<const T*>(I), static_cast<const T*>(EO), static_cast<T*>(out), mode == 2);
    else
      pool_bprop_tiled_kernel<T, 1><<<grid_for(out_elems, c), 256, 0, stream>>>(
          g, static_cast<const T*>(I), static_cast<const T*>(EO), static_cast<T*>(out), mode == 2);
    NG_CHECK_LAUNCH();
    return NG_OK;
  }
  if (mode == 0) {
    T* O = static_cast<T*>(const_cast<void*>(EO));
    if (table)
      pool_table_fprop_kernel<T><<<static_cast<unsigned>((out_elems / VW + 255) / 256), 256, 0, stream>>>(
          g, taps, static_cast<uint32_t>(out_elems / VW), static_cast<const T*>(I), O);
    else if (vec)
      pool_fprop_kernel<T, VW><<<grid_for(out_elems / VW, c), 256, 0, stream>>>(g, static_cast<const T*>(I), O, nullptr, 0);
    else
      pool_fprop_kernel<T, 1><<<grid_for(out_elems, c), 256, 0, stream>>>(g, static_cast<const T*>(I), O, nullptr, 0);
    NG_CHECK_LAUNCH();
  } else {
    if (vec) {
      pool_fprop_kernel<T, VW><<<grid_for(out_elems / VW, c), 256, 0, stream>>>(g, static_cast<const T*>(I), nullptr,
                                                                               arg_ws, mode == 2);
      NG_CHECK_LAUNCH();
      pool_gather_kernel<T, VW><<<grid_for(in_elems / VW, c), 256, 0, stream>>>(g, arg_ws, static_cast<const T*>(EO),
                                                                                static_cast<T*>(out));
    } else {
      pool_fprop_kernel<T, 1><<<grid_for(out_elems, c), 256, 0, stream>>>(g, static_cast<const T*>(I), nullptr, arg_ws,
                                                                          mode == 2);
      NG_CHECK_LAUNCH();
      pool_gather_kernel<T, 1><<<grid_for(in_elems, c), 256, 0, stream>>>(g, arg_ws, static_cast<const T*>(EO),
                                                                          static_cast<T*>(out));
    }
    NG_CHECK_LAUNCH();
  }
  return NG_OK;
}

}  // namespace
}  // namespace ngb

using namespace ngb;

extern "C" {

int ng_pool_output_dims(const ng_pool_desc* d, int* K, int* M, int* P, int* Q) {
  PoolGeo g;
  int rc = make_pool_geo(d, g);
  if (rc != NG_OK) return rc;
  if (K) *K = g.K;
  if (M) *M = g.M;
  if (P) *P = g.P;
  if (Q) *Q = g.Q;
  return NG_OK;
}

int ng_pool_fprop(const ng_pool_desc* d, int dtype_bytes, const void* I, void* O, void* stream) {
  PoolGeo g;
  int rc = make_pool_geo(d, g);
  if (rc != NG_OK) return rc;
  if (!I || !O) return fail(NG_ERR_INVALID_ARG, "null tensor");
  if (1ll * g.C * g.D * g.H * g.W > 0x7fffffffll) return fail(NG_ERR_TOO_LARGE, "too many pixels");
  DeviceCtx* c = current_ctx();
  if (!c) return NG_ERR_CUDA;
  if (dtype_bytes == 2) return run_pool<__half, 8>(g, I, O, O, 0, c, static_cast<cudaStream_t>(stream));
  if (dtype_bytes == 4) return run_pool<float, 4>(g, I, O, O, 0, c, static_cast<cudaStream_t>(stream));
  return fail(NG_ERR_UNSUPPORTED, "pooling supports fp16 and fp32 tensors");
}

int ng_pool_bprop(const ng_pool_desc* d, int dtype_bytes, const void* I, const void* E, void* gradI, void* stream) {
  PoolGeo g;
  int rc = make_pool_geo(d, g);
  if (rc != NG_OK) return rc;
  if (!I || !E || !gradI) return fail(NG_ERR_INVALID_ARG, "null tensor");
  if (1ll * g.C * g.D * g.H * g.W > 0x7fffffffll) return fail(NG_ERR_TOO_LARGE, "too many pixels");
  DeviceCtx* c = current_ctx();
  if (!c) return NG_ERR_CUDA;
  if (dtype_bytes == 2) return run_pool<__half, 8>(g, I, E, gradI, 1, c, static_cast<cudaStream_t>(stream));
  if (dtype_bytes == 4) return run_pool<float, 4>(g, I, E, gradI, 1, c, static_cast<cudaStream_t>(stream));
  return fail(NG_ERR_UNSUPPORTED, "pooling supports fp16 and fp32 tensors");
}

int ng_pool_fprop_op(const ng_pool_desc* d, int op, int dtype_bytes, const void* I, void* O, void* stream) {
  if (op == POOL_MAX) return ng_pool_fprop(d, dtype_bytes, I, O, stream);
  if (op != POOL_AVG && op != POOL_L2) return fail(NG_ERR_INVALID_ARG, "pooling op must be 0 (max), 1 (avg) or 2 (l2)");
  PoolGeo g;
  int rc = make_pool_geo(d, g);
  if (rc != NG_OK) return rc;
  if (!I || !O) return fail(NG_ERR_INVALID_ARG, "null tensor");
  DeviceCtx* c = current_ctx();
  if (!c) return NG_ERR_CUDA;
  if (dtype_bytes == 2) return run_pool_op<__half, 8>(g, op, I, nullptr, O, false, c, static_cast<cudaStream_t>(stream));
  if (dtype_bytes == 4) return run_pool_op<float, 4>(g, op, I, nullptr, O, false, c, static_cast<cudaStream_t>(stream));
  return fail(NG_ERR_UNSUPPORTED, "pooling supports fp16 and fp32 tensors");
}

int ng_pool_bprop_op(const ng_pool_desc* d, int op, int dtype_bytes, const void* I, const void* E, void* gradI,
                     void* stream) {
  if (op == POOL_MAX) return ng_pool_bprop(d, dtype_bytes, I, E, gradI, stream);
  if (op != POOL_AVG && op != POOL_L2) return fail(NG_ERR_INVALID_ARG, "pooling op must be 0 (max), 1 (avg) or 2 (l2)");
  PoolGeo g;
  int rc = make_pool_geo(d, g);
  if (rc != NG_OK) return rc;
  if (!I || !E || !gradI) return fail(NG_ERR_INVALID_ARG, "null tensor");
  DeviceCtx* c = current_ctx();
  if (!c) return NG_ERR_CUDA;
  if (dtype_bytes == 2) return run_pool_op<__half, 8>(g, op, I, E, gradI, true, c, static_cast<cudaStream_t>(stream));
  if (dtype_bytes == 4) return run_pool_op<float, 4>(g, op, I, E, gradI, true, c, static_cast<cudaStream_t>(stream));
  return fail(NG_ERR_UNSUPPORTED, "pooling supports fp16 and fp32 tensors");
}

int ng_pool_argmax_bytes(const ng_pool_desc* d, int dtype_bytes, size_t* bytes) {
  PoolGeo g;
  int rc = make_pool_geo(d, g);
  if (rc != NG_OK) return rc;
  if (!bytes) return fail(NG_ERR_INVALID_ARG, "bytes is null");
  const bool plain = dtype_bytes == 2 && g.J == 1 && g.T == 1 && g.D == 1 && g.str_j == 1 && g.str_d == 1 &&
                     g.pad_j == 0 && g.pad_d == 0 && g.pad_h == 0 && g.pad_w == 0 && g.N % 8 == 0 && g.C <= 65535 &&
                     g.H <= 65535 && g.str_h == g.str_w && g.R == g.S &&
                     ((g.R == 3 && (g.str_h == 2 || g.str_h == 3)) || (g.R == 2 && g.str_h == 2));
  *bytes = plain ? static_cast<size_t>(g.K) * g.M * g.P * g.Q * g.N : 0;
  return NG_OK;
}

int ng_pool_fprop_argmax(const ng_pool_desc* d, int dtype_bytes, const void* I, void* O, void* argmax, void* stream) {
  PoolGeo g;
  int rc = make_pool_geo(d, g);
  if (rc != NG_OK) return rc;
  if (!I || !O || !argmax) return fail(NG_ERR_INVALID_ARG, "null tensor");
  if (dtype_bytes != 2 || (reinterpret_cast<uintptr_t>(argmax) & 7u))
    return fail(NG_ERR_UNSUPPORTED, "recorded argmax needs fp16 tensors and an 8-byte aligned buffer");
  const DeviceCtx* c = current_ctx();
  if (!c) return NG_ERR_CUDA;
  size_t bytes = 0;
  ng_pool_argmax_bytes(d, dtype_bytes, &bytes);
  rc = bytes == 0 ? 1 : try_pool2d<__half, false>(c, g, I, O, O, 3, argmax, static_cast<cudaStream_t>(stream));
  if (rc > 0) return fail(NG_ERR_UNSUPPORTED, "this pooling shape has no recorded-argmax path (see ng_pool_argmax_bytes)");
  return rc;
}

int ng_pool_bprop_argmax(const ng_pool_desc* d, int dtype_bytes, const void* argmax, const void* E, void* gradI,
                         int relu_mask, void* stream) {
  PoolGeo g;
  int rc = make_pool_geo(d, g);
  if (rc != NG_OK) return rc;
  if (!argmax || !E || !gradI) return fail(NG_ERR_INVALID_ARG, "null tensor");
  if (dtype_bytes != 2 || (reinterpret_cast<uintptr_t>(argmax) & 7u))
    return fail(NG_ERR_UNSUPPORTED, "recorded argmax needs fp16 tensors and an 8-byte aligned buffer");
  const DeviceCtx* c = current_ctx();
  if (!c) return NG_ERR_CUDA;
  size_t bytes = 0;
  ng_pool_argmax_bytes(d, dtype_bytes, &bytes);
  rc = bytes == 0 ? 1 : try_pool2d<__half, false>(c, g, nullptr, E, gradI, relu_mask ? 5 : 4, const_cast<void*>(argmax),
                                                  static_cast<cudaStream_t>(stream));
  if (rc > 0) return fail(NG_ERR_UNSUPPORTED, "this pooling shape has no recorded-argmax path (see ng_pool_argmax_bytes)");
  return rc;
}

int ng_pool_bprop_relu(const ng_pool_desc* d, int dtype_bytes, const void* I, const void* E, void* gradI,
                       void* stream) {
  PoolGeo g;
  int rc = make_pool_geo(d, g);
  if (rc != NG_OK) return rc;
  if (!I || !E || !gradI) return fail(NG_ERR_INVALID_ARG, "null tensor");
  if (1ll * g.C * g.D * g.H * g.W > 0x7fffffffll) return fail(NG_ERR_TOO_LARGE, "too many pixels");
  DeviceCtx* c = current_ctx();
  if (!c) return NG_ERR_CUDA;
  if (dtype_bytes == 2) return run_pool<__half, 8>(g, I, E, gradI, 2, c, static_cast<cudaStream_t>(stream));
  if (dtype_bytes == 4) return run_pool<float, 4>(g, I, E, gradI, 2, c, static_cast<cudaStream_t>(stream));
  return fail(NG_ERR_UNSUPPORTED, "pooling supports fp16 and fp32 tensors");
}

}  // extern "C"
