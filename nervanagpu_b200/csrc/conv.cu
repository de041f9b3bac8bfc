// Convolution passes on CDHWN activations / CTRSK filters / KMPQN outputs (fp16 storage).
//   fprop :  O = RN16(relu?(alpha * F (*) I))          nervanagpu/nervanagpu.py:642-650
//   bprop :  dI = RN16(alpha * F^T (*)^T E)             nervanagpu/nervanagpu.py:652-659
//   update:  dF = alpha * sum_{m,p,q,n} Ipatch * E^T    nervanagpu/nervanagpu.py:661-669
// Dimensions follow ConvLayer (nervanagpu/layers.py:281-325): M,P,Q = ceil((X - f + 1 + 2 pad)/stride).
//
// Fast path: the tcgen05 implicit-GEMM engine, fed straight from the activation tensors by TMA
// (padding = out-of-bounds zero fill, no im2col buffer, no filter shuffle):
//   fprop   D[K x MPQN]   = F[crs][k]^T (MN-major A)  *  I patches (MN-major B)
//   bprop   D[C x DHWN]   = F[c][k] per tap (K-major A)  *  E pixels reached through the tap (MN-major B)
//   update  D[C x K]/tap  = I pixels under the tap (K-major A)  *  E (K-major B), reduction over (m,p,q,n)
// A 64-element chunk of the pixel space is either 64 images of one pixel (N % 64 == 0) or, when
// the W stride is 1, 64 consecutive elements of the flattened (x, n) dimension of one image row
// (several pixels of a small minibatch, e.g. the shard of a minibatch that is split over GPUs).
// Image rows that are not a multiple of 64 elements are padded to whole chunks: the last chunk of
// a row runs past its end, where TMA zero-fills (or, between rows of the input, reads pixels
// whose products land in columns that are never stored).
// Strided layers: the backward pass runs phase by phase (the input pixels of one residue modulo the
// strides see a unit-stride layer over their share of the taps), small ones in a single launch
// (bprop_by_phases); with a minibatch that is no multiple of 64 the forward pass and the update read a copy
// of the input whose rows are split by x modulo the stride (phase_split), or, for small updates, a patch
// matrix. Small-C weight updates run as im2col + tensor-core GEMM. The plain CUDA-core kernels serve
// unaligned tensors, small strided backward passes and the tests.
#include <algorithm>
#include <cmath>

#include "../../include/nervana_b200.h"
#include "epilogue.cuh"
#include "host.h"

namespace ngb {

namespace {

struct Geo {
  int N, C, K, D, H, W, T, R, S, M, P, Q;
  int pad_d, pad_h, pad_w, str_d, str_h, str_w;
  __host__ __device__ long long sizeI() const { return 1ll * C * D * H * W * N; }
  __host__ __device__ long long sizeF() const { return 1ll * C * T * R * S * K; }
  __host__ __device__ long long sizeO() const { return 1ll * K * M * P * Q * N; }
};

int out_dim(int x, int f, int pad, int str) {
  // ceil((x - f + 1 + 2 pad) / str), as nervanagpu/layers.py:297-301
  const int num = x - f + 1 + 2 * pad;
  return (num + str - 1) / str;
}

int make_geo(const ng_conv_desc* d, Geo& g) {
  if (!d) return fail(NG_ERR_INVALID_ARG, "conv descriptor is null");
  g.N = d->N; g.C = d->C; g.K = d->K; g.D = d->D; g.H = d->H; g.W = d->W; g.T = d->T; g.R = d->R; g.S = d->S;
  g.pad_d = d->pad_d; g.pad_h = d->pad_h; g.pad_w = d->pad_w;
  g.str_d = d->str_d; g.str_h = d->str_h; g.str_w = d->str_w;
  if (g.N < 1 || g.C < 1 || g.K < 1 || g.D < 1 || g.H < 1 || g.W < 1 || g.T < 1 || g.R < 1 || g.S < 1 ||
      g.str_d < 1 || g.str_h < 1 || g.str_w < 1 || g.pad_d < 0 || g.pad_h < 0 || g.pad_w < 0)
    return fail(NG_ERR_INVALID_ARG, "conv descriptor has a non-positive dimension");
  if (g.N % 8 != 0) return fail(NG_ERR_INVALID_ARG, "N dim must be multiple of 8");
  if (g.K % 8 != 0) return fail(NG_ERR_INVALID_ARG, "K dim must be multiple of 8");
  g.M = out_dim(g.D, g.T, g.pad_d, g.str_d);
  g.P = out_dim(g.H, g.R, g.pad_h, g.str_h);
  g.Q = out_dim(g.W, g.S, g.pad_w, g.str_w);
  if (g.M < 1 || g.P < 1 || g.Q < 1) return fail(NG_ERR_INVALID_ARG, "filter larger than padded input");
  if (g.sizeI() > 0x7fffffffll * 8 || g.sizeO() > 0x7fffffffll * 8) return fail(NG_ERR_TOO_LARGE, "tensor too large");
  return NG_OK;
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// chunking of a (m,p,q,n)-like pixel space with innermost extents (xdim, N)
enum ChunkMode { CH_NONE = 0, CH_PIXEL = 1, CH_FLAT = 2 };
ChunkMode pick_chunk_mode(int N, int str_w) {
  if (N % kChunk == 0) return CH_PIXEL;
  if (str_w == 1) return CH_FLAT;
  return CH_NONE;
}
// chunks per image row of `xdim` pixels
int row_chunks(int N, int xdim, ChunkMode mode) {
  return mode == CH_FLAT ? static_cast<int>((1ll * xdim * N + kChunk - 1) / kChunk) : xdim * (N / kChunk);
}
// Columns of the GEMM view of a (rows, xdim, N) pixel space, and (flattened mode with ragged
// rows) the mapping of its padded columns to memory.
long long pixel_columns(TcParams& p, long long rows, int xdim, int N, ChunkMode mode) {
  const int cpr = row_chunks(N, xdim, mode);
  if (mode == CH_FLAT && (1ll * xdim * N) % kChunk != 0) {
    p.cmap.row_chunks = cpr;
    p.cmap.row_len = xdim * N;
  }
  return rows * cpr * kChunk;
}

// tensor map over an activation tensor (chan, z, y, x, n) seen as (n | x*n, x | 1, y, z, chan)
// (`blocked`: the tensor is the (z, y, chan, x, n) copy made by chan_block, see there)
int act_map(CUtensorMap* m, const void* base, int chan, int Z, int Y, int X, int N, ChunkMode mode, uint32_t box_chan,
            bool blocked = false) {
  uint64_t dims[5], str[4];
  const uint64_t xn = 1ull * X * N * 2;
  if (mode == CH_PIXEL) {
    dims[0] = N; dims[1] = X; str[0] = 1ull * N * 2;
  } else {
    dims[0] = 1ull * X * N; dims[1] = 1; str[0] = xn;
  }
  dims[2] = Y; dims[3] = Z; dims[4] = chan;
  if (blocked) {
    str[1] = xn * chan; str[2] = xn * chan * Y; str[3] = xn;
  } else {
    str[1] = xn; str[2] = xn * Y; str[3] = xn * Y * Z;
  }
  const uint32_t box[5] = {kChunk, 1, 1, 1, box_chan};
  return make_tensor_map(m, base, dims, str, box);
}

// ---- channel planes further apart than a page -------------------------------------------------
// A TMA box of an activation tensor is [channels][64 elements]: one 128-byte row per channel, the
// rows one channel plane (z * y * x * n elements) apart. When a plane is larger than a 2 MB page
// every row of every box lies in another page, and the loads run at less than half their rate:
// with planes of 1.8 MB the 3-D layer 64 -> 64, 3x3x3, 56x56, N = 32 ran at 620 TFLOP/s (with one image
// row per tile), with planes of 2.0 MB at 390, of 3.2 MB at 280, whatever the tensor's total size, and
// with 16 instead of 64 filters (a quarter of the output) in the same time. The remedy is one pass over
// the tensor before the product: a copy in (z, y, chan, x, n) order, whose channel rows are one
// image row (x * n elements) apart, so that a box spans a few hundred KB. The product reads the
// copy through a tensor map with the same dimensions and other strides; nothing in the kernel
// changes. The copy costs one read and one write of the tensor; every tap of the filter reads
// it again, so it pays from a few taps on.
constexpr long long kPlaneBytesBlocked = 1900000;   // between the last fast (1.81 MB) and first slow (2.01 MB) plane
bool wants_chan_block(int Z, int Y, int X, int N, int taps) {
  if (tuning().chan_block == 0) return false;
  const long long row = 2ll * X * N;
  if (row % 16 != 0) return false;
  if (tuning().chan_block == 2) return true;   // (tests: every shape)
  return taps >= 4 && row * Y * Z > kPlaneBytesBlocked;
}
size_t chan_block_bytes(int chan, int Z, int Y, int X, int N) {
  return (static_cast<size_t>(2) * chan * Z * Y * X * N + 255) & ~size_t(255);
}
// dst[(zy * chan + c)][row] = src[(c * zy_count + zy)][row], rows of `rowv` 16-byte vectors; one warp per row
__global__ void chan_block_kernel(const uint4* __restrict__ src, uint4* __restrict__ dst, int chan, long long zy_count,
                                  int rowv) {
  const long long r = blockIdx.x * static_cast<long long>(blockDim.y) + threadIdx.y;
  if (r >= zy_count * chan) return;
  const long long zy = r / chan;
  const int c = static_cast<int>(r - zy * chan);
  const uint4* s = src + (c * zy_count + zy) * rowv;
  uint4* d = dst + r * rowv;
  int v = threadIdx.x;
  for (; v + 96 < rowv; v += 128) {   // four loads in flight per lane
    const uint4 a = s[v], b = s[v + 32], e = s[v + 64], f = s[v + 96];
    d[v] = a; d[v + 32] = b; d[v + 64] = e; d[v + 96] = f;
  }
  for (; v < rowv; v += 32) d[v] = s[v];
}
int chan_block(DeviceCtx* c, cudaStream_t stream, const void* src, void* dst, int chan, int Z, int Y, int X, int N) {
  const long long rows = 1ll * chan * Z * Y;
  const long long blocks = (rows + 7) / 8;
  if (blocks > 0x7fffffffll) return fail(NG_ERR_TOO_LARGE, "tensor too large for the channel-blocked copy");
  (void)c;
  chan_block_kernel<<<static_cast<unsigned>(blocks), dim3(32, 8), 0, stream>>>(
      static_cast<const uint4*>(src), static_cast<uint4*>(dst), chan, 1ll * Z * Y, X * N / 8);
  NG_CHECK_LAUNCH();
  return NG_OK;
}
// ---- strided layers whose minibatch is no multiple of 64 ----------------------------------------
// A chunk then holds several pixels, and consecutive outputs of a row read every str_w-th input pixel.
// The copy splits the rows into their phases: dst[z][y][c][ph][x'][n] = I[c][z][y][str_w * x' + ph -
// pad_w][n], zero outside the row, so that output q of tap s reads x' = q + s / str_w of phase
// s % str_w: consecutive elements again. Channel rows are one split row apart, as in chan_block. The
// product itself needs no other change than this walk over the taps. One read and one write of the
// input; the CUDA-core kernels it replaces ran at 2.3 TFLOP/s: 96 -> 72 channels, 5x5 stride 2,
// 102x102, 88 images, 100.8 -> 0.8 ms.
// The update multiplies a row's last chunk, zeros in the error tensor past the row's end, with whatever the
// copy holds there: with ragged rows its copy has a row of Q pixels for every tap instead (`phases` = S), so
// that a NaN or infinity meets no zero of a tap that does not reach it.
// The CUDA-core kernels skip the taps that fall outside the tensor; here they meet zeros, and a product of zero
// and an infinity or NaN is NaN. Where those kernels ran before and that can show, they run once more over the
// result: forward and backward when a filter value is not finite (nonfinite_scan), and for the elements of a weight
// gradient beyond_patches that are NaN (conv_update_redo). Smaller updates took their patches, zeros included,
// to the tensor cores already.
int update_phases(const Geo& g) { return (1ll * g.Q * g.N) % kChunk == 0 ? g.str_w : std::max(g.str_w, g.S); }
int phase_row(const Geo& g, int phases) { return g.Q + (g.S - 1) / phases; }       // pixels per phase of a row
size_t phase_split_bytes(const Geo& g, int phases) {
  return (static_cast<size_t>(2) * g.C * g.D * g.H * phases * phase_row(g, phases) * g.N + 255) & ~size_t(255);
}
constexpr int kScanFlags = 128;      // blocks that scan a filter, each with a flag of its own (at most a block's threads)
// Whether this block's share of `n` vectors of eight values holds an infinity or NaN, in flags[blockIdx.x]
__device__ __forceinline__ void scan_share(const uint4* F, long long n, int blocks, int* flags) {
  int found = 0;
  for (long long i = blockIdx.x * 1ll * blockDim.x + threadIdx.x; i < n; i += 1ll * blocks * blockDim.x) {
    const uint4 v = __ldg(F + i);
    found |= __vcmpeq2(v.x & 0x7c007c00u, 0x7c007c00u) | __vcmpeq2(v.y & 0x7c007c00u, 0x7c007c00u) |
             __vcmpeq2(v.z & 0x7c007c00u, 0x7c007c00u) | __vcmpeq2(v.w & 0x7c007c00u, 0x7c007c00u);
  }
  found = __syncthreads_or(found);
  if (threadIdx.x == 0) flags[blockIdx.x] = found;
}
__global__ void __launch_bounds__(256) nonfinite_scan(const uint4* __restrict__ F, long long n, int* flags) {
  grid_dependency_wait();
  grid_launch_dependents();   // (the product sets itself up meanwhile)
  scan_share(F, n, gridDim.x, flags);
}
// one block per (z, y, c) row; the first `scans` of them also scan the filter (n_filter vectors)
__global__ void __launch_bounds__(128) phase_split_kernel(Geo g, int phases, int wp, const uint4* __restrict__ I, uint4* __restrict__ dst,
                                                          const uint4* __restrict__ F, long long n_filter, int scans, int* flags) {
  const int nvec = g.N >> 3, c = blockIdx.x % g.C;
  const long long zy = blockIdx.x / g.C;
  const uint4* src = I + (1ll * c * g.D * g.H + zy) * g.W * nvec;
  uint4* out = dst + 1ll * blockIdx.x * phases * wp * nvec;
  for (int i = threadIdx.x; i < phases * wp * nvec; i += 128) {
    const int pix = i / nvec, ph = pix / wp;
    const int x = (pix - ph * wp) * g.str_w + ph - g.pad_w;
    out[i] = x >= 0 && x < g.W ? __ldg(src + x * nvec + (i - pix * nvec)) : make_uint4(0, 0, 0, 0);
  }
  if (blockIdx.x < scans) scan_share(F, n_filter, scans, flags);
}
// F and flags (kScanFlags ints, of which `scans` are set) may be null
int phase_split(const Geo& g, int phases, const void* I, void* dst, const void* F, int* flags, int* scans, cudaStream_t stream) {
  const long long rows = 1ll * g.C * g.D * g.H;
  if (rows > 0x7fffffffll) return fail(NG_ERR_TOO_LARGE, "tensor too large for the phase-split copy");
  const int n = F ? static_cast<int>(std::min<long long>(rows, kScanFlags)) : 0;
  if (scans) *scans = n;
  phase_split_kernel<<<static_cast<unsigned>(rows), 128, 0, stream>>>(g, phases, phase_row(g, phases), static_cast<const uint4*>(I),
                                                                      static_cast<uint4*>(dst), static_cast<const uint4*>(F),
                                                                      g.sizeF() / 8, n, flags);
  NG_CHECK_LAUNCH();
  return NG_OK;
}
// the copy seen as (x' n, phase, y, z, chan)
int phase_map(CUtensorMap* m, const void* base, const Geo& g, int phases, uint32_t box_chan) {
  const uint64_t row = 2ull * phase_row(g, phases) * g.N;
  const uint64_t dims[5] = {1ull * phase_row(g, phases) * g.N, static_cast<uint64_t>(phases), static_cast<uint64_t>(g.H),
                            static_cast<uint64_t>(g.D), static_cast<uint64_t>(g.C)};
  const uint64_t chan = row * phases;
  const uint64_t str[4] = {row, chan * g.C, chan * g.C * g.H, chan};
  const uint32_t box[5] = {kChunk, 1, 1, 1, box_chan};
  return make_tensor_map(m, base, dims, str, box);
}
void fill_phases(TcParams& p, int phases) {
  p.phase_w = phases;
  p.pad_w = 0;         // (part of the copy)
}

size_t round256(size_t b) { return (b + 255) & ~size_t(255); }
// Room for the copies behind the split-K partials of the product `p` (whose tiling and number of
// partitions are final): `n` copies of the given sizes, returned as pointers into the workspace.
// NG_ERR_TOO_LARGE: none to be had, for a product that has a form without scratch (`optional`).
int chan_block_room(DeviceCtx* c, cudaStream_t stream, const TcParams& p, const size_t* bytes, void** ptrs, int n, bool optional = false) {
  const int nz_out = p.nz_out < 1 ? p.nz : p.nz_out;
  size_t off = p.splits > 1 ? static_cast<size_t>(p.splits) * nz_out * p.M * p.N * sizeof(float) : 0;
  off = (off + 255) & ~size_t(255);
  size_t total = off;
  for (int i = 0; i < n; ++i) total += bytes[i];
  if (optional && !scratch_or_none(c, stream, total)) return NG_ERR_TOO_LARGE;
  const int rc = ensure_workspace(c, stream, total);
  if (rc != NG_OK) return rc;
  for (int i = 0; i < n; ++i) {
    ptrs[i] = reinterpret_cast<uint8_t*>(c->ws) + off;
    off += bytes[i];
  }
  return NG_OK;
}

// Tensor map over an activation tensor whose box is a whole column tile of `nb` 64-wide chunks
// that lie in one image row: (n, chan, x, y, z) with a box of nb pixels when a pixel is one chunk
// (N = 64), else (n_lo, chan, n_hi, x, y) for 2-D data. The box lands in shared memory chunk by
// chunk, each [box_chan rows][64], as the per-chunk boxes of act_map would. Returns the value for
// TcParams::b_merge, 0 when the shape has no such map.
int act_map_merged(CUtensorMap* m, const void* base, int chan, int Z, int Y, int X, int N, uint32_t box_chan, int nb,
                   bool blocked = false) {
  if (tuning().merge_boxes == 0 || N % kChunk != 0 || nb < 2) return 0;
  const int cpi = N / kChunk;
  const uint64_t xn = 1ull * X * N * 2;
  const uint64_t chan_str = blocked ? xn : xn * Y * Z, y_str = blocked ? xn * chan : xn;
  uint64_t dims[5], str[4];
  uint32_t box[5];
  if (cpi == 1) {
    dims[0] = N; dims[1] = chan; dims[2] = X; dims[3] = Y; dims[4] = Z;
    str[0] = chan_str; str[1] = 1ull * N * 2; str[2] = y_str; str[3] = y_str * Y;
    box[0] = kChunk; box[1] = box_chan; box[2] = nb; box[3] = 1; box[4] = 1;
    return make_tensor_map(m, base, dims, str, box) == NG_OK ? 1 : 0;
  }
  if (Z != 1 || (nb % cpi != 0 && cpi % nb != 0)) return 0;
  dims[0] = kChunk; dims[1] = chan; dims[2] = cpi; dims[3] = X; dims[4] = Y;
  str[0] = chan_str; str[1] = 128; str[2] = 1ull * N * 2; str[3] = y_str;
  box[0] = kChunk; box[1] = box_chan; box[2] = std::min(cpi, nb); box[3] = std::max(1, nb / cpi); box[4] = 1;
  return make_tensor_map(m, base, dims, str, box) == NG_OK ? 2 : 0;
}

// filter (C, TRS, K) with K a multiple of 64, seen as (k_lo, c, k_hi, trs): a box of two chunks of
// 64 filters lands as [chunk][box_c rows][64]
int filter_map_merged(CUtensorMap* m, const void* base, const Geo& g, uint32_t box_c) {
  const int RST = g.T * g.R * g.S;
  uint64_t dims[5] = {kChunk, static_cast<uint64_t>(g.C), static_cast<uint64_t>(g.K / kChunk),
                      static_cast<uint64_t>(RST), 1};
  uint64_t str[4];
  str[0] = 1ull * g.K * 2 * RST; str[1] = 128; str[2] = 1ull * g.K * 2; str[3] = str[0] * g.C;
  const uint32_t box[5] = {kChunk, box_c, 2, 1, 1};
  return make_tensor_map(m, base, dims, str, box);
}

// tensor map over the filter (C, TRS, K) seen as (k, trs, c)
int filter_map(CUtensorMap* m, const void* base, const Geo& g, uint32_t box_c) {
  const int RST = g.T * g.R * g.S;
  uint64_t dims[5] = {static_cast<uint64_t>(g.K), static_cast<uint64_t>(RST), static_cast<uint64_t>(g.C), 1, 1};
  uint64_t str[4];
  str[0] = 1ull * g.K * 2; str[1] = str[0] * RST; str[2] = str[1] * g.C; str[3] = str[2];
  const uint32_t box[5] = {kChunk, 1, box_c, 1, 1};
  return make_tensor_map(m, base, dims, str, box);
}

// filter (C, T, R, S, K) with T x R x S taps seen as (k, s, r, t, c)
int filter_map_rows(CUtensorMap* m, const void* base, int K, int S, int R, int T, int C, uint32_t box_c) {
  const uint64_t k = 2ull * K;
  const uint64_t dims[5] = {static_cast<uint64_t>(K), static_cast<uint64_t>(S), static_cast<uint64_t>(R),
                            static_cast<uint64_t>(T), static_cast<uint64_t>(C)};
  const uint64_t str[4] = {k, k * S, k * S * R, k * S * R * T};
  const uint32_t box[5] = {kChunk, 1, 1, 1, box_c};
  return make_tensor_map(m, base, dims, str, box);
}

// One phase of the backward pass: the taps t0 + str_d * jt, r0 + str_h * jr, s0 + str_w * js of the
// filter, seen as (k, js, jr, jt, c)
int filter_map_phase(CUtensorMap* m, const void* base, const Geo& g, const int first[3], const int count[3], uint32_t box_c) {
  const uint64_t k = 2ull * g.K;
  const uint64_t dims[5] = {static_cast<uint64_t>(g.K), static_cast<uint64_t>(count[2]), static_cast<uint64_t>(count[1]),
                            static_cast<uint64_t>(count[0]), static_cast<uint64_t>(g.C)};
  const uint64_t str[4] = {k * g.str_w, k * g.S * g.str_h, k * g.R * g.S * g.str_d, k * g.T * g.R * g.S};
  const uint32_t box[5] = {kChunk, 1, 1, 1, box_c};
  const size_t off = k * ((1ull * first[0] * g.R + first[1]) * g.S + first[2]);
  return make_tensor_map(m, static_cast<const uint8_t*>(base) + off, dims, str, box);
}

void fill_taps(TcParams& p, const Geo& g, ChunkMode mode) {
  p.RS = g.R * g.S; p.S = g.S; p.R = g.R;
  p.tap_w = 1; p.tap_h = 1;
  p.pad_d = g.pad_d; p.pad_h = g.pad_h; p.pad_w = g.pad_w;
  p.str_d = g.str_d; p.str_h = g.str_h; p.str_w = g.str_w;
  p.inner_tap = mode == CH_FLAT ? g.N : 0;
  p.x_tap = mode == CH_FLAT ? 0 : 1;
}

void fill_decode(TcParams& p, int N, int X, int Y, int Z, ChunkMode mode) {
  p.dec_cpi = mode == CH_FLAT ? row_chunks(N, X, mode) : N / kChunk;
  p.dec_q = mode == CH_FLAT ? 1 : X;
  p.dec_p = Y;
  p.dec_m = Z;
}

// Two image rows per tile (see kLean 3 of the kernel), or one? Both by the model of tc_pick_tile: tiles run in
// waves of one per SM, a k-block costs the larger of its operand feed and its MMAs. (A layer of less than a
// wave of tiles is split over the SMs in the plain form, and is not with two rows: its waves count in
// parts there, in whole here.) `M` output channels, `a_rows` rows of A that the plain form loads, `taps`
// filter taps in R rows, images of `rows` rows of `row_cols` columns in `planes` planes. 0 = one row, else
// block_n, a multiple of bn_step. Measured, one row -> two: 64 -> 64, 3x3x3, 16x56x56, 32 images forward
// 620 -> 470 us, backward 636 -> 470; 64 -> 128, 3x3, 112x112, 64 images backward 300 -> 212; 64 -> 192, 5x5,
// 27x27, 128 images backward 95 -> 85; 3 -> 64, 11x11 stride 4, 224x224, 128 images forward 56 -> 48; 24 ->
// 16, 7x7, 80x80, 96 images 350 -> 240 and 352 -> 263. Forced on a layer of less than a wave (48 -> 40, 3x3,
// 30x30, 24 images, backward) 15.3 -> 17.3.
int pick_row_stack(const DeviceCtx* c, int M, int a_rows, int taps, int R, int red_chunks, int kb_rows, int rows,
                   long long planes, long long row_cols, float alpha, int bn_step = 64) {
  const int mode = tuning().row_stack;
  if (mode == 0 || tuning().lean_kernels == 0 || M > kChunk || R < 2 || rows < 2 || alpha != 1.0f) return 0;
  const double mma = (kb_rows / 16) * 66.0 + 30.0;
  auto best = [&](int a, long long cols, int num_kb, bool whole, int& block_n) {
    double t_best = -1.0;
    for (int bn = 256; bn >= 128; bn -= bn_step) {
      const long long tiles = (cols + bn - 1) / bn, sm = c->sm_count;
      const double waves = tiles < sm && !whole ? static_cast<double>(tiles) / sm : static_cast<double>((tiles + sm - 1) / sm);
      const double t = waves * (num_kb * std::max((a + bn) * kb_rows * 2.0 / 100, mma) + 600.0);
      if (t_best < 0.0 || t < t_best) { t_best = t; block_n = bn; }
    }
    return t_best;
  };
  int bn1 = 256, bn2 = 256;
  const double one = best(a_rows, planes * rows * row_cols, taps * red_chunks, false, bn1);
  const double two = best(2 * a_rows, planes * ((rows + 1) / 2) * row_cols, taps / R * (R + 1) * red_chunks, true, bn2);
  return mode == 2 || two < 0.95 * one ? bn2 : 0;
}
// The columns of a product over pairs of image rows: `x` elements from pixel to pixel of the output, `y`
// from row to row, `z` from plane to plane.
void fill_row_pairs(TcParams& p, int block_n, int N, int X, int rows, long long planes, ChunkMode mode, int x,
                    long long y, long long z) {
  p.row_stack = 1;
  p.block_n = block_n;
  p.m_halves = p.tiles_m = 1;
  p.cmap.row_chunks = row_chunks(N, X, mode);
  p.cmap.row_len = X * N;
  p.cmap.n = N; p.cmap.x = x; p.cmap.y = 2 * y; p.cmap.z = z;
  p.cmap.y_count = (rows + 1) / 2;
  p.cmap.pair_rows = rows;
  p.N = static_cast<int>(planes * p.cmap.y_count * p.cmap.row_chunks * kChunk);
  p.tiles_n = (p.N + block_n - 1) / block_n;
  p.nz_out = 2;
}

int pick_kb_rows(int C) {
  const int force = tuning().kb_rows;
  if (force >= 16 && force <= 64 && force % 16 == 0) return force;
  int best = 64, best_pad = ((C + 63) / 64) * 64;
  for (int r : {48, 32, 16}) {
    const int pad = ((C + r - 1) / r) * r;
    if (pad < best_pad) { best = r; best_pad = pad; }
  }
  return best;
}

// ------------------------------------------------------------------------------------------
// SIMT fall-backs (one thread per output element, fp32 accumulation)
// ------------------------------------------------------------------------------------------
// With flags (see phase_split): whether the result stands, after a wait for the kernel that made it
__device__ __forceinline__ bool skip_unflagged(const int* flags, int n) {
  if (!flags) return false;
  grid_dependency_wait();
  return !__syncthreads_or(threadIdx.x < n && flags[threadIdx.x] != 0);
}
__global__ void conv_fprop_simt(Geo g, const __half* __restrict__ I, const __half* __restrict__ F, __half* O,
                                float alpha, int relu, const int* flags, int n_flags) {
  if (skip_unflagged(flags, n_flags)) return;
  const long long total = g.sizeO();
  for (long long i = blockIdx.x * 1ll * blockDim.x + threadIdx.x; i < total; i += 1ll * gridDim.x * blockDim.x) {
    long long r = i;
    const int n = r % g.N; r /= g.N;
    const int q = r % g.Q; r /= g.Q;
    const int p = r % g.P; r /= g.P;
    const int m = r % g.M; r /= g.M;
    const int k = static_cast<int>(r);
    float acc = 0.0f;
    for (int c = 0; c < g.C; ++c)
      for (int t = 0; t < g.T; ++t) {
        const int z = m * g.str_d - g.pad_d + t;
        if (z < 0 || z >= g.D) continue;
        for (int rr = 0; rr < g.R; ++rr) {
          const int y = p * g.str_h - g.pad_h + rr;
          if (y < 0 || y >= g.H) continue;
          for (int s = 0; s < g.S; ++s) {
            const int x = q * g.str_w - g.pad_w + s;
            if (x < 0 || x >= g.W) continue;
            const float iv = __half2float(I[(((1ll * c * g.D + z) * g.H + y) * g.W + x) * g.N + n]);
            const float fv = __half2float(F[(((1ll * c * g.T + t) * g.R + rr) * g.S + s) * g.K + k]);
            acc = fmaf(iv, fv, acc);
          }
        }
      }
    acc *= alpha;
    if (relu) acc = fmaxf(acc, 0.0f);
    O[i] = __float2half_rn(acc);
  }
}

__global__ void conv_bprop_simt(Geo g, const __half* __restrict__ F, const __half* __restrict__ E, __half* dI,
                                float alpha, const int* flags, int n_flags) {
  if (skip_unflagged(flags, n_flags)) return;
  const long long total = g.sizeI();
  for (long long i = blockIdx.x * 1ll * blockDim.x + threadIdx.x; i < total; i += 1ll * gridDim.x * blockDim.x) {
    long long r = i;
    const int n = r % g.N; r /= g.N;
    const int x = r % g.W; r /= g.W;
    const int y = r % g.H; r /= g.H;
    const int z = r % g.D; r /= g.D;
    const int c = static_cast<int>(r);
    float acc = 0.0f;
    for (int t = 0; t < g.T; ++t) {
      const int mz = z + g.pad_d - t;
      if (mz < 0 || mz % g.str_d) continue;
      const int m = mz / g.str_d;
      if (m >= g.M) continue;
      for (int rr = 0; rr < g.R; ++rr) {
        const int py = y + g.pad_h - rr;
        if (py < 0 || py % g.str_h) continue;
        const int p = py / g.str_h;
        if (p >= g.P) continue;
        for (int s = 0; s < g.S; ++s) {
          const int qx = x + g.pad_w - s;
          if (qx < 0 || qx % g.str_w) continue;
          const int q = qx / g.str_w;
          if (q >= g.Q) continue;
          const __half* f = F + (((1ll * c * g.T + t) * g.R + rr) * g.S + s) * g.K;
          for (int k = 0; k < g.K; ++k) {
            const float ev = __half2float(E[(((1ll * k * g.M + m) * g.P + p) * g.Q + q) * g.N + n]);
            acc = fmaf(__half2float(f[k]), ev, acc);
          }
        }
      }
    }
    dI[i] = __float2half_rn(acc * alpha);
  }
}

// one filter element by a whole warp: lanes stride over (pixel, n), shuffle reduction
__device__ __forceinline__ void update_element(const Geo& g, const __half* __restrict__ I, const __half* __restrict__ E,
                                               void* dF, int out_f32, float alpha, long long i, int lane) {
  long long r = i;
  const int k = r % g.K; r /= g.K;
  const int s = r % g.S; r /= g.S;
  const int rr = r % g.R; r /= g.R;
  const int t = r % g.T; r /= g.T;
  const int c = static_cast<int>(r);
  float acc = 0.0f;
  const long long span = 1ll * g.M * g.P * g.Q * g.N;
  for (long long j0 = 0; j0 < span; j0 += 32) {
    const long long j = j0 + lane;
    long long rj = j;
    const int n = rj % g.N; rj /= g.N;
    const int q = rj % g.Q; rj /= g.Q;
    const int p = rj % g.P; rj /= g.P;
    const int m = static_cast<int>(rj);
    const int z = m * g.str_d - g.pad_d + t, y = p * g.str_h - g.pad_h + rr, x = q * g.str_w - g.pad_w + s;
    if (j < span && z >= 0 && z < g.D && y >= 0 && y < g.H && x >= 0 && x < g.W) {
      const float iv = __half2float(I[(((1ll * c * g.D + z) * g.H + y) * g.W + x) * g.N + n]);
      const float ev = __half2float(E[1ll * k * span + j]);
      acc = fmaf(iv, ev, acc);
    }
    if (__any_sync(0xffffffffu, acc != acc)) break;   // (NaN whatever follows: a gradient full of them is done at once)
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane == 0) {
    acc *= alpha;
    if (out_f32) static_cast<float*>(dF)[i] = acc;
    else static_cast<__half*>(dF)[i] = __float2half_rn(acc);
  }
}
__global__ void conv_update_simt(Geo g, const __half* __restrict__ I, const __half* __restrict__ E, void* dF,
                                 int out_f32, float alpha) {
  const long long total = g.sizeF();
  const int lane = threadIdx.x & 31;
  const long long warp0 = (blockIdx.x * 1ll * blockDim.x + threadIdx.x) >> 5;
  const long long nwarps = (1ll * gridDim.x * blockDim.x) >> 5;
  for (long long i = warp0; i < total; i += nwarps) update_element(g, I, E, dF, out_f32, alpha, i, lane);
}
// The elements of a gradient that are NaN, again, without the pixels outside the tensor. One read of the gradient
// when there are none.
__global__ void __launch_bounds__(256) conv_update_redo(Geo g, const __half* __restrict__ I, const __half* __restrict__ E,
                                                        void* dF, int out_f32, float alpha) {
  grid_dependency_wait();
  const long long total = g.sizeF();
  const int lane = threadIdx.x & 31;
  const long long warp0 = (blockIdx.x * 1ll * blockDim.x + threadIdx.x) >> 5;
  const long long nwarps = (1ll * gridDim.x * blockDim.x) >> 5;
  for (long long i0 = warp0 * 32; i0 < total; i0 += nwarps * 32) {
    bool nan = false;
    if (i0 + lane < total) {
      const float v = out_f32 ? static_cast<const float*>(dF)[i0 + lane] : __half2float(static_cast<const __half*>(dF)[i0 + lane]);
      nan = v != v;
    }
    for (uint32_t left = __ballot_sync(0xffffffffu, nan); left != 0u; left &= left - 1u)
      update_element(g, I, E, dF, out_f32, alpha, i0 + __ffs(static_cast<int>(left)) - 1, lane);
  }
}

// A kernel that waits for the one before it by itself
template <typename... P, typename... A>
int launch_dependent(int blocks, cudaStream_t stream, void (*kernel)(P...), A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(256);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = tuning().dependent_launch != 0 ? 1 : 0;
  NG_CUDA(cudaLaunchKernelEx(&cfg, kernel, args...));
  NG_CHECK_LAUNCH();
  return NG_OK;
}
int redo_blocks(const DeviceCtx* c) { return 8 * c->sm_count; }    // (that run all at once)

// ------------------------------------------------------------------------------------------
// im2col: col[crst][pixel * N + n] = I[c, z, y, x, n] (zero outside the image); 8 images per thread
// ------------------------------------------------------------------------------------------
// grid: x covers the (m, p, q, 8-image lane) positions of one patch row, y = (c, t, r, s) patch row
// (whole blocks of live threads whatever N is: with 16 images an output row is only 110 lanes wide)
__global__ void __launch_bounds__(256) im2col_kernel(Geo g, const __half* __restrict__ I, __half* __restrict__ col) {
  const int n8 = g.N / 8;
  const long long per_row = 1ll * g.M * g.P * g.Q * n8;
  const long long t0 = blockIdx.x * 256ll + threadIdx.x;
  if (t0 >= per_row) return;
  const int nv = static_cast<int>(t0 % n8);
  long long pix = t0 / n8;
  const int q = static_cast<int>(pix % g.Q); pix /= g.Q;
  const int p = static_cast<int>(pix % g.P);
  const int m = static_cast<int>(pix / g.P);
  int r = blockIdx.y;
  const int s = r % g.S; r /= g.S;
  const int rr = r % g.R; r /= g.R;
  const int t = r % g.T;
  const int c = r / g.T;
  const int z = m * g.str_d - g.pad_d + t, y = p * g.str_h - g.pad_h + rr, x = q * g.str_w - g.pad_w + s;
  uint4 v = make_uint4(0, 0, 0, 0);
  if (z >= 0 && z < g.D && y >= 0 && y < g.H && x >= 0 && x < g.W)
    v = *reinterpret_cast<const uint4*>(I + (((1ll * c * g.D + z) * g.H + y) * g.W + x) * g.N + nv * 8);
  reinterpret_cast<uint4*>(col)[blockIdx.y * per_row + t0] = v;
}

dim3 im2col_grid(const Geo& g) {
  const long long per_row = 1ll * g.M * g.P * g.Q * (g.N / 8);
  return dim3(static_cast<unsigned>((per_row + 255) / 256), g.C * g.T * g.R * g.S, 1);
}

int launch_1d(long long total, int threads, const DeviceCtx* c) {
  long long blocks = (total + threads - 1) / threads;
  return static_cast<int>(std::max<long long>(1, std::min<long long>(blocks, c->sm_count * 32ll)));
}

// ------------------------------------------------------------------------------------------
// Few input channels (first layers): tap blocks.
// One TMA box (64 n, bw x, bh y, 1, C) of the input carries the C*bh*bw rows that a block of
// bh x bw filter taps needs for one output pixel, already in the order (c, dy, dx). With
// rows = C*bh*bw a multiple of 16 this is one k-block of `rows` reduction rows, so a 3-channel
// 11x11 stride-4 layer runs as 9 k-blocks of 48 rows (bh = bw = 4) instead of 121 k-blocks of
// 16 rows holding 3 useful ones. The filter is re-packed (zero padded) to the same row order:
//   Fp[row = (c*bh + dy)*bw + dx][tb = (t*nr + r')*ns + s'][k] = F[c][t][r'*bh+dy][s'*bw+dx][k].
// ------------------------------------------------------------------------------------------
struct TapBlock {
  int bw = 0, bh = 0, rows = 0, nr = 0, ns = 0;
  bool ok = false;
};

// Weight update with few input rows per tap: one work item accumulates `acc_groups` taps at once
// (one TMEM accumulator each), so every chunk of the error tensor is fetched once per group of
// taps instead of once per tap. The group is limited by tensor memory (512 columns), by the
// shared-memory ring (at least four stages must remain) and balanced over the slices.
// Taps with at most 64 rows are also stacked along the 128 rows of one accumulator (`acc_taps`
// boxes of a_rows rows each), which halves (or better) the MMAs a tap costs.
void set_update_groups(TcParams& p, int taps, int a_rows) {
  const int cap = tuning().update_groups, cap_t = tuning().update_stack;   // limits on groups / stacking
  int t = std::max(1, std::min(std::min(kTileM / a_rows, 8), taps));
  if (cap_t > 0) t = std::max(1, std::min(t, cap_t));
  const int accs = (taps + t - 1) / t;                    // accumulators the whole filter needs
  int g = std::min(std::min(8, 512 / p.block_n), accs);
  if (cap > 0) g = std::max(1, std::min(g, cap));
  const int ring = 232448 - 1024 - 512 - static_cast<int>(kEpiStageBytes) - kTileM * 128;
  const int min_stages = tuning().update_min_stages > 0 ? std::max(2, tuning().update_min_stages) : 3;
  while (g > 1 && ((g * t * a_rows * 128 + p.block_n * 128) * min_stages > ring || g * t > 24)) --g;
  // the taps (not the accumulators) are spread evenly over the work items: 9 taps on items of at
  // most 6 become 5 + 4, not 6 + 3
  const int nz = (accs + g - 1) / g;
  p.taps_per_z = (taps + nz - 1) / nz;
  p.nz = (taps + p.taps_per_z - 1) / p.taps_per_z;
  p.acc_groups = (p.taps_per_z + t - 1) / t;
  p.acc_taps = t;
  p.pack_rows = a_rows;
  p.nz_out = taps;
}

// Rows of one tap among the MMA columns of update_swapped: whole groups of 8, and no more than 16 boxes
// per column tile (a lane of the producer warp loads each).
int swap_rows(int C) { return std::max(16, (C + 7) / 8 * 8); }
// Whether the update of a layer with few channels exchanges its operands (update_swapped). Plainly,
// `stack` taps share the 128 rows of an MMA whose columns are the filters, and 64 columns cost what 256
// do; exchanged, `per` taps share the 256 columns. It pays where that halves the MMAs, or with no more than
// 64 filters takes a third of them: 64 -> 64, 3x3x3, 16x56x56, 32 images 1010 -> 724 us; 48 -> 128, 5x5,
// 28x28, 128 images 79 -> 54; 64 -> 64, 3x3, 56x56, 128 images 103 -> 85. Otherwise the operand feed, larger
// by the error boxes, eats the gain (64 -> 128, 3x3, 112x112, 64 images: 237 and 249 us), and so it does
// where 16-row taps stack eight high in the plain form (16 -> 32, 5x5: 34 and 38). Small layers lose the
// 3 us of the transposition (40 -> 48, 3x3, 14x14, 128 images: 21.5 and 23.6).
bool wants_update_swap(const Geo& g, long long chunks) {
  if (tuning().update_swap == 0 || g.C > 64 || g.K > kTileM) return false;
  if (tuning().update_swap == 2) return true;    // (tests: every shape)
  const int rows = swap_rows(g.C), taps = g.T * g.R * g.S;
  const int stack = kTileM / rows, per = 256 / rows;
  const int accs = (taps + stack - 1) / stack, tiles = (taps + per - 1) / per;
  return rows > 16 && 2 * accs >= (g.K <= 64 ? 3 : 4) * tiles && (accs - tiles) * chunks > 3000;
}

// Column tile of the weight update (output channels): the smallest multiple of 64 that covers K
// in the fewest tiles, so that K = 192 or 384 does not pay for 256-wide MMAs.
int update_block_n(int K) {
  const int tiles = (K + 255) / 256;
  const int per = (K + tiles - 1) / tiles;
  return (per + 63) / 64 * 64;
}

TapBlock pick_tap_block(const Geo& g) {
  TapBlock best;
  long long best_cost = 0;
  for (int bh = 1; bh <= 16; ++bh)
    for (int bw = 1; bw <= 16; ++bw) {
      const int rows = g.C * bh * bw;
      if (rows % 16 != 0 || rows > 64) continue;
      const int nr = (g.R + bh - 1) / bh, ns = (g.S + bw - 1) / bw;
      // padded reduction length, plus a fixed charge per k-block
      const long long cost = 1ll * nr * ns * (rows + 8);
      if (!best.ok || cost < best_cost) {
        best.bw = bw; best.bh = bh; best.rows = rows; best.nr = nr; best.ns = ns; best.ok = true;
        best_cost = cost;
      }
    }
  return best;
}

__global__ void filter_repack_kernel(Geo g, TapBlock tb, const __half* __restrict__ F, __half* __restrict__ Fp) {
  const int k8 = g.K / 8;
  const int ntb = g.T * tb.nr * tb.ns;
  const long long total = 1ll * tb.rows * ntb * k8;
  for (long long i = blockIdx.x * 1ll * blockDim.x + threadIdx.x; i < total; i += 1ll * gridDim.x * blockDim.x) {
    long long r = i;
    const int kv = r % k8; r /= k8;
    const int b = r % ntb;
    const int row = static_cast<int>(r / ntb);
    const int dx = row % tb.bw, dy = (row / tb.bw) % tb.bh, c = row / (tb.bw * tb.bh);
    const int sp = b % tb.ns, rp = (b / tb.ns) % tb.nr, t = b / (tb.ns * tb.nr);
    const int rr = rp * tb.bh + dy, s = sp * tb.bw + dx;
    uint4 v = make_uint4(0, 0, 0, 0);
    if (rr < g.R && s < g.S)
      v = *reinterpret_cast<const uint4*>(F + ((((1ll * c * g.T + t) * g.R + rr) * g.S + s) * g.K + kv * 8));
    reinterpret_cast<uint4*>(Fp)[i] = v;
  }
}

// gradient in tap-block order Dp[tb][row][k] (fp32) -> gradF[c][t][r][s][k]
__global__ void filter_unpack_kernel(Geo g, TapBlock tb, const float* __restrict__ Dp, void* gradF, int out_f32) {
  const long long total = g.sizeF();
  for (long long i = blockIdx.x * 1ll * blockDim.x + threadIdx.x; i < total; i += 1ll * gridDim.x * blockDim.x) {
    long long r = i;
    const int k = r % g.K; r /= g.K;
    const int s = r % g.S; r /= g.S;
    const int rr = r % g.R; r /= g.R;
    const int t = r % g.T;
    const int c = static_cast<int>(r / g.T);
    const int b = (t * tb.nr + rr / tb.bh) * tb.ns + s / tb.bw;
    const int row = (c * tb.bh + rr % tb.bh) * tb.bw + s % tb.bw;
    const float v = Dp[(1ll * b * tb.rows + row) * g.K + k];
    if (out_f32) static_cast<float*>(gradF)[i] = v;
    else static_cast<__half*>(gradF)[i] = __float2half_rn(v);
  }
}

// input map whose box carries one tap block: (64 n, bw, bh, 1, C)
int act_map_tapblock(CUtensorMap* m, const void* base, const Geo& g, const TapBlock& tb) {
  const uint64_t xn = 1ull * g.W * g.N * 2;
  uint64_t dims[5] = {static_cast<uint64_t>(g.N), static_cast<uint64_t>(g.W), static_cast<uint64_t>(g.H),
                      static_cast<uint64_t>(g.D), static_cast<uint64_t>(g.C)};
  uint64_t str[4] = {1ull * g.N * 2, xn, xn * g.H, xn * g.H * g.D};
  const uint32_t box[5] = {kChunk, static_cast<uint32_t>(tb.bw), static_cast<uint32_t>(tb.bh), 1,
                           static_cast<uint32_t>(g.C)};
  return make_tensor_map(m, base, dims, str, box);
}

int fprop_tapblock(DeviceCtx* c, const Geo& g, const TapBlock& tb, const void* I, const void* F, void* O, float alpha,
                   int relu, cudaStream_t stream) {
  const int ntb = g.T * tb.nr * tb.ns;
  const long long cols = 1ll * g.M * g.P * g.Q * g.N;
  const size_t fp_bytes = static_cast<size_t>(tb.rows) * ntb * g.K * 2;
  int rc = ensure_workspace(c, stream, fp_bytes);
  if (rc != NG_OK) return rc;
  __half* Fp = reinterpret_cast<__half*>(c->ws);
  filter_repack_kernel<<<launch_1d(1ll * tb.rows * ntb * g.K / 8, 256, c), 256, 0, stream>>>(
      g, tb, static_cast<const __half*>(F), Fp);
  NG_CHECK_LAUNCH();
  TcParams p = {};
  p.mode = TC_FPROP;
  p.block_n = 256;
  p.M = g.K; p.N = static_cast<int>(cols);
  p.tiles_n = static_cast<int>((cols + p.block_n - 1) / p.block_n);
  p.nz = 1; p.splits = 1;
  TcOperandLayout lay = {1, 1, tb.rows};
  p.red_chunks = 1;
  p.num_kb = ntb;
  tc_pick_tile_rows(c, p, p.tiles_n, p.num_kb);
  // fewer, larger boxes: the filters of a 128-row half as one box (K a multiple of 64), the two
  // image groups of a pixel as one box (N = 128, 2-D)
  const bool merge_off = tuning().merge_boxes == 0;
  lay.a_merge = !merge_off && g.K % kChunk == 0 && g.K > kChunk;
  lay.a_chunks = (g.K + kChunk - 1) / kChunk;
  lay.b_pair = !merge_off && g.N == 2 * kChunk && g.D == 1;
  // (tap blocks as high as the stride: the next image row meets the same input rows one block later)
  const int row_cols = row_chunks(g.N, g.Q, CH_PIXEL) * kChunk;
  const int stack = g.str_h == tb.bh ? pick_row_stack(c, g.K, kChunk, ntb, tb.nr, 1, tb.rows, g.P, g.M, row_cols, alpha, lay.b_pair ? 128 : 64) : 0;
  if (stack) {
    fill_row_pairs(p, stack, g.N, g.Q, g.P, g.M, CH_PIXEL, g.N, 1ll * g.Q * g.N, 1ll * g.P * g.Q * g.N);
    p.num_kb = ntb / tb.nr * (tb.nr + 1);
    lay.a_merge = 0;
    lay.a_chunks = 2;
  }
  tc_fill_mma(p, lay);
  fill_taps(p, g, CH_PIXEL);
  p.R = tb.nr + (stack ? 1 : 0); p.S = tb.ns; p.RS = p.R * tb.ns; p.tap_w = tb.bw; p.tap_h = tb.bh;
  if (stack) p.str_h = 2 * g.str_h;
  fill_decode(p, g.N, g.Q, stack ? p.cmap.y_count : g.P, g.M, CH_PIXEL);
  p.oob_y = g.H;
  p.C = O; p.Cold = nullptr; p.ldc = cols; p.c_zstride = stack ? 1ll * g.Q * g.N : 0;
  p.alpha = alpha; p.beta = 0.0f; p.relu = relu; p.sr_bits = 0; p.out_f32 = 0; p.vec_ok = 1;
  CUtensorMap mapA, mapB;
  if (stack) {
    rc = filter_map_rows(&mapA, Fp, g.K, tb.ns, tb.nr, g.T, tb.rows, tb.rows);
    if (rc != NG_OK) return rc;
  } else {  // packed filter seen as (k, tap block, row), or as (k_lo, row, k_hi, tap block)
    uint64_t dims[5] = {static_cast<uint64_t>(g.K), static_cast<uint64_t>(ntb), static_cast<uint64_t>(tb.rows), 1, 1};
    uint64_t str[4];
    str[0] = 1ull * g.K * 2; str[1] = str[0] * ntb; str[2] = str[1] * tb.rows; str[3] = str[2];
    uint32_t box[5] = {kChunk, 1, static_cast<uint32_t>(tb.rows), 1, 1};
    if (lay.a_merge) {
      dims[0] = kChunk; dims[1] = tb.rows; dims[2] = g.K / kChunk; dims[3] = ntb;
      str[0] = 1ull * g.K * 2 * ntb; str[1] = 128; str[2] = 1ull * g.K * 2; str[3] = str[0] * tb.rows;
      box[1] = tb.rows; box[2] = 2;
    }
    rc = make_tensor_map(&mapA, Fp, dims, str, box);
    if (rc != NG_OK) return rc;
  }
  if (lay.b_pair) {  // (n_lo, x, y, chan, n_hi): both image groups of a pixel's tap block in one box
    const uint64_t xn = 1ull * g.W * g.N * 2;
    uint64_t dims[5] = {kChunk, static_cast<uint64_t>(g.W), static_cast<uint64_t>(g.H), static_cast<uint64_t>(g.C), 2};
    uint64_t str[4] = {1ull * g.N * 2, xn, xn * g.H, 128};
    const uint32_t box[5] = {kChunk, static_cast<uint32_t>(tb.bw), static_cast<uint32_t>(tb.bh),
                             static_cast<uint32_t>(g.C), 2};
    rc = make_tensor_map(&mapB, I, dims, str, box);
  } else {
    rc = act_map_tapblock(&mapB, I, g, tb);
  }
  if (rc != NG_OK) return rc;
  return tc_launch(c, mapA, mapB, p, stream);
}

// gradient with the filters along the rows, Dt[k][tile][box][row] (fp32; tile stride 256 columns,
// `per` boxes of tb.rows columns per tile) -> gradF[c][t][r][s][k]
__global__ void filter_unpack_t_kernel(Geo g, TapBlock tb, int per, int ld, const float* __restrict__ Dt, void* gradF,
                                       int out_f32) {
  const long long total = g.sizeF();
  for (long long i = blockIdx.x * 1ll * blockDim.x + threadIdx.x; i < total; i += 1ll * gridDim.x * blockDim.x) {
    long long r = i;
    const int k = r % g.K; r /= g.K;
    const int s = r % g.S; r /= g.S;
    const int rr = r % g.R; r /= g.R;
    const int t = r % g.T;
    const int c = static_cast<int>(r / g.T);
    const int b = (t * tb.nr + rr / tb.bh) * tb.ns + s / tb.bw;
    const int row = (c * tb.bh + rr % tb.bh) * tb.bw + s % tb.bw;
    const float v = Dt[1ll * k * ld + (b / per) * 256 + (b % per) * tb.rows + row];
    if (out_f32) static_cast<float*>(gradF)[i] = v;
    else static_cast<__half*>(gradF)[i] = __float2half_rn(v);
  }
}

// Strided updates that ran on the CUDA cores because their patch matrix would exceed 6 GB (or 65535 rows): their
// sums were serial sums in fp32, rounded, some ten times closer than the tensor cores' truncated ones of the same
// length. Partitions of at most kShortSum k-blocks get there, more of them than fit in the partials' share
// of the workspace: the sum runs in several launches, each adding to the gradient in its second stage. Off the
// sum in 64 bits / time, CUDA cores -> partitions of one wave -> now: 96 -> 72, 5x5 / 2, 224x224, 120 images (7.2 GB) 4.0e-6,
// 1452 ms -> 5.9e-5, 2.0 ms -> 3.2e-7, 4.4 ms; 1400 -> 64, 7x7 / 2, 40x40, 24 images (68600 rows) 3.0e-7, 204 ms -> 5.7e-6,
// 0.29 ms -> 2.6e-7, 0.72 ms.
constexpr int kShortSum = 3;
bool beyond_patches(const Geo& g) {
  const long long rows = 1ll * g.C * g.T * g.R * g.S;
  return rows > 65535 || 2 * rows * g.M * g.P * g.Q * g.N > (6ll << 30) || tuning().stride_phases == 3;   // (3: tests)
}
// Sets p.splits and returns the number of launches.
int short_sums(TcParams& p, long long out_elems) {
  const long long parts = (p.num_kb + kShortSum - 1) / kShortSum;
  if (parts < 2) return 1;
  const long long room = tuning().conv_splits > 1 ? tuning().conv_splits      // (tests: several launches for small sums)
                                                  : std::max<long long>(2, std::min<long long>(kMaxSplits, (256ll << 20) / (out_elems * 4)));
  const long long launches = (parts + room - 1) / room;
  p.splits = static_cast<int>(std::max<long long>(2, (parts + launches - 1) / launches));
  return static_cast<int>(launches);
}
int launch_sums(DeviceCtx* c, const CUtensorMap& mapA, const CUtensorMap& mapB, const TcParams& p, int launches, cudaStream_t stream) {
  for (int i = 0; i < launches; ++i) {
    TcParams q = p;
    q.kb_base = static_cast<int>(1ll * p.num_kb * i / launches);
    q.num_kb = static_cast<int>(1ll * p.num_kb * (i + 1) / launches) - q.kb_base;
    if (i > 0) { q.beta = 1.0f; q.Cold = q.C; }
    const int rc = tc_launch(c, mapA, mapB, q, stream);
    if (rc != NG_OK) return rc;
  }
  return NG_OK;
}
__global__ void round_kernel(const float* __restrict__ src, __half* dst, long long n) {
  for (long long i = blockIdx.x * 1ll * blockDim.x + threadIdx.x; i < n; i += 1ll * gridDim.x * blockDim.x) dst[i] = __float2half_rn(src[i]);
}

// Few filters (K <= 128) as well as few channels: the roles of the operands are exchanged, so that
// the 128 MMA rows carry the filters and the 256 MMA columns carry the rows of several taps or tap
// blocks (an MMA with 64 columns costs nearly as much as one with 256). Column tile j owns tap blocks
// [j * per, (j + 1) * per); its B operand is their input boxes stacked, its A operand the error box.
// `tb`: the tap blocks of a first layer, or single taps (bw = bh = 1) of swap_rows(C) rows each.
int update_swapped(DeviceCtx* c, const Geo& g, const TapBlock& tb, ChunkMode mode, bool phased, const void* I,
                   const void* E, void* gradF, int out_f32, float alpha, cudaStream_t stream) {
  const int ntb = g.T * tb.nr * tb.ns;
  const bool blocks = tb.bw > 1 || tb.bh > 1;
  const int per = 256 / tb.rows;
  const int tiles = (ntb + per - 1) / per;
  const int ld = tiles * 256;
  const bool blocked_i = !blocks && !phased && wants_chan_block(g.D, g.H, g.W, g.N, ntb);
  const bool blocked_e = !blocks && wants_chan_block(g.M, g.P, g.Q, g.N, ntb);
  TcParams p = {};
  p.mode = TC_UPDATE;
  p.swap_ab = 1;
  p.block_n = 256;
  p.M = g.K; p.N = ld;
  p.m_halves = 1; p.tiles_m = 1;
  p.tiles_n = tiles;
  p.nz = 1;
  p.taps_per_z = ntb;
  TcOperandLayout lay = {0, 0, kChunk};
  lay.a_box_rows = std::min(g.K, kTileM);
  lay.b_box_rows = tb.rows;
  lay.b_box_count = per;
  p.num_kb = g.M * g.P * row_chunks(g.N, g.Q, mode);
  tc_fill_mma(p, lay);
  fill_taps(p, g, mode);
  p.R = tb.nr; p.S = tb.ns; p.RS = tb.nr * tb.ns; p.tap_w = tb.bw; p.tap_h = tb.bh;
  if (phased) fill_phases(p, update_phases(g));
  fill_decode(p, g.N, g.Q, g.P, g.M, mode);
  p.oob_y = g.H;
  p.Cold = nullptr; p.ldc = ld; p.c_zstride = 0;
  p.alpha = alpha; p.beta = 0.0f; p.relu = 0; p.sr_bits = 0; p.out_f32 = 1; p.vec_ok = 1;
  p.splits = choose_splits(c, p.tiles_n, p.num_kb, 1ll * g.K * ld);
  if (!blocks) p.splits = shorter_partitions(c, tiles, p.num_kb, p.splits, 1ll * g.K * ld, 2, 64);
  const int launches = phased && beyond_patches(g) ? short_sums(p, 1ll * g.K * ld) : 1;
  // behind the partials: the gradient in tap order and copies of the operands. (Not in the second buffer,
  // where I and the gradient of a layer that was rewritten by space to depth lie.)
  const size_t bytes[3] = {(static_cast<size_t>(g.K) * ld * 4 + 255) & ~size_t(255),
                           phased ? phase_split_bytes(g, update_phases(g)) : (blocked_i ? chan_block_bytes(g.C, g.D, g.H, g.W, g.N) : 0),
                           blocked_e ? chan_block_bytes(g.K, g.M, g.P, g.Q, g.N) : 0};
  void* room[3] = {nullptr, nullptr, nullptr};
  int rc = chan_block_room(c, stream, p, bytes, room, 3, phased);
  if (rc != NG_OK) return rc;
  float* Dt = static_cast<float*>(room[0]);
  p.C = Dt;
  if (phased) rc = phase_split(g, update_phases(g), I, room[1], nullptr, nullptr, nullptr, stream);
  else if (blocked_i) rc = chan_block(c, stream, I, room[1], g.C, g.D, g.H, g.W, g.N);
  if (rc == NG_OK && blocked_e) rc = chan_block(c, stream, E, room[2], g.K, g.M, g.P, g.Q, g.N);
  if (rc != NG_OK) return rc;
  if (bytes[1]) I = room[1];
  if (bytes[2]) E = room[2];
  CUtensorMap mapA, mapB;
  rc = act_map(&mapA, E, g.K, g.M, g.P, g.Q, g.N, mode, lay.a_box_rows, blocked_e);
  if (rc != NG_OK) return rc;
  rc = blocks ? act_map_tapblock(&mapB, I, g, tb)
              : (phased ? phase_map(&mapB, I, g, update_phases(g), tb.rows) : act_map(&mapB, I, g.C, g.D, g.H, g.W, g.N, mode, tb.rows, blocked_i));
  if (rc != NG_OK) return rc;
  rc = launch_sums(c, mapA, mapB, p, launches, stream);
  if (rc != NG_OK) return rc;
  filter_unpack_t_kernel<<<launch_1d(g.sizeF(), 256, c), 256, 0, stream>>>(g, tb, per, ld, Dt, gradF, out_f32);
  NG_CHECK_LAUNCH();
  return NG_OK;
}

int update_tapblock(DeviceCtx* c, const Geo& g, const TapBlock& tb, const void* I, const void* E, void* gradF,
                    int out_f32, float alpha, cudaStream_t stream) {
  const bool swap_ok = tuning().update_swap != 0;
  // (worth it when the tap blocks fill at least half of a 256-column tile)
  if (swap_ok && g.K <= kTileM && g.T * tb.nr * tb.ns * tb.rows >= 128)
    return update_swapped(c, g, tb, CH_PIXEL, false, I, E, gradF, out_f32, alpha, stream);
  const int ntb = g.T * tb.nr * tb.ns;
  const long long span = 1ll * g.M * g.P * g.Q * g.N;
  // workspace: [split-K partials of the engine, at most 32 splits][Dp]
  const size_t dp_bytes = static_cast<size_t>(ntb) * tb.rows * g.K * 4;
  const size_t dp_off = (kMaxSplits * dp_bytes + 255) & ~size_t(255);
  int rc = ensure_workspace(c, stream, dp_off + dp_bytes);
  if (rc != NG_OK) return rc;
  float* Dp = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(c->ws) + dp_off);
  TcParams p = {};
  p.mode = TC_UPDATE;
  p.block_n = update_block_n(g.K);
  p.M = tb.rows; p.N = g.K;
  p.m_halves = 1; p.tiles_m = 1;
  p.tiles_n = (g.K + p.block_n - 1) / p.block_n;
  set_update_groups(p, ntb, tb.rows);
  TcOperandLayout lay = {0, 0, kChunk};
  lay.a_box_rows = tb.rows;
  p.num_kb = static_cast<int>(span / kChunk);
  tc_fill_mma(p, lay);
  fill_taps(p, g, CH_PIXEL);
  p.R = tb.nr; p.S = tb.ns; p.RS = tb.nr * tb.ns; p.tap_w = tb.bw; p.tap_h = tb.bh;
  fill_decode(p, g.N, g.Q, g.P, g.M, CH_PIXEL);
  p.oob_y = g.H;
  p.C = Dp; p.Cold = nullptr; p.ldc = g.K; p.c_zstride = 1ll * tb.rows * g.K;
  p.alpha = alpha; p.beta = 0.0f; p.relu = 0; p.sr_bits = 0; p.out_f32 = 1; p.vec_ok = 1;
  p.splits = choose_splits(c, 1ll * p.tiles_n * p.nz, p.num_kb, 1ll * ntb * tb.rows * g.K);
  CUtensorMap mapA, mapB;
  rc = act_map_tapblock(&mapA, I, g, tb);
  if (rc != NG_OK) return rc;
  rc = act_map(&mapB, E, g.K, g.M, g.P, g.Q, g.N, CH_PIXEL, p.block_n);
  if (rc != NG_OK) return rc;
  rc = tc_launch(c, mapA, mapB, p, stream);
  if (rc != NG_OK) return rc;
  filter_unpack_kernel<<<launch_1d(g.sizeF(), 256, c), 256, 0, stream>>>(g, tb, Dp, gradF, out_f32);
  NG_CHECK_LAUNCH();
  return NG_OK;
}

}  // namespace

}  // namespace ngb

using namespace ngb;

// ------------------------------------------------------------------------------------------
// Strided first layers of a small minibatch: space to depth.
// With fewer than 64 images a chunk holds several pixels, which a strided layer does not read
// from consecutive addresses, and with 3 channels a tap is no k-block. Such a layer (AlexNet
// conv1 on the shard of one of 4 or 8 GPUs) is rewritten as a unit-stride layer over
//   I2[(c, dy, dx)][Y][X][n] = I[c][st * Y + dy - pad_h][st * X + dx - pad_w][n]   (zero outside),
//   F2[(c, dy, dx)][r2][s2][k] = F[c][st * r2 + dy][st * s2 + dx][k]               (zero outside),
// O[k][p][q][n] = sum F2 * I2[..][p + r2][q + s2][n]: C * st * st channels (48 for 3 channels and
// stride 4), ceil(R / st) x ceil(S / st) taps, no padding, which is a shape the flattened-row
// tensor-core path handles at any minibatch. The copies cost a pass over the (small) input; the
// im2col matrix this replaces was R * S / st^2 times larger.
struct SpaceToDepth {
  bool ok = false;
  int st = 1, C2 = 0, H2 = 0, W2 = 0, R2 = 0, S2 = 0;
};
SpaceToDepth pick_space_to_depth(const Geo& g) {
  SpaceToDepth z;
  if (tuning().space_to_depth == 0) return z;
  if (g.D != 1 || g.T != 1 || g.pad_d != 0 || g.str_d != 1 || g.str_h != g.str_w || g.str_w < 2) return z;
  z.st = g.str_w;
  z.C2 = g.C * z.st * z.st;
  z.R2 = (g.R + z.st - 1) / z.st;
  z.S2 = (g.S + z.st - 1) / z.st;
  z.H2 = g.P + z.R2 - 1;
  z.W2 = g.Q + z.S2 - 1;
  z.ok = z.C2 >= 16 && z.C2 <= 4096;
  return z;
}
ng_conv_desc space_to_depth_desc(const Geo& g, const SpaceToDepth& z) {
  ng_conv_desc d = {};
  d.N = g.N; d.C = z.C2; d.K = g.K;
  d.D = 1; d.H = z.H2; d.W = z.W2;
  d.T = 1; d.R = z.R2; d.S = z.S2;
  d.pad_d = d.pad_h = d.pad_w = 0;
  d.str_d = d.str_h = d.str_w = 1;
  return d;
}
// one block row per (channel of I2, Y): the threads walk its X * N / 8 16-byte vectors
__global__ void s2d_input_kernel(Geo g, SpaceToDepth z, const uint4* __restrict__ I, uint4* __restrict__ I2) {
  const int nvec = g.N >> 3;
  const int row = blockIdx.x;                 // c2 * H2 + Y
  const int c2 = row / z.H2, Y = row - c2 * z.H2;
  const int dx = c2 % z.st, dy = (c2 / z.st) % z.st, c = c2 / (z.st * z.st);
  const int y = z.st * Y + dy - g.pad_h;
  const bool row_in = y >= 0 && y < g.H;
  const uint4* src = I + (1ll * c * g.H + (row_in ? y : 0)) * g.W * nvec;
  uint4* dst = I2 + 1ll * row * z.W2 * nvec;
  for (int i = threadIdx.x; i < z.W2 * nvec; i += blockDim.x) {
    const int X = i / nvec, v = i - X * nvec;
    const int x = z.st * X + dx - g.pad_w;
    uint4 val = make_uint4(0, 0, 0, 0);
    if (row_in && x >= 0 && x < g.W) val = __ldg(src + x * nvec + v);
    dst[i] = val;
  }
}
// one 16-byte vector (8 filters) of F2 per thread
__global__ void s2d_filter_kernel(Geo g, SpaceToDepth z, const uint4* __restrict__ F, uint4* __restrict__ F2) {
  const int kvec = g.K >> 3;
  const long long total = 1ll * z.C2 * z.R2 * z.S2 * kvec;
  for (long long i = blockIdx.x * 1ll * blockDim.x + threadIdx.x; i < total; i += 1ll * gridDim.x * blockDim.x) {
    long long r = i;
    const int v = static_cast<int>(r % kvec); r /= kvec;
    const int s2 = static_cast<int>(r % z.S2); r /= z.S2;
    const int r2 = static_cast<int>(r % z.R2);
    const int c2 = static_cast<int>(r / z.R2);
    const int dx = c2 % z.st, dy = (c2 / z.st) % z.st, c = c2 / (z.st * z.st);
    const int rr = z.st * r2 + dy, ss = z.st * s2 + dx;
    uint4 val = make_uint4(0, 0, 0, 0);
    if (rr < g.R && ss < g.S) val = __ldg(F + ((1ll * c * g.R + rr) * g.S + ss) * kvec + v);
    F2[i] = val;
  }
}
// gradF[c][r][s][k] = G2[(c, r % st, s % st)][r / st][s / st][k]
__global__ void s2d_filter_grad_kernel(Geo g, SpaceToDepth z, const float* __restrict__ G2, void* gradF, int out_f32) {
  const long long total = g.sizeF();
  for (long long i = blockIdx.x * 1ll * blockDim.x + threadIdx.x; i < total; i += 1ll * gridDim.x * blockDim.x) {
    long long r = i;
    const int k = static_cast<int>(r % g.K); r /= g.K;
    const int ss = static_cast<int>(r % g.S); r /= g.S;
    const int rr = static_cast<int>(r % g.R);
    const int c = static_cast<int>(r / g.R);
    const int c2 = (c * z.st + rr % z.st) * z.st + ss % z.st;
    const float v = G2[((1ll * c2 * z.R2 + rr / z.st) * z.S2 + ss / z.st) * g.K + k];
    if (out_f32) static_cast<float*>(gradF)[i] = v;
    else static_cast<__half*>(gradF)[i] = __float2half_rn(v);
  }
}
// ------------------------------------------------------------------------------------------
// Backward pass, one phase. Input pixel x of a layer with stride st belongs to phase ph = (x + pad) %
// st and gets error through the taps s = ph + st * j alone: with x' = (x + pad) / st it is
//   dI[x] = sum over j of F[ph + st * j] * E[x' - j],
// a unit-stride layer over the phase's share of the taps, whose outputs are stored every st-th pixel
// (ColumnMap). A unit-stride layer is its only phase. (Issuing every tap for every pixel and letting
// the copy engine fill zeros where the stride does not divide took st^2 times the operands and MMAs.)
// `blocked`: E is its channel-blocked copy. `gather`: the whole layer, every tap for every pixel. `plan`: if
// given, it is filled in and nothing is launched.
// ------------------------------------------------------------------------------------------
struct BpropPlan {
  size_t partials = 0;     // bytes of the split partials, raised to the largest of the phases
  long long steps = 0;     // k-blocks that an SM works on, one after the other
  int splits = 1;
};
int bprop_phase(DeviceCtx* c, const Geo& g, const int first[3], ChunkMode mode, const void* F, const void* E, void* gradI,
                float alpha, bool blocked, bool gather, BpropPlan* plan, cudaStream_t stream) {
  const int str[3] = {g.str_d, g.str_h, g.str_w}, flt[3] = {g.T, g.R, g.S}, pad[3] = {g.pad_d, g.pad_h, g.pad_w},
            ext[3] = {g.D, g.H, g.W};
  int taps[3], lo[3], n[3], off[3];     // taps of the phase; first x' and number of its pixels; first pixel
  for (int i = 0; i < 3; ++i) {
    if (gather) {
      taps[i] = flt[i]; lo[i] = pad[i]; off[i] = 0; n[i] = ext[i];
      continue;
    }
    taps[i] = (flt[i] - first[i] + str[i] - 1) / str[i];
    lo[i] = pad[i] > first[i] ? (pad[i] - first[i] + str[i] - 1) / str[i] : 0;
    off[i] = str[i] * lo[i] + first[i] - pad[i];
    if (off[i] >= ext[i]) return NG_OK;
    n[i] = (ext[i] - off[i] + str[i] - 1) / str[i];
  }
  const bool unit = gather || (str[0] == 1 && str[1] == 1 && str[2] == 1);
  TcParams p = {};
  p.mode = TC_BPROP;
  const long long cols = pixel_columns(p, 1ll * n[0] * n[1], n[2], g.N, mode);
  if (cols > 0x7fffffffll) return fail(NG_ERR_TOO_LARGE, "output too large");
  if (!unit) {
    p.cmap.row_chunks = row_chunks(g.N, n[2], mode);
    p.cmap.row_len = n[2] * g.N;
    p.cmap.n = g.N;
    p.cmap.x = g.str_w * g.N;
    p.cmap.y = 1ll * g.str_h * g.W * g.N;
    p.cmap.z = 1ll * g.str_d * g.H * g.W * g.N;
    p.cmap.y_count = n[1];
  }
  p.M = g.C; p.N = static_cast<int>(cols);
  p.nz = 1; p.splits = 1;
  TcOperandLayout lay = {0, 1, kChunk};
  p.red_chunks = (g.K + kChunk - 1) / kChunk;
  p.num_kb = taps[0] * taps[1] * taps[2] * p.red_chunks;
  tc_pick_tile(c, p, cols, p.num_kb, kChunk);
  // fewer input channels than tile rows (one row tile): the filter box carries the real rows only
  int a_rows = p.tiles_m == 1 ? std::min(kTileM * p.m_halves, (g.C + 7) / 8 * 8) : kTileM * p.m_halves;
  const int n_taps = taps[0] * taps[1] * taps[2];
  const int stack = gather ? 0 : pick_row_stack(c, g.C, a_rows, n_taps, taps[1], p.red_chunks, kChunk, n[1], n[0],
                                                1ll * row_chunks(g.N, n[2], mode) * kChunk, alpha);
  const long long out_row = 1ll * g.str_h * g.W * g.N;
  if (stack) {
    fill_row_pairs(p, stack, g.N, n[2], n[1], n[0], mode, g.str_w * g.N, out_row, 1ll * g.str_d * g.H * g.W * g.N);
    p.num_kb = n_taps / taps[1] * (taps[1] + 1) * p.red_chunks;
    lay.a_box_count = 2;
  }
  lay.a_box_rows = a_rows;
  tc_fill_mma(p, lay);
  p.S = taps[2]; p.R = taps[1] + (stack ? 1 : 0); p.RS = p.R * taps[2];
  p.pad_d = lo[0]; p.pad_h = lo[1] + (stack ? 1 : 0); p.pad_w = lo[2];
  p.inner_tap = mode == CH_FLAT ? g.N : 0;
  p.x_tap = mode == CH_FLAT ? 0 : 1;
  p.gather = gather;
  p.str_d = g.str_d; p.str_h = g.str_h; p.str_w = g.str_w;
  fill_decode(p, g.N, n[2], stack ? p.cmap.y_count : n[1], n[0], mode);
  p.oob_y = g.P;
  p.C = static_cast<__half*>(gradI) + ((1ll * off[0] * g.H + off[1]) * g.W + off[2]) * g.N;
  p.Cold = nullptr; p.ldc = 1ll * g.D * g.H * g.W * g.N; p.c_zstride = stack ? out_row : 0;
  p.alpha = alpha; p.beta = 0.0f; p.relu = 0; p.sr_bits = 0; p.out_f32 = 0; p.vec_ok = 1;
  if (!stack) p.splits = choose_splits(c, 1ll * p.tiles_m * p.tiles_n, p.num_kb, 1ll * g.C * cols, true);
  if (plan) {
    if (p.splits > 1) plan->partials = std::max(plan->partials, static_cast<size_t>(p.splits) * p.M * p.N * sizeof(float));
    plan->splits = p.splits;
    plan->steps = (1ll * p.tiles_m * p.tiles_n + c->sm_count - 1) / c->sm_count * ((p.num_kb + p.splits - 1) / p.splits);
    return NG_OK;
  }
  CUtensorMap mapA, mapB, mapBm;
  int rc = gather ? filter_map_rows(&mapA, F, g.K, g.S, g.R, g.T, g.C, a_rows) : filter_map_phase(&mapA, F, g, first, taps, a_rows);
  if (rc != NG_OK) return rc;
  rc = act_map(&mapB, E, g.K, g.M, g.P, g.Q, g.N, mode, kChunk, blocked);
  if (rc != NG_OK) return rc;
  // the error pixels of a column tile inside one image row as one box
  if (mode == CH_PIXEL && !gather)
    p.b_merge = act_map_merged(&mapBm, E, g.K, g.M, g.P, g.Q, g.N, kChunk, p.block_n / kChunk, blocked);
  return tc_launch(c, mapA, mapB, p, stream, p.b_merge ? &mapBm : nullptr);
}

// Whether the backward pass of a strided layer runs phase by phase. Every phase is a product (and, with few
// tiles, a second stage) of its own, some 5 us before it has done any work. Small layers are shorter as one
// product over every tap of every pixel (`in_place`: minibatches that are multiples of 64), or on the CUDA
// cores. The estimates are fits to 120 layers of 1 to 7 taps and strides 2 to 4, each timed in both forms; by
// phases / the other form, us:
//   one product: 128 -> 64, 4x4 / 4, 8x8, 128 images 82 / 13; 64 -> 64, 3x3 / 2, 14x14, 128 images 22 / 12; 96 -> 32,
//   3x3 / 2, 23x23, 64 images 25 / 15; 64 -> 64, 3x3 / 2, 56x56, 64 images 32 / 52; 96 -> 96, 3x3 / 2, 55x55, 128 images 53 / 169
//   CUDA cores: 16 -> 16, 4x4 / 4, 8x8, 8 images 82 / 7; 32 -> 32, 3x3 / 2, 8x8, 16 images 25 / 11; 24 -> 64, 7x7 / 2, 11x11,
//   48 images 39 / 86; 64 -> 64, 3x3 / 2, 56x56, 24 images 33 / 858
bool bprop_by_phases(DeviceCtx* c, const Geo& g, bool in_place) {
  const int strides = g.str_d * g.str_h * g.str_w, taps = g.T * g.R * g.S;
  if (strides == 1) return true;
  if (tuning().stride_phases >= 0) return tuning().stride_phases != 0;
  const double phases = 1.0 * std::min(g.str_d, g.T) * std::min(g.str_h, g.R) * std::min(g.str_w, g.S);
  const double pixels = 1.0 * g.D * g.H * g.W;
  const int chunks = (g.K + kChunk - 1) / kChunk, row_tiles = (g.C + kTileM - 1) / kTileM;
  auto tiles = [&](double px) { return row_tiles * std::ceil(px * g.N / 256); };
  const double kb = taps / phases * chunks, waves = tiles(pixels / strides) / c->sm_count;
  double by_phases = 3.0 + phases * (5.0 + (waves < 1.0 ? 0.3 * std::min(kb, 8.0 + kb * waves) : 0.5 * std::ceil(waves) * (kb + 1)));
  if (in_place) {       // (the producer takes 0.86 us to find the pixels of a k-block, whatever its size)
    const int first[3] = {0, 0, 0};
    BpropPlan one;
    bprop_phase(c, g, first, g.N % kChunk == 0 ? CH_PIXEL : CH_FLAT, nullptr, nullptr, nullptr, 1.0f, false, true, &one, nullptr);
    return by_phases < 5.0 + (one.splits > 1 ? 3.0 : 0.0) + 0.86 * one.steps;
  }
  by_phases += 5.0;      // (the scan of the filter, the second look at the result)
  const double chain = std::ceil(1.0 * g.T / g.str_d) * std::ceil(1.0 * g.R / g.str_h) * std::ceil(1.0 * g.S / g.str_w) * g.K;
  return by_phases < 7.0 + 0.03 * chain + 1e-6 * g.sizeI() * (17.0 + 0.4 * taps + 1.0 * g.K * taps / strides);
}
// Whether the update of a strided layer whose minibatch is no multiple of 64 reads a phase-split copy, or a
// patch matrix: small ones, and those with about as many input pixels as patch elements or fewer, of which
// patches read only what they need. Phase-split / patches, us (patches, their ratio to the input):
// 128 -> 128, 1x1 / 2, 28x28, 24 images (1.2 MB, 0.25) 17 / 15; 256 -> 32, 3x3 / 2, 16x16, 24 images (7.1 MB, 2.3) 18 / 17; 256 -> 32,
// 7x7 / 3, 19x19, 8 images (9.8 MB, 6.6) 18 / 21; 512 -> 512, 3x3 / 3, 22x22, 32 images (18 MB, 1.2) 41 / 34; 64 -> 64, 3x3 / 2, 56x56,
// 24 images (22 MB, 2.3) 27 / 29; 512 -> 512, 1x1 / 2, 34x34, 96 images (27 MB, 0.25) 76 / 45; 96 -> 512, 3x3 / 4, 85x85, 48 images
// (38 MB, 0.6) 58 / 54; 256 -> 64, 2x2 / 2, 62x62, 32 images (64 MB, 1.1) 46 / 61; 96 -> 72, 5x5 / 2, 51x51, 88 images (284 MB, 6.4) 100 / 218.
// Longest partitions (k-blocks) of the strided updates' sums, so that no gradient is further off the sum in 64
// bits than on the paths these forms replace: patches in one wave / phase-split with up to 64 /
// now, in units of 1e-7: 128 -> 128, 1x1 / 2, 57x57, 120 images 8.5 / 8.2 / 7.9; 512 -> 512, 1x1 / 2, 34x34, 96 images 18.7 / 11.0 / 9.5;
// 128 -> 256, 3x3 / 2, 41x41, 40 images 13.0 / 13.2 / 7.3; 64 -> 64, 3x3 / 2, 14x14, 16 images 3.8 / 3.4 / 2.6; 96 -> 72, 5x5 / 2,
// 51x51, 88 images 47 / 42 / 33. The longer second stage costs 2 % over 70 layers (32 -> 16, 1x1 / 2, 75x75, 96
// images 23 -> 29 us).
constexpr int kLongSum = 16, kLongPatchSum = 3;
constexpr long long kPatchBytes = 8ll << 20;
bool update_by_phases(const Geo& g) {
  if (tuning().stride_phases >= 0) return tuning().stride_phases != 0;
  const long long rows = 1ll * g.C * g.T * g.R * g.S, patches = rows * g.M * g.P * g.Q * g.N;
  if (rows > 65535) return true;          // (the patch kernel has a block row for each)
  return 2 * patches > kPatchBytes && (2 * patches > 3 * g.sizeI() || (2 * patches > 4 * kPatchBytes && 5 * patches > 4 * g.sizeI()));
}


extern "C" {

int ng_conv_output_dims(const ng_conv_desc* d, int* M, int* P, int* Q) {
  Geo g;
  int rc = make_geo(d, g);
  if (rc != NG_OK) return rc;
  if (M) *M = g.M;
  if (P) *P = g.P;
  if (Q) *Q = g.Q;
  return NG_OK;
}

int ng_conv_fprop(const ng_conv_desc* d, const void* I, const void* F, void* O, float alpha, int relu, int path,
                  void* stream_) {
  Geo g;
  int rc = make_geo(d, g);
  if (rc != NG_OK) return rc;
  if (!I || !F || !O) return fail(NG_ERR_INVALID_ARG, "null tensor");
  DeviceCtx* c = current_ctx();
  if (!c) return NG_ERR_CUDA;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  ChunkMode mode = pick_chunk_mode(g.N, g.str_w);
  // a phase-split copy in flattened rows (never slower than the CUDA cores: 16 -> 128, 1x1 / 2, 6x6, 96 images 13 / 15 us)
  const bool phased = mode == CH_NONE && path == NG_PATH_AUTO;
  if (phased) mode = CH_FLAT;
  const bool al = aligned16(I) && aligned16(F) && aligned16(O);
  const bool tc = path != NG_PATH_SIMT && path != NG_PATH_IM2COL && mode != CH_NONE && al;
  if (path == NG_PATH_TENSOR && !tc) return fail(NG_ERR_UNSUPPORTED, "shape not addressable by the tensor-core path");
  if ((path == NG_PATH_AUTO || path == NG_PATH_TENSOR) && g.C < 16 && g.N % kChunk == 0 && al) {
    const TapBlock tb = pick_tap_block(g);
    if (tb.ok) return fprop_tapblock(c, g, tb, I, F, O, alpha, relu, stream);
  }
  if (path == NG_PATH_AUTO && g.C < 16 && g.N % kChunk != 0 && al) {
    const SpaceToDepth z = pick_space_to_depth(g);
    if (z.ok) {
      const size_t i2_bytes = round256(2ull * z.C2 * z.H2 * z.W2 * g.N), f2_bytes = round256(2ull * z.C2 * z.R2 * z.S2 * g.K);
      AuxClaim aux;
      void* room = nullptr;
      rc = aux.room(c, stream, i2_bytes + f2_bytes, &room);
      if (rc != NG_OK) return rc;
      uint4* I2 = static_cast<uint4*>(room);
      uint4* F2 = reinterpret_cast<uint4*>(static_cast<uint8_t*>(room) + i2_bytes);
      s2d_input_kernel<<<z.C2 * z.H2, 256, 0, stream>>>(g, z, static_cast<const uint4*>(I), I2);
      NG_CHECK_LAUNCH();
      s2d_filter_kernel<<<launch_1d(1ll * z.C2 * z.R2 * z.S2 * (g.K / 8), 256, c), 256, 0, stream>>>(
          g, z, static_cast<const uint4*>(F), F2);
      NG_CHECK_LAUNCH();
      const ng_conv_desc d2 = space_to_depth_desc(g, z);
      return ng_conv_fprop(&d2, I2, F2, O, alpha, relu, NG_PATH_AUTO, stream_);
    }
  }
  {
    // Few input channels where tap blocks do not apply: one tap per k-block would feed the tensor
    // core 3 useful rows out of 16, so gather the patches once and run a dense GEMM over all rows:
    //   O[K x span] = F2d[crst][k]^T * col[crst][span]
    const int RST = g.T * g.R * g.S;
    const long long span = 1ll * g.M * g.P * g.Q * g.N;
    const bool small_c = g.C < 16 && path == NG_PATH_AUTO;
    const bool im2col = (small_c || path == NG_PATH_IM2COL) && al && span <= 0x7fffffffll &&
                        1ll * g.C * RST * span * 2 <= (6ll << 30) && g.C * RST <= 65535;
    if (path == NG_PATH_IM2COL && !im2col) return fail(NG_ERR_UNSUPPORTED, "shape not addressable by the im2col path");
    if (im2col) {
      const size_t col_bytes = static_cast<size_t>(g.C) * RST * span * 2;
      AuxClaim aux;              // (the product keeps its partials, if any, in the workspace)
      void* room = nullptr;
      rc = aux.room(c, stream, col_bytes, &room);
      if (rc != NG_OK) return rc;
      __half* col = static_cast<__half*>(room);
      im2col_kernel<<<im2col_grid(g), 256, 0, stream>>>(g, static_cast<const __half*>(I), col);
      NG_CHECK_LAUNCH();
      GemmCall gc = {};
      gc.A = F; gc.B = col; gc.C = O; gc.a_t = 1; gc.b_t = 0;
      gc.m = g.K; gc.n = static_cast<int>(span); gc.k = g.C * RST;
      gc.lda = g.K; gc.ldb = span; gc.ldc = span;
      gc.alpha = alpha; gc.beta = 0.0f; gc.relu = relu; gc.batch = 1; gc.loops = 1;
      return run_gemm(gc, stream);
    }
  }
  auto cuda_cores = [&]() -> int {
    count_fallback_launch();
    conv_fprop_simt<<<launch_1d(g.sizeO(), 256, c), 256, 0, stream>>>(
        g, static_cast<const __half*>(I), static_cast<const __half*>(F), static_cast<__half*>(O), alpha, relu, nullptr, 0);
    NG_CHECK_LAUNCH();
    return NG_OK;
  };
  if (!tc) return cuda_cores();
  const int RST = g.T * g.R * g.S;
  const long long ldo = 1ll * g.M * g.P * g.Q * g.N;
  TcParams p = {};
  p.mode = TC_FPROP;
  const long long cols = pixel_columns(p, 1ll * g.M * g.P, g.Q, g.N, mode);
  if (cols > 0x7fffffffll) return phased ? cuda_cores() : fail(NG_ERR_TOO_LARGE, "output too large");
  p.M = g.K; p.N = static_cast<int>(cols);
  p.nz = 1; p.splits = 1;
  TcOperandLayout lay = {1, 1, pick_kb_rows(g.C)};
  p.red_chunks = (g.C + lay.kb_rows - 1) / lay.kb_rows;
  p.num_kb = RST * p.red_chunks;
  tc_pick_tile(c, p, cols, p.num_kb, lay.kb_rows);
  CUtensorMap mapA, mapB, mapBm;
  // fewer, larger boxes where the shapes allow: the filters of a 128-row half as one box, the
  // pixels of a column tile inside one image row as one box
  const bool merge_off = tuning().merge_boxes == 0;
  lay.a_merge = !merge_off && g.K % kChunk == 0 && g.K > kChunk &&
                filter_map_merged(&mapA, F, g, lay.kb_rows) == NG_OK;
  lay.a_chunks = (g.K + kChunk - 1) / kChunk;
  const int stack = g.str_h == 1 ? pick_row_stack(c, g.K, kChunk, RST, g.R, p.red_chunks, lay.kb_rows, g.P, g.M,
                                                  1ll * row_chunks(g.N, g.Q, mode) * kChunk, alpha)
                                 : 0;
  if (stack) {
    fill_row_pairs(p, stack, g.N, g.Q, g.P, g.M, mode, g.N, 1ll * g.Q * g.N, 1ll * g.P * g.Q * g.N);
    p.num_kb = g.T * (g.R + 1) * g.S * p.red_chunks;
    lay.a_chunks = 2;
  }
  tc_fill_mma(p, lay);
  fill_taps(p, g, mode);
  if (phased) fill_phases(p, g.str_w);
  if (stack) { ++p.R; p.RS += g.S; p.str_h = 2; }
  fill_decode(p, g.N, g.Q, stack ? p.cmap.y_count : g.P, g.M, mode);
  p.oob_y = g.H;
  p.C = O; p.Cold = nullptr; p.ldc = ldo; p.c_zstride = stack ? 1ll * g.Q * g.N : 0;
  p.alpha = alpha; p.beta = 0.0f; p.relu = relu; p.sr_bits = 0; p.out_f32 = 0; p.vec_ok = 1;
  if (!lay.a_merge) {
    rc = stack ? filter_map_rows(&mapA, F, g.K, g.S, g.R, g.T, g.C, lay.kb_rows) : filter_map(&mapA, F, g, lay.kb_rows);
    if (rc != NG_OK) return rc;
  }
  // few tiles (a small minibatch, e.g. the shard of one GPU): the reduction is split over the SMs too
  if (!stack) p.splits = choose_splits(c, 1ll * p.tiles_m * p.tiles_n, p.num_kb, 1ll * g.K * cols, true);
  if (phased) {
    const size_t bytes[2] = {phase_split_bytes(g, g.str_w), kScanFlags * sizeof(int)};
    void* room[2] = {nullptr, nullptr};
    int scans = 0;
    rc = chan_block_room(c, stream, p, bytes, room, 2, true);
    if (rc == NG_ERR_TOO_LARGE) return cuda_cores();
    int* flags = static_cast<int*>(room[1]);
    if (rc == NG_OK) rc = phase_split(g, g.str_w, I, room[0], F, flags, &scans, stream);
    if (rc == NG_OK) rc = phase_map(&mapB, room[0], g, g.str_w, lay.kb_rows);
    if (rc == NG_OK) rc = tc_launch(c, mapA, mapB, p, stream);
    if (rc != NG_OK) return rc;
    return launch_dependent(redo_blocks(c), stream, conv_fprop_simt, g, static_cast<const __half*>(I), static_cast<const __half*>(F),
                       static_cast<__half*>(O), alpha, relu, static_cast<const int*>(flags), scans);
  }
  const bool blocked = wants_chan_block(g.D, g.H, g.W, g.N, RST);
  if (blocked) {   // large channel planes: the product reads a copy in (z, y, chan, x, n) order
    const size_t bytes = chan_block_bytes(g.C, g.D, g.H, g.W, g.N);
    void* copy = nullptr;
    rc = chan_block_room(c, stream, p, &bytes, &copy, 1);
    if (rc == NG_OK) rc = chan_block(c, stream, I, copy, g.C, g.D, g.H, g.W, g.N);
    if (rc != NG_OK) return rc;
    I = copy;
  }
  rc = act_map(&mapB, I, g.C, g.D, g.H, g.W, g.N, mode, lay.kb_rows, blocked);
  if (rc != NG_OK) return rc;
  if (mode == CH_PIXEL && g.str_w == 1)
    p.b_merge = act_map_merged(&mapBm, I, g.C, g.D, g.H, g.W, g.N, lay.kb_rows, p.block_n / kChunk, blocked);
  return tc_launch(c, mapA, mapB, p, stream, p.b_merge ? &mapBm : nullptr);
}

int ng_conv_bprop(const ng_conv_desc* d, const void* F, const void* E, void* gradI, float alpha, int path,
                  void* stream_) {
  Geo g;
  int rc = make_geo(d, g);
  if (rc != NG_OK) return rc;
  if (!F || !E || !gradI) return fail(NG_ERR_INVALID_ARG, "null tensor");
  DeviceCtx* c = current_ctx();
  if (!c) return NG_ERR_CUDA;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  // (the error tensor is read pixel by pixel whatever the strides are; see bprop_phase)
  const ChunkMode mode = g.N % kChunk == 0 ? CH_PIXEL : CH_FLAT;
  const bool in_place = pick_chunk_mode(g.N, g.str_w) != CH_NONE;
  const bool addressable = path != NG_PATH_SIMT && (in_place || path == NG_PATH_AUTO) && aligned16(F) && aligned16(E) && aligned16(gradI);
  if (path == NG_PATH_TENSOR && !addressable) return fail(NG_ERR_UNSUPPORTED, "shape not addressable by the tensor-core path");
  const bool by_phases = addressable && bprop_by_phases(c, g, in_place);
  auto cuda_cores = [&](bool counted) -> int {
    if (counted) count_fallback_launch();
    conv_bprop_simt<<<launch_1d(g.sizeI(), 256, c), 256, 0, stream>>>(
        g, static_cast<const __half*>(F), static_cast<const __half*>(E), static_cast<__half*>(gradI), alpha, nullptr, 0);
    NG_CHECK_LAUNCH();
    return NG_OK;
  };
  if (!addressable || !(by_phases || in_place)) return cuda_cores(!addressable);
  const int str[3] = {g.str_d, g.str_h, g.str_w}, flt[3] = {g.T, g.R, g.S};
  const bool gather = !by_phases;
  const bool blocked = wants_chan_block(g.M, g.P, g.Q, g.N, g.T * g.R * g.S);
  auto phases = [&](BpropPlan* plan) -> int {
    for (int pt = 0; pt < (gather ? 1 : std::min(str[0], flt[0])); ++pt)
      for (int pr = 0; pr < (gather ? 1 : std::min(str[1], flt[1])); ++pr)
        for (int ps = 0; ps < (gather ? 1 : std::min(str[2], flt[2])); ++ps) {
          const int first[3] = {pt, pr, ps};
          const int rc = bprop_phase(c, g, first, mode, F, E, gradI, alpha, blocked, gather, plan, stream);
          if (rc != NG_OK) return rc;
        }
    return NG_OK;
  };
  const bool scan = !in_place;      // (see phase_split)
  const void* E0 = E;
  int* flags = nullptr;
  if (blocked || scan) {   // behind the products' partials: the copy of E, the flags
    BpropPlan plan;
    rc = phases(&plan);
    if (rc == NG_ERR_TOO_LARGE && scan) return cuda_cores(true);
    if (rc != NG_OK) return rc;
    const size_t off = round256(plan.partials);
    const size_t copy_bytes = blocked ? chan_block_bytes(g.K, g.M, g.P, g.Q, g.N) : 0;
    const size_t bytes = off + copy_bytes + kScanFlags * sizeof(int);
    if (scan && !scratch_or_none(c, stream, bytes)) return cuda_cores(true);
    rc = ensure_workspace(c, stream, bytes);
    if (rc != NG_OK) return rc;
    uint8_t* room = reinterpret_cast<uint8_t*>(c->ws) + off;
    if (blocked) {   // large channel planes: the products read a copy in (z, y, chan, x, n) order
      rc = chan_block(c, stream, E, room, g.K, g.M, g.P, g.Q, g.N);
      if (rc != NG_OK) return rc;
      E = room;
    }
    if (scan) {
      flags = reinterpret_cast<int*>(room + copy_bytes);
      rc = launch_dependent(kScanFlags, stream, nonfinite_scan, static_cast<const uint4*>(F), g.sizeF() / 8, flags);
      if (rc != NG_OK) return rc;
    }
  }
  // a phase that no tap falls on, because the stride is larger than the filter, gets no error at all
  if (!gather && (str[0] > flt[0] || str[1] > flt[1] || str[2] > flt[2]))
    NG_CUDA(cudaMemsetAsync(gradI, 0, static_cast<size_t>(g.sizeI()) * 2, stream));
  rc = phases(nullptr);
  if (rc != NG_OK || !scan) return rc;
  return launch_dependent(redo_blocks(c), stream, conv_bprop_simt, g, static_cast<const __half*>(F), static_cast<const __half*>(E0),
                     static_cast<__half*>(gradI), alpha, static_cast<const int*>(flags), kScanFlags);
}

int ng_conv_update(const ng_conv_desc* d, const void* I, const void* E, void* gradF, int out_f32, float alpha,
                   int path, void* stream_) {
  Geo g;
  int rc = make_geo(d, g);
  if (rc != NG_OK) return rc;
  if (!I || !E || !gradF) return fail(NG_ERR_INVALID_ARG, "null tensor");
  DeviceCtx* c = current_ctx();
  if (!c) return NG_ERR_CUDA;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  ChunkMode mode = pick_chunk_mode(g.N, g.str_w);
  const bool al = aligned16(I) && aligned16(E) && aligned16(gradF);
  const int RST = g.T * g.R * g.S;
  const long long span = 1ll * g.M * g.P * g.Q * g.N;
  const bool phased = mode == CH_NONE && path == NG_PATH_AUTO && update_by_phases(g);
  if (phased) mode = CH_FLAT;    // a phase-split copy in flattened rows
  const bool direct = path != NG_PATH_SIMT && path != NG_PATH_IM2COL && mode != CH_NONE && al &&
                      (g.C >= 16 || path == NG_PATH_TENSOR);
  const bool im2col = !direct && path != NG_PATH_SIMT && path != NG_PATH_TENSOR && al &&
                      1ll * g.C * RST * span * 2 <= (6ll << 30) && g.C * RST <= 65535;
  if (path == NG_PATH_TENSOR && !direct) return fail(NG_ERR_UNSUPPORTED, "shape not addressable by the tensor-core path");
  if (path == NG_PATH_IM2COL && !im2col) return fail(NG_ERR_UNSUPPORTED, "shape not addressable by the im2col path");
  if ((path == NG_PATH_AUTO || path == NG_PATH_TENSOR) && g.C < 16 && g.N % kChunk == 0 && al) {
    const TapBlock tb = pick_tap_block(g);
    if (tb.ok) return update_tapblock(c, g, tb, I, E, gradF, out_f32, alpha, stream);
  }
  if (path == NG_PATH_AUTO && g.C < 16 && g.N % kChunk != 0 && al) {
    const SpaceToDepth z = pick_space_to_depth(g);   // see there
    if (z.ok) {
      const size_t i2_bytes = round256(2ull * z.C2 * z.H2 * z.W2 * g.N), g2_bytes = round256(4ull * z.C2 * z.R2 * z.S2 * g.K);
      AuxClaim aux;
      void* room = nullptr;
      rc = aux.room(c, stream, i2_bytes + g2_bytes, &room);
      if (rc != NG_OK) return rc;
      uint4* I2 = static_cast<uint4*>(room);
      float* G2 = reinterpret_cast<float*>(static_cast<uint8_t*>(room) + i2_bytes);
      s2d_input_kernel<<<z.C2 * z.H2, 256, 0, stream>>>(g, z, static_cast<const uint4*>(I), I2);
      NG_CHECK_LAUNCH();
      const ng_conv_desc d2 = space_to_depth_desc(g, z);
      rc = ng_conv_update(&d2, I2, E, G2, 1, alpha, NG_PATH_AUTO, stream_);
      if (rc != NG_OK) return rc;
      s2d_filter_grad_kernel<<<launch_1d(g.sizeF(), 256, c), 256, 0, stream>>>(g, z, G2, gradF, out_f32);
      NG_CHECK_LAUNCH();
      return NG_OK;
    }
  }
  auto cuda_cores = [&, I0 = static_cast<const __half*>(I), E0 = static_cast<const __half*>(E)]() -> int {
    count_fallback_launch();
    conv_update_simt<<<launch_1d(g.sizeF() * 32, 256, c), 256, 0, stream>>>(g, I0, E0, gradF, out_f32, alpha);
    NG_CHECK_LAUNCH();
    return NG_OK;
  };
  auto redo = [&, I0 = static_cast<const __half*>(I), E0 = static_cast<const __half*>(E)] {   // (see phase_split)
    return launch_dependent(redo_blocks(c), stream, conv_update_redo, g, I0, E0, gradF, out_f32, alpha);
  };
  if (direct && wants_update_swap(g, 1ll * g.M * g.P * row_chunks(g.N, g.Q, mode))) {
    TapBlock taps;
    taps.bw = taps.bh = 1; taps.rows = swap_rows(g.C); taps.nr = g.R; taps.ns = g.S; taps.ok = true;
    rc = update_swapped(c, g, taps, mode, phased, I, E, gradF, out_f32, alpha, stream);
    if (rc == NG_ERR_TOO_LARGE && phased) return cuda_cores();
    return rc == NG_OK && phased && beyond_patches(g) ? redo() : rc;
  }
  if (direct) {
    TcParams p = {};
    p.mode = TC_UPDATE;
    p.block_n = update_block_n(g.K);
    p.M = g.C; p.N = g.K;
    p.tiles_n = (g.K + p.block_n - 1) / p.block_n;
    p.nz = RST;
    TcOperandLayout lay = {0, 0, kChunk};
    // one k-block per chunk of the (m, p, q, n) space; ragged image rows are padded to whole
    // chunks, whose tail TMA zero-fills in the error tensor
    p.num_kb = g.M * g.P * row_chunks(g.N, g.Q, mode);
    // the reduction is split to fill the SMs whatever the tile count, so only the operand
    // traffic argues: assume many column tiles
    tc_pick_tile_rows(c, p, 64ll * p.tiles_n * p.nz, p.num_kb);
    int a_rows = kTileM * p.m_halves;
    if (g.C <= 64) {
      // short A boxes leave room in the ring for several taps per work item
      a_rows = (g.C + 7) / 8 * 8;
      lay.a_box_rows = a_rows;
      set_update_groups(p, RST, a_rows);
    }
    tc_fill_mma(p, lay);
    fill_taps(p, g, mode);
    if (phased) fill_phases(p, update_phases(g));
    fill_decode(p, g.N, g.Q, g.P, g.M, mode);
    p.oob_y = g.H;
    p.C = gradF; p.Cold = nullptr; p.ldc = 1ll * RST * g.K; p.c_zstride = g.K;
    p.alpha = alpha; p.beta = 0.0f; p.relu = 0; p.sr_bits = 0; p.out_f32 = out_f32; p.vec_ok = 1;
    p.splits = choose_splits(c, 1ll * p.tiles_m * p.tiles_n * p.nz, p.num_kb, 1ll * g.C * g.K * RST);
    if (phased)
      p.splits = shorter_partitions(c, 1ll * p.tiles_m * p.tiles_n * p.nz, p.num_kb, p.splits, 1ll * g.C * g.K * RST, 4, kLongSum);
    const int launches = phased && beyond_patches(g) ? short_sums(p, 1ll * g.C * g.K * RST) : 1;
    const bool rounded = launches > 1 && !out_f32;      // (summed in fp32, then rounded)
    CUtensorMap mapA, mapB;
    // large channel planes: the product reads copies in (z, y, chan, x, n) order
    const bool blocked_i = !phased && wants_chan_block(g.D, g.H, g.W, g.N, RST);
    const bool blocked_e = wants_chan_block(g.M, g.P, g.Q, g.N, RST);
    if (phased || blocked_i || blocked_e) {
      const size_t bytes[3] = {phased ? phase_split_bytes(g, update_phases(g)) : blocked_i ? chan_block_bytes(g.C, g.D, g.H, g.W, g.N) : 0,
                               blocked_e ? chan_block_bytes(g.K, g.M, g.P, g.Q, g.N) : 0,
                               rounded ? round256(4ull * g.sizeF()) : 0};
      void* copies[3] = {nullptr, nullptr, nullptr};
      rc = chan_block_room(c, stream, p, bytes, copies, 3, phased);
      if (rc == NG_ERR_TOO_LARGE && phased) return cuda_cores();
      if (rc == NG_OK && phased) rc = phase_split(g, update_phases(g), I, copies[0], nullptr, nullptr, nullptr, stream);
      if (rc == NG_OK && blocked_i) rc = chan_block(c, stream, I, copies[0], g.C, g.D, g.H, g.W, g.N);
      if (rc == NG_OK && blocked_e) rc = chan_block(c, stream, E, copies[1], g.K, g.M, g.P, g.Q, g.N);
      if (rc != NG_OK) return rc;
      if (phased || blocked_i) I = copies[0];
      if (blocked_e) E = copies[1];
      if (rounded) { p.C = copies[2]; p.out_f32 = 1; }
    }
    rc = phased ? phase_map(&mapA, I, g, update_phases(g), a_rows) : act_map(&mapA, I, g.C, g.D, g.H, g.W, g.N, mode, a_rows, blocked_i);
    if (rc != NG_OK) return rc;
    rc = act_map(&mapB, E, g.K, g.M, g.P, g.Q, g.N, mode, p.block_n, blocked_e);
    if (rc != NG_OK) return rc;
    rc = launch_sums(c, mapA, mapB, p, launches, stream);
    if (rc == NG_OK && rounded) {
      round_kernel<<<launch_1d(g.sizeF(), 256, c), 256, 0, stream>>>(static_cast<const float*>(p.C), static_cast<__half*>(gradF), g.sizeF());
      NG_CHECK_LAUNCH();
    }
    return rc == NG_OK && phased && beyond_patches(g) ? redo() : rc;
  }
  if (im2col) {
    // dF[crst][k] = col[crst][span] * E[k][span]^T  (both K-major: an "nt" GEMM with split-K)
    const size_t col_bytes = static_cast<size_t>(g.C) * RST * span * 2;
    const size_t col_off = ((static_cast<size_t>(kMaxSplits) * g.C * RST * g.K * 4) + 255) & ~size_t(255);  // room for partials
    rc = ensure_workspace(c, stream, col_off + col_bytes);
    if (rc != NG_OK) return rc;
    __half* col = reinterpret_cast<__half*>(reinterpret_cast<uint8_t*>(c->ws) + col_off);
    const long long total = 1ll * g.C * RST * span / 8;
    (void)total;
    im2col_kernel<<<im2col_grid(g), 256, 0, stream>>>(g, static_cast<const __half*>(I), col);
    NG_CHECK_LAUNCH();
    GemmCall gc = {};
    gc.A = col; gc.B = E; gc.C = gradF; gc.a_t = 0; gc.b_t = 1;
    gc.m = g.C * RST; gc.n = g.K;
    if (span > 0x7fffffffll) return fail(NG_ERR_TOO_LARGE, "reduction too long");
    gc.k = static_cast<int>(span);
    gc.lda = span; gc.ldb = span; gc.ldc = g.K;
    gc.alpha = alpha; gc.beta = 0.0f; gc.batch = 1; gc.loops = 1; gc.out_f32 = out_f32;
    if (mode == CH_NONE) gc.long_kb = kLongPatchSum;
    return run_gemm(gc, stream);
  }
  return cuda_cores();
}

}  // extern "C"
