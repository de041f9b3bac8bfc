// ng.dot on the device: C = relu?(alpha * op(A) * op(B)) + beta * C, fp16 in, fp32 accumulate,
// fp16 out with round-to-nearest-even or stochastic rounding.
// Mirrors NervanaGPU.dot / batched_dot (nervanagpu/nervanagpu.py:820-1105) and the C interface
// nervana_hgemm (nervanagpu/kernels/C_interface/nervana_c_api.h:31-128).
//
// The tcgen05 engine runs them. Operands that TMA cannot address (base not 16-byte aligned, leading
// dimension or batch stride no multiple of 8 elements) are first copied into rows that it can
// (pack_rows_kernel). The plain CUDA-core kernel serves very short products of such operands
// (shorter_unpacked), operands of more than 2^30 packed groups, calls that are both batched and summed
// over a batch, packed and summed products for which there is no scratch memory, and ng_hgemm_simt, the
// second opinion of the tests.
#include <algorithm>

#include "../../include/nervana_b200.h"
#include "epilogue.cuh"
#include "host.h"

namespace ngb {

namespace {

// ------------------------------------------------------------------------------------------
// SIMT fallback: 64x64 tile per CTA, 4x4 outputs per thread, arbitrary strides.
// ------------------------------------------------------------------------------------------
struct SimtGemmArgs {
  const __half* A;
  const __half* B;
  void* C;
  int a_t, b_t;
  int m, n, k;
  long long lda, ldb, ldc;
  long long az, bz, cz;   // batch strides (elements)
  int loops;              // batches accumulated into one output
  long long alz, blz;     // strides between accumulated batches
  int out_f32;
  EpiArgs ea;
};

__global__ void __launch_bounds__(256) gemm_simt_kernel(SimtGemmArgs g) {
  __shared__ float sA[16][64 + 1];
  __shared__ float sB[16][64 + 1];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int m0 = blockIdx.y * 64, n0 = blockIdx.x * 64;
  const int z = blockIdx.z;
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;

  for (int l = 0; l < g.loops; ++l) {
    const __half* A = g.A + z * g.az + l * g.alz;
    const __half* B = g.B + z * g.bz + l * g.blz;
    for (int k0 = 0; k0 < g.k; k0 += 16) {
      for (int i = threadIdx.x; i < 16 * 64; i += 256) {
        int kk, mm;
        if (g.a_t) { mm = i & 63; kk = i >> 6; } else { kk = i & 15; mm = i >> 4; }
        const int gm = m0 + mm, gk = k0 + kk;
        float v = 0.0f;
        if (gm < g.m && gk < g.k) v = __half2float(g.a_t ? A[gk * g.lda + gm] : A[gm * g.lda + gk]);
        sA[kk][mm] = v;
      }
      for (int i = threadIdx.x; i < 16 * 64; i += 256) {
        int kk, nn;
        if (g.b_t) { kk = i & 15; nn = i >> 4; } else { nn = i & 63; kk = i >> 6; }
        const int gn = n0 + nn, gk = k0 + kk;
        float v = 0.0f;
        if (gn < g.n && gk < g.k) v = __half2float(g.b_t ? B[gn * g.ldb + gk] : B[gk * g.ldb + gn]);
        sB[kk][nn] = v;
      }
      __syncthreads();
#pragma unroll
      for (int kk = 0; kk < 16; ++kk) {
        float a[4], b[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = sA[kk][ty * 4 + i];
#pragma unroll
        for (int j = 0; j < 4; ++j) b[j] = sB[kk][tx * 4 + j];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
      }
      __syncthreads();
    }
  }
  for (int i = 0; i < 4; ++i) {
    const int row = m0 + ty * 4 + i;
    if (row >= g.m) continue;
    for (int j = 0; j < 4; ++j) {
      const int col = n0 + tx * 4 + j;
      if (col >= g.n) continue;
      const long long off = z * g.cz + row * g.ldc + col;
      float c = epi_scale(g.ea, acc[i][j]);
      if (g.out_f32) {
        float* out = static_cast<float*>(g.C) + off;
        if (g.ea.beta != 0.0f) c = fmaf(g.ea.beta, *out, c);
        *out = c;
      } else {
        __half* out = static_cast<__half*>(g.C) + off;
        if (g.ea.beta != 0.0f) c = fmaf(g.ea.beta, __half2float(*out), c);
        if (g.ea.sr_bits) {
          const unsigned long long lin = (static_cast<unsigned long long>(z) * g.m + row) * g.n + col;
          uint32_t rnd[8];
          sr_bits8(g.ea, lin >> 3, rnd);
          *out = f2h_sr(c, rnd[lin & 7ull], g.ea.sr_bits);
        } else {
          *out = f2h_rn(c);
        }
      }
    }
  }
}

// ------------------------------------------------------------------------------------------
// Copy of an operand with rows at odd addresses into rows of a multiple of 8 elements.
// ------------------------------------------------------------------------------------------
struct PackArgs {
  const __half* src;
  uint4* dst;
  long long ld, zstride;    // of src, in elements
  uint32_t rows, cols8, cols, total;   // rows per batch entry; 16-byte groups per row; elements per row; groups in all
};

// Each thread moves 8 elements. Their 16 bytes start at any even address: two aligned 16-byte
// loads (the second is the neighbour's first, an L1 hit, and is left out where nothing of it is
// needed, so that no load leaves the 16-byte granules that hold the operand) and a byte shift.
__device__ __forceinline__ void pack_group(const PackArgs& a, uint32_t i) {
  const uint32_t r = i / a.cols8, g = i - r * a.cols8;
  const uint32_t z = r / a.rows;
  const __half* s = a.src + z * a.zstride + static_cast<long long>(r - z * a.rows) * a.ld + g * 8;
  const uint32_t sh = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(s)) & 15u;
  const uint4* q = reinterpret_cast<const uint4*>(reinterpret_cast<uintptr_t>(s) & ~uintptr_t(15));
  const uint32_t need = min(8u, a.cols - g * 8) * 2u;     // bytes that exist
  const uint4 lo = __ldg(q);
  uint4 hi = make_uint4(0u, 0u, 0u, 0u);
  if (sh + need > 16u) hi = __ldg(q + 1);
  uint32_t w0 = lo.x, w1 = lo.y, w2 = lo.z, w3 = lo.w, w4 = hi.x, w5 = hi.y, w6 = hi.z, w7 = hi.w;
  if (sh & 8u) { w0 = w2; w1 = w3; w2 = w4; w3 = w5; w4 = w6; w5 = w7; }
  if (sh & 4u) { w0 = w1; w1 = w2; w2 = w3; w3 = w4; w4 = w5; }
  const uint32_t bits = (sh & 2u) * 8u;
  a.dst[i] = make_uint4(__funnelshift_r(w0, w1, bits), __funnelshift_r(w1, w2, bits), __funnelshift_r(w2, w3, bits),
                        __funnelshift_r(w3, w4, bits));
}

// Both operands in one launch, the groups of the second behind those of the first. Bound by the
// memory traffic (the copies stay in L2 for the product that follows).
__global__ void __launch_bounds__(256) pack_rows_kernel(PackArgs a, PackArgs b) {
  grid_dependency_wait();
  grid_launch_dependents();   // the product sets itself up meanwhile and waits for the copies
  const uint32_t i = blockIdx.x * 256u + threadIdx.x;
  if (i < a.total) pack_group(a, i);
  else if (i - a.total < b.total) pack_group(b, i - a.total);
}

// Fills `a` for an operand of `nz` entries of rows x cols elements; false when it is too large.
bool plan_pack(PackArgs& a, const void* src, long long ld, long long zstride, long long nz, long long rows, long long cols) {
  a.src = static_cast<const __half*>(src);
  a.ld = ld; a.zstride = zstride;
  const long long c8 = (cols + 7) / 8, total = nz * rows * c8;
  if (total > 0x3fffffffll) return false;
  a.rows = static_cast<uint32_t>(rows); a.cols = static_cast<uint32_t>(cols);
  a.cols8 = static_cast<uint32_t>(c8); a.total = static_cast<uint32_t>(total);
  return true;
}

// Whether a product whose operands would have to be packed is shorter on the CUDA cores, which take about
// 2.1 us per 16 rows of the reduction after the first 4.5 while the device holds all tiles, and need no second
// launch. Packing and product take 5.5 to 8.1 us with up to 128 columns and 10 beyond, hardly more for longer
// reductions. CUDA cores / packed, in a recorded sequence (us): 65 x 65 x 9 4.6 / 7.3, x 25 6.6 / 7.3 (one by
// one 8.5 / 7.7), x 33 8.8 / 7.4; 513 x 513 x 9 4.8 / 10.0, x 25 6.7 / 10.2, x 41 9.4 / 10.2 (one by one 10.9 / 10.7);
// 1001 x 1001 x 25 9.3 / 10.4, x 33 12.1 / 10.5.
bool shorter_unpacked(const DeviceCtx* c, const GemmCall& g) {
  if (tuning().pack_odd >= 0) return tuning().pack_odd == 0;
  const long long steps = (g.k + 15ll) / 16 * g.loops;
  const long long tiles = ((g.m + 63ll) / 64) * ((g.n + 63ll) / 64) * g.batch;
  return tiles <= 2ll * c->sm_count && (steps <= 1 || (steps == 2 && g.n > 128));
}

bool tma_ok(const void* p, long long ld, long long zstride) {
  return (reinterpret_cast<uintptr_t>(p) & 15u) == 0 && (ld & 7) == 0 && (zstride & 7) == 0;
}

}  // namespace

int run_gemm(const GemmCall& call, cudaStream_t stream) {
  GemmCall g = call;
  if (!g.A || !g.B || !g.C) return fail(NG_ERR_INVALID_ARG, "null operand");
  if (g.m <= 0 || g.n <= 0 || g.k <= 0) return fail(NG_ERR_INVALID_ARG, "m, n, k must be positive");
  if (g.a_t && g.b_t) return fail(NG_ERR_UNSUPPORTED, "op 'tt' is not supported");
  if (g.sr_bits < 0 || g.sr_bits > 10) return fail(NG_ERR_INVALID_ARG, "stochastic rounding keeps 1..10 mantissa bits");
  const long long min_lda = g.a_t ? g.m : g.k, min_ldb = g.b_t ? g.k : g.n;
  if (g.lda < min_lda || g.ldb < min_ldb || g.ldc < g.n) return fail(NG_ERR_INVALID_ARG, "leading dimension too small");
  DeviceCtx* c = current_ctx();
  if (!c) return NG_ERR_CUDA;

  EpiArgs ea;
  ea.alpha = g.alpha; ea.beta = g.beta; ea.relu = g.relu; ea.sr_bits = g.sr_bits;
  ea.seed_lo = static_cast<uint32_t>(g.seed); ea.seed_hi = static_cast<uint32_t>(g.seed >> 32);
  ea.rng_offset = g.rng_offset;

  // one batch dimension per operand: independent products, or products summed into one output
  const bool sum = g.loops > 1;
  const long long zsa = sum ? g.alz : g.az, zsb = sum ? g.blz : g.bz;
  const int nza = zsa == 0 ? 1 : (sum ? g.loops : g.batch), nzb = zsb == 0 ? 1 : (sum ? g.loops : g.batch);
  PackArgs packA = {}, packB = {};
  bool use_tc = !g.force_simt && !(sum && g.batch > 1);
  if (use_tc && !tma_ok(g.A, g.lda, zsa))
    use_tc = plan_pack(packA, g.A, g.lda, zsa, nza, g.a_t ? g.k : g.m, g.a_t ? g.m : g.k);
  if (use_tc && !tma_ok(g.B, g.ldb, zsb))
    use_tc = plan_pack(packB, g.B, g.ldb, zsb, nzb, g.b_t ? g.n : g.k, g.b_t ? g.k : g.n);
  const bool by_rule = use_tc && (packA.total || packB.total) && shorter_unpacked(c, g);
  auto cuda_cores = [&](bool counted) -> int {
    SimtGemmArgs s;
    s.A = static_cast<const __half*>(g.A); s.B = static_cast<const __half*>(g.B); s.C = g.C;
    s.a_t = g.a_t; s.b_t = g.b_t; s.m = g.m; s.n = g.n; s.k = g.k;
    s.lda = g.lda; s.ldb = g.ldb; s.ldc = g.ldc;
    s.az = g.az; s.bz = g.bz; s.cz = g.cz; s.loops = g.loops; s.alz = g.alz; s.blz = g.blz;
    s.out_f32 = g.out_f32; s.ea = ea;
    dim3 grid((g.n + 63) / 64, (g.m + 63) / 64, g.batch);
    if (counted) count_fallback_launch();
    gemm_simt_kernel<<<grid, 256, 0, stream>>>(s);
    NG_CHECK_LAUNCH();
    return NG_OK;
  };
  if (!use_tc || by_rule) return cuda_cores(!by_rule);

  TcParams p = {};
  p.mode = TC_GEMM;
  p.block_n = g.n <= 64 ? 64 : (g.n <= 128 ? 128 : 256);
  p.M = g.m; p.N = g.n;
  p.tiles_n = (g.n + p.block_n - 1) / p.block_n;
  p.nz = g.batch;
  p.red_chunks = (g.k + kChunk - 1) / kChunk;
  if (static_cast<long long>(p.red_chunks) * g.loops > 0x7fffffffll) return fail(NG_ERR_TOO_LARGE, "reduction too long");
  p.num_kb = p.red_chunks * g.loops;
  tc_pick_tile_rows(c, p, static_cast<long long>(p.tiles_n) * p.nz, p.num_kb);
  // Two or more row tiles and 128 or 256 columns: CTA pairs (a 256-row tile over two SMs, each of
  // which loads half of the B columns).
  if (tuning().pair_mma == 1 && g.m > kTileM && p.block_n >= 128) {
    p.pair = 1;
    p.m_halves = 1;
    p.tiles_m = (g.m + 2 * kTileM - 1) / (2 * kTileM);
  }
  const int bn_cta = p.pair ? p.block_n / 2 : p.block_n;
  TcOperandLayout lay;
  lay.a_mn_major = g.a_t ? 1 : 0;   // stored k x m: m contiguous
  lay.b_mn_major = g.b_t ? 0 : 1;   // stored k x n: n contiguous
  lay.kb_rows = kChunk;
  // an operand whose contiguous dimension is m (or n), a multiple of 64: the map gets the 64-wide
  // chunk number as a dimension of its own, and one box brings a 128-row half (a column tile)
  const bool merge_off = tuning().merge_boxes == 0;
  lay.a_merge = !merge_off && g.a_t && g.m % kChunk == 0;
  lay.b_merge_static = !merge_off && !g.b_t && g.n % kChunk == 0 && bn_cta >= 2 * kChunk;
  tc_fill_mma(p, lay);
  p.a_zmul = !sum && nza > 1; p.b_zmul = !sum && nzb > 1;
  p.a_lmul = sum && nza > 1; p.b_lmul = sum && nzb > 1;
  p.C = g.C; p.Cold = g.beta != 0.0f ? g.C : nullptr;
  p.ldc = g.ldc; p.c_zstride = g.cz;
  p.alpha = g.alpha; p.beta = g.beta; p.relu = g.relu; p.sr_bits = g.sr_bits; p.out_f32 = g.out_f32;
  const int esz = g.out_f32 ? 4 : 2;
  const int vec_elems = 16 / esz;
  p.vec_ok = (reinterpret_cast<uintptr_t>(g.C) & 15u) == 0 && g.ldc % vec_elems == 0 && g.cz % vec_elems == 0;
  p.seed_lo = ea.seed_lo; p.seed_hi = ea.seed_hi; p.rng_offset = g.rng_offset;
  p.splits = choose_splits(c, static_cast<long long>(p.tiles_m) * p.tiles_n * p.nz, p.num_kb,
                           static_cast<long long>(g.m) * g.n * g.batch);
  if (g.long_kb > 0)
    p.splits = shorter_partitions(c, 1ll * p.tiles_m * p.tiles_n * p.nz, p.num_kb, p.splits, 1ll * g.m * g.n * g.batch, 2, g.long_kb);
  if (p.splits > 1 && (g.n & 7)) {
    // partials with whole 16-byte groups per row: they leave through the staged output stage, and
    // the second stage stores the columns that exist
    p.n_store = g.n;
    p.N = (g.n + 7) & ~7;
  }
  size_t off = p.splits > 1 ? static_cast<size_t>(p.splits) * p.nz * p.M * p.N * sizeof(float) : 0;
  off = (off + 255) & ~size_t(255);
  const size_t bytesA = (static_cast<size_t>(packA.total) * 16 + 255) & ~size_t(255);
  const size_t room_bytes = off + bytesA + static_cast<size_t>(packB.total) * 16;
  // (without room, the kernel that needs none)
  if ((packA.total || packB.total || sum) && room_bytes > 0 && !scratch_or_none(c, stream, room_bytes)) return cuda_cores(true);
  if (packA.total || packB.total) {
    uint8_t* room = reinterpret_cast<uint8_t*>(c->ws) + off;
    if (packA.total) {
      packA.dst = reinterpret_cast<uint4*>(room);
      g.A = room; g.lda = packA.cols8 * 8ll; g.az = g.alz = nza > 1 ? g.lda * packA.rows : 0;
    }
    if (packB.total) {
      packB.dst = reinterpret_cast<uint4*>(room + bytesA);
      g.B = room + bytesA; g.ldb = packB.cols8 * 8ll; g.bz = g.blz = nzb > 1 ? g.ldb * packB.rows : 0;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((packA.total + packB.total + 255u) / 256u);
    cfg.blockDim = dim3(256);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = tuning().dependent_launch != 0 ? 1 : 0;
    NG_CUDA(cudaLaunchKernelEx(&cfg, pack_rows_kernel, packA, packB));
    NG_CHECK_LAUNCH();
  }
  const uint64_t zbytesA = static_cast<uint64_t>(sum ? g.alz : g.az) * 2, zbytesB = static_cast<uint64_t>(sum ? g.blz : g.bz) * 2;

  // Tensor maps. Dimension 0 is the contiguous one; dimension 2 walks the batch.
  CUtensorMap mapA, mapB;
  {
    uint64_t dims[5] = {1, 1, 1, 1, 1};
    uint64_t str[4] = {16, 16, 16, 16};
    uint32_t box[5] = {kChunk, 1, 1, 1, 1};
    if (g.a_t) { dims[0] = g.m; dims[1] = g.k; box[1] = kChunk; }
    else       { dims[0] = g.k; dims[1] = g.m; box[1] = kTileM * p.m_halves; }
    dims[2] = nza;
    str[0] = static_cast<uint64_t>(g.lda) * 2;
    str[1] = nza > 1 ? zbytesA : str[0] * dims[1];
    str[2] = str[1] * dims[2];
    str[3] = str[2];
    if (lay.a_merge) {   // (m_lo, k, m_hi, batch)
      dims[0] = kChunk; dims[1] = g.k; dims[2] = g.m / kChunk; dims[3] = nza;
      str[0] = static_cast<uint64_t>(g.lda) * 2; str[1] = 128;
      str[2] = nza > 1 ? zbytesA : str[0] * dims[1];
      str[3] = str[2] * dims[3];
      box[1] = kChunk; box[2] = 2;
    }
    int rc = make_tensor_map(&mapA, g.A, dims, str, box);
    if (rc != NG_OK) return rc;
  }
  {
    uint64_t dims[5] = {1, 1, 1, 1, 1};
    uint64_t str[4] = {16, 16, 16, 16};
    uint32_t box[5] = {kChunk, 1, 1, 1, 1};
    if (g.b_t) { dims[0] = g.k; dims[1] = g.n; box[1] = bn_cta; }
    else       { dims[0] = g.n; dims[1] = g.k; box[1] = kChunk; }
    dims[2] = nzb;
    str[0] = static_cast<uint64_t>(g.ldb) * 2;
    str[1] = nzb > 1 ? zbytesB : str[0] * dims[1];
    str[2] = str[1] * dims[2];
    str[3] = str[2];
    if (lay.b_merge_static) {   // (n_lo, k, n_hi, batch)
      dims[0] = kChunk; dims[1] = g.k; dims[2] = g.n / kChunk; dims[3] = nzb;
      str[0] = static_cast<uint64_t>(g.ldb) * 2; str[1] = 128;
      str[2] = nzb > 1 ? zbytesB : str[0] * dims[1];
      str[3] = str[2] * dims[3];
      box[1] = kChunk; box[2] = bn_cta / kChunk;
    }
    int rc = make_tensor_map(&mapB, g.B, dims, str, box);
    if (rc != NG_OK) return rc;
  }
  return tc_launch(c, mapA, mapB, p, stream);
}

}  // namespace ngb

using namespace ngb;

extern "C" {

int ng_hgemm(const void* A, const void* B, void* C, int a_t, int b_t, int m, int n, int k, int lda, int ldb, int ldc,
             float alpha, float beta, int relu, int sr_bits, unsigned long long seed, unsigned int rng_offset,
             void* stream) {
  GemmCall g = {};
  g.A = A; g.B = B; g.C = C; g.a_t = a_t; g.b_t = b_t; g.m = m; g.n = n; g.k = k;
  g.lda = lda; g.ldb = ldb; g.ldc = ldc; g.alpha = alpha; g.beta = beta; g.relu = relu; g.sr_bits = sr_bits;
  g.seed = seed; g.rng_offset = rng_offset; g.batch = 1; g.loops = 1;
  return run_gemm(g, static_cast<cudaStream_t>(stream));
}

int ng_hgemm_simt(const void* A, const void* B, void* C, int a_t, int b_t, int m, int n, int k, int lda, int ldb,
                  int ldc, float alpha, float beta, int relu, int sr_bits, unsigned long long seed,
                  unsigned int rng_offset, void* stream) {
  GemmCall g = {};
  g.A = A; g.B = B; g.C = C; g.a_t = a_t; g.b_t = b_t; g.m = m; g.n = n; g.k = k;
  g.lda = lda; g.ldb = ldb; g.ldc = ldc; g.alpha = alpha; g.beta = beta; g.relu = relu; g.sr_bits = sr_bits;
  g.seed = seed; g.rng_offset = rng_offset; g.batch = 1; g.loops = 1; g.force_simt = 1;
  return run_gemm(g, static_cast<cudaStream_t>(stream));
}

int ng_hgemm_batched(const void* A, const void* B, void* C, int a_t, int b_t, int m, int n, int k, int lda, int ldb,
                     int ldc, float alpha, float beta, int relu, int sr_bits, unsigned long long seed,
                     unsigned int rng_offset, int batch_grid, int batch_loops, long long ldaz, long long ldbz,
                     long long ldcz, void* stream) {
  if (batch_grid < 1 || batch_loops < 1) return fail(NG_ERR_INVALID_ARG, "batch counts must be >= 1");
  GemmCall g = {};
  g.A = A; g.B = B; g.C = C; g.a_t = a_t; g.b_t = b_t; g.m = m; g.n = n; g.k = k;
  g.lda = lda; g.ldb = ldb; g.ldc = ldc; g.alpha = alpha; g.beta = beta; g.relu = relu; g.sr_bits = sr_bits;
  g.seed = seed; g.rng_offset = rng_offset;
  g.batch = batch_grid; g.loops = batch_loops;
  if (batch_grid > 1) { g.az = ldaz; g.bz = ldbz; g.cz = ldcz; }
  else { g.alz = ldaz; g.blz = ldbz; }
  return run_gemm(g, static_cast<cudaStream_t>(stream));
}

}  // extern "C"
