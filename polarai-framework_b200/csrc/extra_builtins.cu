// The remaining operation builtins of the catalogue
// (include/polarai/core/internal/GenBuiltins.hpp:25-52 of the reference): frelu,
// fsoftmax, fpool, fconv2d, ftranspose, fslice.  2-D single-channel problems: bound by launch and memory latency on
// pictures of the usual sizes.
#include "common.cuh"

namespace polar_b200 {
namespace {

constexpr int kThreads = 256;

// The sum over the CTA, in every thread.
__device__ __forceinline__ double block_sum(double v) {
  __shared__ double warps[kThreads / 32];
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  if ((threadIdx.x & 31) == 0) warps[threadIdx.x >> 5] = v;
  __syncthreads();
  double s = 0.0;
#pragma unroll
  for (int i = 0; i < kThreads / 32; ++i) s += warps[i];
  return s;
}

// fsoftmax, pass 1: one sum of expf(in[i]) per CTA (double accumulation).
__global__ void __launch_bounds__(kThreads) exp_sum_kernel(const float* in, double* partials, uint64_t n, int vec) {
  pdl_enter();
  double acc = 0.0;
  const uint64_t stride = (uint64_t)gridDim.x * kThreads, first = (uint64_t)blockIdx.x * kThreads + threadIdx.x;
  if (vec) {
    for (uint64_t i = first; i < n / 4; i += stride) {
      const float4 x = reinterpret_cast<const float4*>(in)[i];
      acc += ((double)expf(x.x) + (double)expf(x.y)) + ((double)expf(x.z) + (double)expf(x.w));
    }
    if (first < (n & 3)) acc += (double)expf(in[(n & ~3ull) + first]);
  } else {
    for (uint64_t i = first; i < n; i += stride) acc += (double)expf(in[i]);
  }
  acc = block_sum(acc);
  if (threadIdx.x == 0) partials[blockIdx.x] = acc;
}

// fsoftmax, pass 2: every CTA adds the partial sums in the same order (the same bits in every CTA and every run) and
// divides its elements.
__global__ void __launch_bounds__(kThreads) softmax_div_kernel(const float* in, const double* partials, uint32_t count, float* out,
                                                               uint64_t n, int vec) {
  pdl_enter();
  double acc = 0.0;
  for (uint32_t i = threadIdx.x; i < count; i += kThreads) acc += partials[i];
  const float t = (float)block_sum(acc);
  const uint64_t stride = (uint64_t)gridDim.x * kThreads, first = (uint64_t)blockIdx.x * kThreads + threadIdx.x;
  if (vec) {
    for (uint64_t i = first; i < n / 4; i += stride) {
      const float4 x = reinterpret_cast<const float4*>(in)[i];
      reinterpret_cast<float4*>(out)[i] =
          make_float4(__fdiv_rn(expf(x.x), t), __fdiv_rn(expf(x.y), t), __fdiv_rn(expf(x.z), t), __fdiv_rn(expf(x.w), t));
    }
    if (first < (n & 3)) out[(n & ~3ull) + first] = __fdiv_rn(expf(in[(n & ~3ull) + first]), t);
  } else {
    for (uint64_t i = first; i < n; i += stride) out[i] = __fdiv_rn(expf(in[i]), t);
  }
}

// fsoftmax of a vector that fits the registers of one cluster, 8 CTAs x 1024 threads x 32 elements, in one launch: the
// exponentials stay in registers between the sum (through distributed shared memory, in rank order) and the division.
// Bound by latency and, towards its limit, by what eight SMs load and store: the picture
// chain of 28 x 28 ... 640 x 480 pixels takes 15.5 us instead of 20.5 (a launch and the scratch less), 1024 x 768 16.8 instead of 20.0,
// 1024 x 1024, 260100 elements, 19.0 instead of 19.8.
constexpr int kClusterThreads = 1024, kClusterCtas = 8, kClusterVecs = 8;
constexpr uint64_t kClusterElements = 4ull * kClusterThreads * kClusterCtas * kClusterVecs;
template <bool VEC>
__global__ void __launch_bounds__(kClusterThreads, 1) softmax_cluster_kernel(const float* in, float* out, uint32_t n) {
  pdl_enter();
  __shared__ double warps[kClusterThreads / 32], mine;
  const uint32_t first = cluster_rank() * kClusterThreads + threadIdx.x, stride = kClusterThreads * kClusterCtas;
  float e[kClusterVecs][4];
  double acc = 0.0;
#pragma unroll
  for (int v = 0; v < kClusterVecs; ++v) {
    const uint32_t i = first + v * stride;
    if (VEC) {
      const float4 x = i < n / 4 ? reinterpret_cast<const float4*>(in)[i] : make_float4(0.f, 0.f, 0.f, 0.f);
      e[v][0] = x.x, e[v][1] = x.y, e[v][2] = x.z, e[v][3] = x.w;
    } else {
#pragma unroll
      for (int c = 0; c < 4; ++c) e[v][c] = first + (4 * v + c) * stride < n ? in[first + (4 * v + c) * stride] : 0.f;
    }
  }
  const bool tail = VEC && first < (n & 3);                 // the last elements are no vector
  const float t = tail ? expf(in[(n & ~3u) + first]) : 0.f;
#pragma unroll
  for (int v = 0; v < kClusterVecs; ++v)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const bool live = VEC ? first + v * stride < n / 4 : first + (4 * v + c) * stride < n;
      e[v][c] = expf(e[v][c]);
      if (live) acc += (double)e[v][c];
    }
  if (tail) acc += (double)t;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
  if ((threadIdx.x & 31) == 0) warps[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x < 32) {
    acc = warps[threadIdx.x];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    if (threadIdx.x == 0) mine = acc;
  }
  __syncthreads();
  cluster_arrive();
  cluster_wait();
  double part[kClusterCtas], sum = 0.0;
#pragma unroll
  for (int r = 0; r < kClusterCtas; ++r) part[r] = ld_cluster(&mine, (uint32_t)r);
#pragma unroll
  for (int r = 0; r < kClusterCtas; ++r) sum += part[r];
  cluster_arrive();                                         // nobody leaves while another CTA may still read its sum
  const float total = (float)sum;
#pragma unroll
  for (int v = 0; v < kClusterVecs; ++v) {
    const uint32_t i = first + v * stride;
    if (VEC) {
      if (i < n / 4)
        reinterpret_cast<float4*>(out)[i] = make_float4(__fdiv_rn(e[v][0], total), __fdiv_rn(e[v][1], total),
                                                        __fdiv_rn(e[v][2], total), __fdiv_rn(e[v][3], total));
    } else {
#pragma unroll
      for (int c = 0; c < 4; ++c)
        if (first + (4 * v + c) * stride < n) out[first + (4 * v + c) * stride] = __fdiv_rn(e[v][c], total);
    }
  }
  if (tail) out[(n & ~3u) + first] = __fdiv_rn(t, total);
  cluster_wait();
}

// One thread per output, a row of outputs per blockIdx.y (the grid is walked where there are more rows than that).  W > 0:
// square window of that extent, unrolled.
template <int W>
__global__ void __launch_bounds__(kThreads) pool_kernel(const float* in, uint64_t w, uint32_t wh, uint32_t ww, uint64_t sh,
                                                        uint64_t sw, float* out, uint64_t oh, uint64_t ow) {
  pdl_enter();
  const uint64_t j = (uint64_t)blockIdx.x * kThreads + threadIdx.x;
  if (j >= ow) return;
  for (uint64_t i = blockIdx.y; i < oh; i += gridDim.y) {
    const float* src = in + i * sh * w + j * sw;
    float best = -10e5f;
    if (W) {
      float v[W ? W * W : 1];
#pragma unroll
      for (int a = 0; a < W; ++a)
#pragma unroll
        for (int b = 0; b < W; ++b) v[a * W + b] = src[(uint64_t)a * w + b];
#pragma unroll
      for (int e = 0; e < W * W; ++e) best = v[e] > best ? v[e] : best;
    } else {
      for (uint32_t a = 0; a < wh; ++a)
        for (uint32_t b = 0; b < ww; ++b) {
          const float v = src[(uint64_t)a * w + b];
          best = v > best ? v : best;
        }
    }
    out[i * ow + j] = best;
  }
}

// Any kernel extents: one thread per output.
__global__ void __launch_bounds__(kThreads) conv2d_kernel(const float* in, uint64_t w, const float* ker,
                                                          uint32_t kh, uint32_t kw, float* out, uint64_t oh,
                                                          uint64_t ow) {
  pdl_enter();
  const uint64_t j = (uint64_t)blockIdx.x * kThreads + threadIdx.x;
  if (j >= ow) return;
  for (uint64_t i = blockIdx.y; i < oh; i += gridDim.y) {
    float acc = 0.0f;
    for (uint32_t a = 0; a < kh; ++a)
      for (uint32_t b = 0; b < kw; ++b)
        acc = __fadd_rn(__fmul_rn(in[(i + a) * w + j + b], ker[a * kw + b]), acc);   // product rounded, then added
    out[i * ow + j] = acc;
  }
}

// K x K kernels of the usual extents: a CTA computes 128 x 8 outputs from a tile of the picture in shared memory, a thread
// four neighbours of a row: 2 or 3 128-bit loads of the tile serve 4 K products.  One thread per output read every pixel
// K * K times through L1 and spent its time in 64-bit index arithmetic (1024 x 768, K = 5: 17 us, here 4.5).
constexpr int kConvX = 128, kConvY = 8;
template <int K>
__global__ void __launch_bounds__(kThreads) conv2d_tile_kernel(const float* in, uint64_t h, uint64_t w,
                                                               const float* ker, float* out, uint64_t oh,
                                                               uint64_t ow, int vec) {
  constexpr int kRows = kConvY + K - 1, kCols = kConvX + K - 1, kPitch = (kCols + 3) / 4 * 4, kVecs = (K + 3 + 3) / 4;
  __shared__ __align__(16) float tile[kRows][kPitch + 4];
  __shared__ float weight[K * K];
  pdl_enter();
  const uint64_t x0 = (uint64_t)blockIdx.x * kConvX, y0 = (uint64_t)blockIdx.y * kConvY;
  if (threadIdx.x < K * K) weight[threadIdx.x] = ker[threadIdx.x];
  constexpr int kTrips = (kRows * kPitch + kThreads - 1) / kThreads;
  float v[kTrips];
#pragma unroll
  for (int t = 0; t < kTrips; ++t) {
    const int e = threadIdx.x + t * kThreads, r = e / kPitch, c = e % kPitch;
    v[t] = (r < kRows && y0 + r < h && x0 + c < w) ? in[(y0 + r) * w + x0 + c] : 0.f;
  }
#pragma unroll
  for (int t = 0; t < kTrips; ++t) {
    const int e = threadIdx.x + t * kThreads, r = e / kPitch, c = e % kPitch;
    if (r < kRows) tile[r][c] = v[t];
  }
  __syncthreads();
  const int tx = (threadIdx.x & 31) * 4, ty = threadIdx.x >> 5;
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int a = 0; a < K; ++a) {
    float p[kVecs * 4];
#pragma unroll
    for (int q = 0; q < kVecs; ++q) *reinterpret_cast<float4*>(p + 4 * q) = *reinterpret_cast<const float4*>(&tile[ty + a][tx + 4 * q]);
#pragma unroll
    for (int b = 0; b < K; ++b)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[i] = __fadd_rn(__fmul_rn(p[i + b], weight[a * K + b]), acc[i]);   // product rounded, then added
  }
  const uint64_t y = y0 + ty, x = x0 + tx;
  if (y >= oh || x >= ow) return;
  float* dst = out + y * ow + x;
  if (vec && x + 4 <= ow) {
    *reinterpret_cast<float4*>(dst) = make_float4(acc[0], acc[1], acc[2], acc[3]);
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (x + i < ow) dst[i] = acc[i];
  }
}

// out[c, r] = in[r, c] through a 32 x 33 shared-memory tile: both the reads and the writes
// are coalesced rows of 32 floats.  One tile per CTA (32 x 8 threads, four rows each).
constexpr int kTile = 32;
__global__ void __launch_bounds__(kTile * 8) transpose_kernel(const float* in, float* out,
                                                              uint64_t rows, uint64_t cols, uint32_t tiles_c) {
  __shared__ float tile[kTile][kTile + 1];
  pdl_enter();
  const int tx = threadIdx.x % kTile, ty = threadIdx.x / kTile;
  const uint64_t tr = blockIdx.x / tiles_c, tc = blockIdx.x % tiles_c;
  const uint64_t r0 = tr * kTile, c0 = tc * kTile;
  for (int j = ty; j < kTile; j += 8) {
    const uint64_t r = r0 + j, c = c0 + tx;
    if (r < rows && c < cols) tile[j][tx] = in[r * cols + c];
  }
  __syncthreads();
  for (int j = ty; j < kTile; j += 8) {
    const uint64_t c = c0 + j, r = r0 + tx;      // out is [cols, rows]
    if (c < cols && r < rows) out[c * rows + r] = tile[tx][j];
  }
}

dim3 rows_grid(uint64_t oh, uint64_t ow) { return dim3((unsigned)((ow + kThreads - 1) / kThreads), (unsigned)(oh < 65535 ? oh : 65535)); }

}  // namespace
}  // namespace polar_b200

using namespace polar_b200;

extern "C" {

int polar_b200_fsoftmax(const float* in, float* out, uint64_t n, void* workspace, uint64_t workspace_bytes,
                        void* stream) {
  clear_error();
  if (n == 0) return POLAR_B200_OK;
  if (!in || !out) return fail(POLAR_B200_ERR_INVALID, "null device pointer");
  if (workspace && (workspace_bytes < sizeof(double) || (reinterpret_cast<uintptr_t>(workspace) & 7)))
    return fail(POLAR_B200_ERR_WORKSPACE, "fsoftmax needs 8 bytes of 8-byte aligned workspace");
  LaunchDeviceScope on(stream, out);
  cudaStream_t st = as_stream(stream);
  // one partial sum per CTA: as many CTAs as the workspace has room for, or about one per SM
  const int vec = aligned16(in) && aligned16(out);
  uint64_t blocks = (n + 4 * kThreads - 1) / (4 * kThreads);
  if (blocks > (uint64_t)sm_count()) blocks = (uint64_t)sm_count();
  if (workspace && workspace_bytes / sizeof(double) < blocks) blocks = workspace_bytes / sizeof(double);
  if (n <= kClusterElements) {
    const dim3 grid(1, kClusterCtas);
    return vec ? launch_clusters("fsoftmax", softmax_cluster_kernel<true>, grid, kClusterThreads, 0, st, kClusterCtas, in, out, (uint32_t)n)
               : launch_clusters("fsoftmax", softmax_cluster_kernel<false>, grid, kClusterThreads, 0, st, kClusterCtas, in, out, (uint32_t)n);
  }
  double* partials = static_cast<double*>(workspace);
  const bool own = !partials;
  if (own) {
    cudaError_t e = scratch_alloc(reinterpret_cast<void**>(&partials), blocks * sizeof(double), st);
    if (e != cudaSuccess) return fail(POLAR_B200_ERR_CUDA, "scratch (softmax sums)", e);
  }
  int rc = launch("fsoftmax_sum", exp_sum_kernel, (unsigned)blocks, kThreads, 0, st, in, partials, n, vec);
  const uint64_t wide = (n + 4 * kThreads - 1) / (4 * kThreads), cap = (uint64_t)sm_count() * 8;
  if (rc == POLAR_B200_OK)
    rc = launch("fsoftmax", softmax_div_kernel, (unsigned)(wide < cap ? wide : cap), kThreads, 0, st, in, partials, (uint32_t)blocks, out,
                n, vec);
  if (own) scratch_free(partials, st);
  return rc;
}

int polar_b200_fpool(const float* in, uint64_t h, uint64_t w, uint64_t windowH, uint64_t windowW, uint64_t strideH,
                     uint64_t strideW, float* out, void* stream) {
  clear_error();
  if (windowH == 0 || windowW == 0 || strideH == 0 || strideW == 0 || windowH > h || windowW > w)
    return fail(POLAR_B200_ERR_INVALID, "fpool: window and stride must be positive and fit the input");
  const uint64_t oh = (h - windowH) / strideH + 1, ow = (w - windowW) / strideW + 1;
  if (!in || !out) return fail(POLAR_B200_ERR_INVALID, "null device pointer");
  LaunchDeviceScope on(stream, out);
  if (windowH > 0xffffffffull || windowW > 0xffffffffull) return fail(POLAR_B200_ERR_INVALID, "fpool: window too large");
  auto go = [&](auto kernel) {
    return launch("fpool", kernel, rows_grid(oh, ow), kThreads, 0, as_stream(stream), in, w, (uint32_t)windowH, (uint32_t)windowW, strideH,
                  strideW, out, oh, ow);
  };
  if (windowH == 2 && windowW == 2) return go(pool_kernel<2>);
  if (windowH == 3 && windowW == 3) return go(pool_kernel<3>);
  return go(pool_kernel<0>);
}

int polar_b200_fconv2d(const float* in, uint64_t h, uint64_t w, const float* kernel, uint64_t kh, uint64_t kw,
                       float* out, void* stream) {
  clear_error();
  if (kh == 0 || kw == 0 || kh > h || kw > w) return fail(POLAR_B200_ERR_INVALID, "fconv2d: kernel must fit the input");
  // The reference walks offsets -k/2 .. k/2, which is the kernel only when k is odd.
  if ((kh & 1) == 0 || (kw & 1) == 0) return fail(POLAR_B200_ERR_UNSUPPORTED, "fconv2d: kernel extents must be odd");
  if (!in || !kernel || !out) return fail(POLAR_B200_ERR_INVALID, "null device pointer");
  const uint64_t oh = h - kh + 1, ow = w - kw + 1;
  LaunchDeviceScope on(stream, out);
  cudaStream_t st = as_stream(stream);
  const dim3 tiles((unsigned)((ow + kConvX - 1) / kConvX), (unsigned)((oh + kConvY - 1) / kConvY));
  if (kh == kw && (kh == 3 || kh == 5 || kh == 7) && (oh + kConvY - 1) / kConvY <= 65535) {
    const int vec = (ow & 3) == 0 && aligned16(out);
    auto go = [&](auto k) { return launch("fconv2d", k, tiles, kThreads, 0, st, in, h, w, kernel, out, oh, ow, vec); };
    return kh == 3 ? go(conv2d_tile_kernel<3>) : kh == 5 ? go(conv2d_tile_kernel<5>) : go(conv2d_tile_kernel<7>);
  }
  if (kh > 0xffffffffull || kw > 0xffffffffull) return fail(POLAR_B200_ERR_INVALID, "fconv2d: kernel too large");
  return launch("fconv2d", conv2d_kernel, rows_grid(oh, ow), kThreads, 0, st, in, w, kernel, (uint32_t)kh, (uint32_t)kw, out, oh, ow);
}

int polar_b200_ftranspose(const float* in, uint64_t rows, uint64_t cols, float* out, void* stream) {
  clear_error();
  if (rows == 0 || cols == 0) return POLAR_B200_OK;
  if (!in || !out) return fail(POLAR_B200_ERR_INVALID, "null device pointer");
  if (in == out) return fail(POLAR_B200_ERR_INVALID, "ftranspose cannot run in place");
  const uint64_t tiles_r = (rows + kTile - 1) / kTile, tiles_c = (cols + kTile - 1) / kTile;
  if (tiles_r * tiles_c > 0x7fffffffull) return fail(POLAR_B200_ERR_INVALID, "matrix too large");
  LaunchDeviceScope on(stream, out);
  return launch("ftranspose", transpose_kernel, (unsigned)(tiles_r * tiles_c), kTile * 8, 0, as_stream(stream), in, out, rows, cols,
                (uint32_t)tiles_c);
}

int polar_b200_fslice(const float* in, uint64_t first_dim, uint64_t inner, uint64_t index, float* out, void* stream) {
  clear_error();
  if (index >= first_dim) return fail(POLAR_B200_ERR_INVALID, "fslice: index outside the first dimension");
  if (inner && !in) return fail(POLAR_B200_ERR_INVALID, "null device pointer");
  return polar_b200_fcopy(in + index * inner, out, inner, stream);   // a bit-exact copy of one sub-tensor
}

}  // extern "C"
