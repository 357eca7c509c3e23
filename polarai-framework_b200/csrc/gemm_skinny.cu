// fmatmul for shapes with one tiny dimension - the MLP's 10-wide output layer and
// the logistic regression's single column.  A 128 x 256 tensor-core tile would be
// more than 90 % padding there, and the work is bound by streaming the one large
// operand (or the large result) through HBM once, so these run on the CUDA cores
// with 128-bit coalesced accesses of the large matrix and the small one in shared
// memory or registers.
//
//   small_n, left K-contiguous  (left stored [m,k]):   C[m, n<=16] = L . R
//       one warp per group of 4 rows; lanes walk k four floats at a time; R sits
//       transposed in shared memory - all of it, loaded once per persistent CTA,
//       when it fits, else one k-slab at a time; warp-shuffle reduction.
//   small_n, left M-contiguous  (left stored [k,m]):   C[m, n<=16] = L^T . R
//       the sum runs over the long (batch) dimension: the k range is split over
//       CTAs, each thread owns 4 consecutive m and n accumulators each, partial
//       sums go to scratch memory [split][m][n] and a second kernel adds the
//       splits in a fixed order (deterministic; no atomics).
//   small_k (k <= 16):                                  C[m,n] = L . R, result-bound
//       each thread keeps its 4 columns of R in registers and streams rows.
//
// Accumulation is fp32 with fmaf; the order of the k sum differs from the
// reference's sequential order, within the fp32 tolerance used for fmatmul.
#include <mutex>

#include "common.cuh"

namespace polar_b200 {
namespace skinny {

constexpr int kThreads = 256;

// ---------------------------------------------------------------- small n, K-major left

constexpr int KT = 1024;          // k-slab staged in shared memory
static_assert(KT % 256 == 0, "two warps of four floats per lane walk a slab");
constexpr int KT_PAD = KT + 4;    // keeps float4 alignment, staggers banks between columns
constexpr int ROWS_PER_WARP = 4;

// After the xor-shuffle reduction every lane holds all ROWS_PER_WARP x NP sums.  The warp's
// rows are contiguous in `out` (n values each), so lane l stores flat elements l, l + 32, ...:
// coalesced stores, and a fused sigmoid costs each lane one or two evaluations, not forty.
template <int NP>
__device__ __forceinline__ void store_row_sums(const float (&acc)[ROWS_PER_WARP][NP], float* out,
                                               uint64_t row0, uint64_t m, uint64_t n, int lane, int act) {
  if (row0 >= m) return;
  const uint32_t rows = (uint32_t)((m - row0 < ROWS_PER_WARP) ? (m - row0) : ROWS_PER_WARP);
  const uint32_t total = rows * (uint32_t)n;
  for (uint32_t f = lane; f < total; f += 32) {
    float v = 0.f;
#pragma unroll
    for (int r = 0; r < ROWS_PER_WARP; ++r)
#pragma unroll
      for (int j = 0; j < NP; ++j)
        if ((uint32_t)j < (uint32_t)n && (uint32_t)r * (uint32_t)n + (uint32_t)j == f) v = acc[r][j];
    out[row0 * n + f] = act ? sigmoid_clamped(v) : v;
  }
}

// Puts kt x n elements of the small operand into shared memory as [n][pitch], k contiguous.  Read in the order they are
// stored in - whole lines - and eight at a time: one element per trip was one memory latency per trip, 15 us for the
// 4096 x 10 of the MLP's output layer.
template <int THREADS>
__device__ __forceinline__ void stage_small_operand(const float* right, float* bs, int kt, int n, int pitch,
                                                    uint64_t rsk, uint64_t rsj) {
  constexpr int kBatch = 8;
  const bool by_k = rsk == 1;
  const uint32_t inner = by_k ? kt : n, total = (uint32_t)kt * (uint32_t)n;
  const uint32_t step_out = THREADS / inner, step_in = THREADS % inner;
  uint32_t o = threadIdx.x / inner, i = threadIdx.x % inner;   // one division: later elements are THREADS further on
  for (uint32_t e = threadIdx.x; e < total; e += kBatch * THREADS) {
    float v[kBatch];
    uint32_t at[kBatch];
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const uint32_t j = by_k ? o : i, kk = by_k ? i : o;
      at[u] = j * pitch + kk;
      v[u] = e + u * THREADS < total ? right[(uint64_t)kk * rsk + (uint64_t)j * rsj] : 0.f;
      i += step_in;
      o += step_out;
      if (i >= inner) i -= inner, ++o;
    }
#pragma unroll
    for (int u = 0; u < kBatch; ++u)
      if (e + u * THREADS < total) bs[at[u]] = v[u];
  }
}

// Few rows (below kResidentRows), or rows TMA-like loads cannot take as vectors: a CTA computes 4 * RW rows, two warps per
// row group, over one share of k; the CTAs of a cluster hold the shares of the same rows and add them through
// distributed shared memory in rank order.  Bound by latency: what counts is that every SM has a CTA, so the host cuts k
// into up to 8 shares and takes one row per warp until there are enough of them.  (The form with 32 rows
// per CTA had one CTA for 16 rows: 16 x 10 x 4096 61 us, here 4.)
constexpr uint64_t kResidentRows = 4096;
template <int NP, int RW, bool VEC>
__global__ void __launch_bounds__(kThreads)
small_n_rows_kernel(const float* left, const float* right, float* out, uint64_t m,
                    uint64_t n, uint64_t k, uint64_t rsk, uint64_t rsj, int act, uint32_t shares) {
  extern __shared__ float bs[];            // [NP][KT_PAD], k contiguous
  __shared__ float part[2][4 * RW][NP];    // the two k halves of this CTA
  __shared__ float mine[4 * RW][NP];       // its share of the sums
  pdl_enter();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int group = warp & 3, half = warp >> 2;
  const uint64_t row0 = (uint64_t)blockIdx.x * (4 * RW) + (uint64_t)group * RW;
  // shares are whole vectors of 4
  const uint64_t per = ((k + shares - 1) / shares + 3) & ~3ull;
  const uint64_t kbeg = (uint64_t)blockIdx.y * per, kend = kbeg + per < k ? kbeg + per : k;
  float acc[RW][NP];
#pragma unroll
  for (int r = 0; r < RW; ++r)
#pragma unroll
    for (int j = 0; j < NP; ++j) acc[r][j] = 0.f;
  float4 ahead[RW];                        // the next vectors of the thread's rows, asked for before they are needed
  auto fetch = [&](uint64_t kk) {
#pragma unroll
    for (int r = 0; r < RW; ++r)
      ahead[r] = (row0 + r < m && kk < kend) ? *reinterpret_cast<const float4*>(left + (row0 + r) * k + kk)
                                             : make_float4(0.f, 0.f, 0.f, 0.f);
  };
  if (VEC) fetch(kbeg + (half * 32 + lane) * 4);
  for (uint64_t k0 = kbeg; k0 < kend; k0 += KT) {
    const int kt = (int)((kend - k0 < KT) ? (kend - k0) : KT);
    __syncthreads();
    stage_small_operand<kThreads>(right + k0 * rsk, bs, kt, (int)n, KT_PAD, rsk, rsj);
    __syncthreads();
    if (VEC) {
      for (int kk = (half * 32 + lane) * 4; kk < kt; kk += 256) {
        float4 a[RW];
#pragma unroll
        for (int r = 0; r < RW; ++r) a[r] = ahead[r];
        // (KT is a multiple of 256: the first vectors of the next slab follow the last of this one)
        fetch(k0 + kk + 256);
#pragma unroll
        for (int j = 0; j < NP; ++j) {
          if (j >= (int)n) continue;
          const float4 b = *reinterpret_cast<const float4*>(&bs[j * KT_PAD + kk]);
#pragma unroll
          for (int r = 0; r < RW; ++r) {
            acc[r][j] = fmaf(a[r].x, b.x, acc[r][j]);
            acc[r][j] = fmaf(a[r].y, b.y, acc[r][j]);
            acc[r][j] = fmaf(a[r].z, b.z, acc[r][j]);
            acc[r][j] = fmaf(a[r].w, b.w, acc[r][j]);
          }
        }
      }
    } else {
#pragma unroll 4
      for (int kk = half * 32 + lane; kk < kt; kk += 64) {
        float a[RW];
#pragma unroll
        for (int r = 0; r < RW; ++r) a[r] = row0 + r < m ? left[(row0 + r) * k + k0 + kk] : 0.f;
#pragma unroll
        for (int j = 0; j < NP; ++j) {
          if (j >= (int)n) continue;
          const float b = bs[j * KT_PAD + kk];
#pragma unroll
          for (int r = 0; r < RW; ++r) acc[r][j] = fmaf(a[r], b, acc[r][j]);
        }
      }
    }
  }
#pragma unroll
  for (int r = 0; r < RW; ++r)
#pragma unroll
    for (int j = 0; j < NP; ++j) {
      float v = acc[r][j];
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
      if (lane == 0) part[half][group * RW + r][j] = v;
    }
  __syncthreads();
  const int e = threadIdx.x, r = e / NP, j = e % NP;       // 4 * RW * NP <= 256 sums, one per thread
  const bool live = r < 4 * RW;
  float v = live ? part[0][r][j] + part[1][r][j] : 0.f;
  if (shares > 1) {
    if (live) mine[r][j] = v;
    cluster_arrive();
    cluster_wait();
    if (live && cluster_rank() == 0) {
      float other[8];
#pragma unroll
      for (uint32_t c = 1; c < 8; ++c)
        if (c < shares) other[c] = ld_cluster(&mine[r][j], c);
#pragma unroll
      for (uint32_t c = 1; c < 8; ++c)
        if (c < shares) v += other[c];
    }
    cluster_arrive();                      // nobody leaves while the first CTA may still read its sums
    cluster_wait();
    if (cluster_rank() != 0) return;
  }
  const uint64_t row = (uint64_t)blockIdx.x * (4 * RW) + (uint64_t)r;
  if (live && row < m && j < (int)n) out[row * n + j] = act ? sigmoid_clamped(v) : v;
}

// ---------------------------------------------------------------- small n, K-major left, R resident

// When the whole small operand fits in shared memory (n_padded * (k + 4) floats, e.g.
// 164 KB for the MLP's 4096 x 10 output layer) it is loaded ONCE per CTA; one
// persistent 512-thread CTA per SM then streams row groups of the large operand
// with no barrier in the loop.  Each warp owns 4 rows at a time and keeps two
// k chunks (8 x 128-bit loads per lane) in flight.
constexpr int kResidentThreads = 512;

template <int NP>
__global__ void __launch_bounds__(kResidentThreads, 1)
small_n_kmajor_resident_kernel(const float* left, const float* right,
                               float* out, uint64_t m, uint64_t n, uint64_t k, uint64_t rsk,
                               uint64_t rsj, int act) {
  pdl_enter();
  extern __shared__ float bs[];   // [NP][k + 4], k contiguous
  const uint32_t kpad = (uint32_t)k + 4;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint64_t warps_total = (uint64_t)gridDim.x * (kResidentThreads / 32);
  const uint64_t groups = (m + ROWS_PER_WARP - 1) / ROWS_PER_WARP;
  uint64_t g = (uint64_t)blockIdx.x * (kResidentThreads / 32) + warp;
  // The loads of a chunk (two 128-bit loads per row and lane) are issued one chunk ahead of its
  // arithmetic, and the very first ones before the small operand is staged: with one group of
  // rows per warp (8192 rows on 148 SMs) the kernel is otherwise a chain of memory latencies.
  float4 a0[ROWS_PER_WARP], a1[ROWS_PER_WARP];
  auto load_chunk = [&](uint64_t group, uint32_t kk) {
#pragma unroll
    for (int r = 0; r < ROWS_PER_WARP; ++r) {
      const uint64_t row = group * ROWS_PER_WARP + r;
      const float* src = left + (row < m ? row : m - 1) * k;   // clamped: results of padding rows are dropped
      a0[r] = ld_stream(reinterpret_cast<const float4*>(src + kk));
      a1[r] = (kk + 128 < (uint32_t)k) ? ld_stream(reinterpret_cast<const float4*>(src + kk + 128))
                                       : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  if (g < groups && (uint32_t)lane * 4 < (uint32_t)k) load_chunk(g, lane * 4);
  if (n < NP)
    for (uint32_t e = threadIdx.x; e < (NP - (uint32_t)n) * (uint32_t)k; e += kResidentThreads)
      bs[((uint32_t)n + e / (uint32_t)k) * kpad + e % (uint32_t)k] = 0.f;
  stage_small_operand<kResidentThreads>(right, bs, (int)k, (int)n, (int)kpad, rsk, rsj);
  __syncthreads();
  for (; g < groups; g += warps_total) {
    const uint64_t row0 = g * ROWS_PER_WARP;
    float acc[ROWS_PER_WARP][NP];
#pragma unroll
    for (int r = 0; r < ROWS_PER_WARP; ++r)
#pragma unroll
      for (int j = 0; j < NP; ++j) acc[r][j] = 0.f;
    for (uint32_t kk = lane * 4; kk < (uint32_t)k; kk += 256) {
      float4 c0[ROWS_PER_WARP], c1[ROWS_PER_WARP];
#pragma unroll
      for (int r = 0; r < ROWS_PER_WARP; ++r) { c0[r] = a0[r]; c1[r] = a1[r]; }
      const bool second = kk + 128 < (uint32_t)k;
      // the next chunk of this group, or the first chunk of this warp's next group
      if (kk + 256 < (uint32_t)k) load_chunk(g, kk + 256);
      else if (g + warps_total < groups) load_chunk(g + warps_total, lane * 4);
#pragma unroll
      for (int j = 0; j < NP; ++j) {
        const float4 b0 = *reinterpret_cast<const float4*>(&bs[j * kpad + kk]);
#pragma unroll
        for (int r = 0; r < ROWS_PER_WARP; ++r) {
          acc[r][j] = fmaf(c0[r].x, b0.x, acc[r][j]);
          acc[r][j] = fmaf(c0[r].y, b0.y, acc[r][j]);
          acc[r][j] = fmaf(c0[r].z, b0.z, acc[r][j]);
          acc[r][j] = fmaf(c0[r].w, b0.w, acc[r][j]);
        }
      }
      if (second) {
#pragma unroll
        for (int j = 0; j < NP; ++j) {
          const float4 b1 = *reinterpret_cast<const float4*>(&bs[j * kpad + kk + 128]);
#pragma unroll
          for (int r = 0; r < ROWS_PER_WARP; ++r) {
            acc[r][j] = fmaf(c1[r].x, b1.x, acc[r][j]);
            acc[r][j] = fmaf(c1[r].y, b1.y, acc[r][j]);
            acc[r][j] = fmaf(c1[r].z, b1.z, acc[r][j]);
            acc[r][j] = fmaf(c1[r].w, b1.w, acc[r][j]);
          }
        }
      }
    }
#pragma unroll
    for (int r = 0; r < ROWS_PER_WARP; ++r)
#pragma unroll
      for (int j = 0; j < NP; ++j) {
        float v = acc[r][j];
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
        acc[r][j] = v;
      }
    store_row_sums<NP>(acc, out, row0, m, n, lane, act);
  }
}

// ---------------------------------------------------------------- small n, MN-major left (split k)

constexpr int KS = 128;   // rows of R staged per pass
// Sums of at most this many terms are cut over the CTAs of one cluster, longer ones over more CTAs and a second launch.  In a cluster
// against in two launches, us: 784 x 10 x 384 8.8 and 9.5, x 512 10.1 and 10.2, x 768 12.8 and 12.3; 4096 x 10 x 384 9.4 and 19.9,
// x 1024 16.1 and 16.5; 64 x 10 x 256 5.5 and 5.1, x 512 7.3 and 5.3.
constexpr uint64_t kClusterRows = 384;

// Two fused multiply-adds in one instruction (sm_100: fma.rn.f32x2 on register pairs), each
// an IEEE fma like fmaf: (c.lo, c.hi) = (a.lo, a.hi) * (b.lo, b.hi) + (c.lo, c.hi).
__device__ __forceinline__ void ffma2(unsigned long long& c, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}

// The kernel issues one instruction per two multiply-adds and reads each value of the staged
// operand as a ready-made (b, b) pair: at 16 columns the plain form needs every issue slot of
// the SM to keep up with HBM (64 FMA + 16 shared-memory loads per 16 bytes streamed).
// VEC: the thread's four rows are neighbours, one 128-bit load per k; otherwise (rows of `left` that start anywhere) they
// are kThreads apart, four coalesced 32-bit loads.
// `shares` > 1: the splits are the CTAs of a cluster, which add their sums through distributed shared memory (ascending
// split index, the order of reduce_splits_kernel: the same bits) and store the result; one launch and no scratch for
// products of few k, where a second launch costs as much as the first.
template <int NP, bool VEC>
__global__ void __launch_bounds__(kThreads, 2)
small_n_mnmajor_kernel(const float* left, const float* right,
                       float* partial, uint64_t m, uint64_t n, uint64_t k, uint64_t rsk,
                       uint64_t rsj, uint64_t k_per_split, uint32_t shares) {
  __shared__ __align__(16) float2 bs[KS][NP];   // every value twice: one 64-bit load yields the pair
  extern __shared__ float tile[];               // with shares: this CTA's sums, [1024 rows][n]
  pdl_enter();
  const uint64_t block = (uint64_t)blockIdx.x * kThreads * 4;
  const uint64_t m0 = VEC ? block + threadIdx.x * 4 : block + threadIdx.x;
  const uint64_t step = VEC ? 1 : kThreads;     // between the thread's rows
  const uint64_t kbeg = (uint64_t)blockIdx.y * k_per_split;
  const uint64_t kend = (kbeg + k_per_split < k) ? kbeg + k_per_split : k;
  unsigned long long acc01[NP], acc23[NP];      // rows (0,1) and (2,3) of the thread's four
#pragma unroll
  for (int j = 0; j < NP; ++j) acc01[j] = acc23[j] = 0ull;
  const bool live = m0 < m;   // VEC: m is a multiple of 4
  auto load = [&](uint64_t kk) {
    const float* src = left + kk * m + m0;
    if (VEC) return ld_stream(reinterpret_cast<const float4*>(src));
    return make_float4(ld_stream(src), m0 + kThreads < m ? ld_stream(src + kThreads) : 0.f,
                       m0 + 2 * kThreads < m ? ld_stream(src + 2 * kThreads) : 0.f,
                       m0 + 3 * kThreads < m ? ld_stream(src + 3 * kThreads) : 0.f);
  };
  auto multiply = [&](const float4& a, int kk) {
    const unsigned long long a01 = pack2(a.x, a.y), a23 = pack2(a.z, a.w);
#pragma unroll
    for (int j = 0; j + 1 < NP; j += 2) {
      // two pairs per 128-bit load
      const ulonglong2 bb = *reinterpret_cast<const ulonglong2*>(&bs[kk][j]);
      ffma2(acc01[j], a01, bb.x);
      ffma2(acc23[j], a23, bb.x);
      ffma2(acc01[j + 1], a01, bb.y);
      ffma2(acc23[j + 1], a23, bb.y);
    }
    if (NP & 1) {
      const unsigned long long bb = *reinterpret_cast<const unsigned long long*>(&bs[kk][NP - 1]);
      ffma2(acc01[NP - 1], a01, bb);
      ffma2(acc23[NP - 1], a23, bb);
    }
  };
  for (uint64_t k0 = kbeg; k0 < kend; k0 += KS) {
    const int ks = (int)((kend - k0 < KS) ? (kend - k0) : KS);
    __syncthreads();
    for (int e = threadIdx.x; e < ks * NP; e += kThreads) {
      int j = e % NP, kk = e / NP;
      const float v = (uint64_t)j < n ? right[(k0 + kk) * rsk + (uint64_t)j * rsj] : 0.f;
      bs[kk][j] = make_float2(v, v);
    }
    __syncthreads();
    if (live) {
      int kk = 0;
      // eight 128-bit loads in flight per thread: two CTAs of 256 threads per SM then keep
      // 64 KB outstanding, what HBM latency x bandwidth asks of one SM; sixteen where the sums leave registers for it
      constexpr int kBatch = NP <= 4 ? 16 : 8;
      for (; kk + kBatch <= ks; kk += kBatch) {
        float4 a[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) a[u] = load(k0 + kk + u);
#pragma unroll
        for (int u = 0; u < kBatch; ++u) multiply(a[u], kk + u);
      }
      for (; kk < ks; ++kk) multiply(load(k0 + kk), kk);
    }
  }
  float v[4][NP];
#pragma unroll
  for (int j = 0; j < NP; ++j) {
    unpack2(acc01[j], v[0][j], v[1][j]);
    unpack2(acc23[j], v[2][j], v[3][j]);
  }
  if (shares > 1) {
    const uint32_t at = VEC ? threadIdx.x * 4 : threadIdx.x;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < NP; ++j)
        if ((uint64_t)j < n) tile[(at + i * (uint32_t)step) * (uint32_t)n + j] = v[i][j];
    cluster_arrive();
    cluster_wait();
    const uint64_t rows = m - block < 4 * kThreads ? m - block : 4 * kThreads;
    const uint32_t total = (uint32_t)(rows * n), rank = cluster_rank();
    const uint32_t per = (total + shares - 1) / shares, end = (rank + 1) * per < total ? (rank + 1) * per : total;
    for (uint32_t e = rank * per + threadIdx.x; e < end; e += kThreads) {
      float part[8], s = 0.f;
#pragma unroll
      for (uint32_t c = 0; c < 8; ++c)
        if (c < shares) part[c] = ld_cluster(&tile[e], c);
#pragma unroll
      for (uint32_t c = 0; c < 8; ++c)
        if (c < shares) s += part[c];
      partial[block * n + e] = s;          // the result itself
    }
    cluster_arrive();                      // nobody leaves while another CTA may still read its sums
    cluster_wait();
    return;
  }
  float* dst = partial + (uint64_t)blockIdx.y * m * n;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint64_t row = m0 + i * step;
    if (row >= m) continue;
#pragma unroll
    for (int j = 0; j < NP; ++j)
      if ((uint64_t)j < n) dst[row * n + j] = v[i][j];
  }
}

// Sum of one element over the splits, ascending split index (a fixed order); the loads of
// up to 32 splits are issued together, the additions stay in order.
__device__ __forceinline__ float sum_splits(const float* partial, uint64_t elems, uint64_t e,
                                            uint32_t splits) {
  float s = 0.f;
  uint32_t sp = 0;
  for (; sp + 32 <= splits; sp += 32) {
    float v[32];
#pragma unroll
    for (int u = 0; u < 32; ++u) v[u] = ld_l2(partial + (uint64_t)(sp + u) * elems + e);
#pragma unroll
    for (int u = 0; u < 32; ++u) s += v[u];
  }
  for (; sp + 8 <= splits; sp += 8) {
    float v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = ld_l2(partial + (uint64_t)(sp + u) * elems + e);
#pragma unroll
    for (int u = 0; u < 8; ++u) s += v[u];
  }
  for (; sp < splits; ++sp) s += ld_l2(partial + (uint64_t)sp * elems + e);
  return s;
}

// out[e] = sum over splits, ascending split index: a fixed order.
__global__ void __launch_bounds__(kThreads)
reduce_splits_kernel(const float* partial, float* out, uint64_t elems,
                     uint32_t splits) {
  pdl_enter();
  const uint64_t stride = (uint64_t)gridDim.x * kThreads;
  for (uint64_t e = (uint64_t)blockIdx.x * kThreads + threadIdx.x; e < elems; e += stride)
    out[e] = sum_splits(partial, elems, e, splits);
}

// The same sum, stored transposed: partial is [split][m][n], out is [n][m].  Used for the
// last few rows of a product whose left operand is stored [k, rows]: they are computed as
// the small-n product of the transposed problem and land as rows of the result.
__global__ void __launch_bounds__(kThreads)
reduce_splits_transposed_kernel(const float* partial, float* out, uint64_t m,
                                uint64_t n, uint32_t splits) {
  pdl_enter();
  const uint64_t elems = m * n, stride = (uint64_t)gridDim.x * kThreads;
  for (uint64_t e = (uint64_t)blockIdx.x * kThreads + threadIdx.x; e < elems; e += stride) {
    out[(e % n) * m + e / n] = sum_splits(partial, elems, e, splits);
  }
}

// ---------------------------------------------------------------- small k

constexpr int RK = 64;   // rows of the left operand staged per CTA

// L'(i,kk) = left[i*lsi + kk*lsk]; R'(kk,j) = right[kk*rsk + j*rsj]; k <= KP.
template <int KP>
__global__ void __launch_bounds__(kThreads)
small_k_kernel(const float* left, const float* right, float* out,
               uint64_t m, uint64_t n, uint64_t k, uint64_t lsi, uint64_t lsk, uint64_t rsk,
               uint64_t rsj, int vec_store, const float* sig) {
  __shared__ float as[RK][KP];
  pdl_enter();
  // Four columns per thread: one vector, or - rows that are no vectors - a column out of each quarter of the warp's 128, so
  // that a warp's scalar stores are consecutive (the MLP step 2000 x 77 x 1001 x 10, with one such product, 79 -> 68 us)
  const bool vec = vec_store;                // (n is a multiple of four then)
  const uint64_t j0 = (uint64_t)blockIdx.x * kThreads * 4 + (vec ? threadIdx.x * 4u : (threadIdx.x >> 5) * 128u + (threadIdx.x & 31));
  const uint32_t step = vec ? 1 : 32;
  // Each thread's four columns of the small operand stay in registers while the CTA walks
  // over row blocks (gridDim.y CTAs share the rows of one column block).
  float b[4][KP];
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int kk = 0; kk < KP; ++kk)
      b[c][kk] = (j0 + c * step < n && (uint64_t)kk < k) ? right[(uint64_t)kk * rsk + (j0 + c * step) * rsj] : 0.f;
  // The gridDim.y CTAs of a column block split the rows evenly (contiguous ranges, a multiple
  // of four rows each) and stage them RK at a time.
  const uint64_t rows_per_cta = ((m + gridDim.y - 1) / gridDim.y + 3) & ~3ull;
  const uint64_t row_begin = (uint64_t)blockIdx.y * rows_per_cta;
  const uint64_t row_end = row_begin + rows_per_cta < m ? row_begin + rows_per_cta : m;
  for (uint64_t row0 = row_begin; row0 < row_end; row0 += RK) {
    const int rows = (int)((row_end - row0 < RK) ? (row_end - row0) : RK);
    __syncthreads();   // the previous block's rows are no longer read
    for (int e = threadIdx.x; e < RK * KP; e += kThreads) {
      int kk = e % KP, r = e / KP;
      float v = 0.f;
      if (r < rows && (uint64_t)kk < k) v = left[(row0 + r) * lsi + (uint64_t)kk * lsk];
      as[r][kk] = v;
    }
    __syncthreads();
    if (j0 >= n) continue;
    // Rows in groups of four: the four loads of the sigmoid values are issued before any of
    // the arithmetic, so each thread keeps four 128-bit loads in flight.
    for (int rb = 0; rb < rows; rb += 4) {
      float4 sv[4];
      if (sig) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          if (rb + u >= rows) continue;
          const float* sp = sig + (row0 + rb + u) * n + j0;
          if (vec) {
            sv[u] = ld_stream(reinterpret_cast<const float4*>(sp));
          } else {
            sv[u].x = sp[0];
            sv[u].y = (j0 + 32 < n) ? sp[32] : 0.f;
            sv[u].z = (j0 + 64 < n) ? sp[64] : 0.f;
            sv[u].w = (j0 + 96 < n) ? sp[96] : 0.f;
          }
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int r = rb + u;
        if (r >= rows) continue;
        float c0 = 0.f, c1 = 0.f, c2 = 0.f, c3 = 0.f;
#pragma unroll
        for (int kk = 0; kk < KP; ++kk) {
          float a = as[r][kk];
          c0 = fmaf(a, b[0][kk], c0);
          c1 = fmaf(a, b[1][kk], c1);
          c2 = fmaf(a, b[2][kk], c2);
          c3 = fmaf(a, b[3][kk], c3);
        }
        if (sig) {
          // fused Sigmoid derivative: out = product * ((1 - s) * s), s = fsigmoid output
          c0 = sigmoid_grad_chain(c0, sv[u].x); c1 = sigmoid_grad_chain(c1, sv[u].y);
          c2 = sigmoid_grad_chain(c2, sv[u].z); c3 = sigmoid_grad_chain(c3, sv[u].w);
        }
        float* dst = out + (row0 + r) * n + j0;
        if (vec) {
          st_stream(reinterpret_cast<float4*>(dst), make_float4(c0, c1, c2, c3));
        } else {
          dst[0] = c0;
          if (j0 + 32 < n) dst[32] = c1;
          if (j0 + 64 < n) dst[64] = c2;
          if (j0 + 96 < n) dst[96] = c3;
        }
      }
    }
  }   // row ranges
}

// ---------------------------------------------------------------- dense layer backward, one pass
//
// The two products of a dense layer's backward pass that read the layer's INPUT activations
//   dW[kh, n]  = H^T . dZ                      (small n, left M-contiguous: the kernel above)
//   dIn[B, kh] = (dZ . W^T) * ((1 - H) * H)    (small k with the Sigmoid derivative fused)
// share everything: both stream H [B, kh] row by row, both want the dZ rows staged in shared
// memory, and in both a thread owns four consecutive hidden columns.  Done separately H
// crosses HBM twice; here once.  Per row a thread loads its four H values (one 128-bit load),
// reads the dZ row from shared memory, accumulates dW for its columns and stores its four
// dIn values.  The arithmetic, its order and the division of the batch rows into splits are
// those of the two kernels above (same fma per term, rows ascending, splits added in
// ascending order), so both results carry the bits of the separate launches.
template <int NP>
__global__ void __launch_bounds__(kThreads, NP > 10 ? 1 : 2)
dense_grad_kernel(const float* H, const float* dz, const float* W,
                  float* din, float* partial, uint64_t rows, uint64_t kh, uint64_t n,
                  uint64_t rows_per_split) {
  pdl_enter();
  __shared__ __align__(16) float2 bs[KS][NP];   // dZ rows, every value twice: one 64-bit load yields the pair
  const uint64_t m0 = ((uint64_t)blockIdx.x * kThreads + threadIdx.x) * 4;
  const uint64_t rbeg = (uint64_t)blockIdx.y * rows_per_split;
  const uint64_t rend = (rbeg + rows_per_split < rows) ? rbeg + rows_per_split : rows;
  const bool live = m0 < kh;   // kh is a multiple of 4
  // W rows of the thread's four columns, packed as (column 0, column 1) and (column 2, column 3)
  unsigned long long w01[NP], w23[NP], acc01[NP], acc23[NP];
#pragma unroll
  for (int j = 0; j < NP; ++j) {
    float v[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) v[c] = (live && (uint64_t)j < n) ? W[(m0 + c) * n + j] : 0.f;
    w01[j] = pack2(v[0], v[1]);
    w23[j] = pack2(v[2], v[3]);
    acc01[j] = acc23[j] = 0ull;
  }
  for (uint64_t r0 = rbeg; r0 < rend; r0 += KS) {
    const int rs = (int)((rend - r0 < KS) ? (rend - r0) : KS);
    __syncthreads();
    for (int e = threadIdx.x; e < KS * NP; e += kThreads) {
      int j = e % NP, rr = e / NP;
      float v = 0.f;
      if (rr < rs && (uint64_t)j < n) v = dz[(r0 + rr) * n + j];
      bs[rr][j] = make_float2(v, v);
    }
    __syncthreads();
    if (!live) continue;
    // six to eight 128-bit loads in flight per thread (two CTAs of 256 threads per SM then keep
    // 48-64 KB outstanding, what HBM latency x bandwidth asks of one SM)
    constexpr int kBatch = NP == 10 ? 6 : 8;   // at ten columns 128 registers hold six rows without spilling
    for (int rr = 0; rr < rs; rr += kBatch) {
      float4 h[kBatch];
#pragma unroll
      for (int u = 0; u < kBatch; ++u)
        if (rr + u < rs) h[u] = ld_stream(reinterpret_cast<const float4*>(H + (r0 + rr + u) * kh + m0));
#pragma unroll
      for (int u = 0; u < kBatch; ++u) {
        if (rr + u >= rs) continue;
        const unsigned long long h01 = pack2(h[u].x, h[u].y), h23 = pack2(h[u].z, h[u].w);
        unsigned long long c01 = 0ull, c23 = 0ull;   // (dZ . W^T) for the four columns
        auto term = [&](unsigned long long dd, int j) {
          ffma2(c01, dd, w01[j]);
          ffma2(c23, dd, w23[j]);
          ffma2(acc01[j], h01, dd);
          ffma2(acc23[j], h23, dd);
        };
#pragma unroll
        for (int j = 0; j + 1 < NP; j += 2) {              // two pairs per 128-bit load
          const ulonglong2 dd = *reinterpret_cast<const ulonglong2*>(&bs[rr + u][j]);
          term(dd.x, j);
          term(dd.y, j + 1);
        }
        if (NP & 1) term(*reinterpret_cast<const unsigned long long*>(&bs[rr + u][NP - 1]), NP - 1);
        float c0, c1, c2, c3;
        unpack2(c01, c0, c1);
        unpack2(c23, c2, c3);
        const float4 o = make_float4(sigmoid_grad_chain(c0, h[u].x), sigmoid_grad_chain(c1, h[u].y),
                                     sigmoid_grad_chain(c2, h[u].z), sigmoid_grad_chain(c3, h[u].w));
        st_stream(reinterpret_cast<float4*>(din + (r0 + rr + u) * kh + m0), o);
      }
    }
  }
  if (live) {
    float* dst = partial + ((uint64_t)blockIdx.y * kh + m0) * n;
#pragma unroll
    for (int j = 0; j < NP; ++j) {
      float r0, r1, r2, r3;
      unpack2(acc01[j], r0, r1);
      unpack2(acc23[j], r2, r3);
      if ((uint64_t)j < n) {
        dst[j] = r0;
        dst[n + j] = r1;
        dst[2 * n + j] = r2;
        dst[3 * n + j] = r3;
      }
    }
  }
}

// ---------------------------------------------------------------- host side

inline int round_np(uint64_t n) { return n <= 1 ? 1 : n <= 2 ? 2 : n <= 4 ? 4 : n <= 8 ? 8 : n <= 10 ? 10 : 16; }

// Into how many parts the k range of a small-n product with M-contiguous left is cut: about two CTAs per SM, parts of at
// least KS rows - or of 32, as long as the partial sums stay below the 16 MiB that the entry point with built-in scratch
// has (fdense_grad with 4096 columns and 10 outputs: 64 parts of 128 rows left 40 SMs with one CTA at 8192 rows, 16 parts the
// chip half empty at 2048; the step of such a network 208 -> 202 us and 108 -> 102, at 4096 rows 149 -> 132) - or of 16, as
// long as parts of KS rows leave SMs without a CTA.  n = 0: parts of KS rows.
uint32_t splits_for(uint64_t m, uint64_t k, uint64_t n) {
  uint64_t m_blocks = (m + 4 * kThreads - 1) / (4 * kThreads);
  if (m_blocks < 1) m_blocks = 1;
  uint64_t want = ((uint64_t)sm_count() * 2 + m_blocks - 1) / m_blocks;   // about two CTAs per SM
  uint64_t max_by_k = (k + KS - 1) / KS;
  if (max_by_k * m_blocks < (uint64_t)sm_count()) {
    const uint64_t fine = (k + 15) / 16, enough = ((uint64_t)sm_count() + m_blocks - 1) / m_blocks;
    max_by_k = fine < enough ? fine : enough;
    // few enough rows for one cluster: its sums need no second launch
    if (k <= kClusterRows) max_by_k = max_by_k < 8 ? max_by_k : 8;
  }
  uint64_t s = want < max_by_k ? want : max_by_k;
  if (m && n && k > 8 * KS) {
    const uint64_t by_scratch = (16ull << 20) / sizeof(float) / n / m, fine = (k + 31) / 32;
    uint64_t finer = want < fine ? want : fine;
    if (finer > by_scratch) finer = by_scratch;
    if (finer > KS) finer = KS;              // (the error of a sum of sums grows with the longer of the two)
    if (finer > s) s = finer;
  }
  if (s < 1) s = 1;
  if (s > 4096) s = 4096;
  return (uint32_t)s;
}
// Whether the parts run as one cluster that adds them itself.
bool sum_in_cluster(uint64_t k, uint64_t n, uint32_t splits) { return splits > 1 && splits <= 8 && n <= 10 && k <= kClusterRows; }

template <int NP>
int launch_small_n_k(const float* l, const float* r, float* out, uint64_t m, uint64_t n, uint64_t k,
                     uint64_t rsk, uint64_t rsj, cudaStream_t st, int act) {
  // whole small operand resident in shared memory when it fits (and there are rows
  // enough to keep every SM busy); otherwise k slabs
  const size_t resident = (size_t)NP * (k + 4) * sizeof(float);
  if (resident <= 200 * 1024 && m >= kResidentRows && (k & 3) == 0 && aligned16(l)) {
    static bool res_attr[64] = {false};
    int d = 0;
    cudaGetDevice(&d);
    if (d >= 0 && d < 64 && !res_attr[d]) {
      cudaError_t e = cudaFuncSetAttribute(small_n_kmajor_resident_kernel<NP>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
      if (e != cudaSuccess) return fail(POLAR_B200_ERR_CUDA, "cudaFuncSetAttribute(small_n resident)", e);
      res_attr[d] = true;
    }
    return launch("fmatmul_small_n_resident", small_n_kmajor_resident_kernel<NP>, (unsigned)sm_count(), kResidentThreads,
                  resident, st, l, r, out, m, n, k, rsk, rsj, act);
  }
  // one row per warp until every SM has a CTA, then up to four; k in up to 8 shares of at least 128 while SMs are free
  const uint64_t sms = (uint64_t)sm_count();
  const int rw = m >= 16 * sms ? 4 : m >= 8 * sms ? 2 : 1;
  const uint64_t groups = (m + 4 * rw - 1) / (4 * rw);
  uint32_t shares = 1;
  while (shares < 8 && groups * shares * 2 <= 2 * sms && k / (shares * 2) >= 128) shares *= 2;
  if (groups > 0x7fffffffull) return fail(POLAR_B200_ERR_UNSUPPORTED, "too many rows");
  const size_t smem = (size_t)NP * KT_PAD * sizeof(float);
  const bool vec = (k & 3) == 0 && aligned16(l);
  auto go = [&](auto kernel) {
    cudaError_t e = smem > 48 * 1024 - 4096 ? cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) : cudaSuccess;
    if (e != cudaSuccess) return fail(POLAR_B200_ERR_CUDA, "cudaFuncSetAttribute(small_n)", e);
    return launch_clusters("fmatmul_small_n", kernel, dim3((unsigned)groups, shares), kThreads, smem, st, shares, l, r, out, m, n, k,
                           rsk, rsj, act, shares);
  };
  if (vec) return rw == 4 ? go(small_n_rows_kernel<NP, 4, true>) : rw == 2 ? go(small_n_rows_kernel<NP, 2, true>) : go(small_n_rows_kernel<NP, 1, true>);
  return rw == 4 ? go(small_n_rows_kernel<NP, 4, false>) : rw == 2 ? go(small_n_rows_kernel<NP, 2, false>) : go(small_n_rows_kernel<NP, 1, false>);
}

int launch_reduce(const float* ws, float* out, uint64_t elems, uint32_t splits, cudaStream_t st) {
  const uint64_t g = (elems + kThreads - 1) / kThreads, cap = (uint64_t)sm_count() * 4;
  return launch("fmatmul_reduce_splits", reduce_splits_kernel, (unsigned)(g < cap ? g : cap), kThreads, 0, st, ws, out, elems, splits);
}

template <int NP>
int launch_small_n_mn(const float* l, const float* r, float* out, float* ws, uint32_t splits, uint64_t m,
                      uint64_t n, uint64_t k, uint64_t rsk, uint64_t rsj, cudaStream_t st) {
  uint64_t m_blocks = (m + 4 * kThreads - 1) / (4 * kThreads);
  uint64_t k_per_split = (k + splits - 1) / splits;
  k_per_split = (k_per_split + 3) & ~3ull;
  if (m_blocks < 1) m_blocks = 1;
  dim3 grid((unsigned)m_blocks, splits);
  const bool in_cluster = sum_in_cluster(k, n, splits), vec = (m & 3) == 0 && aligned16(l);
  float* dst = splits > 1 && !in_cluster ? ws : out;
  const size_t smem = in_cluster ? (size_t)4 * kThreads * n * sizeof(float) : 0;
  auto go = [&](auto kernel) {
    cudaError_t e = smem + KS * NP * sizeof(float2) > 48 * 1024 ? cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) : cudaSuccess;
    if (e != cudaSuccess) return fail(POLAR_B200_ERR_CUDA, "cudaFuncSetAttribute(small_n split)", e);
    return launch_clusters("fmatmul_small_n_split", kernel, grid, kThreads, smem, st, in_cluster ? splits : 1, l, r, dst, m, n, k, rsk,
                           rsj, k_per_split, in_cluster ? splits : 1);
  };
  int rc = vec ? go(small_n_mnmajor_kernel<NP, true>) : go(small_n_mnmajor_kernel<NP, false>);
  if (rc || splits == 1 || in_cluster) return rc;
  return launch_reduce(ws, out, m * n, splits, st);
}

template <int NP>
int launch_dense_grad_np(const float* H, const float* dz, const float* W, float* din, float* dw, float* ws,
                         uint32_t splits, uint64_t rows, uint64_t kh, uint64_t n, cudaStream_t st) {
  // the same division of the rows as launch_small_n_mn makes for dW = H^T . dZ
  uint64_t m_blocks = (kh / 4 + kThreads - 1) / kThreads;
  uint64_t rows_per_split = (rows + splits - 1) / splits;
  rows_per_split = (rows_per_split + 3) & ~3ull;
  dim3 grid((unsigned)m_blocks, splits);
  float* dst = splits > 1 ? ws : dw;
  int rc = launch("fdense_grad", dense_grad_kernel<NP>, grid, kThreads, 0, st, H, dz, W, din, dst, rows, kh, n, rows_per_split);
  if (rc || splits == 1) return rc;
  return launch_reduce(ws, dw, kh * n, splits, st);
}

}  // namespace skinny

// out_tail[j, i] = sum_kk left_tail[kk*left_pitch + j] * right[kk*n + i]   (j < rem <= 16, i < n):
// `rem` rows of a t_f product, as the small-n product right^T . left_tail stored transposed.
// Scratch: ragged_rows_workspace_bytes.  n a multiple of 4, right 16-byte aligned.
uint64_t ragged_rows_workspace_bytes(uint64_t rem, uint64_t n, uint64_t k) {
  return (uint64_t)skinny::splits_for(n, k, 0) * n * rem * sizeof(float);
}

int launch_ragged_rows(const float* left_tail, uint64_t left_pitch, const float* right, float* out_tail,
                       float* ws, uint64_t rem, uint64_t n, uint64_t k, cudaStream_t st) {
  using namespace skinny;
  const uint32_t splits = splits_for(n, k, 0);
  uint64_t m_blocks = (n / 4 + kThreads - 1) / kThreads;
  uint64_t k_per_split = (k + splits - 1) / splits;
  k_per_split = (k_per_split + 3) & ~3ull;
  dim3 grid((unsigned)m_blocks, splits);
  int rc;
  switch (round_np(rem)) {
#define POLAR_RAGGED(NP) \
  case NP: rc = launch("fmatmul_ragged_rows", small_n_mnmajor_kernel<NP, true>, grid, kThreads, 0, st, right, left_tail, ws, n, rem, k, left_pitch, (uint64_t)1, k_per_split, 1u); break;
    POLAR_RAGGED(1) POLAR_RAGGED(2) POLAR_RAGGED(4) POLAR_RAGGED(8) POLAR_RAGGED(10) POLAR_RAGGED(16)
#undef POLAR_RAGGED
    default: return fail(POLAR_B200_ERR_UNSUPPORTED, "ragged rows: more than 16");
  }
  if (rc) return rc;
  uint64_t g = (n * rem + kThreads - 1) / kThreads;
  uint64_t cap = (uint64_t)sm_count() * 4;
  return launch("fmatmul_ragged_rows_reduce", reduce_splits_transposed_kernel, (unsigned)(g < cap ? g : cap), kThreads, 0, st, ws,
                out_tail, n, rem, splits);
}

// Which skinny kernel, if any, serves this shape: 1 = small n with K-major left,
// 2 = small n with MN-major left (needs scratch), 3 = small k, 0 = none.
int skinny_kind(int tl, int tr, uint64_t m, uint64_t n, uint64_t k, const float* left,
                const float* right, const float* out) {
  (void)tr; (void)right;
  if (n <= 16 && k >= 32) {
    // many unaligned rows stay off: their 32-bit loads would be bound by the re-reads of the small operand
    if (!tl && (((k & 3) == 0 && aligned16(left)) || m < skinny::kResidentRows)) return 1;
    if (tl) return 2;
  }
  if (k <= 16 && n >= 32) return 3;
  (void)out;
  return 0;
}

// What kind 1 (small n, K-major left) takes in microseconds, fitted to measurements on B200 (n = 1 ... 16, k = 128 ... 8192,
// 64 ... 32768 rows; within a third).  Up to 1024 rows the row kernel is a chain of latencies, longer with n and k; the
// resident kernel takes 64 rows per SM at a time; without room for the small operand every CTA reads it again per 32 rows.
double small_n_estimate_us(uint64_t m, uint64_t n, uint64_t k) {
  const uint64_t np = n <= 1 ? 1 : n <= 4 ? 4 : n <= 8 ? 8 : n <= 10 ? 10 : 16;
  const double kd = (double)k, nd = (double)n, md = (double)m;
  if (m >= skinny::kResidentRows && np * (k + 4) * sizeof(float) <= 200 * 1024) {
    const uint64_t at_once = 64ull * (uint64_t)sm_count();
    const double passes = (double)((m + at_once - 1) / at_once) * kd / 4096 * (n <= 10 ? 10.0 + 2.0 * nd : 3.6 * nd);
    const double memory = md * kd * 4e-6 / 6.2;
    return 4.0 + (passes > memory ? passes : memory);
  }
  const double latency = 6.3e-7 * kd * (nd + 3.5) * (m < 1024 ? md : 1024.0), work = 2e-7 * kd * (nd + 3.5) * md;
  return 4.0 + (latency > work ? latency : work);
}

// The same for kind 2 (small n, MN-major left), its summing kernel included.
double small_tn_estimate_us(uint64_t m, uint64_t n, uint64_t k) {
  const double width = (double)(m < 1024 ? m : 1024) * (double)n;
  double doublings = 0;
  for (uint64_t v = k; v > 128; v >>= 1) doublings += 1;
  return 3.5 + 4e-4 * width + (1.4 + 3.6e-4 * width) * doublings + 0.5 * (double)m * (double)k * 4e-6 / 6.2;
}

uint64_t skinny_workspace_bytes(int kind, uint64_t m, uint64_t n, uint64_t k) {
  if (kind != 2) return 0;
  uint32_t s = skinny::splits_for(m, k, n);
  if (skinny::sum_in_cluster(k, n, s)) return 0;
  return s > 1 ? (uint64_t)s * m * n * sizeof(float) : 0;
}

// `sig` (small k only): fuse the Sigmoid derivative with this sigmoid output;
// `sigmoid_out` (small n, K-major left only): store fsigmoid of the product.
int launch_skinny(int kind, int tl, int tr, uint64_t m, uint64_t n, uint64_t k, const float* left,
                  const float* right, float* out, float* ws, cudaStream_t st, const float* sig, int sigmoid_out) {
  using namespace skinny;
  const uint64_t rsk = tr ? 1 : n, rsj = tr ? k : 1;
  if (kind == 1 || kind == 2) {
    const int np = round_np(n);
    const uint32_t splits = kind == 2 ? splits_for(m, k, n) : 1;
#define POLAR_SKINNY_N(NP)                                                                   \
  case NP:                                                                                   \
    return kind == 1 ? launch_small_n_k<NP>(left, right, out, m, n, k, rsk, rsj, st, sigmoid_out) \
                     : launch_small_n_mn<NP>(left, right, out, ws, splits, m, n, k, rsk, rsj, st);
    switch (np) {
      POLAR_SKINNY_N(1)
      POLAR_SKINNY_N(2)
      POLAR_SKINNY_N(4)
      POLAR_SKINNY_N(8)
      POLAR_SKINNY_N(10)
      POLAR_SKINNY_N(16)
    }
#undef POLAR_SKINNY_N
    return fail(POLAR_B200_ERR_UNSUPPORTED, "skinny matmul: unsupported n");
  }
  // small k
  const uint64_t lsi = tl ? 1 : k, lsk = tl ? m : 1;
  // about three CTAs per SM in all, each with an equal share of the rows (a multiple of four)
  uint64_t gx = ((n + 3) / 4 + kThreads - 1) / kThreads, gy = (m + 3) / 4;
  const uint64_t gy_cap = ((uint64_t)sm_count() * 3 + gx - 1) / gx;
  if (gy > gy_cap) gy = gy_cap;
  if (gy > 65535) {
    return fail(POLAR_B200_ERR_UNSUPPORTED, "skinny matmul: more than 65535 row blocks");
  }
  dim3 grid((unsigned)gx, (unsigned)gy);
  int vec = ((n & 3) == 0) && aligned16(out) && (!sig || aligned16(sig));
  auto go = [&](auto kernel) {
    return launch("fmatmul_small_k", kernel, grid, kThreads, 0, st, left, right, out, m, n, k, lsi, lsk, rsk, rsj, vec, sig);
  };
  return k <= 4 ? go(small_k_kernel<4>) : k <= 10 ? go(small_k_kernel<10>) : go(small_k_kernel<16>);
}

// Whether the one-pass dense-layer backward serves these sizes, i.e. whether the two separate
// products would run on the small-n (left M-contiguous) and small-k kernels whose arithmetic it
// reproduces: dZ [rows, n], W [kh, n], H and dIn [rows, kh].
bool dense_grad_ok(uint64_t rows, uint64_t kh, uint64_t n, const float* H, const float* din) {
  return n >= 1 && n <= 16 && rows >= 32 && kh >= 32 && (kh & 3) == 0 && aligned16(H) && aligned16(din);
}
uint64_t dense_grad_workspace_bytes(uint64_t rows, uint64_t kh, uint64_t n) {
  const uint32_t s = skinny::splits_for(kh, rows, n);
  return s > 1 ? (uint64_t)s * kh * n * sizeof(float) : 0;
}
int launch_dense_grad(const float* H, const float* dz, const float* W, float* din, float* dw, float* ws,
                      uint64_t rows, uint64_t kh, uint64_t n, cudaStream_t st) {
  using namespace skinny;
  const uint32_t splits = splits_for(kh, rows, n);
  switch (round_np(n)) {
#define POLAR_DENSE(NP) case NP: return launch_dense_grad_np<NP>(H, dz, W, din, dw, ws, splits, rows, kh, n, st);
    POLAR_DENSE(1) POLAR_DENSE(2) POLAR_DENSE(4) POLAR_DENSE(8) POLAR_DENSE(10) POLAR_DENSE(16)
#undef POLAR_DENSE
  }
  return fail(POLAR_B200_ERR_UNSUPPORTED, "fdense_grad: unsupported n");
}

// ---------------------------------------------------------------- entry point that allocates nothing

// Scratch for polar_b200_fmatmul_tn_small_n_static: the per-split partial sums of
// the split-k kernel above.  It is part of the library image, so every GPU that
// loads the library holds these 16 MiB until the process exits.
constexpr uint64_t kStaticScratchBytes = 16ull << 20;
static __device__ __align__(256) float g_static_scratch[kStaticScratchBytes / sizeof(float)];

namespace {
// In host code `g_static_scratch` is only a handle for the runtime; the address the
// kernels need comes from cudaGetSymbolAddress, asked once per device with that
// device current.
float* static_scratch_for_current_device(int* status) {
  static std::mutex mu;
  static float* cached[64] = {nullptr};
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= 64) {
    *status = fail(POLAR_B200_ERR_CUDA, "cudaGetDevice", e);
    return nullptr;
  }
  std::lock_guard<std::mutex> guard(mu);
  if (!cached[dev]) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_static_scratch);
    if (e != cudaSuccess || !p) {
      *status = fail(POLAR_B200_ERR_CUDA, "cudaGetSymbolAddress(static scratch)", e);
      return nullptr;
    }
    cached[dev] = static_cast<float*>(p);
  }
  *status = POLAR_B200_OK;
  return cached[dev];
}
}  // namespace

}  // namespace polar_b200

extern "C" {

uint64_t polar_b200_static_scratch_bytes(void) { return polar_b200::kStaticScratchBytes; }

int polar_b200_fmatmul_tn_small_n_static(int transRight, uint64_t m, uint64_t n, uint64_t k,
                                         const float* left, const float* right, float* out,
                                         void* stream) {
  using namespace polar_b200;
  clear_error();
  if (transRight != 0 && transRight != 1) return fail(POLAR_B200_ERR_INVALID, "transRight must be 0 or 1");
  if (m == 0 || n == 0) return POLAR_B200_OK;
  if (!left || !right || !out) return fail(POLAR_B200_ERR_INVALID, "null device pointer");
  if (n > 16 || k < 32 || (m & 3) != 0 || !aligned16(left))
    return fail(POLAR_B200_ERR_UNSUPPORTED,
                "static-scratch fmatmul serves left stored [k,m] with m a multiple of 4, a 16-byte aligned "
                "left pointer, n <= 16 and k >= 32");
  if (m > (1ull << 31) || k > (1ull << 31)) return fail(POLAR_B200_ERR_INVALID, "matrix dimension too large");
  const uint64_t need = skinny_workspace_bytes(2, m, n, k);
  if (need > kStaticScratchBytes)
    return fail(POLAR_B200_ERR_WORKSPACE,
                "this product needs more than the 16 MiB of built-in scratch; use polar_b200_fmatmul with a "
                "caller workspace");
  LaunchDeviceScope on(stream, out);   // the array's address is looked up on the device that will run the kernels
  int rc = POLAR_B200_OK;
  float* scratch = static_scratch_for_current_device(&rc);
  if (!scratch) return rc;
  // Every partial sum the reduction reads is written by the first kernel of this
  // call, so nothing in the scratch has to be cleared beforehand.
  return launch_skinny(2, 1, transRight, m, n, k, left, right, out, scratch, as_stream(stream), nullptr, 0);
}

}  // extern "C"
