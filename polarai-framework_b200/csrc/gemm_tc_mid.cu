// fmatmul on the tensor cores for products that are too small, or too oddly shaped, to fill the chip with the
// 256-column tiles of gemm_tc.cu: one output tile of 128 x BN per cluster of CTAs, the k range divided over the
// CTAs of the cluster, the partial tiles added through distributed shared memory.
//
// Why it exists.  1024^3 is 16 tiles of 256 x 256 or 32 of 128 x 256: cut along k they fill 64 of 148 SMs, and
// the partial products travel through global memory and a second kernel.  Here it is 64 tiles of
// 128 x 128 in clusters of two.  An operand whose rows TMA cannot address (a row pitch that is no multiple of 16
// bytes) is first copied to scratch with a padded pitch (pad_kernel); those shapes had only
// the FFMA kernel, at 15 TFLOP/s.
//
// One CTA:
//   warp 0      TMA producer: 32-float k slabs of A (128 rows) and B (BN rows), two instructions per slab;
//   warps 2...   split warps, two or three groups of four: of each landed slab, the hi and lo parts of A to tensor memory and the lo parts of B to
//               shared memory beside the raw words, which are its hi parts (the tensor core ignores the low 13 bits);
//   warp 1      tcgen05.mma issuer: per slab and 8 k the three products of the TF32 split, A from tensor memory;
//   the rest    accumulator warps, eight or four: every `chunk` slabs they read the tensor-memory accumulator and add it to
//               registers in round-to-nearest.  The tensor core's own accumulator rounds toward zero, an error that
//               grows with the length of the sum (8e-9 of the result per term for zero-mean operands);
//               chunks keep it at that of a short sum.
//
// What bounds it: shared memory, 128 bytes per clock.  An instruction of 128 x BN x 8 with both operands there reads
// 4 KB + 32 BN bytes: 64 / 48 / 40 clocks for 128 / 64 / 32 columns, where the tensor core needs 64 / 32 / 16 - all of the
// bandwidth before TMA has written a slab and the split has read it and written the lo parts.  With A in tensor memory
// a 128 x 128 x 32 slab takes 1024 clocks of shared memory instead of 1536 (768 of the tensor core); measured 0.55 us a
// slab.  Narrower tiles are bound by the latencies of their loops: each role asks for its next barrier before it works on the
// current slab (a wait on a barrier long complete took 150 of the 700 clocks per slab), 0.34 us with 64 columns and 0.29
// with 32 (0.60, 0.48, 0.43 us at first).  2001 x 1511 x 999: 60 -> 50 us; 16 x 4096 x 784:
// 8.8 -> 7.5 us.  What is left per tile, 4 to 5 us, is set-up, the first slab's way through the pipeline and the store; the
// exchange in a cluster runs at the 15 bytes per clock an SM gets from another SM's shared memory (pushing the parts
// there instead of reading them was slower: 17.4 against 15.9 us at 1024^3).
//
// The split: A's hi is rounded to the nearest TF32 (it is written anyway), B's is cut off; the dropped lo.lo is below
// 2^-23 |a||b| and of either sign: 9e-8 of the norm for uniform operands, where four products with both cut off left 1.1e-7
// and an FFMA sum has 1.0e-7 (32 terms) to 5.7e-7 (1000 terms).
// A NaN or an infinity always reaches a product: in B as the raw word that is its hi part, in A as its hi part or through the
// difference from it, which is a NaN then.  The sums that it enters come out as NaN or infinite,
// though not always as the right one of the two (an infinity meets lo parts of 0), so a result that is not finite is
// computed again in FFMA, in the order of k (repair_share): the classes of every result are those of an FFMA kernel.
// At the end the tile goes to shared memory in the layout of the result's rows; the cluster's CTAs each
// add one share of it over all CTAs in rank order (the same bits run to run) and store whole lines.
//
// Orientation: rows of a tile are tensor-memory lanes, 128 of them; with `out_t` the kernel was given the
// operands in exchanged roles, and the tile's rows are columns of the result (results of few rows).
//
// Waits are bounded as in gemm_tc.cu; codes 111 ... 117.
#include <cuda.h>

#include <mutex>

#include "common.cuh"
#include "tc_ptx.cuh"

namespace polar_b200 {
namespace tc {
int make_map(CUtensorMap* map, const float* base, uint64_t inner, uint64_t outer, uint32_t box_inner, uint32_t box_outer,
             bool mn_major, int bk, uint64_t pitch);
int make_map_chunks(CUtensorMap* map, const float* base, uint64_t chunks, uint64_t outer, uint32_t box_outer,
                    uint32_t box_chunks, uint64_t pitch);
}  // namespace tc

namespace mid {
using namespace tc;

constexpr int BM = 128, BK = 32;
constexpr int kThreads = 32 * 18;
constexpr uint32_t kBox = 32 * BK * 4;                      // one MN-major chunk of a slab: 32 elements x BK rows

// Shared memory is a ring of raw slabs and a shorter ring of B's lo parts, in step with a ring of A's parts in tensor
// memory.  A raw slab is held from the TMA request to the end of its products (about 2 us: L2 latency, split,
// products), the parts only from the split on, so the raw ring is what has to be deep: at 128 x 128 x 32 a slab's
// products take 0.4 us.
template <int BN> struct Cfg {
  // Groups of four split warps that take the slabs in turn: a slab costs a warp 700 clocks of latencies (barriers, loads, the
  // wait for its stores) whatever its width, more than the products of a narrow tile.
  static constexpr int kGroups = BN == 32 ? 3 : 2, kSplitWarps = 4 * kGroups, kAccWarps = 16 - kSplitWarps;
  static constexpr uint32_t kABytes = BM * BK * 4, kBBytes = BN * BK * 4, kRawBytes = kABytes + kBBytes;
  static constexpr int kRaw = BN == 128 ? 6 : BN == 64 ? 8 : 9, kLo = BN == 128 ? 2 : BN == 64 ? 4 : 6;
  static_assert(kRaw % kGroups == 0 && kLo % kGroups == 0, "a place of a ring belongs to one group");
  static constexpr uint32_t kLoBase = kRaw * kRawBytes;
  static constexpr uint32_t kTileBytes = kLoBase + kLo * kBBytes;
  static constexpr uint32_t kBarBytes = 320, kSmemBytes = kTileBytes + 1024 + kBarBytes;
  // tensor memory: accumulators that take turns, A's parts
  static constexpr int kAccs = BN == 128 ? 2 : 4;
  static constexpr uint32_t kABase = kAccs * BN, kASlab = 2 * BK, kTmemCols = 512;
  static_assert(kABase + kLo * kASlab <= kTmemCols, "tensor memory");
  static_assert(kSmemBytes <= 227 * 1024, "rings must fit shared memory");
  static_assert(BM * (BN + 4) * 4 <= (int)kTileBytes && BN * (BM + 4) * 4 <= (int)kTileBytes, "the tile must fit the rings");
};

// Kept small: a launch pays for every byte of its parameters, on the host and on the way to the SMs.  Extents are 2^31 at most.
struct Params {
  float* out;
  int* status;
  unsigned long long wait_ns;
  const float *a, *b;       // the operands in memory, for repair_share
  uint32_t a_pitch, b_pitch, k;
  uint32_t m, n;            // of the product as the kernel sees it (rows = lanes)
  uint32_t pitch;           // floats per row of the result
  uint32_t tiles_m, slabs;
  uint32_t whole;           // the first tiles, one CTA each whatever the cluster (even; see launch_mid)
  uint32_t b_whole;         // whole 32-element chunks of B's extent: tiles inside them come in one 3-D box
  uint32_t cluster, chunk;
  uint8_t a_mn, b_mn;       // operand stored with m (n) contiguous
  uint8_t out_t, epilogue, vec_out;
};

__device__ __forceinline__ float4 ld_shared_v4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ float4 ld_cluster_v4(uint32_t addr, uint32_t rank) {
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(rank));
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(remote) : "memory");
  return v;
}

// A CTA's share of the finished tile: the parts of all CTAs of the cluster, added in rank order, to the result.
// Eight 128-bit reads of (distributed) shared memory are in flight per thread before the first is used.
// True where one of the thread's results is not finite.
template <int BN, int CL>
__device__ __forceinline__ bool store_share(const Params& p, uint32_t base, uint32_t rank, int m0, int n0) {
  constexpr int kVecs = BM * BN / 4, kShare = kVecs / CL, kBatch = 8 / CL;
  const int shift = p.out_t ? 5 : (BN == 128 ? 5 : BN == 64 ? 4 : 3);       // log2 of the vectors in a row of the result
  const int width = 4 << shift;
  const uint32_t out_rows = p.out_t ? p.n : p.m, out_cols = p.out_t ? p.m : p.n;
  const uint32_t r0 = (uint32_t)(p.out_t ? n0 : m0), c0 = (uint32_t)(p.out_t ? m0 : n0);
  // 0 * y is a NaN where y is not finite; what is stored for such a result is not finite either
  auto act = [](float y) { return fmaf(0.f, y, sigmoid_clamped(y)); };
  float probe = 0.f;
  for (int first = 0; first < kShare; first += kBatch * kThreads) {
    float4 part[kBatch][CL];
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int w = first + u * kThreads + (int)threadIdx.x, v = (int)rank * kShare + w;
      if (w >= kShare) continue;
      const uint32_t at = base + (uint32_t)((v >> shift) * (width + 4) + (v & ((1 << shift) - 1)) * 4) * 4u;
#pragma unroll
      for (int k = 0; k < CL; ++k) part[u][k] = CL == 1 || (uint32_t)k == rank ? ld_shared_v4(at) : ld_cluster_v4(at, (uint32_t)k);
    }
    if (CL > 1 && first + kBatch * kThreads >= kShare) cluster_arrive();     // nothing of another CTA is read after this
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int w = first + u * kThreads + (int)threadIdx.x, v = (int)rank * kShare + w;
      if (w >= kShare) continue;
      const uint32_t r = r0 + (uint32_t)(v >> shift), c = c0 + (uint32_t)(v & ((1 << shift) - 1)) * 4;
      if (r >= out_rows || c >= out_cols) continue;
      float4 y = part[u][0];
#pragma unroll
      for (int k = 1; k < CL; ++k) y.x += part[u][k].x, y.y += part[u][k].y, y.z += part[u][k].z, y.w += part[u][k].w;
      probe = fmaf(0.f, y.x, fmaf(0.f, y.y, fmaf(0.f, y.z, fmaf(0.f, y.w, probe))));
      if (p.epilogue == 1) y = make_float4(act(y.x), act(y.y), act(y.z), act(y.w));
      float* dst = p.out + (uint64_t)r * p.pitch + c;
      if (p.vec_out && c + 4 <= out_cols) {
        *reinterpret_cast<float4*>(dst) = y;
      } else {
        dst[0] = y.x;
        if (c + 1 < out_cols) dst[1] = y.y;
        if (c + 2 < out_cols) dst[2] = y.z;
        if (c + 3 < out_cols) dst[3] = y.w;
      }
    }
  }
  return probe != 0.f;
}

__device__ __forceinline__ void load_terms(const float* p, uint64_t step, float (&v)[4]) {
  if (step == 1 && (reinterpret_cast<uintptr_t>(p) & 15) == 0) {
    const float4 a = *reinterpret_cast<const float4*>(p);
    v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w;
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = p[i * step];
  }
}

// Computes what a thread has stored again where it is not finite: FFMA, ascending k.  A NaN ends a sum.  (Out of the loop
// above, where it cost every launch 0.3 us.)  Four terms are loaded at a time; one by one each waited for the memory
// (2001 x 1511 x 999 with nothing but infinite results 9 to 15 ms, this way 4 to 5).  Kept small: a launch that never comes here
// pays for its code too, 0.05 us more with eight terms.
__device__ __noinline__ void repair_share(const float* a, uint64_t a_row, uint64_t a_k, const float* b, uint64_t b_col, uint64_t b_k,
                                          uint32_t terms, float* out, uint64_t pitch, uint32_t rows, uint32_t cols, uint32_t first_vec,
                                          uint32_t end_vec, int shift, uint32_t r0, uint32_t c0, bool out_t, bool sigmoid) {
#pragma unroll 1
  for (uint32_t v = first_vec + threadIdx.x; v < end_vec; v += kThreads) {
    const uint32_t r = r0 + (v >> shift);
#pragma unroll 1
    for (uint32_t c = c0 + (v & ((1u << shift) - 1)) * 4, end = c + 4; r < rows && c < cols && c < end; ++c) {
      float* dst = out + r * pitch + c;
      if (0.f * *dst == 0.f) continue;
      const float *x = a + (out_t ? c : r) * a_row, *y = b + (out_t ? r : c) * b_col;
      float s = 0.f;
      uint32_t k = 0;
#pragma unroll 1
      for (; k + 4 <= terms && s == s; k += 4, x += 4 * a_k, y += 4 * b_k) {
        float u[4], w[4];
        load_terms(x, a_k, u);
        load_terms(y, b_k, w);
#pragma unroll
        for (int i = 0; i < 4; ++i) s = fmaf(u[i], w[i], s);
      }
#pragma unroll 1
      for (; k < terms && s == s; ++k, x += a_k, y += b_k) s = fmaf(*x, *y, s);
      *dst = sigmoid ? sigmoid_clamped(s) : s;
    }
  }
}

// Two floats in one instruction each (sm_100).
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

template <int BN>
__global__ void __launch_bounds__(kThreads, 1)
fmatmul_mid_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                   const __grid_constant__ CUtensorMap map_b3, const Params p) {
  using C = Cfg<BN>;
  constexpr int kAccs = C::kAccs, kSplitWarps = C::kSplitWarps, kAccWarps = C::kAccWarps;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* gen = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t bars = base + C::kTileBytes;
  auto full_raw = [&](int s) { return bars + 8u * s; };
  auto empty = [&](int s) { return bars + 8u * (C::kRaw + s); };
  auto full_lo = [&](int s) { return bars + 8u * (2 * C::kRaw + s); };
  constexpr int kRings = 2 * C::kRaw + C::kLo;
  auto acc_full = [&](int a) { return bars + 8u * (kRings + a); };
  auto acc_empty = [&](int a) { return bars + 8u * (kRings + kAccs + a); };
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(gen + C::kTileBytes + 8 * (kRings + 2 * kAccs));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  static_assert(8 * (kRings + 2 * kAccs) + 8 <= (int)C::kBarBytes, "barrier block");

  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const bool whole = blockIdx.x < p.whole;
  const uint32_t cluster = whole ? 1u : p.cluster;         // CTAs that share this tile
  const uint32_t rank = cluster > 1 ? cluster_rank() : 0u;
  const uint32_t tile = whole ? blockIdx.x : p.whole + (blockIdx.x - p.whole) / cluster;
  const int m0 = (int)((tile % p.tiles_m) * BM), n0 = (int)((tile / p.tiles_m) * BN);
  const uint32_t kb0 = (uint32_t)((uint64_t)rank * p.slabs / cluster);
  const uint32_t kb1 = (uint32_t)((uint64_t)(rank + 1) * p.slabs / cluster);
  const uint32_t mine = kb1 - kb0, chunks = (mine + p.chunk - 1) / p.chunk;

  constexpr int kBars = kRings + 2 * kAccs;
  static_assert(kBars <= 32, "one lane initialises one barrier");
  if (warp == 0) {
    if (lane < kBars) {
      const bool is_lo = lane >= 2 * C::kRaw && lane < kRings, is_acc_empty = lane >= kRings + kAccs;
      mbar_init(bars + 8u * lane, is_lo ? 4u : is_acc_empty ? (uint32_t)kAccWarps : 1u);
    }
    if (lane == 0) {
      *abort_flag = 0;
      prefetch_map(&map_a);
      prefetch_map(p.b_mn && n0 + BN <= 32 * p.b_whole ? &map_b3 : &map_b);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), C::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);   // (known to be uniform)
  pdl_enter();              // the set-up above overlaps the kernel before; operands and result are touched from here on

  if (warp == 0) {
    const bool leader = elect_one();
    {
      uint32_t s = 0, ph = 1;
      bool free = true;
      for (uint32_t it = 0; it < mine; ++it) {
        if (!free && !mbar_wait(empty(s), ph, abort_flag, p.status, 111, p.wait_ns)) break;
        const uint32_t s_next = s + 1 == C::kRaw ? 0 : s + 1, ph_next = s_next ? ph : ph ^ 1;
        free = mbar_test(empty(s_next), ph_next);
        if (leader) {
          const uint32_t a = base + s * C::kRawBytes, b = a + C::kABytes;
          mbar_expect_tx(full_raw(s), C::kRawBytes);
          const int k0 = (int)((kb0 + it) * BK);
          if (p.a_mn) tma_load_2d(a, &map_a, full_raw(s), m0, k0);
          else tma_load_2d(a, &map_a, full_raw(s), k0, m0);
          if (!p.b_mn) {
            tma_load_2d(b, &map_b, full_raw(s), k0, n0);
          } else if (n0 + BN <= 32 * p.b_whole) {
            tma_load_3d(b, &map_b3, full_raw(s), 0, k0, n0 / 32);
          } else {
            for (int c = 0; c < BN / 32; ++c) tma_load_2d(b + c * kBox, &map_b, full_raw(s), n0 + 32 * c, k0);
          }
        }
        s = s_next, ph = ph_next;
      }
    }
  } else if (warp == 1) {
    const bool leader = elect_one();
    {
      const uint32_t idesc = make_idesc(BM, BN, 0, p.b_mn);
      // K-major: 128-byte rows in the 128-byte swizzle (layout 2), 8-row groups 1 KB apart, 8 k = 32 bytes
      // inside the row.  MN-major: chunks of 32 elements x BK rows (layout 1), chunks kBox apart, 8 k = 1 KB.
      const Operand b_op = make_desc(0, p.b_mn ? kBox : 16u, p.b_mn ? 512u : 1024u, p.b_mn ? 1u : 2u);
      const uint32_t b_step = (p.b_mn ? 1024u : 32u) >> 4;
      // (in a cluster the upper bits of a shared address hold the CTA's rank; a descriptor has no room for them)
      const uint32_t ring = (base & 0x3FFFFu) >> 4;
      uint32_t it = 0, s = 0, l = 0, l_ph = 0;              // slab; its place in either ring
      bool ok = true, split = false, drained = true;        // (the accumulators are empty at first)
      for (uint32_t c = 0; ok && c < chunks; ++c) {
        const int acc = c % kAccs;
        ok = drained || mbar_wait(acc_empty(acc), ((c / kAccs) & 1u) ^ 1u, abort_flag, p.status, 115, p.wait_ns);
        if (!ok) break;
        tc_fence_after();
        drained = mbar_test(acc_empty((c + 1) % kAccs), (((c + 1) / kAccs) & 1u) ^ 1u);
        const uint32_t d = tmem + acc * BN;
        const uint32_t last = it + p.chunk < mine ? it + p.chunk : mine;
        for (uint32_t accumulate = 0; it < last; ++it, accumulate = 1) {
          const uint32_t b_hi = ring + ((s * C::kRawBytes + C::kABytes) >> 4), b_lo = ring + ((C::kLoBase + l * C::kBBytes) >> 4);
          const uint32_t a_hi = tmem + C::kABase + l * C::kASlab, a_lo = a_hi + BK;
          // (the split warps have waited for the raw slab)
          ok = split || mbar_wait(full_lo(l), l_ph, abort_flag, p.status, 113, p.wait_ns);
          if (!ok) break;
          tc_fence_after();
          if (++l == C::kLo) l = 0, l_ph ^= 1;
          split = mbar_test(full_lo(l), l_ph);
          if (leader) {
            // the small products first: what the accumulator cuts off is relative to what it holds
#pragma unroll
            for (int kk = 0; kk < BK / 8; ++kk) {
              tc_mma_tf32_ts(d, a_lo + 8 * kk, b_op, b_hi + kk * b_step, idesc, kk ? 1u : accumulate);
              tc_mma_tf32_ts(d, a_hi + 8 * kk, b_op, b_lo + kk * b_step, idesc, 1u);
            }
#pragma unroll
            for (int kk = 0; kk < BK / 8; ++kk) tc_mma_tf32_ts(d, a_hi + 8 * kk, b_op, b_hi + kk * b_step, idesc, 1u);
            tc_commit(empty(s));
          }
          if (++s == C::kRaw) s = 0;
        }
        if (ok && leader) tc_commit(acc_full(acc));
      }
    }
  } else if (warp < 2 + kSplitWarps) {
    // A: a thread takes one row, the row being the tensor-memory lane its warp may write (warp mod 4).
    // B: vectors of the slab as they lie.
    const int tid = (threadIdx.x - 64) & 127, row = (warp & 3) * 32 + lane;
    constexpr int kVecs = C::kBBytes / 16 / 128 / 2;        // B's vectors of a thread, in two halves like A's 32 k
    static_assert(kVecs * 2 * 128 * 16 == C::kBBytes, "slab must divide over the split warps");
    uint32_t s = (warp - 2) >> 2, ph = 0, l = s, prev = s, prev_ph = 0;   // prev: the slab that used this place of the lo ring before
    bool landed = false;
    for (uint32_t it = s; it < mine; it += C::kGroups) {
      const bool free = it < (uint32_t)C::kLo || mbar_test(empty(prev), prev_ph);
      if (!landed && !mbar_wait(full_raw(s), ph, abort_flag, p.status, 114, p.wait_ns)) break;
      const uint8_t* slab = gen + s * C::kRawBytes;
      const float4* raw = reinterpret_cast<const float4*>(slab + C::kABytes) + tid;
      float4* lo = reinterpret_cast<float4*>(gen + C::kLoBase + l * C::kBBytes) + tid;
      // the tensor core ignores the low 13 bits: adding half of the last one it sees rounds to nearest.  (The largest finite
      // numbers become infinities: their results are computed again like those of an infinity.)
      auto nearest = [](float x) { return __uint_as_float(__float_as_uint(x) + 0x1000u); };
      auto high = [&](float x) { return __uint_as_float(__float_as_uint(nearest(x)) & 0xFFFFE000u); };
      auto low = [&](float x) { return nearest(x - __uint_as_float(__float_as_uint(x) & 0xFFFFE000u)); };
      bool ok = true;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        // all loads before the first store: the compiler cannot tell that the two never meet, and would
        // make one latency of each vector
        float a[16];
        float4 v[kVecs];
        if (p.a_mn) {                                       // rows of 128 m, one per k
#pragma unroll
          for (int j = 0; j < 16; ++j) a[j] = reinterpret_cast<const float*>(slab)[(half * 16 + j) * BM + row];
        } else {                                            // rows of 32 k in the 128-byte swizzle: eight rows cover all banks
#pragma unroll
          for (int j = 0; j < 4; ++j)
            *reinterpret_cast<float4*>(a + 4 * j) = *reinterpret_cast<const float4*>(slab + row * 128 + (((half * 4 + j) ^ (row & 7)) << 4));
        }
#pragma unroll
        for (int i = 0; i < kVecs; ++i) v[i] = raw[(half * kVecs + i) * 128];
        if (half == 0 && it >= (uint32_t)C::kLo) {
          ok = free || mbar_wait(empty(prev), prev_ph, abort_flag, p.status, 117, p.wait_ns);
          if (!ok) break;
          if ((prev += C::kGroups) >= (uint32_t)C::kRaw) prev -= C::kRaw, prev_ph ^= 1;
          tc_fence_after();
        }
        const uint32_t at = tmem + ((uint32_t)((warp & 3) * 32) << 16) + C::kABase + l * C::kASlab + half * 16;
        uint32_t part[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) part[j] = __float_as_uint(high(a[j]));
        tmem_st_32x16(at, part);
        // Two lo parts at a time, and their sum: a NaN, where one of the row's elements is not finite.  (Arithmetic returns the NaN
        // 0x7fffffff, which the rounding makes a zero of; bounding every element below that with a minimum cost 2 % at
        // 1024^3.)
        unsigned long long lost = 0;
#pragma unroll
        for (int j = 0; j < 16; j += 2) {
          const unsigned long long rest = fma2(pack2(__uint_as_float(part[j]), __uint_as_float(part[j + 1])), pack2(-1.f, -1.f), pack2(a[j], a[j + 1]));
          lost = add2(lost, rest);
          float x, y;
          unpack2(rest, x, y);
          part[j] = __float_as_uint(nearest(x));
          part[j + 1] = __float_as_uint(nearest(y));
        }
        float x, y;
        unpack2(lost, x, y);
        part[15] = __float_as_uint(fmaf(0.f, x + y, __uint_as_float(part[15])));
        tmem_st_32x16(at + BK, part);
#pragma unroll
        for (int i = 0; i < kVecs; ++i)
          lo[(half * kVecs + i) * 128] = make_float4(low(v[i].x), low(v[i].y), low(v[i].z), low(v[i].w));
      }
      if (!ok) break;
      if ((s += C::kGroups) >= (uint32_t)C::kRaw) s -= C::kRaw, ph ^= 1;
      landed = mbar_test(full_raw(s), ph);
      fence_async_smem();
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(full_lo(l));               // one arrival per warp
      if ((l += C::kGroups) >= (uint32_t)C::kLo) l -= C::kLo;
    }
  } else {
    // four consecutive warps cover the 128 lanes; with eight, the two warps of a lane quarter take half of the columns each
    const int q = warp & 3, half = (warp - (2 + kSplitWarps)) >> 2;
    constexpr int kCols = BN / (kAccWarps / 4);
    constexpr int kPart = kCols == 32 ? 32 : 16;             // columns in flight: what the register budget allows
    // 32-column tiles have registers for a second level: sums of 16 chunks are added up separately
    constexpr bool kTwoLevels = BN == 32;
    float acc[kCols], sum[kTwoLevels ? kCols : 1];
#pragma unroll
    for (int j = 0; j < kCols; ++j) acc[j] = 0.f;
    if (kTwoLevels) {
#pragma unroll
      for (int j = 0; j < kCols; ++j) sum[j] = 0.f;
    }
    bool ok = true;
    for (uint32_t c = 0; c < chunks; ++c) {
      const int a = c % kAccs;
      ok = mbar_wait(acc_full(a), (c / kAccs) & 1u, abort_flag, p.status, 116, p.wait_ns);
      if (!ok) break;
      tc_fence_after();
      const uint32_t at = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(a * BN + half * kCols);
#pragma unroll
      for (int j0 = 0; j0 < kCols; j0 += kPart) {
        uint32_t r[kPart];
#pragma unroll
        for (int j = 0; j < kPart; j += 16) tmem_ld_32x16(at + j0 + j, r + j);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < kPart; ++j) acc[j0 + j] += __uint_as_float(r[j]);
      }
      if (kTwoLevels && ((c & 15u) == 15u || c + 1 == chunks)) {
        const bool last = c + 1 == chunks;
#pragma unroll
        for (int j = 0; j < kCols; ++j) sum[j] += acc[j], acc[j] = last ? sum[j] : 0.f;
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_empty(a));
    }
    // all products of this CTA are done and every stage has been read: the tile takes their place, in rows of the result
    if (ok) {
      float* t = reinterpret_cast<float*>(gen);
      const int row = q * 32 + lane;
      if (p.out_t) {
#pragma unroll
        for (int j = 0; j < kCols; ++j) t[(half * kCols + j) * (BM + 4) + row] = acc[j];
      } else {
#pragma unroll
        for (int j = 0; j < kCols; j += 4)
          *reinterpret_cast<float4*>(t + row * (BN + 4) + half * kCols + j) = make_float4(acc[j], acc[j + 1], acc[j + 2], acc[j + 3]);
      }
    }
  }

  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (cluster > 1) {
    cluster_arrive();
    cluster_wait();
  }
  if (warp == 1) {
    tc_fence_after();
    if (*abort_flag) {     // let copies and MMAs in flight finish before the tensor memory goes away
      const long long t0 = clock64();
      while (clock64() - t0 < 2000000ll) { }
    }
    tmem_dealloc(tmem, C::kTmemCols);
  }
  bool repair;
  switch (cluster) {
    case 1: repair = store_share<BN, 1>(p, base, 0, m0, n0); break;
    case 2: repair = store_share<BN, 2>(p, base, rank, m0, n0); break;
    case 4: repair = store_share<BN, 4>(p, base, rank, m0, n0); break;
    default: repair = store_share<BN, 8>(p, base, rank, m0, n0);
  }
  if (cluster > 1) cluster_wait();   // nobody leaves while another CTA may still read its part
  if (repair) {
    constexpr uint32_t kVecs = BM * BN / 4;
    const uint64_t a_pitch = p.a_pitch, b_pitch = p.b_pitch;
    repair_share(p.a, p.a_mn ? 1 : a_pitch, p.a_mn ? a_pitch : 1, p.b, p.b_mn ? 1 : b_pitch, p.b_mn ? b_pitch : 1, p.k, p.out, p.pitch,
                 p.out_t ? p.n : p.m, p.out_t ? p.m : p.n, rank * (kVecs / cluster), (rank + 1) * (kVecs / cluster),
                 p.out_t ? 5 : (BN == 128 ? 5 : BN == 64 ? 4 : 3), p.out_t ? n0 : m0, p.out_t ? m0 : n0, p.out_t, p.epilogue == 1);
  }
}

// Copies up to two matrices to scratch with their rows padded to `pitch` floats (a multiple of 32; the
// padding is zero), four floats of the copy per thread.  Bound by memory: 8 bytes per element, 4-byte loads because
// the rows start anywhere.
struct Padded {
  const float* src;
  float* dst;
  uint64_t rows, cols, pitch;
  uint64_t vecs() const { return rows * (pitch / 4); }
};
__global__ void __launch_bounds__(256) pad_kernel(const Padded a, const Padded b, uint64_t vecs_a, uint64_t vecs) {
  pdl_enter();
  uint64_t v = (uint64_t)blockIdx.x * 256 + threadIdx.x;
  if (v >= vecs) return;
  const bool second = v >= vecs_a;
  if (second) v -= vecs_a;
  const float* src = second ? b.src : a.src;
  float* dst = second ? b.dst : a.dst;
  const uint32_t cols = (uint32_t)(second ? b.cols : a.cols), per_row = (uint32_t)((second ? b.pitch : a.pitch) / 4);
  const uint64_t r = v / per_row;
  const uint32_t c = (uint32_t)(v - r * per_row) * 4;
  const float* s = src + r * cols + c;
  float4 x;
  x.x = c < cols ? s[0] : 0.f;
  x.y = c + 1 < cols ? s[1] : 0.f;
  x.z = c + 2 < cols ? s[2] : 0.f;
  x.w = c + 3 < cols ? s[3] : 0.f;
  *reinterpret_cast<float4*>(dst + v * 4) = x;
}

// An operand as it is stored: rows of `cols` contiguous floats, `pitch` floats apart.
struct Stored {
  const float* p;
  uint64_t rows, cols, pitch;
  bool padded;                                              // columns up to the pitch are there, and zero
};

template <int BN>
int launch_cfg(const Stored& left, const Stored& right, bool a_mn, bool b_mn, Params p, uint64_t k, cudaStream_t stream) {
  using C = Cfg<BN>;
  int dev = 0;
  cudaGetDevice(&dev);
  static std::mutex mu;
  static bool attr_done[64] = {false};
  {
    std::lock_guard<std::mutex> guard(mu);
    if (dev >= 0 && dev < 64 && !attr_done[dev]) {
      cudaError_t e = cudaFuncSetAttribute(fmatmul_mid_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::kSmemBytes);
      if (e != cudaSuccess) return fail(POLAR_B200_ERR_CUDA, "cudaFuncSetAttribute(smem)", e);
      attr_done[dev] = true;
    }
  }
  // The extents are the true ones wherever TMA has to cut a box off; a padded MN-major operand offers whole chunks.
  CUtensorMap map_a, map_b, map_b3;
  int rc = a_mn ? make_map(&map_a, left.p, p.m, k, BM, BK, false, 0, left.pitch)       // (the split warps read it: no swizzle)
                : make_map(&map_a, left.p, k, p.m, BK, BM, false, BK, left.pitch);
  if (!rc && !b_mn) {
    rc = make_map(&map_b, right.p, k, p.n, BK, BN, false, BK, right.pitch);
    map_b3 = map_b;
  } else if (!rc) {
    const uint64_t cols = right.padded ? right.pitch : right.cols;
    p.b_whole = (uint32_t)(cols / 32);
    const bool boxes_2d = (p.n + BN - 1) / BN * BN > 32ull * p.b_whole;
    if (p.b_whole) rc = make_map_chunks(&map_b3, right.p, p.b_whole, k, BK, BN / 32, right.pitch);
    if (!rc && (boxes_2d || !p.b_whole)) rc = make_map(&map_b, right.p, cols, k, 32, BK, true, BK, right.pitch);
    else map_b = map_b3;
    if (!p.b_whole) map_b3 = map_b;
  }
  if (rc) return rc;
  p.a_mn = a_mn;
  p.b_mn = b_mn;
  p.a = left.p;
  p.b = right.p;
  p.a_pitch = (uint32_t)left.pitch;
  p.b_pitch = (uint32_t)right.pitch;
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3(p.whole + (p.tiles_m * (uint32_t)((p.n + BN - 1) / BN) - p.whole) * p.cluster);
  c.blockDim = dim3(kThreads);
  c.dynamicSmemBytes = C::kSmemBytes;
  c.stream = stream;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = p.cluster;
  at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
  c.attrs = at;
  c.numAttrs = p.cluster > 1 ? 2 : 1;
  cudaError_t e = cudaLaunchKernelEx(&c, fmatmul_mid_kernel<BN>, map_a, map_b, map_b3, p);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(POLAR_B200_ERR_CUDA, "fmatmul_mid", e);
  }
  count_launch();
  return POLAR_B200_OK;
}

}  // namespace mid

namespace {
uint64_t pad32(uint64_t v) { return (v + 31) & ~31ull; }
bool addressable(const float* p, uint64_t cols) { return aligned16(p) && (cols & 3) == 0; }
}  // namespace

// Scratch for operands that TMA cannot address as they are (0: none).
uint64_t mid_workspace_bytes(int tl, int tr, uint64_t m, uint64_t n, uint64_t k, const float* left, const float* right) {
  const uint64_t lc = tl ? m : k, lr = tl ? k : m, rc = tr ? k : n, rr = tr ? n : k;
  uint64_t floats = 0;
  if (!addressable(left, lc)) floats += lr * pad32(lc);
  if (!addressable(right, rc)) floats += rr * pad32(rc);
  return floats * sizeof(float);
}

// out[m,n] = L'.R' with tiles of 128 x bn, `cluster` CTAs per tile - all but the first `whole` tiles, which get one each:
// where one CTA per tile leaves a last wave at most half full, cutting just its tiles in two shortens the wave by half
// (192 tiles on 148 SMs: one wave and a half instead of two).  swap: the operands exchange roles, the tile's
// rows are columns of the result.  ws: mid_workspace_bytes.  left_pitch: floats between the stored rows of left (0: they
// follow one another), a multiple of 4.
int launch_mid(int tl, int tr, uint64_t m, uint64_t n, uint64_t k, const float* left, const float* right, float* out, int bn,
               int cluster, uint64_t whole, int exact, int swap, int epilogue, float* ws, cudaStream_t stream, uint64_t left_pitch) {
  using namespace mid;
  Stored l{left, tl ? k : m, tl ? m : k, left_pitch ? left_pitch : tl ? m : k, false}, r{right, tr ? n : k, tr ? k : n, tr ? k : n, false};
  Padded copies[2] = {};
  int count = 0;
  for (Stored* s : {&l, &r}) {
    if (addressable(s->p, s->pitch)) continue;
    const uint64_t pitch = pad32(s->cols);
    copies[count++] = Padded{s->p, ws, s->rows, s->cols, pitch};
    s->p = ws;
    s->pitch = pitch;
    s->padded = true;
    ws += s->rows * pitch;
  }
  if (count) {
    const uint64_t va = copies[0].vecs(), v = va + (count > 1 ? copies[1].vecs() : 0);
    if ((v + 255) / 256 > 0x7fffffffull) return fail(POLAR_B200_ERR_UNSUPPORTED, "operand too large");
    int rc = launch("fmatmul_pad", pad_kernel, (unsigned)((v + 255) / 256), 256, 0, stream, copies[0], copies[1], va, v);
    if (rc) return rc;
  }
  int rc = POLAR_B200_OK;
  Params p = {};
  p.status = device_status_word(&rc);
  if (!p.status) return rc;
  p.wait_ns = wait_limit_ns(2000000000ull);
  p.out = out;
  p.pitch = (uint32_t)n;
  p.k = (uint32_t)k;
  p.vec_out = (n & 3) == 0 && aligned16(out);
  p.out_t = swap != 0;
  p.epilogue = (uint8_t)epilogue;
  p.m = (uint32_t)(swap ? n : m);
  p.n = (uint32_t)(swap ? m : n);
  p.tiles_m = (uint32_t)((p.m + BM - 1) / BM);
  p.slabs = (uint32_t)((k + BK - 1) / BK);
  p.cluster = (uint32_t)cluster;
  p.whole = (uint32_t)whole;
  // (32-column tiles replace the narrow kernels too, whose sums are better than FFMA tiles')
  // slabs of 32 terms summed in tensor memory, the rest in registers: `exact` is to stay below the error of FFMA sums
  p.chunk = !exact ? 8 : k < 512 || bn == 32 ? 1 : 2;
  if ((cluster != 1 && cluster != 2 && cluster != 4 && cluster != 8) || p.slabs < p.cluster) return fail(POLAR_B200_ERR_UNSUPPORTED, "fewer slabs than CTAs in a cluster");
  if ((uint64_t)p.tiles_m * ((p.n + bn - 1) / bn) * p.cluster > 0x7fffffffull) return fail(POLAR_B200_ERR_UNSUPPORTED, "too many tiles");
  // exchanged: right' plays the row operand - stored [k, n] is "row extent contiguous" - and left the column operand
  const Stored &a = swap ? r : l, &b = swap ? l : r;
  const bool a_mn = swap ? !tr : tl, b_mn = swap ? tl : !tr;
  switch (bn) {
    case 32: return launch_cfg<32>(a, b, a_mn, b_mn, p, k, stream);
    case 64: return launch_cfg<64>(a, b, a_mn, b_mn, p, k, stream);
    case 128: return launch_cfg<128>(a, b, a_mn, b_mn, p, k, stream);
  }
  return fail(POLAR_B200_ERR_INVALID, "tile width must be 32, 64 or 128");
}

}  // namespace polar_b200
