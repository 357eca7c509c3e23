// Shared host-side helpers of the kernel library: status recording, launch
// accounting and launch-geometry constants for B200.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/polar_b200.h"

namespace polar_b200 {

// B200: 148 SMs.  Grids of persistent (grid-stride) kernels are sized as a
// multiple of the SM count the device reports.
int sm_count();

// Records `msg` (and the CUDA error text, if any) as the calling thread's last
// error and returns `status`.
int fail(int status, const char* msg, cudaError_t err = cudaSuccess);
void clear_error();
void count_launch(uint64_t n = 1);

// Checks the launch that was just issued.
inline int check_launch(const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(POLAR_B200_ERR_CUDA, what, e);
  count_launch();
  return POLAR_B200_OK;
}

// ---- status words and wait limits of the bounded device-side waits -----------------------
// One status word per device, in pinned host memory every device can write (so the host reads
// it without a CUDA call, even while a kernel is still running).  A kernel whose wait gives
// up stores its code with atomicCAS(word, 0, code): the first code since the last clear stays.
// Returns the device-visible pointer of the CURRENT device's word (nullptr + *rc on failure).
int* device_status_word(int* rc);
int device_status_read(int device);     // device < 0: the first non-zero word of any device
void device_status_clear_all();
// The host's wait bound in nanoseconds, or `fallback` when none was set.
unsigned long long wait_limit_ns(unsigned long long fallback);

inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// Every launching entry point opens one of these.  A kernel must be launched with the device
// of its stream current; a caller that drives several GPUs from one thread (or a plugin that
// enumerated them) may arrive with another device current.  With a real stream handle the
// stream's own device is made current for the duration of the call; with the NULL (legacy
// default) stream, which every device has, the device that owns `ptr` (one of the call's
// device buffers) decides.  The caller's current device is put back on exit.  Costs two
// runtime queries per launch when nothing needs switching.
class LaunchDeviceScope {
public:
  LaunchDeviceScope(void* stream, const void* ptr) {
    int want = -1, cur = -1;
    if (cudaGetDevice(&cur) != cudaSuccess) {
      cudaGetLastError();
      return;
    }
    if (stream && stream != (void*)cudaStreamLegacy && stream != (void*)cudaStreamPerThread) {
      // A stream under capture is left alone (only the capture-status query is allowed on it
      // without risk to the capture): whoever captures has made the stream's device current.
      cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
      if (cudaStreamIsCapturing(as_stream(stream), &capturing) != cudaSuccess) {
        cudaGetLastError();
        return;
      }
      if (capturing != cudaStreamCaptureStatusNone) return;
      if (cudaStreamGetDevice(as_stream(stream), &want) != cudaSuccess) {
        cudaGetLastError();
        return;
      }
    } else if (ptr) {
      cudaPointerAttributes attr;
      if (cudaPointerGetAttributes(&attr, ptr) != cudaSuccess) {
        cudaGetLastError();
        return;
      }
      if (attr.type != cudaMemoryTypeDevice && attr.type != cudaMemoryTypeManaged) return;
      want = attr.device;
    }
    if (want >= 0 && want != cur && cudaSetDevice(want) == cudaSuccess) {
      prev_ = cur;
      switched_ = true;
    }
  }
  ~LaunchDeviceScope() {
    if (switched_ && cudaSetDevice(prev_) != cudaSuccess) cudaGetLastError();
  }
  LaunchDeviceScope(const LaunchDeviceScope&) = delete;
  LaunchDeviceScope& operator=(const LaunchDeviceScope&) = delete;

private:
  int prev_ = -1;
  bool switched_ = false;
};

// While it lives, the calling thread may allocate and create streams and graphs although another thread captures in the
// global mode (torch.cuda.graph's default): in that mode such a call from any thread fails and ends the other's capture with
// an error.  None of the calls that it is used for touches what that thread captures.
struct RelaxedCaptureMode {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  RelaxedCaptureMode() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~RelaxedCaptureMode() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

// ---- scratch ------------------------------------------------------------------------------
// Device memory for the length of one launch sequence, when the caller hands in no workspace:
// from a pool of the library's own (one per device, made on first use), so that blocks survive a
// synchronisation.  The device's default pool gives everything back at each one, and the next
// call pays for mapping it again: 0.45 ms on B200, thirteen times what a 1024^3 product takes.
// The pool keeps at most kScratchKeepBytes across a synchronisation; polar_b200_trim_scratch
// gives the rest back too.  Stream-ordered, so it is safe with any number of threads and streams.
constexpr uint64_t kScratchKeepBytes = 256ull << 20;
cudaError_t scratch_alloc(void** p, uint64_t bytes, cudaStream_t stream);
inline cudaError_t scratch_free(void* p, cudaStream_t stream) {
  RelaxedCaptureMode relaxed;
  return cudaFreeAsync(p, stream);
}

#ifdef __CUDACC__
// ---- programmatic dependent launch -------------------------------------------------------------
// Kernels of a step follow one another on one stream, each a few microseconds long, and the gap
// between two of them is as long as the small ones.  launch() lets a kernel's CTAs be set up
// while the kernel before it drains; in return every kernel launched this way calls
// pdl_enter() before its first access to global memory, which waits until everything earlier in
// the stream has finished and written its results.  Measured on B200 for back-to-back kernels of
// 2^14 elements: 3.06 us each without, 1.97 us with (the host's launch rate).
// "Before its first access" is something the compiler has to keep to as well, since the kernel before may still be writing
// what this one reads.  So no pointer of such a kernel is __restrict__ (which would promise that nobody writes the data
// while the kernel runs, and allow loads through the read-only path and above the wait), and loads and stores with a
// cache hint are the volatile ones below instead of the intrinsics.
__device__ __forceinline__ void pdl_enter() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Streaming (evict-first) loads and stores of data that is touched once; a load from L2, past L1.
__device__ __forceinline__ float ld_stream(const float* p) {
  float v;
  asm volatile("ld.global.cs.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ float4 ld_stream(const float4* p) {
  float4 v;
  asm volatile("ld.global.cs.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_stream(float4* p, float4 v) {
  asm volatile("st.global.cs.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
__device__ __forceinline__ float ld_l2(const float* p) {
  float v;
  asm volatile("ld.global.cg.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
  return v;
}

// `cluster`: CTAs per cluster along y (1: no clusters).
template <typename... P, typename... A>
int launch_clusters(const char* what, void (*kernel)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t stream,
                    unsigned cluster, A... args) {
  cudaLaunchConfig_t c = {};
  c.gridDim = grid;
  c.blockDim = dim3(threads);
  c.dynamicSmemBytes = smem;
  c.stream = stream;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = at[1].val.clusterDim.z = 1;
  at[1].val.clusterDim.y = cluster;
  c.attrs = at;
  c.numAttrs = cluster > 1 ? 2 : 1;
  cudaError_t e = cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(POLAR_B200_ERR_CUDA, what, e);
  }
  count_launch();
  return POLAR_B200_OK;
}
template <typename... P, typename... A>
int launch(const char* what, void (*kernel)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t stream,
           A... args) {
  return launch_clusters(what, kernel, grid, threads, smem, stream, 1, args...);
}

// ---- clusters: the CTA's rank, the two halves of the cluster barrier, a read of another CTA's shared memory
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ float ld_cluster(const float* p, uint32_t rank) {
  uint32_t remote;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(remote) : "memory");
  return v;
}
__device__ __forceinline__ double ld_cluster(const double* p, uint32_t rank) {
  uint32_t remote;
  double v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(remote) : "memory");
  return v;
}

// fsigmoid's arithmetic, shared by the elementwise builtin and the fused matmul
// epilogue so that both give the same bits: r = 1/(1+exp(-x)), then the reference's
// clamp to [1e-5, 1-1e-5] (opencl/kernels.h:141-156 of the reference).
__device__ __forceinline__ float sigmoid_clamped(float x) {
  // Six instructions, two of them on the special-function unit: ex2.approx of -x * log2 e, 1 + e,
  // rcp.approx, and the clamp as one min and one max.  In the tensor-core epilogue, which cannot
  // overlap the next tile's k loop with 256-row tiles, the sigmoid is a large part of the drain,
  // and a dozen instructions per element (IEEE reciprocal, compare-and-select clamp) made the
  // drain issue-bound.
  //  - Error: ex2.approx is good to 2 ulp, the product -x * log2 e adds |x| * 6e-8 relative to the
  //    exponential (at most 8e-7 where it still matters: |x| < 11.6, beyond which the clamp takes
  //    over), rcp.approx 1 ulp: within the 1e-5 the builtin is held to, by a factor 10.
  //  - The clamp: r lies in [0, 1], so the reference's "|r - 1| < eps -> 1 - eps, else |r| < eps
  //    -> eps" is min(r, fl(1 - eps)) followed by max(., eps); the .NaN forms keep a NaN a NaN,
  //    as the reference's comparisons (all false) do.
  const float eps = 1e-5f;
  const float hi = 1.0f - eps;   // folded at compile time, the same float as fadd(1, -eps)
  float d = __fadd_rn(1.0f, __expf(-x)), r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
  asm("min.NaN.f32 %0, %0, %1;" : "+f"(r) : "f"(hi));
  asm("max.NaN.f32 %0, %0, %1;" : "+f"(r) : "f"(eps));
  return r;
}
// The reference's Sigmoid derivative chain on one element, with its three roundings:
// fadd(ones,1,s,-1) -> fmul(.,s) -> fmul(grad,.)  (SigmoidOperationInternal.cpp:107-135).
__device__ __forceinline__ float sigmoid_grad_chain(float g, float s) {
  float one_minus = __fadd_rn(__fmul_rn(1.0f, 1.0f), __fmul_rn(s, -1.0f));
  return __fmul_rn(g, __fmul_rn(one_minus, s));
}
#endif

}  // namespace polar_b200
