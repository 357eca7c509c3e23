// Arithmetic of the elementwise builtins, one functor each, shared by the single-builtin kernels
// (elementwise.cu) and the kernel that runs a whole chain of them in one pass (program.cu), so that a
// chain gives the bits of its builtins launched one by one.
#pragma once
#include "common.cuh"

namespace polar_b200 {
namespace ew {

struct FillOp {
  float v;
  __device__ __forceinline__ float operator()(float, float) const { return v; }
};
struct CopyOp {
  __device__ __forceinline__ float operator()(float a, float) const { return a; }
};
struct AddOp {
  float sa, sb;
  __device__ __forceinline__ float operator()(float a, float b) const {
    return __fadd_rn(__fmul_rn(a, sa), __fmul_rn(b, sb));
  }
};
struct MulOp {
  __device__ __forceinline__ float operator()(float a, float b) const { return __fmul_rn(a, b); }
};
struct DivOp {
  __device__ __forceinline__ float operator()(float a, float b) const { return __fdiv_rn(a, b); }
};
template <bool CLAMP>
struct SigmoidOp {
  __device__ __forceinline__ float operator()(float x, float) const {
    if (CLAMP) return sigmoid_clamped(x);
    return __fdiv_rn(1.0f, __fadd_rn(1.0f, expf(-x)));
  }
};
struct LogLossOp {
  // out = fl(fl(-y * log(p + eps)) - fl((1 - y) * log(1 - p + eps))), eps = 1e-5: the general
  // form, two full-precision logarithms (scalar fallback kernel, and soft labels in the
  // vector kernel below).
  __device__ __forceinline__ float operator()(float p, float y) const {
    const float eps = 1e-5f;
    float t0 = __fmul_rn(-y, logf(__fadd_rn(p, eps)));
    float t1 = __fmul_rn(__fadd_rn(1.0f, -y), logf(__fadd_rn(__fadd_rn(1.0f, -p), eps)));
    return __fadd_rn(t0, -t1);
  }
};
// flogloss for labels that are exactly 0 or 1 (what LogLoss is fed): one of the two weights
// -y and 1-y is then an exact zero, and its product with a logarithm is a signed zero, NaN
// or NaN - whatever the logarithm's low bits are.  So only the OTHER logarithm needs full
// precision; the one under the zero weight comes from the special-function unit
// (lg2.approx), which returns the same NaN / -inf / +inf classes and the same sign.  (The
// sign of that zero is only visible when the full-precision term is itself zero, i.e. its
// argument is exactly 1; the two arguments sum to 1 + 2 eps, so the other one is then about
// 2e-5, far from where an approximate logarithm could have the wrong sign.)  Same bits as
// the two-logarithm form at roughly 60 % of its instructions - two full logf per element make
// the builtin issue-bound instead of HBM-bound.  Branch-free, so the unrolled elements
// interleave.
__device__ __forceinline__ float logloss_binary(float p, float y) {
  const float eps = 1e-5f;
  const float a0 = __fadd_rn(p, eps);
  const float a1 = __fadd_rn(__fadd_rn(1.0f, -p), eps);
  const float w0 = -y, w1 = __fadd_rn(1.0f, -y);
  const bool first = (w1 == 0.0f);                       // y == 1: log(a0) carries the result
  const float fine = logf(first ? a0 : a1);
  const float coarse = __logf(first ? a1 : a0);
  const float t0 = __fmul_rn(w0, first ? fine : coarse);
  const float t1 = __fmul_rn(w1, first ? coarse : fine);
  return __fadd_rn(t0, -t1);
}
// Extended builtin: the three launches the reference's Sigmoid derivative compiles to
// (SigmoidOperationInternal.cpp:107-135: fadd(ones,1,s,-1) -> fmul(.,s) -> fmul(grad,.))
// in one pass, with the same three roundings, so the result is bit-identical.
struct SigmoidGradOp {
  __device__ __forceinline__ float operator()(float g, float s) const {
    return sigmoid_grad_chain(g, s);
  }
};
// Extended builtin: dZ = dL/dP * dP/dZ for LogLoss on a Sigmoid output, the seven launches
// the reference's derivatives compile to (LogLossOperationInternal.cpp:127-170:
// fadd(p,1,y,-1), fmul(p,p), fadd(p,1,pp,-1), fdivide; SigmoidOperationInternal.cpp:107-135:
// fadd(ones,1,p,-1), fmul(.,p), fmul(dLdP,.)) in one pass with the same seven roundings.
struct SigmoidLogLossGradOp {
  __device__ __forceinline__ float operator()(float p, float y) const {
    const float pmy = __fadd_rn(__fmul_rn(p, 1.0f), __fmul_rn(y, -1.0f));
    const float pp = __fmul_rn(p, p);
    const float den = __fadd_rn(__fmul_rn(p, 1.0f), __fmul_rn(pp, -1.0f));
    const float dldp = __fdiv_rn(pmy, den);
    return sigmoid_grad_chain(dldp, p);
  }
};
struct ScaleByFirstOp {  // fmulconcat: the scalar is read once per thread
  float g;
  __device__ __forceinline__ float operator()(float l, float) const { return __fmul_rn(g, l); }
};
struct ReluOp {
  // ordered compare: NaN gives 0, as the reference's select does
  __device__ __forceinline__ float operator()(float v, float) const { return v > 0.0f ? v : 0.0f; }
};

}  // namespace ew
}  // namespace polar_b200
