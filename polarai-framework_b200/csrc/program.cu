// Builtin programs: a list of builtin launches, prepared once and run many times.
//
// What a small program costs is not its arithmetic but its launches: on B200 about 2.5 us of host time
// each and 3 us of GPU time from one short kernel to the next.  Two things take them out:
//
//  - Two neighbouring short chains (or single elementwise builtins) over different element counts share a launch where
//    neither touches what the other writes.
//  - Consecutive elementwise builtins over the same element count become ONE launch (chain_kernel): each
//    thread carries four elements through the whole chain.  Every tensor a builtin of the chain names as its
//    result is still written, with the bits its own launch gives; what goes away is reading a
//    tensor back that the same pass has just computed or read (the four-builtin chain of
//    (a + b) * c / d -> sigmoid moves 32 instead of 44 bytes per element).
//  - From its third run on, a program of many short launches is replayed as a CUDA graph: one host call instead of 2 us
//    of host time per launch.  Programs of up to three steps, and programs with tensors of two million elements or
//    more, whose kernels outlast their launches, stay with launches: programmatic dependent launch overlaps them more
//    closely in a stream than in a graph (inference on 16 rows, two launches: 17.3 us against 19.9).  The 12-launch MLP step by its
//    largest tensor, as a graph and launched: 0.8 M elements 63.3 and 66.0 us, 2.1 M 120.8 and 119.1, 8.4 M 255.7 and
//    249.6; the ragged step takes 29 instead of 57 us of host time at the same 52 us in all.  The first two runs are
//    launched one by one, so that a program run once or twice never pays for the instantiation; a run under the caller's
//    own stream capture is always launched one by one.
#include <cstring>
#include <exception>
#include <memory>
#include <mutex>
#include <new>
#include <string>
#include <vector>

#include "elementwise_ops.cuh"

namespace polar_b200 {
// dispatch.cu: while a thread captures a program, its forks take this stream set instead of the device's
// shared one, which other threads may be using at the same time.
bool use_capture_side_stream(bool on);

namespace {

constexpr int kChainThreads = 128;
constexpr int kChainOps = 16;
constexpr int kChainInputs = 8;
constexpr uint8_t kPrevious = 0xff;   // operand = the result of the instruction before
constexpr uint8_t kNoSlot = 0xff;

enum Code : uint8_t { kFill, kCopy, kAdd, kMul, kDivide, kSigmoid, kLogLoss, kMulConcat, kRelu, kSigmoidGrad, kSigmoidLogLossGrad };

struct ChainOp {
  uint8_t code, a, b;      // operands: slot numbers (inputs first, then kept results), or kPrevious
  uint8_t result;          // slot of the result, or kNoSlot
  float s0, s1;            // fadd's scales, ffill's value
  const float* scalar;     // fmulconcat's factor, in device memory
  float* out;
};
struct ChainParams {
  uint64_t n;
  uint32_t inputs, ops;
  const float* in[kChainInputs];
  ChainOp op[kChainOps];
};

template <int CHAINS>
struct ChainLaunch {
  ChainParams chain[CHAINS];
  uint32_t first_blocks;
};

template <class Op>
__device__ __forceinline__ float4 map4(Op op, float4 a, float4 b) {
  return make_float4(op(a.x, b.x), op(a.y, b.y), op(a.z, b.z), op(a.w, b.w));
}

// A chain of elementwise builtins on one vector of four elements per thread.  HBM-bound for long vectors, one launch
// latency for short ones.  (Two vectors per thread halve the decoding and are no faster anywhere: 8.2 us against 6.6 at
// 2^20 elements, the same from 2^22 on.)
// Values live in shared memory, [slot][thread]: a thread only ever touches its own column, so there
// is no barrier, and consecutive lanes touch consecutive 16 bytes.
// Measured, four-builtin chain, 32 bytes per element: 2^20 elements 18.4 us as four launches, 6.6 us as one;
// 2^25 elements 158 us, 6.8 TB/s.
// CHAINS == 2: two short chains of different lengths that have nothing to do with each other, as the updates of two layers'
// weights; the second one's blocks follow the first one's.  (The step 999 x 301 x 514 x 7 55.0 -> 53.7 us.)
template <int CHAINS>
__global__ void __launch_bounds__(kChainThreads) chain_kernel(const __grid_constant__ ChainLaunch<CHAINS> l) {
  extern __shared__ float4 slots[];
  pdl_enter();
  const bool second = CHAINS == 2 && blockIdx.x >= l.first_blocks;
  const ChainParams& p = l.chain[second];
  const uint64_t e0 = ((uint64_t)(blockIdx.x - (second ? l.first_blocks : 0u)) * kChainThreads + threadIdx.x) * 4;
  if (e0 >= p.n) return;
  const bool full = e0 + 4 <= p.n;
  const int left = full ? 4 : (int)(p.n - e0);             // the last vector of an n that is no multiple of four
  float4* mine = slots + threadIdx.x;
#pragma unroll
  for (int first = 0; first < kChainInputs; first += 4) {  // four inputs' loads in flight at a time
    if (first >= (int)p.inputs) break;
    float4 v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (first + i >= (int)p.inputs) continue;
      const float* src = p.in[first + i] + e0;
      v[i] = full ? *reinterpret_cast<const float4*>(src)
                  : make_float4(src[0], left > 1 ? src[1] : 0.f, left > 2 ? src[2] : 0.f, 0.f);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (first + i < (int)p.inputs) mine[(first + i) * kChainThreads] = v[i];
  }
  float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
  for (uint32_t i = 0; i < p.ops; ++i) {
    const ChainOp& o = p.op[i];
    const float4 a = o.a == kPrevious ? r : mine[o.a * kChainThreads];
    const float4 b = o.b == kPrevious ? r : mine[o.b * kChainThreads];
    switch (o.code) {   // the same for all threads
      case kFill: r = map4(ew::FillOp{o.s0}, a, b); break;
      case kCopy: r = a; break;
      case kAdd: r = map4(ew::AddOp{o.s0, o.s1}, a, b); break;
      case kMul: r = map4(ew::MulOp{}, a, b); break;
      case kDivide: r = map4(ew::DivOp{}, a, b); break;
      case kSigmoid: r = map4(ew::SigmoidOp<true>{}, a, a); break;
      case kLogLoss: {
        auto hard = [](float y) { return y == 0.0f || y == 1.0f; };
        r = hard(b.x) && hard(b.y) && hard(b.z) && hard(b.w)
                ? make_float4(ew::logloss_binary(a.x, b.x), ew::logloss_binary(a.y, b.y), ew::logloss_binary(a.z, b.z),
                              ew::logloss_binary(a.w, b.w))
                : map4(ew::LogLossOp{}, a, b);
        break;
      }
      case kMulConcat: r = map4(ew::ScaleByFirstOp{*o.scalar}, a, a); break;
      case kRelu: r = map4(ew::ReluOp{}, a, a); break;
      case kSigmoidGrad: r = map4(ew::SigmoidGradOp{}, a, b); break;
      default: r = map4(ew::SigmoidLogLossGradOp{}, a, b); break;
    }
    if (o.result != kNoSlot) mine[o.result * kChainThreads] = r;
    float* dst = o.out + e0;
    if (full) {
      *reinterpret_cast<float4*>(dst) = r;
    } else {
      dst[0] = r.x;
      if (left > 1) dst[1] = r.y;
      if (left > 2) dst[2] = r.z;
    }
  }
}

// ---- host side

struct Op {                    // one builtin, its argument list owned by the program
  std::string name;
  std::vector<polar_b200_arg> args;
  std::vector<std::vector<uint64_t>> shapes;
};
struct Step {                  // one builtin, a chain, or two chains
  int op = -1;
  ChainParams chain = {}, second = {};   // (one elementwise builtin is a chain of one, for pairing)
  size_t smem = 0;
};
struct Program {
  std::vector<Op> ops;
  std::vector<Step> steps;
  const void* any_pointer = nullptr;
  void* workspace = nullptr;
  uint64_t workspace_bytes = 0;
  std::mutex mu;
  int runs = 0;
  bool short_launches = true;   // worth a graph
  bool graph_failed = false;
  cudaGraphExec_t graph = nullptr;
  uint64_t graph_launches = 0;
  unsigned long long graph_limit = 0;   // polar_b200_set_wait_limit_ns when the graph was made: its launches carry it
};

uint64_t elements(const polar_b200_tensor& t) {
  uint64_t n = 1;
  for (uint64_t d = 0; d < t.dims; ++d) n *= t.shape[d];
  return n;
}

// An elementwise builtin in the form the chain takes; false for anything else.
struct Elementwise {
  Code code;
  uint64_t n;
  const float* in[2] = {nullptr, nullptr};
  const float* scalar = nullptr;
  float s0 = 0.f, s1 = 0.f;
  float* out;
};
bool elementwise(const Op& op, Elementwise* e) {
  struct Form { const char* name; Code code; const char* args; };
  static const Form forms[] = {
      {"ffill", kFill, "fT"}, {"fcopy", kCopy, "TT"}, {"fadd", kAdd, "TfTfT"}, {"fmul", kMul, "TTT"}, {"fdivide", kDivide, "TTT"},
      {"fsigmoid", kSigmoid, "TT"}, {"flogloss", kLogLoss, "TTT"}, {"fmulconcat", kMulConcat, "TTT"}, {"frelu", kRelu, "TT"},
      {"fsigmoid_grad", kSigmoidGrad, "TTT"}, {"fsigmoid_logloss_grad", kSigmoidLogLossGrad, "TTT"}};
  for (const Form& f : forms) {
    if (op.name != f.name) continue;
    if (op.args.size() != std::strlen(f.args)) return false;
    const polar_b200_arg& result = op.args.back();
    if (!result.is_tensor) return false;
    e->code = f.code;
    e->out = result.tensor.data;
    e->n = elements(result.tensor);
    if (e->n == 0 || e->n > (1ull << 40) || !e->out || !aligned16(e->out)) return false;
    int tensors = 0, scalars = 0;
    for (size_t i = 0; i + 1 < op.args.size(); ++i) {
      const polar_b200_arg& a = op.args[i];
      if ((f.args[i] == 'T') != (a.is_tensor != 0)) return false;
      if (!a.is_tensor) {
        (scalars++ == 0 ? e->s0 : e->s1) = a.scalar;
      } else if (f.code == kMulConcat && tensors == 0 && !e->scalar) {
        if (elements(a.tensor) < 1 || !a.tensor.data) return false;
        e->scalar = a.tensor.data;
      } else {
        if (elements(a.tensor) != e->n || !a.tensor.data || !aligned16(a.tensor.data)) return false;
        e->in[tensors++] = a.tensor.data;
      }
    }
    return !(e->scalar && e->scalar >= e->out && e->scalar < e->out + e->n);
  }
  return false;
}

// Builds chains.  An instruction joins the open one when it covers the same number of elements and
// nothing it touches overlaps what the chain touches other than as the same whole tensor: a thread
// sees its own four elements only.
class ChainBuilder {
public:
  bool add(const Elementwise& e) {
    if (!ops_.empty() && (e.n != n_ || ops_.size() == kChainOps || !compatible(e))) return false;
    size_t fresh = e.in[0] && find(e.in[0]) < 0;
    fresh += e.in[1] && e.in[1] != e.in[0] && find(e.in[1]) < 0;
    if (inputs_.size() + fresh > kChainInputs) return false;
    n_ = e.n;
    Entry t{e, {-1, -1}};
    for (int i = 0; i < 2; ++i) {
      if (!e.in[i]) continue;
      int v = find(e.in[i]);
      if (v < 0) {
        inputs_.push_back(e.in[i]);
        values_.push_back({e.in[i], false, (int)inputs_.size() - 1});
        v = (int)values_.size() - 1;
      }
      t.operand[i] = v;
    }
    values_.push_back({e.out, true, (int)ops_.size()});
    ops_.push_back(t);
    return true;
  }
  size_t size() const { return ops_.size(); }
  Step finish() {
    Step s;
    ChainParams& p = s.chain;
    p.n = n_;
    p.inputs = (uint32_t)inputs_.size();
    p.ops = (uint32_t)ops_.size();
    for (size_t i = 0; i < inputs_.size(); ++i) p.in[i] = inputs_[i];
    // a result gets a slot when something later than the next instruction reads it
    std::vector<int> slot_of(ops_.size(), -1);
    size_t slots = inputs_.size();
    for (size_t i = 0; i < ops_.size(); ++i)
      for (int v : ops_[i].operand)
        if (v >= 0 && values_[v].computed && values_[v].index + 1 != (int)i) slot_of[values_[v].index] = 0;
    for (int& n : slot_of)
      if (n == 0) n = (int)slots++;
    for (size_t i = 0; i < ops_.size(); ++i) {
      const Entry& t = ops_[i];
      ChainOp& o = p.op[i];
      o.code = t.e.code;
      o.s0 = t.e.s0;
      o.s1 = t.e.s1;
      o.scalar = t.e.scalar;
      o.out = t.e.out;
      o.result = slot_of[i] < 0 ? kNoSlot : (uint8_t)slot_of[i];
      auto operand = [&](int v) -> uint8_t {
        if (v < 0) return kPrevious;                       // no such operand: any value will do
        const Value& val = values_[v];
        if (!val.computed) return (uint8_t)val.index;
        return val.index + 1 == (int)i ? kPrevious : (uint8_t)slot_of[val.index];
      };
      o.a = operand(t.operand[0]);
      o.b = t.operand[1] < 0 ? o.a : operand(t.operand[1]);
    }
    s.smem = slots * kChainThreads * sizeof(float4);
    *this = ChainBuilder();
    return s;
  }

private:
  struct Entry { Elementwise e; int operand[2]; };
  struct Value { const float* tensor; bool computed; int index; };   // index: input number, or instruction number
  // The value the tensor holds at this point of the chain.
  int find(const float* tensor) const {
    for (int i = (int)values_.size() - 1; i >= 0; --i)
      if (values_[i].tensor == tensor) return i;
    return -1;
  }
  static bool overlap(const float* a, uint64_t na, const float* b, uint64_t nb) { return a < b + nb && b < a + na; }
  bool compatible(const Elementwise& e) const {
    auto partial = [&](const float* a, const float* b) { return a && b && a != b && overlap(a, n_, b, n_); };
    for (const Value& v : values_) {
      if (partial(e.in[0], v.tensor) || partial(e.in[1], v.tensor) || partial(e.out, v.tensor)) return false;
      // fmulconcat's factor is read by every thread: nothing in the chain may write it
      if (e.scalar && v.computed && overlap(e.scalar, 1, v.tensor, n_)) return false;
    }
    for (const Entry& t : ops_)
      if (t.e.scalar && overlap(t.e.scalar, 1, e.out, n_)) return false;
    return true;
  }
  uint64_t n_ = 0;
  std::vector<const float*> inputs_;
  std::vector<Value> values_;
  std::vector<Entry> ops_;
};

// Whether two chains are short - longer ones outlast a launch, and a single builtin's own kernel has more loads in
// flight - and neither touches a tensor that the other one writes: then their order does not matter.  Two fadds of n and n / 2
// elements, together against apart: n = 2^18 2.5 against 4.6 us, 2^19 2.9 and 4.5, 2^20 4.4 and 4.6, 2^21 7.7 and 5.3.
constexpr uint64_t kPairElements = 1ull << 19;
bool may_pair(const ChainParams& a, const ChainParams& b) {
  if (a.n > kPairElements || b.n > kPairElements) return false;
  auto writes_into = [](const ChainParams& w, const ChainParams& o) {
    for (uint32_t i = 0; i < w.ops; ++i) {
      auto hits = [&](const float* t, uint64_t n) { return t && w.op[i].out < t + n && t < w.op[i].out + w.n; };
      for (uint32_t j = 0; j < o.inputs; ++j)
        if (hits(o.in[j], o.n)) return true;
      for (uint32_t j = 0; j < o.ops; ++j)
        if (hits(o.op[j].out, o.n) || hits(o.op[j].scalar, 1)) return true;
    }
    return false;
  };
  return !writes_into(a, b) && !writes_into(b, a);
}

void plan(Program* p) {
  ChainBuilder chain;
  int first = -1;                                          // the builtin a one-instruction chain stands for
  auto flush = [&] {
    if (chain.size() == 0) return;
    Step s = chain.finish();
    if (s.chain.ops == 1) s.op = first;                    // (its own kernel, unless it finds a partner)
    if (!p->steps.empty()) {
      Step& last = p->steps.back();
      if (last.chain.ops && !last.second.ops && may_pair(last.chain, s.chain)) {
        last.op = -1;
        last.second = s.chain;
        if (s.smem > last.smem) last.smem = s.smem;
        return;
      }
    }
    p->steps.push_back(s);
  };
  for (size_t i = 0; i < p->ops.size(); ++i) {
    Elementwise e;
    const bool ok = elementwise(p->ops[i], &e);
    if (!ok || !chain.add(e)) {
      flush();
      if (!ok || !chain.add(e)) {
        Step s;
        s.op = (int)i;
        p->steps.push_back(s);
        continue;
      }
    }
    if (chain.size() == 1) first = (int)i;
  }
  flush();
}

int run_steps(Program* p, cudaStream_t stream) {
  for (const Step& s : p->steps) {
    int rc;
    if (s.op >= 0) {
      const Op& op = p->ops[s.op];
      rc = polar_b200_launch_by_name(op.name.c_str(), op.args.data(), op.args.size(), p->workspace, p->workspace_bytes, stream);
    } else {
      auto blocks = [](uint64_t n) { return ((n + 3) / 4 + kChainThreads - 1) / kChainThreads; };
      const uint64_t first = blocks(s.chain.n), second = s.second.ops ? blocks(s.second.n) : 0;
      if (first + second > 0x7fffffffull) return fail(POLAR_B200_ERR_INVALID, "element count too large");
      rc = second ? launch("two chains of elementwise builtins", chain_kernel<2>, (unsigned)(first + second), kChainThreads, s.smem,
                           stream, ChainLaunch<2>{{s.chain, s.second}, (uint32_t)first})
                  : launch("chain of elementwise builtins", chain_kernel<1>, (unsigned)first, kChainThreads, s.smem, stream,
                           ChainLaunch<1>{{s.chain}, (uint32_t)first});
    }
    if (rc) return rc;
  }
  return POLAR_B200_OK;
}

uint64_t kernel_nodes(cudaGraph_t g) {
  size_t nodes = 0;
  cudaGraphGetNodes(g, nullptr, &nodes);
  std::unique_ptr<cudaGraphNode_t[]> list(new (std::nothrow) cudaGraphNode_t[nodes]);
  if (!list || cudaGraphGetNodes(g, list.get(), &nodes) != cudaSuccess) return 0;
  uint64_t kernels = 0;
  for (size_t i = 0; i < nodes; ++i) {
    cudaGraphNodeType type;
    if (cudaGraphNodeGetType(list[i], &type) == cudaSuccess && type == cudaGraphNodeTypeKernel) kernels++;
  }
  return kernels;
}

// Captures one pass on a stream of the program's own and instantiates it.  Thread-local capture mode: other
// threads may go on launching and allocating.
bool make_graph(Program* p) {
  static std::mutex one_at_a_time;                         // the capture side stream is one per device
  std::lock_guard<std::mutex> guard(one_at_a_time);
  RelaxedCaptureMode relaxed;
  cudaStream_t s = nullptr;
  if (cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  bool ok = false;
  if (use_capture_side_stream(true) && cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
    const int rc = run_steps(p, s);
    cudaGraph_t g = nullptr;
    const bool ended = cudaStreamEndCapture(s, &g) == cudaSuccess && g;
    if (rc == POLAR_B200_OK && ended) {
      ok = cudaGraphInstantiate(&p->graph, g, 0) == cudaSuccess;
      p->graph_launches = kernel_nodes(g);
      count_launch(0 - p->graph_launches);                 // captured, not launched
    }
    if (g) cudaGraphDestroy(g);
  }
  use_capture_side_stream(false);
  cudaGetLastError();
  cudaStreamDestroy(s);
  return ok;
}

}  // namespace
}  // namespace polar_b200

using namespace polar_b200;

extern "C" {

int polar_b200_program_create(const polar_b200_op* ops, uint64_t count, void* workspace, uint64_t workspace_bytes,
                              void** program) {
  clear_error();
  if (!program || (count && !ops)) return fail(POLAR_B200_ERR_INVALID, "null program or operation list");
  *program = nullptr;
  try {
    std::unique_ptr<Program> p(new Program);
    for (uint64_t i = 0; i < count; ++i) {
      const polar_b200_op& o = ops[i];
      if (!o.name || (o.argc && !o.args)) return fail(POLAR_B200_ERR_INVALID, "null kernel name or argument list");
      Op op;
      op.name = o.name;
      op.args.assign(o.args, o.args + o.argc);
      op.shapes.resize(o.argc);
      for (uint64_t a = 0; a < o.argc; ++a) {
        if (!o.args[a].is_tensor) continue;
        const polar_b200_tensor& t = o.args[a].tensor;
        if (t.dims && !t.shape) return fail(POLAR_B200_ERR_INVALID, "tensor without a shape");
        op.shapes[a].assign(t.shape, t.shape + t.dims);
        if (!p->any_pointer) p->any_pointer = t.data;
        if (elements(t) >= 2000000) p->short_launches = false;
      }
      p->ops.push_back(std::move(op));
      Op& kept = p->ops.back();
      for (uint64_t a = 0; a < o.argc; ++a)
        if (kept.args[a].is_tensor) kept.args[a].tensor.shape = kept.shapes[a].data();
    }
    p->workspace = workspace;
    p->workspace_bytes = workspace_bytes;
    plan(p.get());
    *program = p.release();
  } catch (const std::exception&) {                        // (no exception may leave a C entry)
    return fail(POLAR_B200_ERR_INVALID, "out of host memory");
  }
  return POLAR_B200_OK;
}

static int run_program(Program* p, cudaStream_t st) {
  if (p->steps.size() > 3 && p->short_launches) {
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    // (a query on the legacy stream fails while some other stream is capturing: then launch one by one)
    const bool eager = cudaStreamIsCapturing(st, &capturing) != cudaSuccess || capturing != cudaStreamCaptureStatusNone;
    if (eager) {
      cudaGetLastError();
    } else {
      std::lock_guard<std::mutex> guard(p->mu);
      if (p->graph && p->graph_limit != wait_limit_ns(0)) {
        cudaGraphExecDestroy(p->graph);                    // (a run in flight is not disturbed)
        p->graph = nullptr;
      }
      if (p->runs < 2) {
        ++p->runs;
      } else if (!p->graph && !p->graph_failed) {
        p->graph_limit = wait_limit_ns(0);
        p->graph_failed = !make_graph(p);
      }
      if (p->graph) {
        cudaError_t e = cudaGraphLaunch(p->graph, st);
        if (e != cudaSuccess) {
          cudaGetLastError();
          return fail(POLAR_B200_ERR_CUDA, "cudaGraphLaunch", e);
        }
        count_launch(p->graph_launches);
        return POLAR_B200_OK;
      }
    }
  }
  return run_steps(p, st);
}

int polar_b200_program_run(void* program, void* stream) {
  clear_error();
  Program* p = static_cast<Program*>(program);
  if (!p) return fail(POLAR_B200_ERR_INVALID, "null program");
  LaunchDeviceScope on(stream, p->any_pointer);
  try {
    return run_program(p, as_stream(stream));
  } catch (const std::exception&) {
    return fail(POLAR_B200_ERR_INVALID, "out of host memory");
  }
}

uint64_t polar_b200_program_steps(const void* program) {
  return program ? static_cast<const Program*>(program)->steps.size() : 0;
}

void polar_b200_program_destroy(void* program) {
  Program* p = static_cast<Program*>(program);
  if (!p) return;
  if (p->graph) cudaGraphExecDestroy(p->graph);
  delete p;
}

}  // extern "C"
