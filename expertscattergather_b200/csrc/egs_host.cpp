// Native host path of the package: tensor-level operators, autograd functions and the explicit training step over the C ABI
// of libegs_b200.so.  Python (ops.py, kernels.py, torch_interface.py, step.py) only parses arguments and calls in here.
//
// Why it is native: a training step of a small block is eight to ten kernels of 5-30 us, and issuing them from Python costs
// 400-570 us per step (argument handling, ctypes marshalling, Python autograd functions, stream contexts), several times the
// device time.  Issued from here a step of a tiny float32 block takes 105 us, device time included, against 420 us from Python.
//
// Conventions, shared by everything in this file:
//   * buffers (outputs, workspaces, gradients) come from torch's caching allocator on the CURRENT stream; work that runs on
//     the helper stream is forked from it and joined to it before the call returns, so stream order on the current stream
//     covers every buffer;
//   * nothing synchronises with the device (the first call on a device waits for a 4-byte fill on a stream of its own);
//   * one status word per device (see egs_b200.h) with a mapped host mirror that kernels write when they report invalid
//     results: every operator call looks at the mirror first and raises.
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/extension.h>

#include <ATen/core/dispatch/Dispatcher.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>
#include <dlfcn.h>

#include <array>
#include <atomic>
#include <mutex>
#include <optional>
#include <stdexcept>
#include <string>

#include "../../include/egs_b200.h"

namespace {

using at::Tensor;
using OptTensor = std::optional<Tensor>;

// ---- the C ABI, resolved from the library instance ctypes has loaded ---------------------------------------------------
struct Api {
#define EGS_API(X)                                                                                                        \
  X(egs_status_string) X(egs_last_cuda_error) X(egs_gather_gemm_bias) X(egs_gemm_scatter_bias) X(egs_gemm_scatter_prepared) \
  X(egs_scatter_workspace_bytes) X(egs_dweight) X(egs_dweight_prezeroed) X(egs_dw_workspace_bytes)                          \
  X(egs_gather_scatter_pair) X(egs_fused_pair_eligible) X(egs_route_topk) X(egs_index_csr) X(egs_index_csr_scratch_bytes)   \
  X(egs_fill_zero) X(egs_set_status_mirror) X(egs_expert_row_sum)
#define EGS_FIELD(name) decltype(&::name) name = nullptr;
  EGS_API(EGS_FIELD)
#undef EGS_FIELD
  bool loaded = false;
} api;

void init(const std::string& path) {
  if (api.loaded) return;
  void* h = dlopen(path.c_str(), RTLD_NOW | RTLD_LOCAL);
  if (!h) throw std::runtime_error(std::string("cannot load ") + path + ": " + dlerror());
#define EGS_RESOLVE(name)                                                          \
  api.name = reinterpret_cast<decltype(api.name)>(dlsym(h, #name));                \
  if (!api.name) throw std::runtime_error("missing symbol " #name " in " + path);
  EGS_API(EGS_RESOLVE)
#undef EGS_RESOLVE
  api.loaded = true;
}

[[noreturn]] void value_error(const std::string& s) { throw py::value_error(s); }

void check(int rc, const char* what) {
  if (rc == EGS_OK) return;
  std::string text = std::string(what) + ": " + api.egs_status_string(rc);
  if (rc == EGS_ERR_CUDA) text += std::string(": ") + api.egs_last_cuda_error();
  if (rc == EGS_ERR_INVALID_ARGUMENT || rc == EGS_ERR_UNSUPPORTED || rc == EGS_ERR_TOO_LARGE) value_error(text);
  throw std::runtime_error(text);
}

// ---- module-wide defaults (set_precision / set_path of ops.py) -----------------------------------------------------------
std::atomic<int> g_precision{EGS_PREC_STRICT}, g_path{EGS_PATH_AUTO};
std::atomic<bool> g_debug{false};
void configure(int precision, int path, bool debug) {
  g_precision = precision;
  g_path = path;
  g_debug = debug;
}
int prec_of(int p) { return p >= 0 ? p : g_precision.load(std::memory_order_relaxed); }
int path_of(int p) { return p >= 0 ? p : g_path.load(std::memory_order_relaxed); }

// ---- per-device state: status word, its host mirror, the helper stream ---------------------------------------------------
constexpr int kMaxDevices = 64;
struct DeviceState {
  Tensor word;                                  // int32[1] on the device
  volatile int32_t* mirror = nullptr;           // mapped host memory, written by kernels that report invalid results
  std::optional<c10::cuda::CUDAStream> side;
};
std::array<std::atomic<DeviceState*>, kMaxDevices> g_devices{};
std::mutex g_devices_mutex;

DeviceState& device_state(int idx) {
  TORCH_CHECK(idx >= 0 && idx < kMaxDevices, "device index out of range");
  if (DeviceState* s = g_devices[idx].load(std::memory_order_acquire)) return *s;
  std::lock_guard<std::mutex> lock(g_devices_mutex);
  if (DeviceState* s = g_devices[idx].load(std::memory_order_acquire)) return *s;
  c10::cuda::CUDAGuard guard(static_cast<c10::DeviceIndex>(idx));
  // The first call on a device may come while this or another thread captures a graph: the allocations are allowed then, and the
  // word is neither the graph's memory nor zeroed by a node of it.
  c10::cuda::CUDAStreamCaptureModeGuard relaxed(cudaStreamCaptureModeRelaxed);
  auto ok = [](cudaError_t e, const char* what) {
    if (e != cudaSuccess) throw std::runtime_error(std::string(what) + ": " + cudaGetErrorString(e));
  };
  void *host = nullptr, *word = nullptr;
  cudaStream_t once = nullptr;
  ok(cudaHostAlloc(&host, sizeof(int32_t), cudaHostAllocMapped | cudaHostAllocPortable), "cudaHostAlloc");
  ok(cudaMalloc(&word, sizeof(int32_t)), "cudaMalloc");
  ok(cudaStreamCreateWithFlags(&once, cudaStreamNonBlocking), "cudaStreamCreate");
  ok(cudaMemsetAsync(word, 0, sizeof(int32_t), once), "cudaMemsetAsync");
  ok(cudaStreamSynchronize(once), "cudaStreamSynchronize");
  cudaStreamDestroy(once);
  *static_cast<volatile int32_t*>(host) = 0;
  auto* s = new DeviceState;                    // lives as long as the process, like the device's context
  s->word = at::from_blob(word, {1}, at::TensorOptions().dtype(at::kInt).device(at::kCUDA, idx));
  s->mirror = static_cast<volatile int32_t*>(host);
  check(api.egs_set_status_mirror(s->word.data_ptr<int32_t>(), static_cast<int32_t*>(host)), "egs_set_status_mirror");
  s->side = c10::cuda::getStreamFromPool(/*isHighPriority=*/false, static_cast<c10::DeviceIndex>(idx));
  g_devices[idx].store(s, std::memory_order_release);
  return *s;
}

std::string status_text(int idx, int v) {
  std::string msgs;
  auto add = [&](const char* m) { msgs += (msgs.empty() ? "" : "; ") + std::string(m); };
  if (v & EGS_STATUS_INDEX_OUT_OF_RANGE) add("an Ind value outside [0, T) was met (slot skipped)");
  if (v & EGS_STATUS_PIPELINE_TIMEOUT) add("a bounded wait inside a tensor-core kernel ran out (results invalid)");
  if (v & EGS_STATUS_INTERNAL) add("a tensor-core kernel found its shared memory misaligned and did no work (results invalid)");
  return "egs kernels on cuda:" + std::to_string(idx) + " reported: " + msgs;
}

void reset_status(int device) {
  for (int i = 0; i < kMaxDevices; ++i) {
    if (device >= 0 && device != i) continue;
    if (DeviceState* s = g_devices[i].load(std::memory_order_acquire)) {
      s->word.zero_();
      *s->mirror = 0;
    }
  }
}

// Reads the status word (synchronises) and raises if a kernel flagged a problem.
void check_status(int device) {
  for (int i = 0; i < kMaxDevices; ++i) {
    if (device >= 0 && device != i) continue;
    DeviceState* s = g_devices[i].load(std::memory_order_acquire);
    if (!s) continue;
    const int v = s->word.item<int>();
    if (v) {
      s->word.zero_();
      *s->mirror = 0;
      throw std::runtime_error(status_text(i, v));
    }
  }
}

// What every operator call does first: device checks and a look at the mirror (no synchronisation).
struct Call {
  c10::cuda::OptionalCUDAGuard guard;
  int idx;
  DeviceState* st;
  cudaStream_t stream;
  template <class... Ts>
  explicit Call(const Tensor& first, const Ts&... more) {
    const auto dev = first.device();
    auto one = [&](const Tensor& t) {
      if (!t.is_cuda()) throw std::runtime_error("expert gather/scatter kernels need CUDA tensors (there is no CPU path)");
      if (t.device() != dev) throw std::runtime_error("all tensors must be on the same CUDA device");
    };
    one(first);
    (one(more), ...);
    idx = dev.index();
    guard.set_index(idx);
    st = &device_state(idx);
    if (const int v = *st->mirror; v & (EGS_STATUS_PIPELINE_TIMEOUT | EGS_STATUS_INTERNAL)) {
      *st->mirror = 0;
      st->word.zero_();
      throw std::runtime_error(status_text(idx, v));
    }
    stream = c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(idx)).stream();
  }
  int32_t* status() const { return st->word.data_ptr<int32_t>(); }
  void debug() const {
    if (g_debug.load(std::memory_order_relaxed)) check_status(idx);
  }
};

// Runs independent work of one call on the device's helper stream: forks at construction, joins when it goes out of scope.
class SideStream {
 public:
  explicit SideStream(const Call& c) : idx_(static_cast<c10::DeviceIndex>(c.idx)), main_(c.stream), side_(c.st->side->stream()) {
    events_ = &events_for(c.idx);
    sync_from_main();
  }
  SideStream(const SideStream&) = delete;
  ~SideStream() { join(); }
  cudaStream_t stream() const { return side_; }
  // later work on the side stream starts after what the main stream holds now
  void sync_from_main() {
    c10::cuda::CUDAGuard guard(idx_);                  // (the default stream's handle means the current device's)
    ok(cudaEventRecord(events_->fork, main_));
    ok(cudaStreamWaitEvent(side_, events_->fork, 0));
  }
  void join() {
    if (joined_) return;
    joined_ = true;
    c10::cuda::CUDAGuard guard(idx_);
    if (cudaEventRecord(events_->join, side_) == cudaSuccess) cudaStreamWaitEvent(main_, events_->join, 0);
  }

 private:
  struct Events {
    cudaEvent_t fork = nullptr, join = nullptr;
    ~Events() {
      if (fork) cudaEventDestroy(fork);
      if (join) cudaEventDestroy(join);
    }
  };
  static void ok(cudaError_t e) {
    if (e != cudaSuccess) throw std::runtime_error(std::string("CUDA error: ") + cudaGetErrorString(e));
  }
  static Events& events_for(int idx) {
    static thread_local std::array<Events, kMaxDevices> ev;
    Events& e = ev[idx];
    if (!e.fork) {
      ok(cudaEventCreateWithFlags(&e.fork, cudaEventDisableTiming));
      ok(cudaEventCreateWithFlags(&e.join, cudaEventDisableTiming));
    }
    return e;
  }
  c10::DeviceIndex idx_;
  cudaStream_t main_, side_;
  Events* events_;
  bool joined_ = false;
};

// ---- small helpers ---------------------------------------------------------------------------------------------------------
int type_id(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return EGS_F32;
    case at::kHalf: return EGS_F16;
    case at::kBFloat16: return EGS_BF16;
    default: value_error("Unknown dtype");
  }
}
struct Index {
  Tensor t;
  int type;
};
Index index_tensor(const Tensor& Ind) {
  switch (Ind.scalar_type()) {
    case at::kLong: return {Ind.contiguous(), EGS_I64};
    case at::kInt: return {Ind.contiguous(), EGS_I32};
    case at::kShort: return {Ind.contiguous(), EGS_I16};
    case at::kChar:
    case at::kByte: return {Ind.to(at::kInt).contiguous(), EGS_I32};
    default: value_error(std::string("Ind must be an integer tensor, got ") + toString(Ind.scalar_type()));
  }
}
int index_type(at::ScalarType t) {
  switch (t) {
    case at::kLong: return EGS_I64;
    case at::kInt: return EGS_I32;
    case at::kShort: return EGS_I16;
    default: value_error("index_dtype must be int64, int32 or int16");
  }
}
Tensor empty(at::IntArrayRef sizes, at::ScalarType dtype, int idx) {
  if (torch::jit::tracer::isTracing())     // a trace has to know its outputs
    return at::empty(sizes, at::TensorOptions().dtype(dtype).device(at::kCUDA, static_cast<c10::DeviceIndex>(idx)));
  return at::detail::empty_cuda(sizes, dtype, c10::Device(c10::kCUDA, static_cast<c10::DeviceIndex>(idx)), std::nullopt);
}
// device scratch of `bytes` (undefined tensor for none)
Tensor scratch(size_t bytes, int idx) {
  return bytes ? empty({static_cast<int64_t>((bytes + 3) / 4)}, at::kInt, idx) : Tensor();
}
void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }

struct WDims {
  int64_t E, C, N;
};
WDims w_dims(const Tensor& W, int layout) {
  return layout == EGS_W_CN ? WDims{W.size(0), W.size(1), W.size(2)} : WDims{W.size(0), W.size(2), W.size(1)};
}
std::string shape_of(const Tensor& t) {
  std::string s = "(";
  for (int64_t i = 0; i < t.dim(); ++i) s += (i ? ", " : "") + std::to_string(t.size(i));
  return s + ")";
}
const char* layout_name(int layout) { return layout == EGS_W_CN ? "cn" : "nc"; }

Tensor bias_rows(const OptTensor& bias, int64_t E, int64_t N, at::ScalarType dtype, const Call& c) {
  if (!bias || !bias->defined()) return Tensor();
  if (bias->numel() != E * N || bias->dim() < 1 || bias->size(0) != E || bias->size(-1) != N)
    value_error("bias must be [E, N] or [E, 1, N] = [" + std::to_string(E) + ", " + std::to_string(N) + "], got " + shape_of(*bias));
  if (!bias->is_cuda() || bias->get_device() != c.idx) throw std::runtime_error("bias must be on the tensors' CUDA device");
  return bias->reshape({E, N}).to(dtype).contiguous();
}

// ---- operators -------------------------------------------------------------------------------------------------------------
Tensor gather_gemm(const Tensor& X, const Tensor& W, const Tensor& Ind, int layout, int precision, int path, const OptTensor& bias) {
  if (X.dim() != 3 || W.dim() != 3 || Ind.dim() != 3) value_error("expected X[B,T,C], W[E,.,.], Ind[B,E,K]");
  Call c(X, W, Ind);
  if (W.scalar_type() != X.scalar_type()) value_error("X and W must have the same dtype");
  const int dt = type_id(X.scalar_type());
  const WDims w = w_dims(W, layout);
  const int64_t B = X.size(0), T = X.size(1), K = Ind.size(2);
  if (X.size(2) != w.C || Ind.size(1) != w.E || Ind.size(0) != B)
    value_error("shape mismatch: X" + shape_of(X) + " W" + shape_of(W) + " Ind" + shape_of(Ind) + " (" + layout_name(layout) + ")");
  const Tensor Xc = X.contiguous(), Wc = W.contiguous();
  const Index I = index_tensor(Ind);
  Tensor Y = empty({B, w.E, K, w.N}, X.scalar_type(), c.idx);
  const Tensor b = bias_rows(bias, w.E, w.N, X.scalar_type(), c);
  const egs_dims d{B, T, w.E, K, w.C, w.N};
  check(api.egs_gather_gemm_bias(ptr(Xc), ptr(Wc), ptr(b), ptr(I.t), ptr(Y), &d, layout, dt, I.type, prec_of(precision), path_of(path),
                                 c.status(), c.stream),
        "egs_gather_gemm");
  c.debug();
  return Y;
}

Tensor gemm_scatter(const Tensor& Y, const Tensor& W, const Tensor& Ind, int64_t T, int layout, const OptTensor& given, int precision,
                    int path, const OptTensor& bias, const OptTensor& csr_info) {
  if (Y.dim() != 4 || W.dim() != 3 || Ind.dim() != 3) value_error("expected Y[B,E,K,C], W[E,.,.], Ind[B,E,K]");
  Call c(Y, W, Ind);
  if (W.scalar_type() != Y.scalar_type()) value_error("Y and W must have the same dtype");
  const int dt = type_id(Y.scalar_type());
  const WDims w = w_dims(W, layout);
  const int64_t B = Y.size(0), K = Y.size(2);
  if (Y.size(3) != w.C || Y.size(1) != w.E || Ind.size(0) != B || Ind.size(1) != w.E || Ind.size(2) != K)
    value_error("shape mismatch: Y" + shape_of(Y) + " W" + shape_of(W) + " Ind" + shape_of(Ind) + " (" + layout_name(layout) + ")");
  const Tensor Yc = Y.contiguous(), Wc = W.contiguous();
  const Index I = index_tensor(Ind);
  Tensor out;
  if (given && given->defined()) {
    out = *given;
    if (out.dim() != 3 || out.size(0) != B || out.size(1) != T || out.size(2) != w.N || out.scalar_type() != Y.scalar_type() ||
        !out.is_contiguous())
      value_error("out must be a contiguous [B,T,N] tensor of Y's dtype");
  }
  const int zero = out.defined() ? 0 : 1;
  if (zero) out = empty({B, T, w.N}, Y.scalar_type(), c.idx);
  const egs_dims d{B, T, w.E, K, w.C, w.N};
  const size_t ws_bytes = api.egs_scatter_workspace_bytes(B, T, w.N, dt);
  const Tensor ws = scratch(ws_bytes, c.idx);
  const Tensor b = bias_rows(bias, w.E, w.N, Y.scalar_type(), c);
  if (csr_info && csr_info->defined())
    check(api.egs_gemm_scatter_prepared(ptr(Yc), ptr(Wc), ptr(b), ptr(I.t), static_cast<const int*>(ptr(*csr_info)), ptr(out), &d, layout,
                                        zero, dt, I.type, prec_of(precision), path_of(path), ptr(ws), ws_bytes, c.status(), c.stream),
          "egs_gemm_scatter");
  else
    check(api.egs_gemm_scatter_bias(ptr(Yc), ptr(Wc), ptr(b), ptr(I.t), ptr(out), &d, layout, zero, dt, I.type, prec_of(precision),
                                    path_of(path), ptr(ws), ws_bytes, c.status(), c.stream),
          "egs_gemm_scatter");
  c.debug();
  return out;
}

// on_stream: where the kernels go.  The buffers belong to the current stream either way, and the other stream knows nothing of what the
// current one does behind the fork: all that it writes is allocated before a temporary of a later operator could be freed and its block
// handed out again, so work for it is issued right behind the fork.  The caller forks and joins the two, passes contiguous inputs, and keeps
// *shared_ws - the scratch, one buffer for the weight gradients of one pass, which run one after the other and are of one size - until it has joined.
Tensor dweight_on(const Tensor& Xsrc, const Tensor& Ysrc, const Tensor& Ind, int out_layout, int precision, int path, const OptTensor& zeroed,
                  std::optional<cudaStream_t> on_stream, Tensor* shared_ws) {
  if (Xsrc.dim() != 3 || Ysrc.dim() != 4 || Ind.dim() != 3) value_error("expected Xsrc[B,T,FG], Ysrc[B,E,K,FD], Ind[B,E,K]");
  Call c(Xsrc, Ysrc, Ind);
  if (Xsrc.scalar_type() != Ysrc.scalar_type()) value_error("Xsrc and Ysrc must have the same dtype");
  const int dt = type_id(Xsrc.scalar_type());
  const int64_t B = Xsrc.size(0), T = Xsrc.size(1), FG = Xsrc.size(2), E = Ysrc.size(1), K = Ysrc.size(2), FD = Ysrc.size(3);
  if (Ysrc.size(0) != B || Ind.size(0) != B || Ind.size(1) != E || Ind.size(2) != K)
    value_error("shape mismatch: Xsrc" + shape_of(Xsrc) + " Ysrc" + shape_of(Ysrc) + " Ind" + shape_of(Ind));
  const std::array<int64_t, 3> shape = out_layout == EGS_DW_GATHERED_ROWS ? std::array<int64_t, 3>{E, FG, FD} : std::array<int64_t, 3>{E, FD, FG};
  const Tensor Xc = Xsrc.contiguous(), Yc = Ysrc.contiguous();
  const Index I = index_tensor(Ind);
  Tensor out;
  auto fn = api.egs_dweight;
  if (zeroed && zeroed->defined()) {
    out = *zeroed;
    if (out.sizes() != at::IntArrayRef(shape) || out.scalar_type() != at::kFloat || Xsrc.scalar_type() != at::kFloat || !out.is_contiguous())
      value_error("zeroed_out must be a contiguous float32 tensor of the output's shape");
    fn = api.egs_dweight_prezeroed;
  } else {
    out = empty(shape, Xsrc.scalar_type(), c.idx);
  }
  const size_t ws_bytes = api.egs_dw_workspace_bytes(E, FG, FD, dt);
  Tensor ws = shared_ws ? *shared_ws : Tensor();
  if (!ws.defined()) ws = scratch(ws_bytes, c.idx);
  if (shared_ws) *shared_ws = ws;
  check(fn(ptr(Xc), ptr(Yc), ptr(I.t), ptr(out), B, T, E, K, FG, FD, out_layout, dt, I.type, prec_of(precision), path_of(path), ptr(ws),
           ws_bytes, c.status(), on_stream ? *on_stream : c.stream),
        "egs_dweight");
  c.debug();
  return out;
}
Tensor dweight(const Tensor& Xsrc, const Tensor& Ysrc, const Tensor& Ind, int out_layout, int precision, int path, const OptTensor& zeroed) {
  return dweight_on(Xsrc, Ysrc, Ind, out_layout, precision, path, zeroed, std::nullopt, nullptr);
}

std::tuple<Tensor, Tensor> gather_scatter_pair(const Tensor& Src, const Tensor& W1, const Tensor& W2, const Tensor& Ind, int layout,
                                               const OptTensor& given, int precision) {
  if (Src.dim() != 3 || W1.dim() != 3 || W2.dim() != 3 || Ind.dim() != 3)
    value_error("expected Src[B,T,C1], W1[E,.,.], W2[E,.,.], Ind[B,E,K]");
  Call c(Src, W1, W2, Ind);
  if (W1.scalar_type() != Src.scalar_type() || W2.scalar_type() != Src.scalar_type()) value_error("Src, W1 and W2 must have the same dtype");
  const int dt = type_id(Src.scalar_type());
  const WDims a = w_dims(W1, layout), b = w_dims(W2, layout);
  const int64_t B = Src.size(0), T = Src.size(1), K = Ind.size(2);
  if (Src.size(2) != a.C || b.E != a.E || b.C != a.N || Ind.size(1) != a.E || Ind.size(0) != B)
    value_error("shape mismatch: Src" + shape_of(Src) + " W1" + shape_of(W1) + " W2" + shape_of(W2) + " Ind" + shape_of(Ind) + " (" +
                layout_name(layout) + ")");
  const Tensor Sc = Src.contiguous(), W1c = W1.contiguous(), W2c = W2.contiguous();
  const Index I = index_tensor(Ind);
  Tensor Mid = empty({B, a.E, K, a.N}, Src.scalar_type(), c.idx), out;
  if (given && given->defined()) {
    out = *given;
    if (out.dim() != 3 || out.size(0) != B || out.size(1) != T || out.size(2) != b.N || out.scalar_type() != Src.scalar_type() ||
        !out.is_contiguous())
      value_error("out must be a contiguous [B,T,N2] tensor of Src's dtype");
  }
  const int zero = out.defined() ? 0 : 1;
  if (zero) out = empty({B, T, b.N}, Src.scalar_type(), c.idx);
  const size_t ws_bytes = api.egs_scatter_workspace_bytes(B, T, b.N, dt);
  const Tensor ws = scratch(ws_bytes, c.idx);
  check(api.egs_gather_scatter_pair(ptr(Sc), ptr(W1c), ptr(W2c), ptr(I.t), ptr(Mid), ptr(out), B, T, a.E, K, a.C, a.N, b.N, layout, zero,
                                    dt, I.type, prec_of(precision), ptr(ws), ws_bytes, c.status(), c.stream),
        "egs_gather_scatter_pair");
  c.debug();
  return {Mid, out};
}

bool fused_pair_eligible(int64_t C1, int64_t N1, int64_t N2, int dt, int layout, int precision) {
  if (g_path.load(std::memory_order_relaxed) == EGS_PATH_GENERIC) return false;
  return api.egs_fused_pair_eligible(C1, N1, N2, layout, dt, prec_of(precision)) != 0;
}

// See ops.fused_pair_preferred.
constexpr int64_t kSmCount = 148;
bool fused_pair_preferred(const Tensor& X, const Tensor& Wg, const Tensor& Ind) {
  if (!X.is_cuda() || X.scalar_type() != at::kFloat || X.dim() != 3 || Wg.dim() != 3 || Ind.dim() != 3) return false;
  const int64_t I = X.size(2), J = Wg.size(2);
  if (Wg.size(0) * ((X.size(0) * Ind.size(2) + 127) / 128) > kSmCount) return false;
  return fused_pair_eligible(I, J, I, EGS_F32, EGS_W_CN, -1) && fused_pair_eligible(I, J, I, EGS_F32, EGS_W_NC, -1);
}

Tensor route_topk(const Tensor& scores, int64_t K, at::ScalarType index_dtype) {
  if (scores.dim() != 3) value_error("expected scores[B,T,E]");
  Call c(scores);
  const int it = index_type(index_dtype);
  const Tensor sc = scores.to(at::kFloat).contiguous();
  const int64_t B = sc.size(0), T = sc.size(1), E = sc.size(2);
  if (K < 0) value_error("K must not be negative");
  Tensor Ind = empty({B, E, K}, index_dtype, c.idx);
  check(api.egs_route_topk(static_cast<const float*>(ptr(sc)), ptr(Ind), B, T, E, K, it, c.stream), "egs_route_topk");
  return Ind;
}

std::tuple<Tensor, Tensor, Tensor, Tensor> build_index_csr(const Tensor& Ind, int64_t T) {
  if (Ind.dim() != 3) value_error("expected Ind[B,E,K]");
  Call c(Ind);
  const int64_t B = Ind.size(0), E = Ind.size(1), K = Ind.size(2);
  const Index I = index_tensor(Ind);
  Tensor counts = empty({B * T}, at::kInt, c.idx), offsets = empty({B * T + 1}, at::kInt, c.idx), entries = empty({B * E * K}, at::kInt, c.idx),
         info = empty({4}, at::kInt, c.idx);
  const size_t sb = api.egs_index_csr_scratch_bytes(B, T);
  const Tensor ws = scratch(sb, c.idx);
  check(api.egs_index_csr(ptr(I.t), I.type, B, T, E, K, counts.data_ptr<int>(), offsets.data_ptr<int>(), entries.data_ptr<int>(),
                          info.data_ptr<int>(), ptr(ws), sb, c.stream),
        "egs_index_csr");
  return {counts, offsets, entries, info};
}

void fill_zero(const Tensor& t) {
  if (!t.is_cuda() || !t.is_contiguous()) value_error("fill_zero needs a contiguous CUDA tensor");
  c10::cuda::OptionalCUDAGuard guard(t.device());
  check(api.egs_fill_zero(t.data_ptr(), t.numel() * t.element_size(), c10::cuda::getCurrentCUDAStream(t.get_device()).stream()), "egs_fill_zero");
}

// [E, N]: per expert, the sum of its slot rows of Src (no Ind) or of the token rows of Src that Ind names; on_stream as in dweight_on
Tensor expert_row_sum(const Tensor& Src, const OptTensor& Ind, int64_t B, int64_t T, int64_t E, int64_t K, std::optional<cudaStream_t> on_stream) {
  Call c(Src);
  const int64_t N = Src.size(-1);
  Tensor out = empty({E, N}, Src.scalar_type(), c.idx);
  const Index I = Ind ? index_tensor(*Ind) : Index{Tensor(), EGS_I64};
  check(api.egs_expert_row_sum(ptr(Src), ptr(I.t), ptr(out), B, T, E, K, N, type_id(Src.scalar_type()), I.type, c.status(),
                               on_stream ? *on_stream : c.stream),
        "egs_expert_row_sum");
  return out;
}

// ---- backward passes of the two operators ------------------------------------------------------------------------------------
// The weight gradient runs on the helper stream next to the dX / dY kernel: the two are independent and share the SMs.  The fork and
// the join cost the host 3 us, which small passes, bound by the host, would only pay for.  Where the line lies depends on the kernels:
// forward and backward of two modules take 110 us with and 107 without the fork at 2^26 multiply-adds on the tensor cores (float32: 105
// and 101), at 2^27 the fills of long sequences turn it (T=16384: 101 and 104 us); on the generic kernels 141 and 158 us at 2^26, and
// at 2^25 the same.
constexpr double kSmallTensorWork = 1 << 26, kSmallGenericWork = 1 << 25;
bool worth_a_side_stream(const Tensor& slot_rows, const Tensor& W) {      // [B,E,K,J] and a weight tensor of E * I * J elements
  if (g_debug.load(std::memory_order_relaxed)) return false;             // every operator is checked behind its own kernels
  const double slots = static_cast<double>(slot_rows.size(0)) * slot_rows.size(2);
  const int64_t per16 = 16 / W.element_size();                           // whole 16-byte chunks in both widths: see rowgemm_tensor_ok
  const bool tensor = W.size(1) % per16 == 0 && W.size(2) % per16 == 0 && g_path.load(std::memory_order_relaxed) != EGS_PATH_GENERIC;
  return slots * W.numel() > (tensor ? kSmallTensorWork : kSmallGenericWork);
}
// Bias gradients of 16-bit tensors follow the weight gradient there: their row sums read memory under the end of the dX / dY kernel, whose last
// wave leaves SMs free, where they stood alone behind it before.  Forward and backward in bf16 through both modules, ten processes each, with
// both sums on the main and both on the helper stream: 32 experts, 768 and 192 features 238 and 231 us, 192 and 768 265 and 264, 64 of 1024 and 128
// 262 and 254, 24 of ragged sizes 179.5 and 181; with the scatter's alone on the main stream 239, 263, 254 and 179, in one process of ten 226, 257, 250
// and 174.  Through the ExpertScatter alone, whose dY kernel ends before the weight gradient, the main stream would be the better one: 129 and
// 134, 115 and 123, 142 and 148.  Where there is no dX / dY kernel the sum belongs on the main stream, beside the weight gradient (an ExpertGather
// alone 70.1 us, behind it on the helper stream 78.6).  The float32 weight gradients take longer than the dX / dY kernels, and sums behind them
// 1-4 % of a large pass (1024 and 256 features 674 and 695 us).
struct Grads {
  Tensor in, w, b;
};
std::optional<cudaStream_t> row_sum_stream(const std::optional<SideStream>& side, const Tensor& rows) {
  return side && rows.element_size() == 2 ? std::optional<cudaStream_t>(side->stream()) : std::nullopt;
}

Grads gather_backward(const Tensor& X_, const Tensor& W, const Tensor& Ind_, const Tensor& dY_, bool need_x, bool need_w, bool need_b) {
  const Tensor dY = dY_.contiguous(), X = X_.contiguous(), Ind = index_tensor(Ind_).t;
  Grads g;
  Tensor ws;
  std::optional<SideStream> side;
  if (need_w) {
    std::optional<cudaStream_t> on;
    if ((need_x || need_b) && worth_a_side_stream(dY, W)) {
      side.emplace(Call(X, dY));
      on = side->stream();
    }
    g.w = dweight_on(X, dY, Ind, EGS_DW_GATHERED_ROWS, -1, -1, std::nullopt, on, &ws);
  }
  auto bias_gradient = [&](std::optional<cudaStream_t> on) { g.b = expert_row_sum(dY, std::nullopt, dY.size(0), X.size(1), dY.size(1), dY.size(2), on); };
  const auto sums_on = need_x ? row_sum_stream(side, dY) : std::nullopt;
  if (need_b && sums_on) bias_gradient(sums_on);                  // (before the dX kernel's scratch comes and goes, see dweight_on)
  if (need_x) g.in = gemm_scatter(dY, W, Ind, X.size(1), EGS_W_NC, std::nullopt, -1, -1, std::nullopt, std::nullopt);
  if (need_b && !sums_on) bias_gradient(std::nullopt);
  return g;
}

Grads scatter_backward(const Tensor& Y_, const Tensor& W, const Tensor& Ind_, const Tensor& dOut_, bool need_y, bool need_w, bool need_b) {
  const Tensor dOut = dOut_.contiguous(), Y = Y_.contiguous(), Ind = index_tensor(Ind_).t;
  Grads g;
  Tensor ws;
  std::optional<SideStream> side;
  if (need_w) {
    std::optional<cudaStream_t> on;
    if ((need_y || need_b) && worth_a_side_stream(Y, W)) {
      side.emplace(Call(Y, dOut));
      on = side->stream();
    }
    g.w = dweight_on(dOut, Y, Ind, EGS_DW_DIRECT_ROWS, -1, -1, std::nullopt, on, &ws);
  }
  auto bias_gradient = [&](std::optional<cudaStream_t> on) { g.b = expert_row_sum(dOut, Ind, Y.size(0), dOut.size(1), Y.size(1), Y.size(2), on); };
  const auto sums_on = need_y ? row_sum_stream(side, dOut) : std::nullopt;
  if (need_b && sums_on) bias_gradient(sums_on);                  // (before a copy of the weights comes and goes, see dweight_on)
  if (need_y) g.in = gather_gemm(dOut, W, Ind, EGS_W_NC, -1, -1, std::nullopt);
  if (need_b && !sums_on) bias_gradient(std::nullopt);
  return g;
}

// ---- autograd functions ------------------------------------------------------------------------------------------------------
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

// Under create_graph a backward pass runs as the dispatcher op, as it does behind the Python functions, so that torch's fallback for
// ops without a derivative of their own (a warning, zero second derivatives) is what a caller meets either way.
std::string g_namespace;               // of the dispatcher ops
variable_list through_dispatcher(const char* op, const Tensor& A, const Tensor& W, const Tensor& Ind, const Tensor& grad) {
  using Fn = std::tuple<Tensor, Tensor>(const Tensor&, const Tensor&, const Tensor&, const Tensor&, at::ScalarType);
  const std::string name = g_namespace + "::" + op;
  auto r = c10::Dispatcher::singleton().findSchemaOrThrow(name.c_str(), "").typed<Fn>().call(A, W, Ind, grad, at::kFloat);
  return {std::get<0>(r), std::get<1>(r)};
}
bool wants_graph(const Tensor& A, const Tensor& W) { return at::GradMode::is_enabled() && A.requires_grad() && W.requires_grad(); }

struct GatherFunction : torch::autograd::Function<GatherFunction> {
  static Tensor forward(AutogradContext* ctx, const Tensor& X, const Tensor& W, const Tensor& Ind) {
    Tensor Y = gather_gemm(X, W, Ind, EGS_W_CN, -1, -1, std::nullopt);
    ctx->save_for_backward({X, W, Ind});
    return Y;
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& g) {
    const auto s = ctx->get_saved_variables();
    if (wants_graph(s[0], s[1])) {
      variable_list d = through_dispatcher("expert_gather_backward_call_fn", s[0], s[1], s[2], g[0]);
      return {d[0], d[1], Tensor()};
    }
    Grads r = gather_backward(s[0], s[1], s[2], g[0], ctx->needs_input_grad(0), ctx->needs_input_grad(1), false);
    return {r.in, r.w, Tensor()};
  }
};

struct ScatterFunction : torch::autograd::Function<ScatterFunction> {
  static Tensor forward(AutogradContext* ctx, const Tensor& Y, const Tensor& W, const Tensor& Ind, int64_t T) {
    Tensor out = gemm_scatter(Y, W, Ind, T, EGS_W_CN, std::nullopt, -1, -1, std::nullopt, std::nullopt);
    ctx->save_for_backward({Y, W, Ind});
    return out;
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& g) {
    const auto s = ctx->get_saved_variables();
    if (wants_graph(s[0], s[1])) {
      variable_list d = through_dispatcher("expert_scatter_backward_call_fn", s[0], s[1], s[2], g[0]);
      return {d[0], d[1], Tensor(), Tensor()};
    }
    Grads r = scatter_backward(s[0], s[1], s[2], g[0], ctx->needs_input_grad(0), ctx->needs_input_grad(1), false);
    return {r.in, r.w, Tensor(), Tensor()};
  }
};

struct GatherBiasFunction : torch::autograd::Function<GatherBiasFunction> {
  static Tensor forward(AutogradContext* ctx, const Tensor& X, const Tensor& W, const Tensor& bias, const Tensor& Ind) {
    Tensor Y = gather_gemm(X, W, Ind, EGS_W_CN, -1, -1, bias);
    ctx->save_for_backward({X, W, Ind});
    ctx->saved_data["bias_shape"] = bias.sizes().vec();
    return Y;
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& g) {
    const auto s = ctx->get_saved_variables();
    Grads r = gather_backward(s[0], s[1], s[2], g[0], ctx->needs_input_grad(0), ctx->needs_input_grad(1), ctx->needs_input_grad(2));
    if (r.b.defined()) r.b = r.b.reshape(ctx->saved_data["bias_shape"].toIntVector());
    return {r.in, r.w, r.b, Tensor()};
  }
};

struct ScatterBiasFunction : torch::autograd::Function<ScatterBiasFunction> {
  static Tensor forward(AutogradContext* ctx, const Tensor& Y, const Tensor& W, const Tensor& bias, const Tensor& Ind, int64_t T) {
    Tensor out = gemm_scatter(Y, W, Ind, T, EGS_W_CN, std::nullopt, -1, -1, bias, std::nullopt);
    ctx->save_for_backward({Y, W, Ind});
    ctx->saved_data["bias_shape"] = bias.sizes().vec();
    return out;
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& g) {
    const auto s = ctx->get_saved_variables();
    Grads r = scatter_backward(s[0], s[1], s[2], g[0], ctx->needs_input_grad(0), ctx->needs_input_grad(1), ctx->needs_input_grad(2));
    if (r.b.defined()) r.b = r.b.reshape(ctx->saved_data["bias_shape"].toIntVector());
    return {r.in, r.w, r.b, Tensor(), Tensor()};
  }
};

// The block: Y, Out and whether the fused kernel ran.
std::tuple<Tensor, Tensor, bool> gather_scatter_forward(const Tensor& X, const Tensor& Wg, const Tensor& Ws, const Tensor& Ind) {
  const bool fused = fused_pair_preferred(X, Wg, Ind);
  Tensor Y, out;
  if (fused) {
    std::tie(Y, out) = gather_scatter_pair(X, Wg, Ws, Ind, EGS_W_CN, std::nullopt, -1);
  } else {
    Y = gather_gemm(X, Wg, Ind, EGS_W_CN, -1, -1, std::nullopt);
    out = gemm_scatter(Y, Ws, Ind, X.size(1), EGS_W_CN, std::nullopt, -1, -1, std::nullopt, std::nullopt);
  }
  return {Y, out, fused};
}

// dX, dWg, dWs; those not needed stay undefined
std::array<Tensor, 3> gather_scatter_backward(const Tensor& X_, const Tensor& Wg, const Tensor& Ws, const Tensor& Ind_, const Tensor& Y_,
                                              const Tensor& dOut_, bool fused, bool need_x, bool need_wg, bool need_ws) {
  const Tensor X = X_.contiguous(), dOut = dOut_.contiguous(), Y = Y_.contiguous(), Ind = index_tensor(Ind_).t;
  Tensor dX, dWg, dWs, dY, ws;
  std::optional<SideStream> side;
  const bool fork = worth_a_side_stream(Y, Wg);
  std::optional<cudaStream_t> on;
  if (need_ws) {                                     // needs only dOut and Y
    if (fork) {
      side.emplace(Call(X, dOut));
      on = side->stream();
    }
    dWs = dweight_on(dOut, Y, Ind, EGS_DW_DIRECT_ROWS, -1, -1, std::nullopt, on, &ws);
  }
  if (need_x && fused)
    std::tie(dY, dX) = gather_scatter_pair(dOut, Ws, Wg, Ind, EGS_W_NC, std::nullopt, -1);
  else if (need_x || need_wg)
    dY = gather_gemm(dOut, Ws, Ind, EGS_W_NC, -1, -1, std::nullopt);
  if (need_wg) {
    if (side) {
      side->sync_from_main();
    } else if (fork) {
      side.emplace(Call(X, dOut));
      on = side->stream();
    }
    dWg = dweight_on(X, dY, Ind, EGS_DW_GATHERED_ROWS, -1, -1, std::nullopt, on, &ws);
  }
  if (need_x && !dX.defined()) dX = gemm_scatter(dY, Wg, Ind, X.size(1), EGS_W_NC, std::nullopt, -1, -1, std::nullopt, std::nullopt);
  return {dX, dWg, dWs};
}

struct GatherScatterFunction : torch::autograd::Function<GatherScatterFunction> {
  static Tensor forward(AutogradContext* ctx, const Tensor& X_, const Tensor& Wg_, const Tensor& Ws_, const Tensor& Ind) {
    const Tensor X = X_.contiguous(), Wg = Wg_.contiguous(), Ws = Ws_.contiguous();
    auto [Y, out, fused] = gather_scatter_forward(X, Wg, Ws, Ind);
    ctx->saved_data["fused"] = fused;
    ctx->save_for_backward({X, Wg, Ws, Ind, Y});
    return out;
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    const auto s = ctx->get_saved_variables();
    auto d = gather_scatter_backward(s[0], s[1], s[2], s[3], s[4], grads[0], ctx->saved_data["fused"].toBool(), ctx->needs_input_grad(0),
                                     ctx->needs_input_grad(1), ctx->needs_input_grad(2));
    return {d[0], d[1], d[2], Tensor()};
  }
};

// Tensors this path takes as they are: plain tensors outside any tracing, transform or dispatch mode.  (Fake tensors, tensor
// subclasses and functorch wrappers go through the Python functions and their dispatcher ops.)
bool plain(const Tensor& t) {
  const auto ks = t.key_set();
  return !(ks.has(c10::DispatchKey::Python) || ks.has(c10::DispatchKey::FuncTorchBatched) ||
           ks.has(c10::DispatchKey::FuncTorchGradWrapper) || ks.has(c10::DispatchKey::Functionalize) || t.is_meta());
}
template <class... Ts>
bool native_ok(const Ts&... ts) {
  return !c10::impl::dispatch_mode_enabled() && !torch::jit::tracer::isTracing() && (plain(ts) && ...);
}
bool native_ok_bias(const OptTensor& bias) { return !bias || plain(*bias); }

OptTensor gather_autograd(const Tensor& X, const Tensor& W, const OptTensor& bias, const Tensor& Ind) {
  if (!native_ok(X, W, Ind) || !native_ok_bias(bias)) return std::nullopt;
  return bias ? GatherBiasFunction::apply(X, W, *bias, Ind) : GatherFunction::apply(X, W, Ind);
}
OptTensor scatter_autograd(const Tensor& Y, const Tensor& W, const OptTensor& bias, const Tensor& Ind, int64_t T) {
  if (!native_ok(Y, W, Ind) || !native_ok_bias(bias)) return std::nullopt;
  return bias ? ScatterBiasFunction::apply(Y, W, *bias, Ind, T) : ScatterFunction::apply(Y, W, Ind, T);
}
OptTensor gather_scatter_autograd(const Tensor& X, const Tensor& Wg, const Tensor& Ws, const Tensor& Ind) {
  if (!native_ok(X, Wg, Ws, Ind)) return std::nullopt;
  return GatherScatterFunction::apply(X, Wg, Ws, Ind);
}

// The backward passes for the Python functions: gradients that are not needed come back as None.
OptTensor opt(const Tensor& t) { return t.defined() ? OptTensor(t) : std::nullopt; }
using OptGrads = std::tuple<OptTensor, OptTensor, OptTensor>;
OptGrads gather_backward_op(const Tensor& X, const Tensor& W, const Tensor& Ind, const Tensor& dY, bool need_x, bool need_w, bool need_b) {
  Grads g = gather_backward(X, W, Ind, dY, need_x, need_w, need_b);
  return {opt(g.in), opt(g.w), opt(g.b)};
}
OptGrads scatter_backward_op(const Tensor& Y, const Tensor& W, const Tensor& Ind, const Tensor& dOut, bool need_y, bool need_w, bool need_b) {
  Grads g = scatter_backward(Y, W, Ind, dOut, need_y, need_w, need_b);
  return {opt(g.in), opt(g.w), opt(g.b)};
}
OptGrads gather_scatter_backward_op(const Tensor& X, const Tensor& Wg, const Tensor& Ws, const Tensor& Ind, const Tensor& Y, const Tensor& dOut,
                                    bool fused, bool need_x, bool need_wg, bool need_ws) {
  auto d = gather_scatter_backward(X, Wg, Ws, Ind, Y, dOut, fused, need_x, need_wg, need_ws);
  return {opt(d[0]), opt(d[1]), opt(d[2])};
}

// ---- the explicit step ---------------------------------------------------------------------------------------------------------
// Y, Out, dY, dX, dWg, dWs (see step.train_step).
using Step = std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor, Tensor>;
Step train_step(const Tensor& X_, const Tensor& Wg, const Tensor& Ws, const Tensor& Ind_, const Tensor& G_, bool overlap, bool fused_pairs) {
  const Tensor X = X_.contiguous(), G = G_.contiguous(), Ind = index_tensor(Ind_).t;
  const int64_t T = X.size(1);
  const auto none = std::nullopt;
  Tensor Y, Out, dY, dX, dWg, dWs;
  if (!overlap || g_debug.load(std::memory_order_relaxed)) {
    Y = gather_gemm(X, Wg, Ind, EGS_W_CN, -1, -1, none);
    Out = gemm_scatter(Y, Ws, Ind, T, EGS_W_CN, none, -1, -1, none, none);
    dY = gather_gemm(G, Ws, Ind, EGS_W_NC, -1, -1, none);
    dWs = dweight(G, Y, Ind, EGS_DW_DIRECT_ROWS, -1, -1, none);
    dX = gemm_scatter(dY, Wg, Ind, T, EGS_W_NC, none, -1, -1, none, none);
    dWg = dweight(X, dY, Ind, EGS_DW_GATHERED_ROWS, -1, -1, none);
    return {Y, Out, dY, dX, dWg, dWs};
  }
  const bool fused = fused_pairs && fused_pair_preferred(X, Wg, Ind);
  if (fused) {
    std::tie(Y, Out) = gather_scatter_pair(X, Wg, Ws, Ind, EGS_W_CN, none, -1);
  } else {
    Y = gather_gemm(X, Wg, Ind, EGS_W_CN, -1, -1, none);
    Out = gemm_scatter(Y, Ws, Ind, T, EGS_W_CN, none, -1, -1, none, none);
  }
  Tensor ws;
  SideStream side(Call(X, G));                         // dW_s next to dY, dW_g next to dX
  dWs = dweight_on(G, Y, Ind, EGS_DW_DIRECT_ROWS, -1, -1, none, side.stream(), &ws);
  if (fused) std::tie(dY, dX) = gather_scatter_pair(G, Ws, Wg, Ind, EGS_W_NC, none, -1);
  else dY = gather_gemm(G, Ws, Ind, EGS_W_NC, -1, -1, none);
  side.sync_from_main();
  dWg = dweight_on(X, dY, Ind, EGS_DW_GATHERED_ROWS, -1, -1, none, side.stream(), &ws);
  if (!fused) dX = gemm_scatter(dY, Wg, Ind, T, EGS_W_NC, none, -1, -1, none, none);
  side.join();
  return {Y, Out, dY, dX, dWg, dWs};
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  using nogil = py::call_guard<py::gil_scoped_release>;
  m.def("init", &init);
  m.def("configure", &configure);
  m.def("set_namespace", [](const std::string& ns) { g_namespace = ns; });
  m.def("status_word", [](int idx) { return device_state(idx).word; });
  m.def("reset_status", &reset_status);
  m.def("check_status", &check_status, nogil());
  m.def("raise_if_flagged", [](const Tensor& t) { Call c(t); });
  m.def("gather_gemm", &gather_gemm, nogil());
  m.def("gemm_scatter", &gemm_scatter, nogil());
  m.def("dweight", &dweight, nogil());
  m.def("gather_scatter_pair", &gather_scatter_pair, nogil());
  m.def("fused_pair_preferred", &fused_pair_preferred);
  m.def("route_topk", &route_topk, nogil());
  m.def("build_index_csr", &build_index_csr, nogil());
  m.def("fill_zero", &fill_zero, nogil());
  m.def("gather_autograd", &gather_autograd, nogil());
  m.def("scatter_autograd", &scatter_autograd, nogil());
  m.def("gather_scatter_autograd", &gather_scatter_autograd, nogil());
  m.def("gather_backward", &gather_backward_op, nogil());
  m.def("scatter_backward", &scatter_backward_op, nogil());
  m.def("gather_scatter_forward", &gather_scatter_forward, nogil());
  m.def("gather_scatter_backward", &gather_scatter_backward_op, nogil());
  m.def("train_step", &train_step, nogil());
}
