// Host path of the hot entry points: argument checks, output allocation, autograd bookkeeping and the call
// into libgca_b200.so, without a Python frame per step.
//
// What this bounds: a decode-sized call is 5-15 us of device work, and the ctypes path in front of it (one
// Python object per argument field, a Python allocation call per output, Python autograd.Function) was
// 35-40 us per call and ~220 us for a forward + backward.  Here the same checks run in C++ on the tensors'
// own metadata; the C ABI of include/gca_b200.h stays the only way to the kernels.
//
// The library is not linked: `bind` receives the addresses of its entry points from the ctypes loader, so that
// the build of the library that the process selected is the one that runs.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/core/LegacyTypeDispatch.h>
#include <ATen/ops/empty.h>
#include <ATen/ops/empty_like.h>
#include <ATen/ops/empty_strided.h>
#include <ATen/ops/arange.h>
#include <ATen/ops/constant_pad_nd.h>
#include <ATen/ops/nan_to_num.h>
#include <ATen/ops/softmax.h>
#include <ATen/ops/zeros.h>
#include <ATen/ops/zeros_like.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <nvtx3/nvToolsExt.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>

#include <array>
#include <atomic>
#include <cmath>
#include <mutex>

#include "gca_b200.h"

namespace {

using at::Tensor;
using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

// ------------------------------------------------------------------------------------------- the library
struct Api {
#define GCA_API(name) decltype(&::name) name = nullptr;
#define GCA_API_LIST                                                                                          \
  GCA_API(gca_fwd) GCA_API(gca_decode) GCA_API(gca_bwd_stages) GCA_API(gca_bwd_workspace_bytes)               \
  GCA_API(lmk_score_topk_kept) GCA_API(lmk_topk_workspace_bytes) GCA_API(lmk_weights_backward) GCA_API(gca_kv_project_append) GCA_API(gca_row_rms) \
  GCA_API(gca_linear) GCA_API(gca_linear_batched) GCA_API(gca_rms_linear_batched) GCA_API(gca_linear_few_rows) GCA_API(gca_layer_decode) GCA_API(gca_silu_mul) GCA_API(gca_window_decode)            \
  GCA_API(gca_window_ring_decode) GCA_API(gca_strerror)
  GCA_API_LIST
#undef GCA_API
};
Api api;
PyObject* gca_error = nullptr;                  // the package's GcaError class
std::atomic<bool> nvtx_on{false}, check_on{false};

// A code returned by the library: negative -> ValueError, positive -> GcaError.
struct LibraryError {
  int code;
  const char* what;
};

// CUDA error text and argument-rule text come from the library itself
void set_python_error(const LibraryError& e) {
  const char* msg = api.gca_strerror ? api.gca_strerror(e.code) : "";
  if (e.code < 0) PyErr_Format(PyExc_ValueError, "%s: %s (code %d)", e.what, msg, e.code);
  else PyErr_Format(gca_error ? gca_error : PyExc_RuntimeError, "%s: CUDA error %d: %s", e.what, e.code, msg);
}

struct TimeoutError {};
void set_python_error(const TimeoutError&) {
  PyErr_SetString(gca_error ? gca_error : PyExc_RuntimeError,
                  "a GCA kernel gave up a bounded wait (GCA_STATUS_TIMEOUT): its outputs are not valid");
}

template <class F>
void call(const char* name, F&& f) {
  const bool range = nvtx_on.load(std::memory_order_relaxed);
  if (range) nvtxRangePushA(name);
  const int rc = f();
  if (range) nvtxRangePop();
  if (rc) throw LibraryError{rc, name};
}

struct NoGil {
  PyThreadState* save = PyEval_SaveThread();
  ~NoGil() { PyEval_RestoreThread(save); }
};

// ------------------------------------------------------------------------------------------- status words
constexpr int MAX_DEVICES = 64;
std::mutex status_mu;
Tensor status_words[MAX_DEVICES];
std::atomic<int32_t*> status_ptrs[MAX_DEVICES];

const Tensor& status_word(int dev) {
  TORCH_CHECK(dev >= 0 && dev < MAX_DEVICES, "device index out of range");
  std::lock_guard<std::mutex> lock(status_mu);
  if (!status_words[dev].defined()) {
    status_words[dev] = at::zeros({1}, at::TensorOptions().dtype(at::kInt).device(at::kCUDA, (c10::DeviceIndex)dev));
    status_ptrs[dev].store(status_words[dev].data_ptr<int32_t>());
  }
  return status_words[dev];
}
int32_t* status_ptr(int dev) {
  int32_t* p = dev >= 0 && dev < MAX_DEVICES ? status_ptrs[dev].load(std::memory_order_acquire) : nullptr;
  return p ? p : status_word(dev).data_ptr<int32_t>();
}

// With checks on, read the status word after a launch; a bounded wait that ran out raises.
void maybe_check(int dev) {
  if (!check_on.load(std::memory_order_relaxed)) return;
  at::AutoDispatchBelowADInplaceOrView below;
  Tensor word = status_word(dev);
  const int bits = word.item<int32_t>();
  word.zero_();
  if (bits & GCA_STATUS_TIMEOUT) throw TimeoutError{};
}

// The device guard and stream of a call: the current stream of the device that holds the tensor.
struct Launch {
  c10::cuda::OptionalCUDAGuard guard;
  int dev;
  void* stream;
  explicit Launch(const Tensor& t) : dev(t.get_device()) {
    guard.set_index((c10::DeviceIndex)dev);
    stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream();
  }
};

// Dual numbers of forward-mode differentiation, which no kernel here knows about.
bool has_tangent(std::initializer_list<const Tensor*> ts) {
  for (const Tensor* t : ts)
    if (t->_fw_grad(0).defined()) return true;
  return false;
}

Tensor inner_contiguous(const Tensor& t) { return t.stride(-1) == 1 ? t : t.contiguous(); }
Tensor as_int32(const Tensor& t) { return (t.scalar_type() == at::kInt ? t : t.to(at::kInt)).contiguous(); }
Tensor as_float(const Tensor& t) { return (t.scalar_type() == at::kFloat ? t : t.to(at::kFloat)).contiguous(); }

int dtype_code(const Tensor& t) {
  if (t.scalar_type() == at::kBFloat16) return GCA_BF16;
  if (t.scalar_type() == at::kFloat) return GCA_F32;
  TORCH_CHECK_VALUE(false, "unsupported dtype ", t.scalar_type(), ": the GCA kernels take bfloat16 or float32");
}

// ------------------------------------------------------------------------------------------- GCA
// One GCA problem as the kernels see it: q (N, J, Hq, S, D), caches (N, C, L, Hkv, D), whatever the shapes
// the caller's tensors have.
struct Problem {
  int64_t N, J, Hq, S, D, C, L, Hkv, K;
  int64_t qs[4], ks[4], vs[4];     // strides {n, j, h, s} and {n, c, l, h}
};

// (N, C, L, Hkv*D) token-major or (N, C, L, Hkv, D)
void cache_view(const Tensor& t, int64_t head_dim, int64_t dims[4], int64_t st[4]) {
  TORCH_CHECK_VALUE(t.dim() == 5 || (t.dim() == 4 && t.size(3) % head_dim == 0),
                    "cache must be (N, C, L, Hkv*D) or (N, C, L, Hkv, D), got ", t.sizes());
  dims[0] = t.size(0); dims[1] = t.size(1); dims[2] = t.size(2);
  dims[3] = t.dim() == 5 ? t.size(3) : t.size(3) / head_dim;
  TORCH_CHECK_VALUE(t.dim() == 4 || t.size(4) == head_dim, "head dims of q and the cache differ");
  st[0] = t.stride(0); st[1] = t.stride(1); st[2] = t.stride(2);
  st[3] = t.dim() == 5 ? t.stride(3) : head_dim;
}

Problem indexed_problem(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& idx, const Tensor& w) {
  TORCH_CHECK_VALUE(q.dim() == 5, "expected q (N,J,Hq,S,D) and caches (N,C,L,Hkv,D)");
  Problem p;
  p.N = q.size(0); p.J = q.size(1); p.Hq = q.size(2); p.S = q.size(3); p.D = q.size(4);
  int64_t kd[4], vd[4];
  cache_view(k, p.D, kd, p.ks);
  cache_view(v, p.D, vd, p.vs);
  for (int i = 0; i < 4; ++i) TORCH_CHECK_VALUE(kd[i] == vd[i], "k_cache and v_cache must have the same shape");
  TORCH_CHECK_VALUE(q.scalar_type() == k.scalar_type() && q.scalar_type() == v.scalar_type(), "q, k_cache and v_cache must share one dtype");
  TORCH_CHECK_VALUE(idx.dim() == 3 && idx.size(0) == p.N && idx.size(1) == p.J && w.sizes() == idx.sizes() && kd[0] == p.N,
                    "indices/weights must be (N, J, K) = (", p.N, ", ", p.J, ", K); got ", idx.sizes(), ", ", w.sizes());
  p.C = kd[1]; p.L = kd[2]; p.Hkv = kd[3]; p.K = idx.size(2);
  TORCH_CHECK_VALUE(p.Hkv > 0 && p.Hq % p.Hkv == 0, "number of q heads must be a multiple of the number of kv heads");
  for (int i = 0; i < 4; ++i) p.qs[i] = q.stride(i);
  return p;
}

// q (Z, Hq, S, D), k / v (Z, Hkv, K, L, D): every row block has a cache of its own whose K chunks are all "retrieved"
Problem gathered_problem(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& w) {
  TORCH_CHECK_VALUE(q.dim() == 4 && k.dim() == 5 && v.dim() == 5, "expected q (Z,Hq,S,D), k/v (Z,Hkv,K,L,D)");
  TORCH_CHECK_VALUE(w.dim() == 2, "weights must be 2-D (Z, K)");                                        // ltriton/gca.py:699
  TORCH_CHECK_VALUE(q.size(3) == k.size(4) && k.sizes() == v.sizes(), "head dims / k,v shapes differ");   // ltriton/gca.py:697
  TORCH_CHECK_VALUE(w.size(0) == k.size(0) && w.size(1) == k.size(2), "weights must be (Z, K)");
  Problem p;
  p.N = q.size(0); p.J = 1; p.Hq = q.size(1); p.S = q.size(2); p.D = q.size(3);
  p.C = p.K = k.size(2); p.L = k.size(3); p.Hkv = k.size(1);
  p.qs[0] = q.stride(0); p.qs[1] = q.stride(0); p.qs[2] = q.stride(1); p.qs[3] = q.stride(2);
  for (int i = 0; i < 2; ++i) {
    const Tensor& t = i ? v : k;
    int64_t* s = i ? p.vs : p.ks;
    s[0] = t.stride(0); s[1] = t.stride(2); s[2] = t.stride(3); s[3] = t.stride(1);
  }
  TORCH_CHECK_VALUE(k.size(0) == p.N, "q and k / v must have the same number of row blocks");
  TORCH_CHECK_VALUE(q.scalar_type() == k.scalar_type() && q.scalar_type() == v.scalar_type(), "q, k_cache and v_cache must share one dtype");
  TORCH_CHECK_VALUE(p.Hkv > 0 && p.Hq % p.Hkv == 0, "number of q heads must be a multiple of the number of kv heads");
  return p;
}

void copy4(int64_t dst[4], const int64_t src[4]) { for (int i = 0; i < 4; ++i) dst[i] = src[i]; }

GcaFwdArgs fwd_args(const Problem& p, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& idx, const Tensor& w,
                    const Tensor& out, const int64_t os[4], float* lse, double sm_scale, double off_by_one, int64_t algo, int dev) {
  GcaFwdArgs a;
  a.q = q.const_data_ptr(); a.k_cache = k.const_data_ptr(); a.v_cache = v.const_data_ptr();
  a.indices = idx.defined() ? idx.const_data_ptr<int32_t>() : nullptr;
  a.weights = w.const_data_ptr<float>();
  a.out = out.mutable_data_ptr(); a.lse = lse; a.status = status_ptr(dev);
  copy4(a.q_stride, p.qs); copy4(a.o_stride, os); copy4(a.k_stride, p.ks); copy4(a.v_stride, p.vs);
  a.N = (int32_t)p.N; a.J = (int32_t)p.J; a.Hq = (int32_t)p.Hq; a.Hkv = (int32_t)p.Hkv; a.S = (int32_t)p.S; a.L = (int32_t)p.L;
  a.D = (int32_t)p.D; a.K = (int32_t)p.K; a.C = (int32_t)p.C;
  a.dtype = dtype_code(q); a.algo = (int32_t)algo; a.sm_scale = (float)sm_scale; a.off_by_one = (float)off_by_one;
  return a;
}

// The output tensor in the caller's shape -- (N, J, Hq, S, D), or (Z, Hq, S, D) -- and its {n, j, h, s} strides.
// token_major: memory order (n, j, s, h, d), so that the caller flattens it to (N, J*S, H*D) for free.
Tensor make_out(const Problem& p, const Tensor& q, bool gathered, bool token_major, int64_t os[4]) {
  if (token_major) { os[3] = p.Hq * p.D; os[2] = p.D; os[1] = p.S * os[3]; os[0] = p.J * os[1]; }
  else { os[3] = p.D; os[2] = p.S * p.D; os[1] = p.Hq * os[2]; os[0] = p.J * os[1]; }
  if (gathered) return at::empty_strided({p.N, p.Hq, p.S, p.D}, {os[0], os[2], os[3], 1}, q.options());
  return at::empty_strided({p.N, p.J, p.Hq, p.S, p.D}, {os[0], os[1], os[2], os[3], 1}, q.options());
}

struct Grads { Tensor dq, dk, dv, dw; };

Tensor grad_like(const Tensor& t) {
  Tensor g = at::empty_like(t);
  return g.stride(-1) == 1 ? g : at::empty(t.sizes(), t.options());
}

// The backward's tensors and argument block.  `ws` undefined: outputs and workspace are allocated here.
void backward_call(const Problem& p, bool gathered, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& idx, const Tensor& w,
                   const Tensor& dout_in, const Tensor& lse, double sm_scale, double off_by_one, int64_t algo, unsigned stages, Grads& g,
                   Tensor& ws) {
  const Tensor dout = inner_contiguous(dout_in);
  TORCH_CHECK_VALUE(dout.dim() == q.dim() && dout.scalar_type() == q.scalar_type(), "dout must be like q");
  Launch on(q);
  GcaBwdArgs a;
  a.q = q.const_data_ptr(); a.k_cache = k.const_data_ptr(); a.v_cache = v.const_data_ptr();
  a.indices = idx.defined() ? idx.const_data_ptr<int32_t>() : nullptr;
  a.weights = w.const_data_ptr<float>(); a.dout = dout.const_data_ptr(); a.lse = lse.const_data_ptr<float>();
  a.N = (int32_t)p.N; a.J = (int32_t)p.J; a.Hq = (int32_t)p.Hq; a.Hkv = (int32_t)p.Hkv; a.S = (int32_t)p.S; a.L = (int32_t)p.L;
  a.D = (int32_t)p.D; a.K = (int32_t)p.K; a.C = (int32_t)p.C;
  a.dtype = dtype_code(q); a.algo = (int32_t)algo; a.sm_scale = (float)sm_scale; a.off_by_one = (float)off_by_one;
  if (!ws.defined()) {
    g.dq = grad_like(q); g.dk = grad_like(k); g.dv = grad_like(v);
    g.dw = at::empty(w.sizes(), w.options());
    const int64_t need = (int64_t)api.gca_bwd_workspace_bytes(&a);
    ws = at::empty({need + 256}, q.options().dtype(at::kByte));
  }
  a.dq = g.dq.mutable_data_ptr(); a.dk_cache = g.dk.mutable_data_ptr(); a.dv_cache = g.dv.mutable_data_ptr();
  a.dw = g.dw.mutable_data_ptr<float>();
  a.status = status_ptr(on.dev);
  auto like_q = [&](const Tensor& t, int64_t s[4]) {
    if (gathered) { s[0] = s[1] = t.stride(0); s[2] = t.stride(1); s[3] = t.stride(2); }
    else for (int i = 0; i < 4; ++i) s[i] = t.stride(i);
  };
  auto like_cache = [&](const Tensor& t, int64_t s[4]) {
    if (gathered) { s[0] = t.stride(0); s[1] = t.stride(2); s[2] = t.stride(3); s[3] = t.stride(1); }
    else { int64_t d[4]; cache_view(t, p.D, d, s); }
  };
  copy4(a.q_stride, p.qs); copy4(a.k_stride, p.ks); copy4(a.v_stride, p.vs);
  like_q(dout, a.do_stride); like_q(g.dq, a.dq_stride);
  like_cache(g.dk, a.dk_stride); like_cache(g.dv, a.dv_stride);
  const uintptr_t base = (reinterpret_cast<uintptr_t>(ws.mutable_data_ptr()) + 255) / 256 * 256;
  a.workspace = reinterpret_cast<void*>(base);
  a.workspace_bytes = (size_t)(ws.numel() - 256);
  call("gca_bwd_stages", [&] { return api.gca_bwd_stages(&a, stages, on.stream); });
  maybe_check(on.dev);
}

// The autograd node of one GCA call: edges to q, k, v and the weights.
struct GcaBackward : public Node {
  SavedVariable q, k, v, idx, w, lse;
  bool gathered = false, released = false;
  double sm_scale = 0, off_by_one = 0;
  int64_t algo = 0;
  std::mutex mu;

  std::string name() const override { return "GcaBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mu);
    released = true;
    for (SavedVariable* s : {&q, &k, &v, &idx, &w, &lse}) s->reset_data();
  }
  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mu);
    TORCH_CHECK(!released, torch::autograd::ERR_BACKWARD_TWICE);
    variable_list out(4);
    if (!grads[0].defined()) return out;
    const Tensor tq = q.unpack(), tk = k.unpack(), tv = v.unpack(), ti = idx.unpack(), tw = w.unpack(), tl = lse.unpack();
    unsigned stages = GCA_BWD_STAGE_Q;                                  // the caches may be constants
    if (task_should_compute_output(1) || task_should_compute_output(2)) stages = GCA_BWD_STAGE_ALL;
    at::AutoDispatchBelowADInplaceOrView below;
    Grads g;
    Tensor ws;
    try {
      const Problem p = gathered ? gathered_problem(tq, tk, tv, tw) : indexed_problem(tq, tk, tv, ti, tw);
      backward_call(p, gathered, tq, tk, tv, ti, tw, grads[0], tl, sm_scale, off_by_one, algo, stages, g, ws);
    } catch (const LibraryError& e) { raise(e); }
    catch (const TimeoutError& e) { raise(e); }
    out[0] = g.dq; out[3] = g.dw;
    if (stages == GCA_BWD_STAGE_ALL) { out[1] = g.dk; out[2] = g.dv; }
    return out;
  }
  // an error of the package's own class, through the engine to the thread that called backward
  template <class E>
  [[noreturn]] static void raise(const E& e) {
    PyGILState_STATE gil = PyGILState_Ensure();
    set_python_error(e);
    python_error err;
    err.persist();
    PyGILState_Release(gil);
    throw err;
  }
};

// gca_indexed / attention: forward, recorded for autograd when a gradient can be asked for.
Tensor gca_autograd(Tensor q, Tensor k, Tensor v, const Tensor& idx_in, const Tensor& w_in, double sm_scale, double off_by_one, int64_t algo,
                    bool gathered, bool token_major) {
  TORCH_CHECK_NOT_IMPLEMENTED(!has_tangent({&q, &k, &v, &w_in}), "GCA has no forward-mode derivative");
  q = inner_contiguous(q);
  k = inner_contiguous(k);
  v = inner_contiguous(v);
  const Tensor idx = gathered ? Tensor() : as_int32(idx_in);
  const Tensor w = as_float(w_in);
  const Problem p = gathered ? gathered_problem(q, k, v, w) : indexed_problem(q, k, v, idx, w);
  std::shared_ptr<GcaBackward> node;
  if (torch::autograd::compute_requires_grad(q, k, v, w)) {
    node = std::shared_ptr<GcaBackward>(new GcaBackward(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(q, k, v, w));
    node->q = SavedVariable(q, false); node->k = SavedVariable(k, false); node->v = SavedVariable(v, false);
    node->idx = SavedVariable(idx, false); node->w = SavedVariable(w, false);
    node->gathered = gathered; node->sm_scale = sm_scale; node->off_by_one = off_by_one; node->algo = algo;
  }
  Tensor out, lse;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    Launch on(q);
    int64_t os[4];
    out = make_out(p, q, gathered, token_major, os);
    if (node) lse = at::empty({p.N * p.J, p.Hq, p.K, p.S}, w.options());       // only the backward reads it
    const GcaFwdArgs a =
        fwd_args(p, q, k, v, idx, w, out, os, node ? lse.mutable_data_ptr<float>() : nullptr, sm_scale, off_by_one, algo, on.dev);
    call("gca_fwd", [&] { return api.gca_fwd(&a, on.stream); });
    maybe_check(on.dev);
  }
  if (node) {
    node->lse = SavedVariable(lse, false);
    torch::autograd::set_history(out, node);
  }
  return out;
}

// Inference: up to 16 query rows take the decode kernels.
Tensor gca_nograd(const Tensor& q_in, const Tensor& k_in, const Tensor& v_in, const Tensor& idx_in, const Tensor& w_in, double sm_scale,
                  double off_by_one, int64_t algo, bool gathered, bool token_major) {
  at::AutoDispatchBelowADInplaceOrView below;
  const Tensor q = inner_contiguous(q_in), k = inner_contiguous(k_in), v = inner_contiguous(v_in);
  const Tensor idx = gathered ? Tensor() : as_int32(idx_in);
  const Tensor w = as_float(w_in);
  const Problem p = gathered ? gathered_problem(q, k, v, w) : indexed_problem(q, k, v, idx, w);
  Launch on(q);
  int64_t os[4];
  const Tensor out = make_out(p, q, gathered, token_major, os);
  if (p.S <= 16) {
    const GcaFwdArgs a = fwd_args(p, q, k, v, idx, w, out, os, nullptr, sm_scale, off_by_one, algo, on.dev);
    call("gca_decode", [&] { return api.gca_decode(&a, on.stream); });
  } else {
    const int64_t pick = p.S != 64 && algo == GCA_ALGO_AUTO ? (int64_t)GCA_ALGO_SIMT : algo;
    const GcaFwdArgs a = fwd_args(p, q, k, v, idx, w, out, os, nullptr, sm_scale, off_by_one, pick, on.dev);
    call("gca_fwd", [&] { return api.gca_fwd(&a, on.stream); });
  }
  maybe_check(on.dev);
  return out;
}

// Forward with the log-sum-exps returned, and the backward without autograd (tests, tools, stage timing).
std::tuple<Tensor, Tensor> gca_forward_lse(const Tensor& q_in, const Tensor& k_in, const Tensor& v_in, const Tensor& idx_in, const Tensor& w_in,
                                           double sm_scale, double off_by_one, int64_t algo) {
  at::AutoDispatchBelowADInplaceOrView below;
  const Tensor q = inner_contiguous(q_in), k = inner_contiguous(k_in), v = inner_contiguous(v_in);
  const Tensor idx = as_int32(idx_in), w = as_float(w_in);
  const Problem p = indexed_problem(q, k, v, idx, w);
  Launch on(q);
  int64_t os[4];
  const Tensor out = make_out(p, q, false, false, os);
  const Tensor lse = at::empty({p.N * p.J, p.Hq, p.K, p.S}, w.options());
  const GcaFwdArgs a = fwd_args(p, q, k, v, idx, w, out, os, lse.mutable_data_ptr<float>(), sm_scale, off_by_one, algo, on.dev);
  call("gca_fwd", [&] { return api.gca_fwd(&a, on.stream); });
  return {out, lse};
}

// ------------------------------------------------------------------------------------------- projections
void require_bf16(const Tensor& t, const char* name) {
  TORCH_CHECK(t.is_cuda(), name, ": the fused projections run on a CUDA device only (no CPU fallback)");
  TORCH_CHECK_VALUE(t.scalar_type() == at::kBFloat16, name, ": expected bfloat16, got ", t.scalar_type());
}

// (..., D) as M rows with one row stride; `hold` keeps a copy alive when no such view exists
struct Rows { int64_t m, stride; Tensor hold; };
Rows rows_of(const Tensor& t) {
  const int64_t d = t.size(-1);
  if (t.dim() == 2 && t.stride(1) == 1) return {t.size(0), t.stride(0), t};
  if (t.is_contiguous()) return {d ? t.numel() / d : 0, d, t};
  const Tensor c = t.contiguous();
  return {d ? c.numel() / d : 0, d, c};
}

Tensor row_rms(const Tensor& x, double eps) {
  at::AutoDispatchBelowADInplaceOrView below;
  const Rows r = rows_of(x);
  Launch on(x);
  const Tensor out = at::empty({r.m}, x.options().dtype(at::kFloat));
  RowRmsArgs a;
  a.x = r.hold.const_data_ptr(); a.row_scale = out.mutable_data_ptr<float>(); a.M = r.m; a.x_stride = r.stride;
  a.D = (int32_t)x.size(-1); a.eps = (float)eps;
  call("gca_row_rms", [&] { return api.gca_row_rms(&a, on.stream); });
  return out;
}

Tensor linear(const Tensor& x, const Tensor& weight, const Tensor& row_scale, const Tensor& residual, const Tensor& out_in) {
  at::AutoDispatchBelowADInplaceOrView below;
  const Rows r = rows_of(x);
  const int64_t n = weight.size(0);
  Launch on(x);
  Tensor out = out_in;
  if (!out.defined()) {
    c10::SmallVector<int64_t, 6> shape(x.sizes().begin(), x.sizes().end());
    shape.back() = n;
    out = at::empty(shape, x.options());
  }
  const Rows o = rows_of(out);
  TORCH_CHECK_VALUE(o.hold.const_data_ptr() == out.const_data_ptr(), "linear: `out` must be viewable as (M, N) rows");
  LinearArgs a{};
  a.x = r.hold.const_data_ptr(); a.w = weight.const_data_ptr(); a.out = o.hold.mutable_data_ptr();
  a.M = r.m; a.N = (int32_t)n; a.K = (int32_t)x.size(-1);
  a.x_stride = r.stride; a.w_stride = weight.stride(0); a.out_stride = o.stride;
  Rows res;
  if (residual.defined()) {
    require_bf16(residual, "linear residual");
    res = rows_of(residual);
    TORCH_CHECK_VALUE(res.m == o.m && residual.size(-1) == out.size(-1), "linear: residual ", residual.sizes(), " does not match the output ",
                      out.sizes());
    a.residual = res.hold.const_data_ptr(); a.residual_stride = res.stride;
  }
  if (row_scale.defined()) {
    TORCH_CHECK_VALUE(row_scale.scalar_type() == at::kFloat && row_scale.numel() == r.m && row_scale.is_contiguous(),
                      "linear: row_scale must be contiguous float32 with one value per row");
    a.row_scale = row_scale.const_data_ptr<float>();
  }
  a.status = status_ptr(on.dev);
  call("gca_linear", [&] { return api.gca_linear(&a, on.stream); });
  return out;
}

// RMSNorm(x) w^T with the norm's gain in w: a few rows take the latency-bound kernel, more the GEMM that sums the squares up on the way.
Tensor rmsnorm_linear(const Tensor& x, const Tensor& weight, double eps) {
  at::AutoDispatchBelowADInplaceOrView below;
  const Rows r = rows_of(x);
  Launch on(x);
  c10::SmallVector<int64_t, 6> shape(x.sizes().begin(), x.sizes().end());
  shape.back() = weight.size(0);
  const Tensor out = at::empty(shape, x.options());
  LinearBatchedArgs lp{};
  lp.one.x = r.hold.const_data_ptr(); lp.one.w = weight.const_data_ptr(); lp.one.out = out.mutable_data_ptr();
  lp.one.M = r.m; lp.one.N = (int32_t)weight.size(0); lp.one.K = (int32_t)x.size(-1);
  lp.one.x_stride = r.stride; lp.one.w_stride = weight.stride(0); lp.one.out_stride = weight.size(0);
  lp.batches = 1; lp.rms_eps = (float)eps;
  if (api.gca_linear_few_rows(r.m, (int32_t)weight.size(0), (int32_t)x.size(-1), 1))
    call("gca_linear", [&] { return api.gca_linear_batched(&lp, on.stream); });
  else {
    const Tensor scratch = at::empty({r.m}, x.options().dtype(at::kFloat));
    call("gca_linear", [&] { return api.gca_rms_linear_batched(&lp, scratch.mutable_data_ptr<float>(), on.stream); });
  }
  return out;
}

// One GCA sub-layer for inference: residual + o_proj(GCA(q_proj(RMSNorm(hidden)))) on hidden (n, chunks, s, dim).
// The q rows and the attention's output are token-major buffers, so nothing is re-laid out between the
// three steps, and the rows of a skipped first chunk (nothing retrieved: the residual alone, or zeros) are written by
// the output projection's launch.
Tensor layer_fused(const Tensor& hidden_in, const Tensor& q_weight, double eps, const Tensor& k, const Tensor& v, const Tensor& idx_in,
                   const Tensor& w_in, const Tensor& o_weight, const Tensor& residual_in, bool first_chunk_retrieves, int64_t heads,
                   double sm_scale) {
  at::AutoDispatchBelowADInplaceOrView below;
  const Tensor hidden = hidden_in.contiguous();
  TORCH_CHECK_VALUE(hidden.dim() == 4, "forward_fused: hidden_states must be (N, D, S, dim)");
  const int64_t n = hidden.size(0), chunks = hidden.size(1), s = hidden.size(2), dim = hidden.size(3), head_dim = dim / heads;
  Launch on(hidden);
  const Tensor out = at::empty({n, chunks * s, dim}, hidden.options());
  Tensor residual = residual_in;
  if (residual.defined()) {
    require_bf16(residual, "linear residual");
    TORCH_CHECK_VALUE(residual.sizes() == out.sizes(), "linear: residual ", residual.sizes(), " does not match the output ", out.sizes());
    if (residual.stride(2) != 1) residual = residual.contiguous();
  }
  if (idx_in.size(1) * idx_in.size(2) == 0 || out.numel() == 0) {         // nothing retrieved at all
    if (residual.defined()) out.copy_(residual);
    else out.zero_();
    return out;
  }
  const int64_t skip = chunks > 1 && !first_chunk_retrieves ? 1 : 0, J = chunks - skip, rows = J * s;
  const Tensor idx = as_int32(idx_in), w = as_float(w_in);
  Problem p;
  int64_t kd[4], vd[4];
  cache_view(k, head_dim, kd, p.ks);
  cache_view(v, head_dim, vd, p.vs);
  for (int i = 0; i < 4; ++i) TORCH_CHECK_VALUE(kd[i] == vd[i], "k_cache and v_cache must have the same shape");
  TORCH_CHECK_VALUE(k.scalar_type() == at::kBFloat16 && v.scalar_type() == at::kBFloat16, "q, k_cache and v_cache must share one dtype");
  TORCH_CHECK_VALUE(idx.dim() == 3 && idx.size(0) == n && idx.size(1) == J && w.sizes() == idx.sizes() && kd[0] == n,
                    "indices/weights must be (N, J, K) = (", n, ", ", J, ", K); got ", idx.sizes(), ", ", w.sizes());
  TORCH_CHECK_VALUE(kd[3] > 0 && heads % kd[3] == 0, "number of q heads must be a multiple of the number of kv heads");
  p.N = n; p.J = J; p.Hq = heads; p.S = s; p.D = head_dim; p.C = kd[1]; p.L = kd[2]; p.Hkv = kd[3]; p.K = idx.size(2);
  // a decode step of a few sequences is one launch
  if (chunks == 1 && skip == 0 && s <= 2 && head_dim == 64 && dim == heads * 64 && p.L == 64 && q_weight.size(0) == dim && o_weight.size(0) == dim) {
    LayerDecodeArgs d;
    d.x = hidden.const_data_ptr(); d.wq = q_weight.const_data_ptr(); d.wo = o_weight.const_data_ptr();
    d.k_cache = k.const_data_ptr(); d.v_cache = v.const_data_ptr(); d.indices = idx.const_data_ptr<int32_t>(); d.weights = w.const_data_ptr<float>();
    d.residual = nullptr; d.residual_batch_stride = d.residual_stride = 0;
    if (residual.defined()) {
      d.residual = residual.const_data_ptr(); d.residual_batch_stride = residual.stride(0); d.residual_stride = residual.stride(1);
    }
    d.out = out.mutable_data_ptr(); d.status = status_ptr(on.dev);
    d.wq_stride = q_weight.stride(0); d.wo_stride = o_weight.stride(0);
    copy4(d.k_stride, p.ks); copy4(d.v_stride, p.vs);
    d.N = (int32_t)n; d.S = (int32_t)s; d.H = (int32_t)heads; d.Hkv = (int32_t)p.Hkv; d.K = (int32_t)p.K; d.C = (int32_t)p.C;
    d.eps = (float)eps; d.sm_scale = (float)sm_scale;
    bool done = true;
    call("gca_layer_decode", [&] {
      const int rc = api.gca_layer_decode(&d, on.stream);
      done = rc != GCA_ERR_ALGO;
      return done ? rc : 0;
    });
    if (done) {
      maybe_check(on.dev);
      return out;
    }
  }
  const bool few = skip == 0 && api.gca_linear_few_rows(n * rows, (int32_t)q_weight.size(0), (int32_t)dim, 1);       // the norm rides on the projection
  const Tensor q = at::empty({2, n, J, s, dim}, hidden.options());      // [0]: q, [1]: the attention's output
  void* const vals = static_cast<char*>(q.mutable_data_ptr()) + q.stride(0) * 2;
  LinearBatchedArgs lp{};
  LinearArgs& a = lp.one;
  a.x = static_cast<const char*>(hidden.const_data_ptr()) + skip * s * dim * 2; a.w = q_weight.const_data_ptr(); a.out = q.mutable_data_ptr();
  a.M = rows; a.N = (int32_t)q_weight.size(0); a.K = (int32_t)dim;
  a.x_stride = dim; a.w_stride = q_weight.stride(0); a.out_stride = dim;
  lp.rms_eps = (float)eps;
  a.status = status_ptr(on.dev);
  lp.batches = (int32_t)n; lp.x_batch_stride = chunks * s * dim; lp.out_batch_stride = rows * dim;
  if (few) call("gca_linear", [&] { return api.gca_linear_batched(&lp, on.stream); });
  else {
    const Tensor scratch = at::empty({n * rows}, hidden.options().dtype(at::kFloat));
    call("gca_linear", [&] { return api.gca_rms_linear_batched(&lp, scratch.mutable_data_ptr<float>(), on.stream); });
  }
  // q as (n, J, heads, s, head_dim) by strides
  p.qs[0] = rows * dim; p.qs[1] = s * dim; p.qs[2] = head_dim; p.qs[3] = dim;
  GcaFwdArgs f = fwd_args(p, q, k, v, idx, w, q, p.qs, nullptr, sm_scale, 0.0, GCA_ALGO_AUTO, on.dev);
  f.out = vals;
  if (s <= 16) call("gca_decode", [&] { return api.gca_decode(&f, on.stream); });
  else {
    if (s != 64) f.algo = GCA_ALGO_SIMT;
    call("gca_fwd", [&] { return api.gca_fwd(&f, on.stream); });
  }
  a.x = vals; a.w = o_weight.const_data_ptr(); a.w_stride = o_weight.stride(0); a.N = (int32_t)o_weight.size(0);
  a.out = static_cast<char*>(out.mutable_data_ptr()) + skip * s * dim * 2;
  a.row_scale = nullptr;
  lp.rms_eps = 0.f;
  lp.x_batch_stride = rows * dim; lp.out_batch_stride = chunks * s * dim;
  lp.lead_rows = (int32_t)(skip * s);
  if (residual.defined()) {
    a.residual = static_cast<const char*>(residual.const_data_ptr()) + skip * s * residual.stride(1) * 2;
    a.residual_stride = residual.stride(1); lp.residual_batch_stride = residual.stride(0);
  }
  call("gca_linear", [&] { return api.gca_linear_batched(&lp, on.stream); });
  maybe_check(on.dev);
  return out;
}

Tensor silu_mul(const Tensor& gate_up) {
  at::AutoDispatchBelowADInplaceOrView below;
  const Rows r = rows_of(gate_up);
  const int64_t inter = gate_up.size(-1) / 2;
  TORCH_CHECK_VALUE(gate_up.size(-1) == 2 * inter, "silu_mul: the last dimension must hold gate and up halves of equal width");
  Launch on(gate_up);
  c10::SmallVector<int64_t, 6> shape(gate_up.sizes().begin(), gate_up.sizes().end());
  shape.back() = inter;
  const Tensor out = at::empty(shape, gate_up.options());
  call("gca_silu_mul", [&] {
    return api.gca_silu_mul(r.hold.const_data_ptr(), out.mutable_data_ptr(), r.m, (int32_t)inter, r.stride, inter, on.stream);
  });
  return out;
}

// ------------------------------------------------------------------------------------------- windowed attention
Tensor window_args(WindowDecodeArgs& a, const Tensor& q, const Tensor& k, const Tensor& v, int64_t window, const Tensor& slopes, double sm_scale) {
  const Tensor* ts[3] = {&q, &k, &v};
  const char* names[3] = {"window_decode q", "window_decode k", "window_decode v"};
  for (int i = 0; i < 3; ++i) {
    require_bf16(*ts[i], names[i]);
    TORCH_CHECK_VALUE(ts[i]->dim() == 4 && ts[i]->size(3) == 64 && ts[i]->stride(3) == 1, names[i],
                      " must be (N, H, L, 64) with contiguous head dimension");
  }
  TORCH_CHECK_VALUE(v.sizes() == k.sizes() && k.size(0) == q.size(0), "window_decode: k and v must be (N, Hkv, T, 64)");
  const int64_t n = q.size(0), hq = q.size(1), sq = q.size(2);
  const Tensor out = at::empty({n, hq, sq, 64}, q.options());
  a.q = q.const_data_ptr(); a.k = k.const_data_ptr(); a.v = v.const_data_ptr(); a.out = out.mutable_data_ptr();
  a.alibi_slopes = nullptr;
  if (slopes.defined()) {
    TORCH_CHECK_VALUE(slopes.scalar_type() == at::kFloat && slopes.numel() == hq && slopes.is_contiguous() && slopes.is_cuda(),
                      "window_decode: slopes must be contiguous float32 (Hq,) on the device");
    a.alibi_slopes = slopes.const_data_ptr<float>();
  }
  for (int i = 0; i < 3; ++i) {
    a.q_stride[i] = q.stride(i); a.o_stride[i] = out.stride(i); a.k_stride[i] = k.stride(i); a.v_stride[i] = v.stride(i);
  }
  a.N = (int32_t)n; a.Hq = (int32_t)hq; a.Hkv = (int32_t)k.size(1); a.Sq = (int32_t)sq; a.T = (int32_t)k.size(2); a.window = (int32_t)window;
  a.sm_scale = (float)sm_scale;
  return out;
}

Tensor window_decode(const Tensor& q, const Tensor& k, const Tensor& v, int64_t window, const Tensor& slopes, double sm_scale) {
  at::AutoDispatchBelowADInplaceOrView below;
  WindowDecodeArgs a;
  require_bf16(q, "window_decode q");
  Launch on(q);
  const Tensor out = window_args(a, q, k, v, window, slopes, sm_scale);
  call("gca_window_decode", [&] { return api.gca_window_decode(&a, on.stream); });
  return out;
}

Tensor window_ring_decode(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& k_new, const Tensor& v_new, const Tensor& rows_written,
                          int64_t window, const Tensor& slopes, double sm_scale) {
  at::AutoDispatchBelowADInplaceOrView below;
  require_bf16(k_new, "window_ring_decode k_new");
  require_bf16(v_new, "window_ring_decode v_new");
  TORCH_CHECK(rows_written.is_cuda(), "window_ring_decode rows_written: the fused projections run on a CUDA device only (no CPU fallback)");
  TORCH_CHECK_VALUE(rows_written.scalar_type() == at::kLong && rows_written.numel() == 1, "window_ring_decode: rows_written must be one int64 on the device");
  require_bf16(q, "window_decode q");
  Launch on(q);
  WindowRingDecodeArgs a;
  const Tensor out = window_args(a.attn, q, k, v, window, slopes, sm_scale);
  const int64_t n = k.size(0), h = k.size(1);
  // (N, Hkv, 1, 64) or (N, Hkv, 64): strides of (n, kv head)
  auto new_rows = [&](const Tensor& t, int64_t st[2]) {
    TORCH_CHECK_VALUE((t.dim() == 3 || (t.dim() == 4 && t.size(2) == 1)) && t.size(0) == n && t.size(1) == h && t.size(-1) == 64 && t.stride(-1) == 1,
                      "window_ring_decode: new rows must be bf16 with a contiguous head dimension and equal strides");
    st[0] = t.stride(0); st[1] = t.stride(1);
  };
  int64_t vs[2];
  new_rows(k_new, a.new_stride);
  new_rows(v_new, vs);
  TORCH_CHECK_VALUE(vs[0] == a.new_stride[0] && vs[1] == a.new_stride[1],
                    "window_ring_decode: new rows must be bf16 with a contiguous head dimension and equal strides");
  a.k_new = k_new.const_data_ptr(); a.v_new = v_new.const_data_ptr(); a.rows_written = rows_written.const_data_ptr<int64_t>();
  call("gca_window_ring_decode", [&] { return api.gca_window_ring_decode(&a, on.stream); });
  return out;
}

// ------------------------------------------------------------------------------------------- landmark retrieval
Tensor bf16_rows(const Tensor& t) {
  const Tensor b = t.scalar_type() == at::kBFloat16 ? t : t.to(at::kBFloat16);
  return b.stride(-1) == 1 ? b : b.contiguous();
}

// A contiguous tensor over part of a storage of its own kind of bytes: the five outputs of a retrieval are one
// allocation (they live and die together, and each allocator call is ~1 us of a call that takes 10).
Tensor carve(const c10::Storage& st, size_t byte_offset, at::IntArrayRef sizes, at::ScalarType dt) {
  Tensor t = at::detail::make_tensor<c10::TensorImpl>(c10::Storage(st), c10::DispatchKeySet(c10::DispatchKey::CUDA), c10::scalarTypeToTypeMeta(dt));
  t.unsafeGetTensorImpl()->set_storage_offset((int64_t)(byte_offset / c10::elementSize(dt)));
  t.unsafeGetTensorImpl()->set_sizes_contiguous(sizes);
  return t;
}

struct Retrieved { Tensor keys, indices, scores, weights, n_valid; };
struct Selection { Tensor indices, weights; };       // a selection that the caller never sees

// `kept`: the selection is written twice, for a backward pass that the caller's in-place changes to its own tensors must not reach.
Retrieved score_topk(const Tensor& q_in, const Tensor& k_in, int64_t topk, bool has_pos0, int64_t q_pos0, int64_t e_base, const Tensor& noise_in,
                     int64_t head_dim, int64_t score_round, int64_t splits, Selection* kept = nullptr) {
  at::AutoDispatchBelowADInplaceOrView below;
  const Tensor q = bf16_rows(q_in), k = bf16_rows(k_in);
  const int64_t n = q.size(0), cq = q.size(1), d = q.size(2), e = k.size(1);
  Launch on(q);
  c10::SmallVector<int64_t, 4> shape{n, cq};
  int64_t rows = n * cq;
  if (head_dim > 0) { shape.push_back(d / head_dim); rows *= d / head_dim; }
  const c10::SmallVector<int64_t, 4> row_shape = shape;
  shape.push_back(topk);
  const int64_t m = rows * topk;
  const Tensor block = at::empty({m * (kept ? 28 : 20) + rows * 4}, q.options().dtype(at::kByte));
  const c10::Storage& st = block.storage();
  Retrieved r;
  r.keys = carve(st, 0, shape, at::kLong);
  r.indices = carve(st, (size_t)m * 8, shape, at::kInt);
  r.scores = carve(st, (size_t)m * 12, shape, at::kFloat);
  r.weights = carve(st, (size_t)m * 16, shape, at::kFloat);
  r.n_valid = carve(st, (size_t)m * 20, row_shape, at::kInt);
  if (kept) {
    const size_t at = (size_t)m * 20 + (size_t)rows * 4;
    kept->indices = carve(st, at, shape, at::kInt);
    kept->weights = carve(st, at + (size_t)m * 4, shape, at::kFloat);
  }
  if (n * cq == 0) return r;
  LmkTopkArgs a{};
  Tensor noise;
  if (noise_in.defined()) {
    noise = as_float(noise_in);
    TORCH_CHECK_VALUE(noise.dim() == 3 && noise.size(0) == n && noise.size(1) == cq && noise.size(2) == e, "noise must be (N, Cq, E)");
    a.noise = noise.const_data_ptr<float>();
  }
  a.lmk_q = q.const_data_ptr(); a.lmk_k = k.const_data_ptr();
  a.out_keys = reinterpret_cast<uint64_t*>(r.keys.mutable_data_ptr()); a.out_indices = static_cast<int32_t*>(r.indices.mutable_data_ptr());
  a.out_scores = static_cast<float*>(r.scores.mutable_data_ptr()); a.out_weights = static_cast<float*>(r.weights.mutable_data_ptr());
  a.out_nvalid = static_cast<int32_t*>(r.n_valid.mutable_data_ptr());
  a.q_batch_stride = q.stride(0); a.q_row_stride = q.stride(1); a.k_batch_stride = k.stride(0); a.k_row_stride = k.stride(1);
  a.q_pos0 = has_pos0 ? q_pos0 : e - cq; a.e_base = e_base;
  a.N = (int32_t)n; a.Cq = (int32_t)cq; a.E = (int32_t)e; a.D = (int32_t)d; a.K = (int32_t)topk;
  a.head_dim = (int32_t)head_dim; a.score_round = (int32_t)score_round; a.splits = (int32_t)splits;
  const size_t need = api.lmk_topk_workspace_bytes(&a);
  const Tensor ws = at::empty({(int64_t)(need > 16 ? need : 16)}, q.options().dtype(at::kByte));
  a.workspace = ws.mutable_data_ptr(); a.workspace_bytes = need;
  call("lmk_score_topk", [&] {
    return api.lmk_score_topk_kept(&a, kept ? kept->indices.mutable_data_ptr<int32_t>() : nullptr,
                                   kept ? kept->weights.mutable_data_ptr<float>() : nullptr, on.stream);
  });
  return r;
}

// A tensor over the storage of `t` without its last row (axis 1 of a contiguous (N, Cq, K)); an in-place change to either counts for both.
Tensor without_last_row(const Tensor& t) {
  Tensor s = carve(t.storage(), (size_t)t.storage_offset() * t.element_size(), {0}, t.scalar_type());
  const int64_t cq = t.size(1);
  s.unsafeGetTensorImpl()->set_sizes_and_strides({t.size(0), cq > 0 ? cq - 1 : 0, t.size(2)}, t.strides());
  torch::autograd::impl::set_version_counter(s, torch::autograd::impl::version_counter(t));
  return s;
}

// The retrieval weights as a function of the landmarks: outputs the whole weights, then those without the last row.  The selection is the
// node's own copy.
struct WeightsBackward : public Node {
  SavedVariable q, k, indices, w;
  bool released = false;
  std::mutex mu;

  std::string name() const override { return "RetrievalWeightsBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mu);
    released = true;
    for (SavedVariable* s : {&q, &k, &indices, &w}) s->reset_data();
  }
  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mu);
    TORCH_CHECK(!released, torch::autograd::ERR_BACKWARD_TWICE);
    variable_list out(2);
    if (!grads[0].defined() && !grads[1].defined()) return out;
    const Tensor tq = q.unpack(), tk = k.unpack(), ti = indices.unpack(), tw = w.unpack();
    // gradients that are to be differentiated again, or come batched from vmap
    const auto plain = [](const Tensor& t) { return !t.defined() || t.has_storage(); };
    if (at::GradMode::is_enabled() || !plain(grads[0]) || !plain(grads[1])) return by_operations(tq, tk, ti, grads);
    at::AutoDispatchBelowADInplaceOrView below;
    const Tensor cq = inner_contiguous(tq), ck = inner_contiguous(tk);
    Launch on(cq);
    LmkGradArgs a{};
    a.lmk_q = cq.const_data_ptr(); a.lmk_k = ck.const_data_ptr();
    a.indices = ti.const_data_ptr<int32_t>(); a.weights = tw.const_data_ptr<float>();
    if (grads[0].defined()) {
      a.dw_all = grads[0].const_data_ptr<float>();
      for (int i = 0; i < 3; ++i) a.dw_all_stride[i] = grads[0].stride(i);
    }
    if (grads[1].defined()) {
      a.dw_rows = grads[1].const_data_ptr<float>(); a.rows = (int32_t)grads[1].size(1);
      for (int i = 0; i < 3; ++i) a.dw_rows_stride[i] = grads[1].stride(i);
    }
    if (task_should_compute_output(0)) { out[0] = at::empty(cq.sizes(), cq.options()); a.dlmk_q = out[0].mutable_data_ptr(); }
    if (task_should_compute_output(1)) { out[1] = at::empty(ck.sizes(), ck.options()); a.dlmk_k = out[1].mutable_data_ptr(); }
    a.q_batch_stride = cq.stride(0); a.q_row_stride = cq.stride(1); a.k_batch_stride = ck.stride(0); a.k_row_stride = ck.stride(1);
    a.N = (int32_t)cq.size(0); a.Cq = (int32_t)cq.size(1); a.E = (int32_t)ck.size(1); a.D = (int32_t)cq.size(2); a.K = (int32_t)ti.size(2);
    a.q_pos0 = ck.size(1) - cq.size(1);
    try {
      call("lmk_weights_backward", [&] { return api.lmk_weights_backward(&a, on.stream); });
    } catch (const LibraryError& e) { GcaBackward::raise(e); }
    return out;
  }
  // The same gradient as differentiable operations in float32, the weights among them.
  variable_list by_operations(const Tensor& tq, const Tensor& tk, const Tensor& ti, const variable_list& grads) {
    const double scale = 1.0 / std::sqrt((double)tq.size(2));
    const Tensor lq = tq.to(at::kFloat), lk = tk.to(at::kFloat), padding = ti < 0;
    const c10::List<std::optional<Tensor>> at_rows({at::arange(tq.size(0), ti.options().dtype(at::kLong)).view({-1, 1, 1}), ti.clamp_min(0).to(at::kLong)});
    const Tensor rows = lk.index(at_rows);                                                       // (N, Cq, K, D)
    const Tensor s = ((lq.unsqueeze(2) * rows).sum(-1) * scale).masked_fill(padding, -INFINITY);
    const Tensor weights = at::nan_to_num(at::softmax(s, -1), 0.0);
    Tensor dw = grads[0];
    if (grads[1].defined()) {
      const Tensor whole = at::constant_pad_nd(grads[1], {0, 0, 0, 1});                          // the last row is in the first output only
      dw = dw.defined() ? dw + whole : whole;
    }
    const Tensor ds = weights * (dw - (dw * weights).sum(-1, true)) * scale;
    variable_list out(2);
    if (task_should_compute_output(0)) out[0] = (ds.unsqueeze(-1) * rows).sum(2).to(tq.scalar_type());
    if (task_should_compute_output(1))
      out[1] = at::zeros_like(lk).index_put(at_rows, ds.unsqueeze(-1) * lq.unsqueeze(2), true).to(tk.scalar_type());
    return out;
  }
};

struct Retrieving { Tensor indices, weights; Retrieved full; };

// Selection and weights for query chunks 1 .. Cq - 1 (row i serves query chunk i + 1), recorded for autograd when a landmark
// needs a gradient.
Retrieving retrieve(const Tensor& q, const Tensor& k, int64_t topk, const Tensor& noise, int64_t score_round) {
  Retrieving r;
  const bool record = torch::autograd::compute_requires_grad(q, k);
  Selection kept;
  r.full = score_topk(q, k, topk, false, 0, 0, noise, 0, score_round, 0, record ? &kept : nullptr);
  r.indices = without_last_row(r.full.indices);
  r.weights = without_last_row(r.full.weights);
  if (record) {
    auto node = std::shared_ptr<WeightsBackward>(new WeightsBackward(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(q, k));
    node->q = SavedVariable(q, false); node->k = SavedVariable(k, false);
    node->indices = SavedVariable(kept.indices, false); node->w = SavedVariable(kept.weights, false);
    torch::autograd::set_history(r.full.weights, node);
    // the rows are a view of the whole with an edge of their own: an in-place change to either is recorded for both
    r.weights = torch::autograd::make_variable_differentiable_view(r.weights, torch::autograd::ViewInfo(r.full.weights, nullptr, nullptr),
                                                                   std::nullopt, false, torch::autograd::CreationMeta::DEFAULT);
    torch::autograd::set_history(r.weights, node);
  }
  return r;
}

// The projection + append of `count` chunks at chunk position `pos` of the caches.
void kv_project_append(const Tensor& x, const Tensor& wk, const Tensor& wv, const Tensor& k_cache, const Tensor& v_cache, const Tensor& lmk,
                       int64_t pos, int64_t capacity, bool zero_landmark) {
  at::AutoDispatchBelowADInplaceOrView below;
  Launch on(x);
  const Tensor ck = wk.contiguous(), cv = wv.contiguous();
  KvProjectArgs a;
  a.x = x.const_data_ptr(); a.wk = ck.const_data_ptr(); a.wv = cv.const_data_ptr();
  a.k_cache = k_cache.mutable_data_ptr(); a.v_cache = v_cache.mutable_data_ptr(); a.lmk_cache = lmk.mutable_data_ptr();
  a.status = status_ptr(on.dev);
  a.cache_batch_stride = k_cache.stride(0); a.lmk_cache_batch_stride = lmk.stride(0);
  a.N = (int32_t)x.size(0); a.count = (int32_t)x.size(1); a.pos = (int32_t)pos; a.D = (int32_t)x.size(3);
  a.capacity = (int32_t)capacity; a.lmk_capacity = (int32_t)lmk.size(1);
  a.zero_landmark = zero_landmark;
  call("gca_kv_project_append", [&] { return api.gca_kv_project_append(&a, on.stream); });
}

// K, V (N, capacity, L, HD) like `k` (N, D, L, HD) and landmarks (N, capacity, Dm) like `lmk` (.., Dm).
std::array<Tensor, 3> cache_buffers(const Tensor& k, const Tensor& lmk, int64_t capacity) {
  TORCH_CHECK_VALUE(k.dim() == 4 && lmk.dim() > 0, "cache_buffers: expected (N, D, L, HD) and (.., Dm)");
  at::AutoDispatchBelowADInplaceOrView below;
  c10::cuda::OptionalCUDAGuard guard;
  guard.set_index(k.device().index());
  const int64_t shape[4] = {k.size(0), capacity, k.size(2), k.size(3)}, rows[3] = {k.size(0), capacity, lmk.size(-1)};
  return {at::empty(shape, k.options()), at::empty(shape, k.options()), at::empty(rows, lmk.options())};
}

// ------------------------------------------------------------------------------------------- Python glue
// Positional arguments only; the Python functions in front of these give them their names and defaults.
struct Args {
  PyObject* const* v;
  Py_ssize_t n;
  Args(const char* name, PyObject* const* v_, Py_ssize_t n_, Py_ssize_t want) : v(v_), n(n_) {
    TORCH_CHECK_TYPE(n == want, name, ": expected ", want, " arguments, got ", n);
  }
  const Tensor& tensor(int i) const {
    TORCH_CHECK_TYPE(THPVariable_Check(v[i]), "argument ", i + 1, " must be a tensor, got ", Py_TYPE(v[i])->tp_name);
    return THPVariable_Unpack(v[i]);
  }
  Tensor maybe(int i) const { return v[i] == Py_None ? Tensor() : tensor(i); }
  int64_t integer(int i) const {
    const long long x = PyLong_AsLongLong(v[i]);
    if (x == -1 && PyErr_Occurred()) throw python_error();
    return x;
  }
  double real(int i) const {
    const double x = PyFloat_AsDouble(v[i]);
    if (x == -1.0 && PyErr_Occurred()) throw python_error();
    return x;
  }
  bool flag(int i) const { return PyObject_IsTrue(v[i]) == 1; }
};

void require_cuda(std::initializer_list<const Tensor*> ts) {
  for (const Tensor* t : ts) TORCH_CHECK(t->is_cuda(), "GCA runs on CUDA tensors only (there is no CPU path)");
}

template <class F>
PyObject* guarded(F&& f) {
  HANDLE_TH_ERRORS
  try {
    return f();
  } catch (const LibraryError& e) {
    set_python_error(e);
  } catch (const TimeoutError& e) {
    set_python_error(e);
  }
  return nullptr;
  END_HANDLE_TH_ERRORS
}

// The work itself runs without the interpreter lock (a launch can block when the stream's queue is full).
template <class F>
auto unlocked(F&& f) {
  NoGil no_gil;
  return f();
}

PyObject* wrap(const Tensor& t) { return THPVariable_Wrap(t); }
PyObject* wrap_tuple(std::initializer_list<Tensor> ts) {
  PyObject* out = PyTuple_New((Py_ssize_t)ts.size());
  if (!out) throw python_error();
  Py_ssize_t i = 0;
  for (const Tensor& t : ts) PyTuple_SET_ITEM(out, i++, wrap(t));
  return out;
}

#define ENTRY(name, count) PyObject* py_##name(PyObject*, PyObject* const* argv, Py_ssize_t argc) { \
  return guarded([&]() -> PyObject* { const Args a(#name, argv, argc, count);
#define ENTRY_END }); }

ENTRY(gca_indexed, 9)
  const Tensor &q = a.tensor(0), &k = a.tensor(1), &v = a.tensor(2), &idx = a.tensor(3), &w = a.tensor(4);
  require_cuda({&q, &k, &v, &idx, &w});
  const double scale = a.real(5), obo = a.real(6);
  const int64_t algo = a.integer(7);
  const bool token_major = a.flag(8);
  return wrap(unlocked([&] { return gca_autograd(q, k, v, idx, w, scale, obo, algo, false, token_major); }));
ENTRY_END

ENTRY(attention, 5)
  const Tensor &q = a.tensor(0), &k = a.tensor(1), &v = a.tensor(2), &w = a.tensor(3);
  require_cuda({&q, &k, &v, &w});
  const double scale = a.real(4);
  return wrap(unlocked([&] { return gca_autograd(q, k, v, Tensor(), w, scale, 0.0, GCA_ALGO_AUTO, true, false); }));
ENTRY_END

ENTRY(gca_nograd, 9)
  const Tensor &q = a.tensor(0), &k = a.tensor(1), &v = a.tensor(2), &idx = a.tensor(3), &w = a.tensor(4);
  require_cuda({&q, &k, &v, &idx, &w});
  const double scale = a.real(5), obo = a.real(6);
  const int64_t algo = a.integer(7);
  const bool token_major = a.flag(8);
  return wrap(unlocked([&] { return gca_nograd(q, k, v, idx, w, scale, obo, algo, false, token_major); }));
ENTRY_END

ENTRY(gca_kv_cache, 5)
  const Tensor &q = a.tensor(0), &k = a.tensor(1), &v = a.tensor(2), &w = a.tensor(3);
  require_cuda({&q, &k, &v, &w});
  const double scale = a.real(4);
  return wrap(unlocked([&] { return gca_nograd(q, k, v, Tensor(), w, scale, 0.0, GCA_ALGO_AUTO, true, false); }));
ENTRY_END

ENTRY(gca_forward_lse, 8)
  const Tensor &q = a.tensor(0), &k = a.tensor(1), &v = a.tensor(2), &idx = a.tensor(3), &w = a.tensor(4);
  require_cuda({&q, &k, &v, &idx, &w});
  const double scale = a.real(5), obo = a.real(6);
  const int64_t algo = a.integer(7);
  const auto r = unlocked([&] { return gca_forward_lse(q, k, v, idx, w, scale, obo, algo); });
  return wrap_tuple({std::get<0>(r), std::get<1>(r)});
ENTRY_END

// (q, k, v, idx, w, dout, lse, scale, off_by_one, algo, stages, bufs or None) -> (dq, dk, dv, dw, workspace)
ENTRY(gca_backward, 12)
  const Tensor &q_in = a.tensor(0), &k_in = a.tensor(1), &v_in = a.tensor(2), &idx_in = a.tensor(3), &w_in = a.tensor(4);
  const Tensor &dout = a.tensor(5), &lse = a.tensor(6);
  require_cuda({&q_in, &k_in, &v_in, &idx_in, &w_in, &dout, &lse});
  const double scale = a.real(7), obo = a.real(8);
  const int64_t algo = a.integer(9), stages = a.integer(10);
  Grads g;
  Tensor ws;
  if (argv[11] != Py_None) {
    TORCH_CHECK_TYPE(PyTuple_Check(argv[11]) && PyTuple_GET_SIZE(argv[11]) == 5, "bufs must be (dq, dk, dv, dw, workspace)");
    Tensor* const to[5] = {&g.dq, &g.dk, &g.dv, &g.dw, &ws};
    for (int i = 0; i < 5; ++i) {
      PyObject* o = PyTuple_GET_ITEM(argv[11], i);
      TORCH_CHECK_TYPE(THPVariable_Check(o), "bufs must hold tensors");
      *to[i] = THPVariable_Unpack(o);
    }
  }
  unlocked([&] {
    at::AutoDispatchBelowADInplaceOrView below;
    const Tensor q = inner_contiguous(q_in), idx = as_int32(idx_in), w = as_float(w_in);
    Tensor k = inner_contiguous(k_in), v = inner_contiguous(v_in);
    const Problem p = indexed_problem(q, k, v, idx, w);
    for (Tensor* t : {&k, &v})                                         // gradients with the head axis apart
      if (t->dim() == 4) *t = t->unflatten(3, {p.Hkv, p.D});
    backward_call(p, false, q, k, v, idx, w, dout, lse, scale, obo, algo, (unsigned)stages, g, ws);
    return 0;
  });
  return wrap_tuple({g.dq, g.dk, g.dv, g.dw, ws});
ENTRY_END

ENTRY(row_rms, 2)
  const Tensor& x = a.tensor(0);
  require_bf16(x, "row_rms");
  const double eps = a.real(1);
  return wrap(unlocked([&] { return row_rms(x, eps); }));
ENTRY_END

ENTRY(linear, 5)
  const Tensor &x = a.tensor(0), &w = a.tensor(1);
  require_bf16(x, "linear");
  require_bf16(w, "linear weight");
  const Tensor scale = a.maybe(2), residual = a.maybe(3), out = a.maybe(4);
  return wrap(unlocked([&] { return linear(x, w, scale, residual, out); }));
ENTRY_END

// (q, landmarks, topk, noise or None, score_round) -> (indices[:, :-1], weights[:, :-1], keys, indices, scores, weights, n_valid);
// None when the landmarks carry tangents
ENTRY(retrieve, 5)
  const Tensor &q = a.tensor(0), &k = a.tensor(1);
  TORCH_CHECK(q.is_cuda() && k.is_cuda(), "landmark retrieval runs on CUDA tensors only (there is no CPU path)");
  TORCH_CHECK_VALUE(q.dim() == 3 && k.dim() == 3 && q.size(0) == k.size(0) && q.size(2) == k.size(2), "expected lmk_q (N, Cq, D) and lmk_k (N, E, D)");
  const int64_t topk = a.integer(2), round = a.integer(4);
  const Tensor noise = a.maybe(3);
  if (has_tangent({&q, &k})) Py_RETURN_NONE;
  const Retrieving r = unlocked([&] { return retrieve(q, k, topk, noise, round); });
  return wrap_tuple({r.indices, r.weights, r.full.keys, r.full.indices, r.full.scores, r.full.weights, r.full.n_valid});
ENTRY_END

ENTRY(rmsnorm_linear, 3)
  const Tensor &x = a.tensor(0), &w = a.tensor(1);
  require_bf16(x, "linear");
  require_bf16(w, "linear weight");
  const double eps = a.real(2);
  return wrap(unlocked([&] { return rmsnorm_linear(x, w, eps); }));
ENTRY_END

// (hidden, q weight with the norm's gain, eps, k, v, idx, w, o weight, residual or None, first chunk retrieves, heads, scale)
ENTRY(layer_fused, 12)
  const Tensor &x = a.tensor(0), &qw = a.tensor(1), &k = a.tensor(3), &v = a.tensor(4), &idx = a.tensor(5), &w = a.tensor(6), &ow = a.tensor(7);
  require_bf16(x, "linear");
  require_bf16(qw, "linear weight");
  require_bf16(ow, "linear weight");
  require_cuda({&k, &v, &idx, &w});
  const double eps = a.real(2), scale = a.real(11);
  const Tensor residual = a.maybe(8);
  const bool first = a.flag(9);
  const int64_t heads = a.integer(10);
  return wrap(unlocked([&] { return layer_fused(x, qw, eps, k, v, idx, w, ow, residual, first, heads, scale); }));
ENTRY_END

ENTRY(silu_mul, 1)
  const Tensor& x = a.tensor(0);
  require_bf16(x, "silu_mul");
  return wrap(unlocked([&] { return silu_mul(x); }));
ENTRY_END

ENTRY(window_decode, 6)
  const Tensor &q = a.tensor(0), &k = a.tensor(1), &v = a.tensor(2);
  const int64_t window = a.integer(3);
  const Tensor slopes = a.maybe(4);
  const double scale = a.real(5);
  return wrap(unlocked([&] { return window_decode(q, k, v, window, slopes, scale); }));
ENTRY_END

ENTRY(window_ring_decode, 9)
  const Tensor &q = a.tensor(0), &k = a.tensor(1), &v = a.tensor(2), &kn = a.tensor(3), &vn = a.tensor(4), &count = a.tensor(5);
  const int64_t window = a.integer(6);
  const Tensor slopes = a.maybe(7);
  const double scale = a.real(8);
  return wrap(unlocked([&] { return window_ring_decode(q, k, v, kn, vn, count, window, slopes, scale); }));
ENTRY_END

// (q, landmarks, topk, q_pos0 or None, e_base, noise or None, head_dim, score_round, splits)
ENTRY(lmk_score_topk, 9)
  const Tensor &q = a.tensor(0), &k = a.tensor(1);
  TORCH_CHECK(q.is_cuda() && k.is_cuda(), "landmark retrieval runs on CUDA tensors only (there is no CPU path)");
  TORCH_CHECK_VALUE(q.dim() == 3 && k.dim() == 3 && q.size(0) == k.size(0) && q.size(2) == k.size(2), "expected lmk_q (N, Cq, D) and lmk_k (N, E, D)");
  const int64_t topk = a.integer(2), pos0 = argv[3] == Py_None ? 0 : a.integer(3), e_base = a.integer(4), head_dim = a.integer(6),
                round = a.integer(7), splits = a.integer(8);
  const bool has_pos0 = argv[3] != Py_None;
  const Tensor noise = a.maybe(5);
  const Retrieved r = unlocked([&] { return score_topk(q, k, topk, has_pos0, pos0, e_base, noise, head_dim, round, splits); });
  return wrap_tuple({r.keys, r.indices, r.scores, r.weights, r.n_valid});
ENTRY_END

ENTRY(kv_project_append, 9)
  const Tensor &x = a.tensor(0), &wk = a.tensor(1), &wv = a.tensor(2), &k = a.tensor(3), &v = a.tensor(4), &lmk = a.tensor(5);
  const int64_t pos = a.integer(6), capacity = a.integer(7);
  const bool zero = a.flag(8);
  unlocked([&] { kv_project_append(x, wk, wv, k, v, lmk, pos, capacity, zero); return 0; });
  Py_RETURN_NONE;
ENTRY_END

ENTRY(cache_buffers, 3)
  const Tensor &k = a.tensor(0), &lmk = a.tensor(1);
  const int64_t capacity = a.integer(2);
  const auto t = unlocked([&] { return cache_buffers(k, lmk, capacity); });
  return wrap_tuple({t[0], t[1], t[2]});
ENTRY_END

ENTRY(status_word, 1)
  const int64_t dev = a.integer(0);
  return wrap(unlocked([&] { return status_word((int)dev); }));
ENTRY_END

ENTRY(set_switches, 2)                      // (NVTX ranges, status check after every call)
  nvtx_on = a.flag(0);
  check_on = a.flag(1);
  Py_RETURN_NONE;
ENTRY_END

// ({entry point name: address}, GcaError)
ENTRY(bind, 2)
  TORCH_CHECK_TYPE(PyDict_Check(argv[0]), "bind: expected a dict of addresses");
  auto address = [&](const char* name) {
    PyObject* o = PyDict_GetItemString(argv[0], name);
    TORCH_CHECK_VALUE(o, "bind: the library has no ", name);
    void* p = PyLong_AsVoidPtr(o);
    if (!p) { if (PyErr_Occurred()) throw python_error(); TORCH_CHECK_VALUE(false, "bind: null address for ", name); }
    return p;
  };
#define GCA_API(name) api.name = reinterpret_cast<decltype(api.name)>(address(#name));
  GCA_API_LIST
#undef GCA_API
  Py_INCREF(argv[1]);
  Py_XSETREF(gca_error, argv[1]);
  Py_RETURN_NONE;
ENTRY_END

#define METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(&py_##name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    METHOD(bind), METHOD(set_switches), METHOD(status_word), METHOD(gca_indexed), METHOD(attention), METHOD(gca_nograd), METHOD(gca_kv_cache),
    METHOD(gca_forward_lse), METHOD(gca_backward), METHOD(row_rms), METHOD(linear), METHOD(rmsnorm_linear), METHOD(layer_fused), METHOD(silu_mul),
    METHOD(window_decode), METHOD(window_ring_decode), METHOD(lmk_score_topk), METHOD(retrieve), METHOD(kv_project_append), METHOD(cache_buffers), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_host", "Host path of the hot entry points.", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) { return PyModule_Create(&module_def); }
