// The single-device operator as PyTorch sees it: argument checks, head-dimension slices, allocation, the C-ABI
// calls and the autograd node, in native code.  The kernels of an ordinary layer take tens of microseconds; the same
// steps as a Python autograd function with ctypes calls took the host about 210 us for a forward and a backward
// pass (57 us for a forward pass alone) and set the pace of every call below about 50 MB of inputs.
//
// Interface of LightningAttention, lasp/lightning_attention.py:396-504, with the wrapper's head-dimension slicing
// (:510-531: a sum over 128-wide q,k slices, v slices side by side): every 128-wide slice pair is read and written
// where it lies in the wide tensors (row pitch in the problem), later contributions to a slice of o, dq, dk, dv
// are added by the kernels' own stores.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/SavedTensorHooks.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/CUDAGraphsUtils.cuh>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/library.h>

#include <nvtx3/nvToolsExt.h>

#include <cmath>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <mutex>
#include <tuple>
#include <utility>
#include <vector>

#include "lasp_b200.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

constexpr int64_t kSlice = 128;      // widest q/k (d) or v (e) slice one kernel call takes
constexpr int64_t kSyncBytes = 4096; // synchronisation words of a launch (lasp_call_options.sync)

struct Range {   // NVTX range around a library call (LASP_B200_NVTX=1)
  bool on;
  explicit Range(const char* name) : on(enabled()) {
    if (on) nvtxRangePushA(name);
  }
  ~Range() {
    if (on) nvtxRangePop();
  }
  static bool enabled() {
    static const bool v = [] {
      const char* e = std::getenv("LASP_B200_NVTX");
      return e && e[0] == '1';
    }();
    return v;
  }
};

// A negative status becomes lasp_b200._cabi.LaspStatusError, on whatever thread this is (autograd's workers too).
void check_status(const char* fn, int status) {
  if (status >= 0) return;
  std::string text = lasp_b200_strerror(status);
  if (status == LASP_ERR_CUDA) text += std::string(": ") + lasp_b200_last_cuda_error();
  PyGILState_STATE gil = PyGILState_Ensure();
  PyObject* mod = PyImport_ImportModule("lasp_b200._cabi");
  PyObject* cls = mod ? PyObject_GetAttrString(mod, "LaspStatusError") : nullptr;
  PyObject* exc = cls ? PyObject_CallFunction(cls, "sis", fn, status, text.c_str()) : nullptr;
  if (exc) PyErr_SetObject(cls, exc);
  Py_XDECREF(exc);
  Py_XDECREF(cls);
  Py_XDECREF(mod);
  python_error err;
  err.persist();
  PyGILState_Release(gil);
  throw err;
}

int32_t lasp_dtype_of(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return LASP_F32;
    case at::kBFloat16: return LASP_BF16;
    case at::kHalf: return LASP_F16;
    default: TORCH_CHECK_TYPE(false, "unsupported dtype ", t, "; use float32, bfloat16 or float16");
  }
}

int32_t requested_path() {   // env LASP_B200_PATH, looked at on every call as the Python launcher does
  const char* p = std::getenv("LASP_B200_PATH");
  if (!p || !*p || !std::strcmp(p, "auto")) return LASP_PATH_AUTO;
  if (!std::strcmp(p, "simt")) return LASP_PATH_SIMT;
  if (!std::strcmp(p, "tensor")) return LASP_PATH_TENSOR;
  TORCH_CHECK_VALUE(false, "unknown kernel path '", p, "'; use auto, simt or tensor");
}

// The 4 KB of synchronisation words of the current stream's launches: zeroed once, then kept consistent by the
// kernels.  Launches of one stream do not overlap, so they share a block; a capturing stream gets a block per call,
// zeroed by the graph itself, because the graph may be replayed anywhere.  At most kMaxBlocks are kept, the oldest
// going first; a block comes from its stream's allocator pool, so giving it back is ordered behind its last use.
Tensor sync_words(const at::Device& device, const at::cuda::CUDAStream& stream) {
  const auto fresh = [&] { return at::zeros({kSyncBytes}, at::TensorOptions().dtype(at::kByte).device(device)); };
  if (at::cuda::currentStreamCaptureStatusMayInitCtx() != at::cuda::CaptureStatus::None) return fresh();
  struct Block {
    int64_t device;
    unsigned long long stream;
    Tensor words;
  };
  constexpr size_t kMaxBlocks = 64;
  static std::mutex lock;
  static auto* blocks = new std::deque<Block>;   // never destroyed: the process may end after the CUDA context
  unsigned long long id = 0;
  C10_CUDA_CHECK(cudaStreamGetId(stream.stream(), &id));   // unique, unlike a handle that a later stream may reuse
  std::lock_guard<std::mutex> guard(lock);
  for (const Block& b : *blocks)
    if (b.stream == id && b.device == device.index()) return b.words;
  if (blocks->size() >= kMaxBlocks) blocks->pop_front();
  blocks->push_back({device.index(), id, fresh()});
  return blocks->back().words;
}

struct Shape {
  int64_t b, h, n, d, e;
};

Shape check_inputs(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& s) {
  TORCH_CHECK_VALUE(q.dim() == 4 && k.sizes() == q.sizes() && v.dim() == 4 && v.sizes().slice(0, 3) == q.sizes().slice(0, 3),
                    "expected q,k (b,h,n,d) and v (b,h,n,e); got ", q.sizes(), ", ", k.sizes(), ", ", v.sizes());
  TORCH_CHECK_TYPE(k.scalar_type() == q.scalar_type() && v.scalar_type() == q.scalar_type(), "q, k, v must share one dtype");
  TORCH_CHECK_VALUE(s.numel() == q.size(1), "decay tensor has ", s.numel(), " entries for ", q.size(1), " heads");
  for (const auto& [name, width] : {std::pair<const char*, int64_t>{"q/k", q.size(3)}, {"v", v.size(3)}})
    TORCH_CHECK_VALUE(width % 16 == 0, "head dimension of ", name, " is ", width, ": it must be a multiple of 16 (wider than ",
                      kSlice, ": cut in ", kSlice, "-wide slices)");
  TORCH_CHECK_VALUE(q.size(0) * q.size(1) <= 65535, "batch x heads = ", q.size(0) * q.size(1), " exceeds 65535");
  lasp_dtype_of(q.scalar_type());
  // (a width of zero is a multiple of 16: it would leave no slice to run and the output as it was allocated)
  if (q.size(3) == 0 || v.size(3) == 0) check_status("lasp_b200_resolve_path", LASP_ERR_SHAPE);
  // (a call without gradients does not pass through the autograd function, which would refuse a tangent)
  for (const Tensor* t : {&q, &k, &v, &s})
    TORCH_CHECK_NOT_IMPLEMENTED(!t->_fw_grad(0).defined(), "lasp_b200 has no forward-mode derivative");
  for (const Tensor* t : {&q, &k, &v})
    TORCH_CHECK(t->is_cuda(), "lasp_b200 runs on CUDA tensors only (there is no CPU fallback); got a tensor on ", t->device());
  return {q.size(0), q.size(1), q.size(2), q.size(3), v.size(3)};
}

lasp_problem problem_of(const Shape& m, int64_t d, int64_t e, int32_t dtype, double scale, int64_t map, bool pitched) {
  TORCH_CHECK_VALUE(m.n <= INT32_MAX, "sequence of ", m.n, " tokens is too long");
  lasp_problem p = {};
  p.b = (int32_t)m.b, p.h = (int32_t)m.h, p.n = (int32_t)m.n, p.d = (int32_t)d, p.e = (int32_t)e;
  p.dtype = dtype, p.path = requested_path();
  p.qk_map = (int32_t)map, p.qk_scale = (float)scale;
  if (pitched) p.pitch_d = (int32_t)m.d, p.pitch_e = (int32_t)m.e;
  return p;
}

// One 128-wide slice pair of the head dimensions: columns [d0, d1) of q,k and [e0, e1) of v, where they lie in the
// wide tensors.
struct Pair {
  int64_t d0, d1, e0, e1;
  lasp_problem problem;
  size_t ws_bytes;
};

bool resolve(lasp_problem& p) {
  const int path = lasp_b200_resolve_path(&p);
  if (path < 0) return false;
  p.path = path;
  return true;
}

std::vector<Pair> slice_pairs(const Shape& m, int32_t dtype, double scale, int64_t map) {
  std::vector<Pair> pairs;
  const bool wide = m.d > kSlice || m.e > kSlice;
  for (int64_t e0 = 0; e0 < m.e; e0 += kSlice)
    for (int64_t d0 = 0; d0 < m.d; d0 += kSlice) {
      Pair p{d0, std::min(d0 + kSlice, m.d), e0, std::min(e0 + kSlice, m.e), {}, 0};
      p.problem = problem_of(m, p.d1 - p.d0, p.e1 - p.e0, dtype, scale, map, wide);
      if (!resolve(p.problem)) check_status("lasp_b200_resolve_path", lasp_b200_resolve_path(&p.problem));
      p.ws_bytes = lasp_b200_fwd_workspace_bytes(&p.problem);
      pairs.push_back(p);
    }
  return pairs;
}

char* column(const Tensor& t, int64_t col) { return static_cast<char*>(t.data_ptr()) + col * t.element_size(); }

// Heads of 256: whether each result is made in one pass (1) or slice by slice
bool in_one_pass(const Shape& m, int32_t dtype, double scale, int64_t map, bool backward, lasp_problem* p) {
  if (m.d != 256 || m.e != 256) return false;
  *p = problem_of(m, m.d, m.e, dtype, scale, map, false);
  return lasp_b200_wide_ok(p, backward ? 1 : 0) == 1;
}

std::vector<Tensor> run_forward(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& s, const Shape& m,
                                double scale, int64_t map, bool keep) {
  const c10::cuda::CUDAGuard guard(q.device());
  const auto stream = at::cuda::getCurrentCUDAStream();
  Tensor o = at::empty({m.b, m.h, m.n, m.e}, q.options());
  lasp_problem wide;
  if (keep && in_one_pass(m, lasp_dtype_of(q.scalar_type()), scale, map, true, &wide)) keep = false;   // such a backward pass needs no states
  if (!keep && in_one_pass(m, lasp_dtype_of(q.scalar_type()), scale, map, false, &wide)) {
    lasp_fwd_args a = {};
    a.q = q.data_ptr(), a.k = k.data_ptr(), a.v = v.data_ptr(), a.s = s.const_data_ptr<float>(), a.o = o.data_ptr();
    Range range("lasp_b200_forward");
    check_status("lasp_b200_forward_wide", lasp_b200_forward_wide(&wide, &a, stream.stream()));
    return {o};
  }
  const Tensor sync = sync_words(q.device(), stream);
  std::vector<Tensor> out{o};
  Tensor ws;
  for (const Pair& p : slice_pairs(m, lasp_dtype_of(q.scalar_type()), scale, map)) {
    // (nothing is kept without a backward pass: the slices then share a workspace)
    if (keep || !ws.defined() || (size_t)ws.numel() < p.ws_bytes)
      ws = at::empty({(int64_t)p.ws_bytes}, q.options().dtype(at::kByte));
    if (keep) out.push_back(ws);
    lasp_fwd_args a = {};
    a.q = column(q, p.d0), a.k = column(k, p.d0), a.v = column(v, p.e0), a.s = s.const_data_ptr<float>();
    a.o = column(o, p.e0);
    a.ws = ws.data_ptr(), a.ws_bytes = (size_t)ws.numel();
    lasp_call_options opt = {};
    opt.sync = static_cast<uint32_t*>(sync.data_ptr());
    opt.keep_states = keep ? 1 : 0;
    opt.accumulate = p.d0 > 0 ? LASP_ACCUMULATE_V : 0;   // a v slice collects from every q/k slice
    opt.alone = 1;
    Range range("lasp_b200_forward");
    check_status("lasp_b200_forward", lasp_b200_forward_opt(&p.problem, &a, &opt, stream.stream()));
  }
  return out;
}

// Whether q and k go through elu(x) + 1 in a pass of their own, ahead of the kernels, or tile by tile inside them.  The
// kernels of a training step map a tile up to five times and evaluate the exponential of the chain rule twice more; the pass
// costs a launch and 8 bytes of memory traffic an element.  Passes through the operator, training, 64-wide 4 x 16 x 4096 272 -> 198
// us, 2 x 16 x 2048 92 -> 87, 2 x 16 x 1024 83 -> 86; 128-wide 8 x 32 x 2048 754 -> 610, 2 x 16 x 1024 93 -> 87, 1 x 16 x 1024 81 -> 86:
// from 2^22 elements of q on.  A forward pass alone: v 64 wide 4 x 16 x 4096 80 -> 73, 2 x 16 x 2048 29 -> 28, 2 x 16 x 1024 even; 128
// wide never.  Those are without decay; with it tiles next to a span's border alone are read twice, which moves the line
// little.  Launches alone, inside -> ahead, without / with decay: training 64-wide 4 x 16 x 4096 251 -> 180 / 241 -> 176, 2 x 16 x 1024
// 52 -> 45 / 52 -> 44, 128-wide 8 x 32 x 2048 699 -> 543 / 700 -> 535, 1 x 16 x 16384 394 -> 311 / 372 -> 287; forward 64-wide 4 x 16 x 4096
// 71 -> 64 / 67 -> 62, 128-wide 8 x 32 x 2048 174 -> 174 / 172 -> 176.
bool map_first(const Shape& m, bool train) { return m.b * m.h * m.n * m.d >= (int64_t{1} << 22) && (train || m.e <= 64); }

std::pair<Tensor, Tensor> mapped_qk(const Tensor& q, const Tensor& k) {
  const c10::cuda::CUDAGuard guard(q.device());
  const auto stream = at::cuda::getCurrentCUDAStream();
  Tensor qm = at::empty(q.sizes(), q.options()), km = at::empty(k.sizes(), k.options());
  check_status("lasp_b200_map_qk", lasp_b200_map_qk(q.data_ptr(), k.data_ptr(), qm.data_ptr(), km.data_ptr(), q.numel(), stream.stream()));
  return {qm, km};
}

// What autograd asks of a saved tensor when it is taken out again, for q and k whose mapped copies are saved in their place:
// that nobody has written to them since.  (Saving them beside the copies would hold twice the memory until the backward
// pass.)  Under saved-tensor hooks it does not ask, what they have packed being theirs.
struct Unwritten : torch::CustomClassHolder {
  c10::VariableVersion counter[2];
  uint32_t at[2];
  Unwritten(const Tensor& q, const Tensor& k)
      : counter{torch::autograd::impl::version_counter(q), torch::autograd::impl::version_counter(k)},
        at{counter[0].current_version(), counter[1].current_version()} {}
  void check() const {
    for (int i = 0; i < 2; ++i)
      TORCH_CHECK(counter[i].current_version() == at[i],
                  "one of the variables needed for gradient computation has been modified by an inplace operation: ", i ? "k" : "q",
                  " of lasp_b200 attention is at version ", counter[i].current_version(), "; expected version ", at[i], " instead");
  }
};

class Lightning : public torch::autograd::Function<Lightning> {
 public:
  static Tensor forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& s,
                        double scale, int64_t map) {
    const Shape m{q.size(0), q.size(1), q.size(2), q.size(3), v.size(3)};
    variable_list saved{q, k, v, s};
    std::vector<Tensor> out;
    if (map == LASP_QK_ELU1 && map_first(m, true)) {
      for (const Tensor* t : {&q, &k})   // (as for a tensor that is saved)
        TORCH_CHECK(!t->is_inference(), "Inference tensors cannot be saved for backward. To work around you can make a clone to get a "
                                        "normal tensor and use it in autograd.");
      if (!at::SavedTensorDefaultHooks::get_hooks())
        ctx->saved_data["unwritten"] = c10::IValue::make_capsule(c10::make_intrusive<Unwritten>(q, k));
      std::tie(saved[0], saved[1]) = mapped_qk(q, k);   // all that the backward pass takes
      map = LASP_QK_ELU1_MAPPED;
      out = run_forward(saved[0], saved[1], v, s, m, scale, map, true);
    } else {
      out = run_forward(q, k, v, s, m, scale, map, true);
    }
    saved.insert(saved.end(), out.begin() + 1, out.end());
    ctx->save_for_backward(std::move(saved));
    ctx->saved_data["scale"] = scale;
    ctx->saved_data["map"] = map;
    return out[0];
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list saved = ctx->get_saved_variables();
    const auto unwritten = ctx->saved_data.find("unwritten");
    if (unwritten != ctx->saved_data.end()) c10::static_intrusive_pointer_cast<Unwritten>(unwritten->second.toCapsule())->check();
    if (!grads[0].defined()) return {Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
    // What was saved may have been through a saved-tensor hook (offloading, compression): it can come back with other
    // strides, or not as what it was.
    const int64_t map = ctx->saved_data["map"].toInt();
    constexpr size_t first_ws = 4;
    const Tensor q = saved[0].contiguous(), k = saved[1].contiguous(), v = saved[2].contiguous(), d_o = grads[0].contiguous();
    TORCH_CHECK(q.is_cuda() && k.is_cuda() && v.is_cuda() && d_o.is_cuda(), "lasp_b200: a saved tensor is not on a GPU any more");
    TORCH_CHECK_TYPE(q.scalar_type() == d_o.scalar_type() && k.scalar_type() == q.scalar_type() && v.scalar_type() == q.scalar_type(),
                     "lasp_b200: a saved tensor has changed its dtype");
    Tensor s = saved[3];
    if (s.device() != q.device() || s.scalar_type() != at::kFloat) s = s.to(q.device(), at::kFloat);
    s = s.contiguous();
    const Shape m{q.size(0), q.size(1), q.size(2), q.size(3), v.size(3)};
    TORCH_CHECK_VALUE(k.sizes() == q.sizes() && v.sizes() == d_o.sizes() && v.sizes().slice(0, 3) == q.sizes().slice(0, 3) && s.numel() == m.h,
                      "lasp_b200: a saved tensor has changed its shape");
    const c10::cuda::CUDAGuard guard(q.device());
    const auto stream = at::cuda::getCurrentCUDAStream();
    Tensor dq = at::empty(q.sizes(), q.options()), dk = at::empty(k.sizes(), k.options()), dv = at::empty(v.sizes(), v.options());
    if (saved.size() == first_ws) {   // the forward pass has left no states: each result in one pass
      lasp_problem wide = problem_of(m, m.d, m.e, lasp_dtype_of(q.scalar_type()), 1.0, LASP_QK_IDENTITY, false);
      wide.path = LASP_PATH_TENSOR;
      lasp_bwd_args a = {};
      a.q = q.data_ptr(), a.k = k.data_ptr(), a.v = v.data_ptr(), a.d_o = d_o.data_ptr(), a.s = s.const_data_ptr<float>();
      a.dq = dq.data_ptr(), a.dk = dk.data_ptr(), a.dv = dv.data_ptr();
      Range range("lasp_b200_backward");
      check_status("lasp_b200_backward_wide", lasp_b200_backward_wide(&wide, &a, stream.stream()));
      return {dq, dk, dv, Tensor(), Tensor(), Tensor()};
    }
    const Tensor sync = sync_words(q.device(), stream);
    Tensor ws;
    const std::vector<Pair> pairs = slice_pairs(m, lasp_dtype_of(q.scalar_type()), ctx->saved_data["scale"].toDouble(), map);
    for (size_t i = 0; i < pairs.size(); ++i) {
      const Pair& p = pairs[i];
      const Tensor fwd_ws = saved[first_ws + i].contiguous();
      TORCH_CHECK(fwd_ws.is_cuda() && fwd_ws.scalar_type() == at::kByte && (size_t)fwd_ws.numel() >= p.ws_bytes,
                  "lasp_b200: the states saved by the forward pass did not come back as the bytes that they are");
      if (!ws.defined() || (size_t)ws.numel() < p.ws_bytes)
        ws = at::empty({(int64_t)p.ws_bytes}, q.options().dtype(at::kByte));
      lasp_bwd_args a = {};
      a.q = column(q, p.d0), a.k = column(k, p.d0), a.v = column(v, p.e0), a.d_o = column(d_o, p.e0);
      a.s = s.const_data_ptr<float>();
      a.dq = column(dq, p.d0), a.dk = column(dk, p.d0), a.dv = column(dv, p.e0);
      a.fwd_ws = fwd_ws.data_ptr(), a.fwd_ws_bytes = (size_t)fwd_ws.numel();
      a.ws = ws.data_ptr(), a.ws_bytes = (size_t)ws.numel();
      lasp_call_options opt = {};
      opt.sync = static_cast<uint32_t*>(sync.data_ptr());
      // a q/k slice collects from every v slice, a v slice from every q/k slice
      opt.accumulate = (p.e0 > 0 ? LASP_ACCUMULATE_QK : 0) | (p.d0 > 0 ? LASP_ACCUMULATE_V : 0);
      opt.alone = 1;
      Range range("lasp_b200_backward");
      check_status("lasp_b200_backward", lasp_b200_backward_opt(&p.problem, &a, &opt, stream.stream()));
    }
    return {dq, dk, dv, Tensor(), Tensor(), Tensor()};
  }
};

Tensor preprocess(const Tensor& x, double scale, int64_t map) {   // what a caller would write in front of the operator
  Tensor y = map ? at::elu(x) + 1.0 : x;
  return scale == 1.0 ? y : y * scale;
}

Tensor attention(Tensor q, Tensor k, Tensor v, const Tensor& ed, double scale, int64_t map) {
  const Shape m = check_inputs(q, k, v, ed);
  if (scale != 1.0 || map != 0) {
    // kernels that cannot take the preprocessing over get preprocessed tensors
    lasp_problem p = problem_of(m, std::min(m.d, kSlice), std::min(m.e, kSlice), lasp_dtype_of(q.scalar_type()), scale, map, false);
    if (!resolve(p)) q = preprocess(q, scale, map), k = preprocess(k, scale, map), scale = 1.0, map = 0;
  }
  Tensor s = ed.reshape({-1});
  if (s.device() != q.device() || s.scalar_type() != at::kFloat) s = s.to(q.device(), at::kFloat);
  s = s.contiguous();
  q = q.contiguous(), k = k.contiguous(), v = v.contiguous();
  // (the decay rates get no gradient, but a result that depends on them through a graph says so)
  if (at::GradMode::is_enabled() && (q.requires_grad() || k.requires_grad() || v.requires_grad() || s.requires_grad()))
    return Lightning::apply(q, k, v, s, scale, map);
  if (map == LASP_QK_ELU1 && map_first(m, false)) {
    std::tie(q, k) = mapped_qk(q, k);
    map = LASP_QK_ELU1_MAPPED;
  }
  return run_forward(q, k, v, s, m, scale, map, false)[0];
}

// The operator as a node of a traced graph: torch.jit.trace records what goes through the dispatcher, and the launches do
// not (it would keep the allocation of o alone).  Calls outside a trace spare themselves the dispatcher.
Tensor attention_op(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& s, double scale, int64_t map) {
  return attention(q, k, v, s, scale, map);
}
TORCH_LIBRARY(lasp_b200, m) {
  m.def("attention(Tensor q, Tensor k, Tensor v, Tensor s, float qk_scale, int map) -> Tensor");
  m.impl("attention", c10::DispatchKey::CompositeImplicitAutograd, TORCH_FN(attention_op));
}
Tensor traced_attention(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& s, double scale, int64_t map) {
  static const auto op = c10::Dispatcher::singleton()
                             .findSchemaOrThrow("lasp_b200::attention", "")
                             .typed<Tensor(const Tensor&, const Tensor&, const Tensor&, const Tensor&, double, int64_t)>();
  return op.call(q, k, v, s, scale, map);
}

// attention(q, k, v, s, qk_scale, map) -> o
PyObject* py_attention(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  TORCH_CHECK_TYPE(nargs == 6, "attention(q, k, v, s, qk_scale, map) takes 6 arguments");
  for (int i = 0; i < 4; ++i)
    TORCH_CHECK_TYPE(THPVariable_Check(args[i]), "q, k, v and the decay rates must be tensors");
  const double scale = PyFloat_AsDouble(args[4]);
  const long map = PyLong_AsLong(args[5]);
  if (PyErr_Occurred()) return nullptr;
  const Tensor &q = THPVariable_Unpack(args[0]), &k = THPVariable_Unpack(args[1]), &v = THPVariable_Unpack(args[2]),
               &s = THPVariable_Unpack(args[3]);
  Tensor o;
  {
    pybind11::gil_scoped_release no_gil;
    o = torch::jit::tracer::isTracing() ? traced_attention(q, k, v, s, scale, map) : attention(q, k, v, s, scale, map);
  }
  return THPVariable_Wrap(std::move(o));
  END_HANDLE_TH_ERRORS
}

PyMethodDef kMethods[] = {
    {"attention", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_attention)), METH_FASTCALL,
     "attention(q, k, v, s, qk_scale, map) -> o: decay-masked causal linear attention on scale * map(q), scale * map(k)"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_torch_ops", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__torch_ops(void) { return PyModule_Create(&kModule); }
