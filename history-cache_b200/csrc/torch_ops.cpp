// Python module hiscache_backend._native: the operators of libhiscache_b200 on torch tensors.
//
// The C ABI stays the boundary of the kernel library (include/hiscache_b200.h); this module only
// checks tensors, allocates results and scratch from torch's allocator and calls it.  It exists
// because a training step is some ninety calls of a few microseconds of GPU time each: argument
// checks and ctypes conversions in Python cost 8-12 us a call and an autograd.Function written in
// Python 60-90 us for its two directions, so the small layers of a batch waited for the host
// (1 000 x 5 edges of 1 KB, forward + backward: 119 us per pass, 11 us of it on the GPU).  Here a
// call is a few microseconds and the backward passes run on the autograd thread without the
// interpreter lock.
//
// The library's functions are looked up in the handle that the ctypes binding opened, so an
// overridden library (the index-checking build) is the one that runs.
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <dlfcn.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/extension.h>

#include <atomic>
#include <mutex>

#include "hiscache_b200.h"

namespace py = pybind11;
using at::Tensor;
using OptTensor = std::optional<Tensor>;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

namespace {

// ---------------------------------------------------------------------------
// the library's entry points
// ---------------------------------------------------------------------------
#define HC_FUNCTIONS(X)                                                                            \
  X(hc_error_string) X(hc_aggr_fwd) X(hc_aggr_bwd) X(hc_transpose_scratch_bytes)                   \
  X(hc_transpose_block) X(hc_gather_scratch_bytes) X(hc_aggr_bwd_gather)                           \
  X(hc_aggr_bwd_source_scratch_bytes) X(hc_aggr_bwd_source) X(hc_norm_scratch_bytes)               \
  X(hc_norm_act_fwd) X(hc_norm_act_bwd)

struct Lib {
#define X(f) decltype(&::f) f = nullptr;
  HC_FUNCTIONS(X)
#undef X
} lib;

void open_library(uintptr_t handle) {
  void* h = reinterpret_cast<void*>(handle);
#define X(f)                                                              \
  lib.f = reinterpret_cast<decltype(lib.f)>(dlsym(h, #f));                \
  TORCH_CHECK(lib.f != nullptr, "hiscache_backend: library lacks ", #f);
  HC_FUNCTIONS(X)
#undef X
}

void check(int rc, const char* what) {
  if (rc != 0) {
    const char* msg = lib.hc_error_string(rc);
    TORCH_CHECK(false, what, " failed (", rc, "): ", msg ? msg : "?");
  }
}

// ---------------------------------------------------------------------------
// launch counter and timing spans
// ---------------------------------------------------------------------------
std::atomic<int64_t> g_launches{0};
std::atomic<bool> g_timed{false};      // a KernelTimer is set: every call is bracketed by two events
py::object* g_span = nullptr;          // hiscache_backend._span (never destroyed)

std::string tag_of(const char* name, const Tensor& t) {
  return std::string(name) + "[" + (t.scalar_type() == at::kHalf ? "f16" : "f32") + ",F=" +
         std::to_string(t.size(-1)) + "]";
}

// Brackets one library call; with no timer set this is one relaxed load.
struct Span {
  std::unique_ptr<py::object> ctx;
  template <typename Name>
  Span(Name&& name, const at::Device& dev) {
    if (C10_UNLIKELY(g_timed.load(std::memory_order_relaxed))) {
      py::gil_scoped_acquire gil;
      ctx = std::make_unique<py::object>((*g_span)(py::str(name()), py::cast(dev)));
      ctx->attr("__enter__")();
    }
  }
  ~Span() {
    if (ctx) {
      py::gil_scoped_acquire gil;
      try {
        ctx->attr("__exit__")(py::none(), py::none(), py::none());
      } catch (py::error_already_set&) {
      }
      ctx.reset();
    }
  }
};
#define HC_SPAN(name, dev) Span span_([&] { return std::string(name); }, dev)
#define HC_SPAN_ROWS(name, t, dev) Span span_([&] { return tag_of(name, t); }, dev)

// ---------------------------------------------------------------------------
// tensor helpers
// ---------------------------------------------------------------------------
struct Where {       // all given tensors must live on one CUDA device
  at::Device dev{at::kCPU};
  bool any = false;
  Where& add(const Tensor& t) {
    if (!t.defined()) return *this;
    TORCH_CHECK(t.is_cuda(), "hiscache_backend: tensors must be CUDA tensors "
                             "(this library has no CPU implementation)");
    if (!any) {
      dev = t.device();
      any = true;
    } else {
      TORCH_CHECK(t.device() == dev, "hiscache_backend: tensors on different devices (", dev, ", ", t.device(), ")");
    }
    return *this;
  }
  Where& add(const OptTensor& t) { return t ? add(*t) : *this; }
};
template <typename... T>
at::Device require_cuda(const T&... t) {
  Where w;
  (w.add(t), ...);
  TORCH_CHECK(w.any, "hiscache_backend: no CUDA tensor given");
  return w.dev;
}

int dtype_code(const Tensor& t) {
  if (t.scalar_type() == at::kFloat) return HC_F32;
  if (t.scalar_type() == at::kHalf) return HC_F16;
  throw py::type_error("hiscache_backend: rows must be float32 or float16, got " +
                       std::string(c10::toString(t.scalar_type())));
}

Tensor i64c(const Tensor& t, const char* name = "index") {
  if (!t.defined()) return t;
  if (t.scalar_type() != at::kLong)
    throw py::type_error(std::string("hiscache_backend: ") + name + " must be int64, got " +
                         c10::toString(t.scalar_type()));
  return t.is_contiguous() ? t : t.contiguous();
}

// row-major with unit inner stride
Tensor rows2d(const Tensor& t) {
  if (!t.defined()) return t;
  return (t.stride(-1) != 1 && t.numel() > 0) ? t.contiguous() : t;
}

Tensor some(const OptTensor& t) { return t ? *t : Tensor(); }
Tensor some_nonempty(const OptTensor& t) { return t && t->defined() && t->numel() > 0 ? *t : Tensor(); }

template <typename T = void>
T* data(const Tensor& t) {
  return t.defined() ? static_cast<T*>(t.data_ptr()) : nullptr;
}
const int64_t* idata(const Tensor& t) { return data<int64_t>(t); }
float* fdata(const Tensor& t) { return data<float>(t); }

void* stream_of(const at::Device& dev) { return c10::cuda::getCurrentCUDAStream(dev.index()).stream(); }

Tensor new_cuda(at::IntArrayRef shape, at::ScalarType type, const at::Device& dev) {
  return at::detail::empty_cuda(shape, type, dev, std::nullopt);
}
Tensor new_f32(at::IntArrayRef shape, const at::Device& dev) { return new_cuda(shape, at::kFloat, dev); }
Tensor new_i64(at::IntArrayRef shape, const at::Device& dev) { return new_cuda(shape, at::kLong, dev); }
// Scratch comes from torch's caching allocator for the length of the call: its block goes back to
// the pool of the stream it was used on, so calls on several streams or threads never share one.
Tensor new_scratch(int64_t bytes, const at::Device& dev) {
  return new_cuda({std::max<int64_t>(bytes, 16)}, at::kByte, dev);
}

// ---------------------------------------------------------------------------
// aggregation
// ---------------------------------------------------------------------------
// Where the aggregation's backward pass leaves the per-row admission score.
// `fresh` turns true when a backward pass has written `tensor` since the last reset.
struct ScoreSink {
  Tensor tensor;
  bool fresh = false;
};

struct Block {      // the tensors of one aggregation call
  Tensor inp, ptr, idx, ev, hmap, hbuf, smap, salt;
  int64_t num_node = 0;
  bool indexed = false;
};

int64_t row_stride(const Tensor& t, int64_t row) { return t.size(0) > 1 ? t.stride(0) : row; }

hc_aggr_args aggr_args(const Block& b) {
  hc_aggr_args a{};
  a.struct_size = sizeof(hc_aggr_args);
  const int64_t H = b.inp.dim() == 3 ? b.inp.size(1) : 1, F = b.inp.size(-1);
  a.ptr = idata(b.ptr);
  a.idx = idata(b.idx);
  a.num_node = b.num_node;
  a.input = data(b.inp);
  a.in_dtype = dtype_code(b.inp);
  a.feat = (int32_t)F;
  a.num_head = (int32_t)H;
  a.n_src = b.inp.size(0);
  a.in_stride = row_stride(b.inp, H * F);
  if (b.smap.defined()) {
    a.src_map = idata(b.smap);
    a.src_alt = data(b.salt);
    a.alt_dtype = dtype_code(b.salt);
    a.alt_stride = row_stride(b.salt, H * F);
    a.alt_rows = b.salt.size(0);
  }
  a.edge_value = fdata(b.ev);
  if (b.hmap.defined()) {
    a.hmap = idata(b.hmap);
    a.hbuf = data(b.hbuf);
    a.h_dtype = dtype_code(b.hbuf);
    a.h_indexed = b.indexed ? 1 : 0;
    a.hsize = b.hbuf.dim() > 1 && b.hbuf.size(0) > 1 ? b.hbuf.stride(0) : b.hbuf.size(-1);
    a.h_rows = b.hbuf.dim() > 1 ? b.hbuf.size(0) : 1;
  }
  return a;
}

// ---- transposition of a block, shared by the layers of a declared batch -------
struct Transposed {
  Tensor t_ptr, t_dst, t_w;
  int64_t n_edges = 0;
};

Transposed transpose_block(const hc_aggr_args& a, int64_t max_edges, const at::Device& dev) {
  Transposed t;
  t.n_edges = max_edges;
  const int64_t n = std::max<int64_t>(max_edges, 1);
  t.t_ptr = new_i64({a.n_src + 1}, dev);
  t.t_dst = new_i64({n}, dev);
  t.t_w = new_f32({n}, dev);
  Tensor sc = new_scratch(lib.hc_transpose_scratch_bytes(a.n_src, n), dev);
  {
    HC_SPAN("hc_transpose_block", dev);
    check(lib.hc_transpose_block(&a, max_edges, data<int64_t>(t.t_ptr), data<int64_t>(t.t_dst), fdata(t.t_w),
                                 data(sc), stream_of(dev)),
          "hc_transpose_block");
  }
  int bits = 0;
  for (int64_t v = std::max<int64_t>(a.n_src, 1); v; v >>= 1) ++bits;
  g_launches += 2 + 5 * std::max(1, (bits + 7) / 8);
  return t;
}

struct GraphKey {
  void *ptr = nullptr, *idx = nullptr;
  int64_t rows = -1, edges = -1, v_ptr = 0, v_idx = 0;
  bool operator==(const GraphKey& o) const {
    return ptr == o.ptr && idx == o.idx && rows == o.rows && edges == o.edges && v_ptr == o.v_ptr && v_idx == o.v_idx;
  }
};
int64_t version_of(const Tensor& t) { return t.is_inference() ? 0 : (int64_t)t._version(); }
GraphKey graph_key(const Tensor& ptr, const Tensor& idx) {
  return {ptr.data_ptr(), idx.data_ptr(), ptr.size(0), idx.size(0), version_of(ptr), version_of(idx)};
}

struct Declared {
  GraphKey key;
  int64_t n_nodes = 0;
  bool built = false;
  Transposed t;
  Tensor keep_ptr, keep_idx;     // the tensors stay alive with the entry
};
std::mutex g_declared_mutex;
Declared g_declared[64];

Declared& declared_slot(const at::Device& dev) {
  TORCH_CHECK(dev.index() >= 0 && dev.index() < 64, "hiscache_backend: device index");
  return g_declared[dev.index()];
}

void declare_batch(const Tensor& ptr, const Tensor& idx, int64_t n_nodes) {
  if (!ptr.is_cuda()) return;
  Declared d;
  d.key = graph_key(ptr, idx);
  d.n_nodes = n_nodes;
  std::lock_guard<std::mutex> lock(g_declared_mutex);
  // a declaration opens a new batch: the same buffers may have been refilled by a library call
  // (which leaves no trace in the tensors' version counters), and a step that is being captured
  // must record its own transposition instead of borrowing the one of the warm-up
  std::swap(declared_slot(ptr.device()), d);
}

// The declared batch's transposition, or n_edges = -1 when (ptr, idx) was not declared.
Transposed shared_transpose(const Tensor& ptr, const Tensor& idx) {
  const at::Device dev = ptr.device();
  const GraphKey key = graph_key(ptr, idx);
  std::lock_guard<std::mutex> lock(g_declared_mutex);
  Declared& d = declared_slot(dev);
  Transposed none;
  none.n_edges = -1;
  if (!(d.key == key)) return none;
  if (!d.built) {
    hc_aggr_args a{};
    a.struct_size = sizeof(hc_aggr_args);
    a.ptr = idata(ptr);
    a.idx = idata(idx);
    a.num_node = ptr.size(0) - 1;
    a.feat = 4;
    a.num_head = 1;
    a.n_src = d.n_nodes;
    d.t = transpose_block(a, idx.size(0), dev);
    d.keep_ptr = ptr;
    d.keep_idx = idx;
    d.built = true;
  }
  return d.t;
}

void aggr_bwd_gather(const hc_aggr_args& a, const Transposed& t, const Tensor& grad_out, const Tensor& grad_input,
                     const at::Device& dev, const Tensor& tag) {
  Tensor sc;
  if (t.n_edges > 64) sc = new_scratch(lib.hc_gather_scratch_bytes(t.n_edges, a.feat), dev);
  {
    HC_SPAN_ROWS("hc_aggr_bwd_gather", tag, dev);
    check(lib.hc_aggr_bwd_gather(&a, idata(t.t_ptr), idata(t.t_dst), fdata(t.t_w), t.t_ptr.size(0) - 1, t.n_edges,
                                 fdata(grad_out), fdata(grad_input), data(sc), stream_of(dev)),
          "hc_aggr_bwd_gather");
  }
  g_launches += t.n_edges > 64 ? 4 : 1;
}

// which backward a call takes (see the Python module for the measured limits)
struct BwdRule {
  bool deterministic = false;
  int64_t gather_min_bytes = 0, gather_min_feat = 0;
};

// Counterpart of AggrHistoryFunction / AggrHistoryEdgeValueFunction
// (src/cpp/src/history_aggr.cu:475-596).  Saves the index tensors themselves (the reference keeps
// raw device pointers across forward and backward, history_aggr.cu:406-408).
struct AggrBackward : public torch::autograd::Node {
  SavedVariable inp, ptr, idx, ev, hmap, hbuf, smap, salt;
  int64_t num_node = 0;
  bool indexed = false, released = false;
  std::shared_ptr<ScoreSink> sink;
  Tensor score;
  int score_kind = HC_SCORE_L2;
  BwdRule rule;

  std::string name() const override { return "AggrBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    for (SavedVariable* v : {&inp, &ptr, &idx, &ev, &hmap, &hbuf, &smap, &salt}) v->reset_data();
    released = true;
  }
  variable_list apply(variable_list&& grads) override;
};

variable_list AggrBackward::apply(variable_list&& grads) {
  std::lock_guard<std::mutex> lock(mutex_);
  TORCH_CHECK(!released, torch::autograd::ERR_BACKWARD_TWICE);
  at::NoGradGuard no_grad;
  Block b;
  b.inp = inp.unpack(); b.ptr = ptr.unpack(); b.idx = idx.unpack(); b.ev = ev.unpack();
  b.hmap = hmap.unpack(); b.hbuf = hbuf.unpack(); b.smap = smap.unpack(); b.salt = salt.unpack();
  b.num_node = num_node;
  b.indexed = indexed;
  const at::Device dev = b.inp.device();
  c10::cuda::CUDAGuard guard(dev);
  const bool multi = b.inp.dim() == 3;
  Tensor go = grads[0];
  if (!go.defined()) {
    go = multi ? at::zeros({num_node, b.inp.size(1), b.inp.size(2)}, b.inp.options().dtype(at::kFloat))
               : at::zeros({num_node, b.inp.size(1)}, b.inp.options().dtype(at::kFloat));
  }
  if (go.scalar_type() != at::kFloat) go = go.to(at::kFloat);
  go = go.contiguous();
  const bool need_in = task_should_compute_output(0);
  const bool need_ev = b.ev.defined() && task_should_compute_output(1);
  const bool need_h = b.hbuf.defined() && task_should_compute_output(2);
  TORCH_CHECK(!(need_h && indexed), "gradients w.r.t. an indexed history table are not defined; "
                                    "pass a row-aligned history_buffer");
  hc_aggr_args a = aggr_args(b);
  variable_list out(4);
  Tensor row_score = multi ? Tensor() : score;
  if (!(need_in || need_ev || need_h || row_score.defined())) return out;
  Tensor g_in, g_ev, g_h;
  if (need_in) g_in = new_f32(b.inp.sizes(), dev);
  if (need_ev) g_ev = new_f32(b.ev.sizes(), dev);
  // Three forms.  A reproducible backward gathers over the sorted transposition.  Otherwise blocks
  // that gather enough are differentiated by source, and the rest scatter.
  bool gathered = false, edges_done = false;
  if (need_in && rule.deterministic && !b.ev.defined() && !multi && a.feat % 4 == 0 && a.feat <= 1024) {
    Transposed t = shared_transpose(b.ptr, b.idx);
    if (t.n_edges < 0 || t.t_ptr.size(0) - 1 < a.n_src)      // a block nobody declared: its own transposition
      t = transpose_block(a, b.idx.numel(), dev);
    aggr_bwd_gather(a, t, go, g_in, dev, b.inp);
    gathered = true;
  } else if ((need_in || need_ev) && !rule.deterministic && (int64_t)a.feat * a.num_head >= rule.gather_min_feat &&
             a.n_src * (int64_t)a.feat * a.num_head * 4 >= rule.gather_min_bytes) {
    const int64_t bytes = lib.hc_aggr_bwd_source_scratch_bytes(&a, b.idx.numel(), g_ev.defined());
    if (bytes >= 0) {
      Tensor sc = new_scratch(bytes, dev);
      HC_SPAN_ROWS("hc_aggr_bwd_source", b.inp, dev);
      check(lib.hc_aggr_bwd_source(&a, b.idx.numel(), fdata(go), fdata(g_in), fdata(g_ev), data(sc), stream_of(dev)),
            "hc_aggr_bwd_source");
      g_launches += 5;
      gathered = edges_done = true;
    }
  }
  if (need_h) {
    g_h = at::zeros(b.hbuf.sizes(), b.hbuf.options().dtype(at::kFloat));
    a.hsize = b.hbuf.size(-1);  // grad_history is dense
  }
  if (!gathered || need_h || row_score.defined()) {
    HC_SPAN_ROWS("hc_aggr_bwd", b.inp, dev);
    check(lib.hc_aggr_bwd(&a, fdata(go), gathered ? nullptr : fdata(g_in), 1, fdata(g_h), edges_done ? nullptr : fdata(g_ev),
                          fdata(row_score), score_kind, stream_of(dev)),
          "hc_aggr_bwd");
    ++g_launches;
  }
  if (row_score.defined() && sink) sink->fresh = true;
  if (g_in.defined()) out[0] = g_in.scalar_type() == b.inp.scalar_type() ? g_in : g_in.to(b.inp.scalar_type());
  if (g_ev.defined()) out[1] = g_ev;
  if (g_h.defined()) out[2] = g_h.scalar_type() == b.hbuf.scalar_type() ? g_h : g_h.to(b.hbuf.scalar_type());
  return out;
}

// forward; score_out is None, a ScoreSink or a tensor
Tensor aggr(const Tensor& input, const Tensor& ptr, const Tensor& idx, int64_t num_node, const OptTensor& history_map,
            const OptTensor& history_buffer, bool indexed, const OptTensor& edge_value, const OptTensor& src_map,
            const OptTensor& src_alt, const py::object& score_out, int score_kind, bool force_grad,
            bool deterministic, int64_t gather_min_bytes, int64_t gather_min_feat) {
  Block b;
  b.inp = input;
  b.ptr = ptr;
  b.idx = idx;
  b.hmap = some_nonempty(history_map);
  b.hbuf = some_nonempty(history_buffer);
  if (!b.hmap.defined() || !b.hbuf.defined()) b.hmap = b.hbuf = Tensor();
  b.ev = some_nonempty(edge_value);
  b.smap = some_nonempty(src_map);
  b.salt = b.smap.defined() ? some(src_alt) : Tensor();
  b.num_node = num_node == 0 ? ptr.size(0) - 1 : num_node;
  b.indexed = indexed;
  const at::Device dev = require_cuda(b.inp, b.ptr, b.idx, b.ev, b.hmap, b.hbuf, b.smap, b.salt);
  std::shared_ptr<AggrBackward> node;
  if (torch::autograd::compute_requires_grad(b.inp, b.ev, b.hbuf, b.salt)) {
    node = std::shared_ptr<AggrBackward>(new AggrBackward(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(b.inp, b.ev, b.hbuf, b.salt));
  }
  at::NoGradGuard no_grad;
  b.inp = rows2d(b.inp);
  b.ptr = i64c(b.ptr, "ptr");
  b.idx = i64c(b.idx, "idx");
  b.hmap = i64c(b.hmap, "history_map");
  b.smap = i64c(b.smap, "src_map");
  if (b.ev.defined()) {
    b.ev = b.ev.contiguous();
    if (b.ev.scalar_type() != at::kFloat) throw py::type_error("edge_value must be float32");
  }
  b.hbuf = rows2d(b.hbuf);
  b.salt = rows2d(b.salt);
  const bool multi = b.inp.dim() == 3;
  c10::cuda::CUDAGuard guard(dev);
  if (b.idx.numel() == 0) b.idx = at::zeros({1}, b.idx.options());  // a block without edges still needs an address
  TORCH_CHECK(b.ptr.size(0) >= b.num_node + 1, "aggr_forward: ptr has ", b.ptr.size(0), " entries, need ", b.num_node + 1);
  if (b.hmap.defined()) {
    TORCH_CHECK(b.hmap.size(0) >= b.num_node, "aggr_forward: history_map shorter than num_node");
    TORCH_CHECK(indexed || b.hbuf.size(0) >= b.num_node,
                "aggr_forward: row-aligned history_buffer shorter than num_node");
  }
  Tensor out = multi ? new_f32({b.num_node, b.inp.size(1), b.inp.size(2)}, dev) : new_f32({b.num_node, b.inp.size(1)}, dev);
  const hc_aggr_args a = aggr_args(b);
  {
    HC_SPAN_ROWS("hc_aggr_fwd", b.inp, dev);
    check(lib.hc_aggr_fwd(&a, fdata(out), stream_of(dev)), "hc_aggr_fwd");
  }
  ++g_launches;
  if (node) {
    node->inp = SavedVariable(b.inp, false);
    node->ptr = SavedVariable(b.ptr, false);
    node->idx = SavedVariable(b.idx, false);
    node->ev = SavedVariable(b.ev, false);
    node->hmap = SavedVariable(b.hmap, false);
    node->hbuf = SavedVariable(b.hbuf, false);
    node->smap = SavedVariable(b.smap, false);
    node->salt = SavedVariable(b.salt, false);
    node->num_node = b.num_node;
    node->indexed = indexed;
    if (!score_out.is_none()) {
      if (py::isinstance<ScoreSink>(score_out)) {
        node->sink = score_out.cast<std::shared_ptr<ScoreSink>>();
        node->score = node->sink->tensor;
      } else {
        node->score = score_out.cast<Tensor>();
      }
    }
    node->score_kind = score_kind;
    node->rule = {deterministic, gather_min_bytes, gather_min_feat};
    torch::autograd::set_history(out, node);
  } else if (force_grad) {
    out.set_requires_grad(true);
  }
  return out;
}

// ---------------------------------------------------------------------------
// batch norm + ReLU + dropout
// ---------------------------------------------------------------------------
struct NormCfg {
  double momentum, eps, p;
  bool relu;
  uint64_t seed;
};

hc_norm_args norm_args(const Tensor& x, const Tensor& valid, const Tensor& weight, const Tensor& bias,
                       const Tensor& rmean, const Tensor& rvar, const NormCfg& c, const Tensor& state,
                       const Tensor& save) {
  hc_norm_args a{};
  const int64_t F = x.size(1);
  a.struct_size = sizeof(hc_norm_args);
  a.x = fdata(x);
  a.n = x.size(0);
  a.feat = (int32_t)F;
  a.x_stride = row_stride(x, F);
  a.valid = data<uint8_t>(valid);
  a.weight = fdata(weight);
  a.bias = fdata(bias);
  a.running_mean = fdata(rmean);
  a.running_var = fdata(rvar);
  a.momentum = (float)c.momentum;
  a.eps = (float)c.eps;
  a.drop_p = (float)c.p;
  a.relu = c.relu ? 1 : 0;
  a.seed = c.seed;
  a.state = data<int64_t>(state);
  // one buffer: mean [feat], 1 / std [feat], row count [1], all on 16-byte boundaries (feat % 4 == 0)
  a.save_mean = fdata(save);
  a.save_rstd = fdata(save) + F;
  a.save_count = fdata(save) + 2 * F;
  return a;
}

struct NormActBackward : public torch::autograd::Node {
  SavedVariable x, weight, bias, valid, state;
  Tensor save;
  NormCfg cfg{};
  bool released = false;

  std::string name() const override { return "NormActBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    for (SavedVariable* v : {&x, &weight, &bias, &valid, &state}) v->reset_data();
    save = Tensor();
    released = true;
  }
  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    TORCH_CHECK(!released, torch::autograd::ERR_BACKWARD_TWICE);
    at::NoGradGuard no_grad;
    const Tensor xt = x.unpack(), w = weight.unpack(), bi = bias.unpack(), va = valid.unpack(), stt = state.unpack();
    const at::Device dev = xt.device();
    c10::cuda::CUDAGuard guard(dev);
    Tensor gy = grads[0].defined() ? grads[0].contiguous() : at::zeros(xt.sizes(), xt.options());
    Tensor gx = new_f32(xt.sizes(), dev), gw, gb;
    if (w.defined() && task_should_compute_output(1)) gw = new_f32(w.sizes(), dev);
    if (bi.defined() && task_should_compute_output(2)) gb = new_f32(bi.sizes(), dev);
    const hc_norm_args a = norm_args(xt, va, w, bi, Tensor(), Tensor(), cfg, stt, save);
    Tensor sc = new_scratch(lib.hc_norm_scratch_bytes(a.feat), dev);
    {
      HC_SPAN("hc_norm_act_bwd", dev);
      check(lib.hc_norm_act_bwd(&a, fdata(gy), fdata(gx), fdata(gw), fdata(gb), data(sc), stream_of(dev)),
            "hc_norm_act_bwd");
    }
    g_launches += 2;
    return {gx, gw, gb};
  }
};

Tensor norm_act(const Tensor& x_in, const OptTensor& weight, const OptTensor& bias, const Tensor& state,
                const OptTensor& valid_in, const OptTensor& running_mean, const OptTensor& running_var,
                double momentum, double eps, double p, bool relu, uint64_t seed) {
  const Tensor w = some(weight), bi = some(bias), rm = some(running_mean), rv = some(running_var);
  Tensor valid = some(valid_in);
  const at::Device dev = require_cuda(x_in, w, bi, valid, rm, rv, state);
  std::shared_ptr<NormActBackward> node;
  if (torch::autograd::compute_requires_grad(x_in, w, bi)) {
    node = std::shared_ptr<NormActBackward>(new NormActBackward(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(x_in, w, bi));
  }
  at::NoGradGuard no_grad;
  const Tensor x = rows2d(x_in);
  if (x.scalar_type() != at::kFloat || x.dim() != 2) throw py::type_error("norm_act: x must be a float32 matrix");
  if (valid.defined()) {
    valid = valid.contiguous();
    TORCH_CHECK(valid.size(0) >= x.size(0), "norm_act: row mask shorter than x");
  }
  c10::cuda::CUDAGuard guard(dev);
  const int64_t F = x.size(1);
  Tensor y = new_f32({x.size(0), F}, dev), save = new_f32({2 * F + 4}, dev);
  const NormCfg cfg{momentum, eps, p, relu, seed};
  const hc_norm_args a = norm_args(x, valid, w, bi, rm, rv, cfg, state, save);
  Tensor sc = new_scratch(lib.hc_norm_scratch_bytes((int32_t)F), dev);
  {
    HC_SPAN("hc_norm_act_fwd", dev);
    check(lib.hc_norm_act_fwd(&a, fdata(y), data(sc), stream_of(dev)), "hc_norm_act_fwd");
  }
  g_launches += 2;
  if (node) {
    node->x = SavedVariable(x, false);
    node->weight = SavedVariable(w, false);
    node->bias = SavedVariable(bi, false);
    node->valid = SavedVariable(valid, false);
    node->state = SavedVariable(state, false);
    node->save = save;
    node->cfg = cfg;
    torch::autograd::set_history(y, node);
  }
  return y;
}

}  // namespace

PYBIND11_MODULE(_native, m) {
  m.doc() = "operators of libhiscache_b200 on torch tensors";
  m.def("open_library", &open_library);
  m.def("launches", [] { return g_launches.load(); });
  m.def("add_launches", [](int64_t n) { g_launches += n; }, py::arg("n") = 1);
  m.def("set_span", [](py::object span) { g_span = new py::object(std::move(span)); });
  m.def("set_timed", [](bool on) { g_timed = on; });
  py::class_<ScoreSink, std::shared_ptr<ScoreSink>>(
      m, "ScoreSink",
      "Where the aggregation's backward pass leaves the per-row admission score.  `fresh` turns True when a "
      "backward pass has written `tensor` since the last reset.")
      .def(py::init([](const Tensor& t) {
             auto s = std::make_shared<ScoreSink>();
             s->tensor = t;
             return s;
           }),
           py::arg("tensor"))
      .def_readwrite("tensor", &ScoreSink::tensor)
      .def_readwrite("fresh", &ScoreSink::fresh);
  m.def("aggr", &aggr);
  m.def("declare_batch", &declare_batch);
  m.def("shared_transpose", [](const Tensor& ptr, const Tensor& idx) -> py::object {
    if (!ptr.is_cuda()) return py::none();
    Transposed t = shared_transpose(ptr, idx);
    if (t.n_edges < 0) return py::none();
    return py::make_tuple(t.t_ptr, t.t_dst, t.t_w, t.n_edges);
  });
  m.def("norm_act", &norm_act);
}
