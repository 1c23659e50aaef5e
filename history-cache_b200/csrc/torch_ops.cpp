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
#include <ATen/cuda/CUDAEvent.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <dlfcn.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/extension.h>

#include <array>
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
  X(hc_score_rows) X(hc_select_scratch_bytes) X(hc_select_threshold)                               \
  X(hc_select_threshold_counted) X(hc_select_threshold_masked) X(hc_admit_scratch_bytes)           \
  X(hc_record_history_masked) X(hc_cache_admit) X(hc_evict_stale) X(hc_evict_stale_dev)            \
  X(hc_evict_by_score) X(hc_evict_both) X(hc_stamp_checkin) X(hc_used_masks_scratch_bytes)         \
  X(hc_used_masks_together) X(hc_count_num) X(hc_map_lookup) X(hc_map_lookup_masked)               \
  X(hc_cache_lookup) X(hc_gather_rows) X(hc_load_rows) X(hc_load_rows_staged)                      \
  X(hc_stage_host_rows) X(hc_sample_fixed_scratch_bytes) X(hc_sample_batch) X(hc_sample_counts)    \
  X(hc_sample_picks) X(hc_relabel_scratch_bytes) X(hc_relabel) X(hc_relabel_seed)                  \
  X(hc_relabel_reset) X(hc_edge_types) X(hc_rgcn_group_scratch_bytes) X(hc_rgcn_group)             \
  X(hc_aggr_bwd_rooted) X(hc_rgcn_rows_scratch_bytes) X(hc_rgcn_rows) X(hc_override_rows)          \
  X(hc_adam_step) X(hc_sage_pack) X(hc_slab_sums_scratch_bytes) X(hc_slab_sums) X(hc_nll_fwd)      \
  X(hc_nll_bwd)                                                                                    \
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

// What the layer behind an aggregation leaves for its backward pass: the gradient of the destination rows
// that the layer read directly ([num_node, feat], rows may be part of a wider product).  The aggregation's
// gradient then starts from it, instead of autograd padding it to all sources and adding it up.
struct RootGrad {
  Tensor rows;
};

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
  const c10::TensorImpl* source = nullptr;       // the input tensor (only compared)
  std::shared_ptr<RootGrad> root;

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
  Tensor root_rows;
  if (root) std::swap(root_rows, root->rows);
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
  // one scatter takes rows that are part of a wider product as they lie
  const bool by_source = (need_in || need_ev) && !rule.deterministic &&
                         (int64_t)a.feat * a.num_head >= rule.gather_min_feat &&
                         a.n_src * (int64_t)a.feat * a.num_head * 4 >= rule.gather_min_bytes;
  const bool plain = !multi && !b.ev.defined() && a.feat % 4 == 0 && !by_source && !rule.deterministic;
  if (!(plain && go.stride(-1) == 1 && go.stride(0) % 4 == 0 && ((uintptr_t)go.data_ptr() & 15) == 0)) go = go.contiguous();
  Tensor root_start = plain && root_rows.defined() && need_in && root_rows.stride(-1) == 1 && root_rows.stride(0) % 4 == 0 &&
                              ((uintptr_t)root_rows.data_ptr() & 15) == 0
                          ? root_rows : Tensor();
  // Three forms.  A reproducible backward gathers over the sorted transposition.  Otherwise blocks
  // that gather enough are differentiated by source, and the rest scatter.
  bool gathered = false, edges_done = false;
  if (need_in && rule.deterministic && !b.ev.defined() && !multi && a.feat % 4 == 0 && a.feat <= 1024) {
    Transposed t = shared_transpose(b.ptr, b.idx);
    if (t.n_edges < 0 || t.t_ptr.size(0) - 1 < a.n_src)      // a block nobody declared: its own transposition
      t = transpose_block(a, b.idx.numel(), dev);
    aggr_bwd_gather(a, t, go, g_in, dev, b.inp);
    gathered = true;
  } else if (by_source) {
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
    check(lib.hc_aggr_bwd_rooted(&a, fdata(go), multi ? 0 : go.stride(0), fdata(root_start),
                                 root_start.defined() ? root_start.stride(0) : 0, gathered ? nullptr : fdata(g_in), 1,
                                 fdata(g_h), edges_done ? nullptr : fdata(g_ev), fdata(row_score), score_kind,
                                 stream_of(dev)),
          "hc_aggr_bwd");
    ++g_launches;
  }
  if (g_in.defined() && root_rows.defined() && !root_start.defined()) g_in.slice(0, 0, num_node).add_(root_rows);
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
    node->source = input.unsafeGetTensorImpl();
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
                double momentum, double eps, double p, bool relu, uint64_t seed, const OptTensor& tracked_in) {
  const Tensor w = some(weight), bi = some(bias), rm = some(running_mean), rv = some(running_var), tracked = some(tracked_in);
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
  hc_norm_args a = norm_args(x, valid, w, bi, rm, rv, cfg, state, save);
  if (tracked.defined()) {
    TORCH_CHECK(tracked.device() == dev && tracked.scalar_type() == at::kLong && tracked.numel() == 1,
                "norm_act: num_batches_tracked must be an int64 CUDA scalar");
    if (a.n) {
      a.batches_tracked = data<int64_t>(tracked);
      torch::autograd::impl::bump_version(tracked);
    } else {
      tracked.add_(1);
    }
  }
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


// ---------------------------------------------------------------------------
// scores, threshold, admission, eviction
// ---------------------------------------------------------------------------
#define HC_ON(dev) c10::cuda::CUDAGuard guard_(dev)

Tensor f32_rows(const Tensor& t) {
  Tensor x = rows2d(t);
  return x.scalar_type() == at::kFloat ? x : x.to(at::kFloat);
}
// a row mask: one byte per row
Tensor byte_mask(const OptTensor& m, int64_t n, const char* what) {
  Tensor t = some(m);
  if (!t.defined()) return t;
  TORCH_CHECK(t.element_size() == 1 && t.size(0) >= n, what, " must have one byte per row");
  return t.is_contiguous() ? t : t.contiguous();
}

Tensor score_rows(const Tensor& x_in, int kind, const OptTensor& out_in) {
  const at::Device dev = require_cuda(x_in);
  HC_ON(dev);
  at::NoGradGuard no_grad;
  const Tensor x = f32_rows(x_in);
  const int64_t n = x.size(0), F = x.size(1);
  Tensor out = out_in ? *out_in : new_f32({n}, dev);
  {
    HC_SPAN("hc_score_rows", dev);
    check(lib.hc_score_rows(fdata(x), n, (int32_t)F, row_stride(x, F), kind, fdata(out), stream_of(dev)), "hc_score_rows");
  }
  ++g_launches;
  return out;
}

Tensor select_threshold(const Tensor& score_in, double q, const OptTensor& out_in, const OptTensor& n_valid,
                        const OptTensor& valid_in) {
  const at::Device dev = require_cuda(score_in);
  HC_ON(dev);
  const Tensor score = score_in.contiguous();
  if (score.scalar_type() != at::kFloat) throw py::type_error("select_threshold: scores must be float32");
  Tensor out = out_in ? *out_in : new_f32({1}, dev);
  const int64_t n = score.size(0), bytes = lib.hc_select_scratch_bytes(n);
  const Tensor valid = byte_mask(valid_in, n, "select_threshold: valid");
  Tensor sc;
  if (bytes) sc = new_scratch(bytes, dev);
  {
    HC_SPAN("hc_select_threshold", dev);
    if (valid.defined())
      check(lib.hc_select_threshold_masked(fdata(score), data<uint8_t>(valid), n, (float)q, fdata(out), data(sc),
                                           stream_of(dev)), "hc_select_threshold_masked");
    else if (n_valid)
      check(lib.hc_select_threshold_counted(fdata(score), n, idata(*n_valid), (float)q, fdata(out), data(sc),
                                            stream_of(dev)), "hc_select_threshold_counted");
    else
      check(lib.hc_select_threshold(fdata(score), n, (float)q, fdata(out), data(sc), stream_of(dev)),
            "hc_select_threshold");
  }
  g_launches += bytes ? 9 : 1;
  return out;
}

void record_history(const Tensor& new_in, const Tensor& buffer_all, const OptTensor& used_in, const Tensor& sub_to_full,
                    const Tensor& sub_to_history, const Tensor& history_to_full, const Tensor& full_to_history,
                    const Tensor& header, const Tensor& score_in, const Tensor& thres_in, const Tensor& checkin_iter,
                    int64_t glb_iter, const OptTensor& n_admitted, const OptTensor& valid_in) {
  const at::Device dev = require_cuda(new_in, buffer_all, sub_to_full, sub_to_history, history_to_full, full_to_history,
                                      header, score_in, thres_in, checkin_iter);
  HC_ON(dev);
  at::NoGradGuard no_grad;
  const Tensor rows = f32_rows(new_in);
  const int64_t n = rows.size(0), hs = rows.size(1);
  TORCH_CHECK(buffer_all.is_contiguous(), "record_history: buffer_all must be contiguous");
  TORCH_CHECK(buffer_all.size(1) == hs, "record_history: row widths differ");
  const std::pair<const char*, const Tensor*> maps[] = {{"history_to_full", &history_to_full},
                                                        {"full_to_history", &full_to_history},
                                                        {"header", &header},
                                                        {"checkin_iter", &checkin_iter}};
  for (auto& m : maps)
    if (m.second->scalar_type() != at::kLong || !m.second->is_contiguous())
      throw py::type_error(std::string("record_history: ") + m.first + " must be contiguous int64");
  Tensor used = some(used_in);
  if (used.defined()) {
    if (used.scalar_type() != at::kBool && used.scalar_type() != at::kByte)
      throw py::type_error("record_history: used_mask must be bool");
    used = used.contiguous();
    TORCH_CHECK(used.size(0) >= n, "record_history: used_mask shorter than buffer_new");
  }
  const Tensor valid = byte_mask(valid_in, n, "record_history: valid");
  TORCH_CHECK(sub_to_full.size(0) >= n && sub_to_history.size(0) >= n && score_in.size(0) >= n,
              "record_history: per-row arguments shorter than buffer_new");
  const Tensor thres = thres_in.scalar_type() == at::kFloat ? thres_in : thres_in.to(at::kFloat);
  const Tensor score = (score_in.scalar_type() == at::kFloat ? score_in : score_in.to(at::kFloat)).contiguous();
  const Tensor s2f = i64c(sub_to_full), s2h = i64c(sub_to_history);
  Tensor sc = new_scratch(lib.hc_admit_scratch_bytes(n), dev);
  {
    HC_SPAN("hc_record_history", dev);
    check(lib.hc_record_history_masked(fdata(rows), row_stride(rows, hs), n, data(buffer_all), dtype_code(buffer_all),
                                       buffer_all.size(0), (int32_t)hs, data<uint8_t>(used), data<uint8_t>(valid),
                                       idata(s2f), idata(s2h), data<int64_t>(history_to_full),
                                       data<int64_t>(full_to_history), data<int64_t>(header), fdata(score),
                                       fdata(thres), data<int64_t>(checkin_iter), glb_iter,
                                       n_admitted ? data<int64_t>(*n_admitted) : nullptr, data(sc), stream_of(dev)),
          "hc_record_history");
  }
  ++g_launches;
}

void cache_admit(const Tensor& produced, const Tensor& buffer, int64_t hidden, int64_t in_feat, int64_t embed_capacity,
                 const Tensor& sub_to_full, const Tensor& sub2embed, const Tensor& score, const Tensor& thres,
                 const Tensor& full2embed, int64_t total_num_node, const Tensor& embed2full, const OptTensor& feat2full,
                 const Tensor& header, bool reset_header, const OptTensor& n_admitted, const OptTensor& valid) {
  const at::Device dev = require_cuda(produced, buffer, sub_to_full, sub2embed, score, thres, full2embed, embed2full, header);
  HC_ON(dev);
  at::NoGradGuard no_grad;
  const Tensor rows = f32_rows(produced);
  const int64_t n = rows.size(0);
  const Tensor s2f = i64c(sub_to_full), s2e = i64c(sub2embed), f2f = some(feat2full), v = some(valid);
  Tensor sc = new_scratch(lib.hc_admit_scratch_bytes(n), dev);
  {
    HC_SPAN("hc_cache_admit", dev);
    check(lib.hc_cache_admit(fdata(rows), row_stride(rows, hidden), n, data(buffer), dtype_code(buffer), (int32_t)hidden,
                             (int32_t)in_feat, embed_capacity, idata(s2f), idata(s2e), fdata(score), fdata(thres),
                             data<int64_t>(full2embed), total_num_node, data<int64_t>(embed2full), idata(f2f),
                             f2f.defined() ? f2f.size(0) : 0, data<int64_t>(header), reset_header ? 1 : 0,
                             data<uint8_t>(v), n_admitted ? data<int64_t>(*n_admitted) : nullptr, data(sc),
                             stream_of(dev)),
          "hc_cache_admit");
  }
  ++g_launches;
}

void evict_stale(const Tensor& checkin, const Tensor& h2f, const Tensor& f2h, int64_t glb_iter, int64_t limit) {
  const at::Device dev = require_cuda(checkin, h2f, f2h);
  HC_ON(dev);
  HC_SPAN("hc_evict_stale", dev);
  check(lib.hc_evict_stale(data<int64_t>(checkin), data<int64_t>(h2f), data<int64_t>(f2h), checkin.size(0), glb_iter, limit,
                           stream_of(dev)), "hc_evict_stale");
  ++g_launches;
}
void evict_stale_dev(const Tensor& checkin, const Tensor& h2f, const Tensor& f2h, const Tensor& iter_dev, int64_t limit) {
  const at::Device dev = require_cuda(checkin, h2f, f2h, iter_dev);
  HC_ON(dev);
  HC_SPAN("hc_evict_stale", dev);
  check(lib.hc_evict_stale_dev(data<int64_t>(checkin), data<int64_t>(h2f), data<int64_t>(f2h), checkin.size(0),
                               idata(iter_dev), limit, stream_of(dev)), "hc_evict_stale_dev");
  ++g_launches;
}
void stamp_checkin(const Tensor& checkin, const Tensor& iter_dev, int64_t marker) {
  const at::Device dev = require_cuda(checkin, iter_dev);
  HC_ON(dev);
  HC_SPAN("hc_stamp_checkin", dev);
  check(lib.hc_stamp_checkin(data<int64_t>(checkin), checkin.size(0), marker, idata(iter_dev), stream_of(dev)),
        "hc_stamp_checkin");
  ++g_launches;
}
void evict_by_score(const Tensor& s2h_in, const Tensor& score_in, const Tensor& thres, const Tensor& checkin,
                    const Tensor& h2f, const Tensor& f2h) {
  const at::Device dev = require_cuda(s2h_in, score_in, thres, checkin);
  HC_ON(dev);
  const Tensor s2h = i64c(s2h_in), score = score_in.contiguous();
  HC_SPAN("hc_evict_by_score", dev);
  check(lib.hc_evict_by_score(idata(s2h), fdata(score), fdata(thres), std::min(s2h.size(0), score.size(0)),
                              data<int64_t>(checkin), data<int64_t>(h2f), data<int64_t>(f2h), stream_of(dev)),
        "hc_evict_by_score");
  ++g_launches;
}
// evict_by_score and the eviction by age in one launch; iter_dev (or None) replaces glb_iter
void evict_both(const Tensor& s2h_in, const Tensor& score_in, const Tensor& thres, const Tensor& checkin,
                const Tensor& h2f, const Tensor& f2h, int64_t glb_iter, const OptTensor& iter_dev, int64_t limit) {
  const at::Device dev = require_cuda(s2h_in, score_in, thres, checkin, h2f, f2h, iter_dev);
  HC_ON(dev);
  const Tensor s2h = i64c(s2h_in), score = score_in.contiguous();
  HC_SPAN("hc_evict_both", dev);
  check(lib.hc_evict_both(idata(s2h), fdata(score), fdata(thres), std::min(s2h.size(0), score.size(0)),
                          data<int64_t>(checkin), data<int64_t>(h2f), data<int64_t>(f2h), checkin.size(0), glb_iter,
                          iter_dev ? idata(*iter_dev) : nullptr, limit, stream_of(dev)),
        "hc_evict_both");
  ++g_launches;
}

// ---------------------------------------------------------------------------
// receptive-field bookkeeping, lookup, row assembly
// ---------------------------------------------------------------------------
std::vector<Tensor> used_masks(const Tensor& ptr_in, const Tensor& idx_in, const OptTensor& maps, int64_t num_node,
                               int64_t num_seed, int num_layer) {
  const at::Device dev = require_cuda(ptr_in, idx_in);
  HC_ON(dev);
  const Tensor ptr = i64c(ptr_in, "ptr"), idx = i64c(idx_in, "idx"), hm = i64c(some_nonempty(maps), "history_maps");
  Tensor buf = new_cuda({num_layer + 1, num_node}, at::kBool, dev);
  Tensor sc = new_scratch(lib.hc_used_masks_scratch_bytes(), dev);
  {
    HC_SPAN("hc_used_masks", dev);
    check(lib.hc_used_masks_together(idata(ptr), idata(idx), ptr.size(0) - 1, idata(hm), hm.defined() ? hm.size(0) : 0,
                                     num_node, num_seed, num_layer, data<uint8_t>(buf), data(sc), stream_of(dev)),
          "hc_used_masks");
  }
  ++g_launches;
  return buf.unbind(0);
}

Tensor count_num(const Tensor& arr_in, int64_t mmax) {
  const at::Device dev = require_cuda(arr_in);
  HC_ON(dev);
  const Tensor arr = i64c(arr_in, "arr");
  Tensor out = new_cuda({mmax + 1}, at::kInt, dev);
  HC_SPAN("hc_count_num", dev);
  check(lib.hc_count_num(idata(arr), arr.size(0), mmax, data<int32_t>(out), stream_of(dev)), "hc_count_num");
  ++g_launches;
  return out;
}

Tensor map_lookup(const Tensor& map, const Tensor& ids_in, int64_t offset, int64_t force_miss_below,
                  const OptTensor& out_in, const OptTensor& valid_in) {
  const at::Device dev = require_cuda(map, ids_in);
  HC_ON(dev);
  const Tensor ids = i64c(ids_in, "ids");
  const int64_t n = ids.size(0);
  const Tensor valid = byte_mask(valid_in, n, "map_lookup: valid");
  Tensor out = out_in ? *out_in : new_i64({n}, dev);
  {
    HC_SPAN("hc_map_lookup", dev);
    if (valid.defined()) {
      TORCH_CHECK(offset == 0, "map_lookup: a row mask needs offset 0");
      check(lib.hc_map_lookup_masked(idata(map), map.size(0), idata(ids), n, force_miss_below, data<uint8_t>(valid),
                                     data<int64_t>(out), stream_of(dev)), "hc_map_lookup_masked");
    } else {
      check(lib.hc_map_lookup(idata(map), map.size(0), idata(ids), n, offset, force_miss_below, data<int64_t>(out),
                              stream_of(dev)), "hc_map_lookup");
    }
  }
  ++g_launches;
  return out;
}

// (sub2embed [n1], sub2feat [n])
std::tuple<Tensor, Tensor> cache_lookup(const Tensor& map, const Tensor& ids_in, int64_t n1, int64_t offset) {
  const at::Device dev = require_cuda(map, ids_in);
  HC_ON(dev);
  const Tensor ids = i64c(ids_in, "ids");
  const int64_t n = ids.size(0);
  Tensor embed = new_i64({n1}, dev), feat = new_i64({n}, dev);
  {
    HC_SPAN("hc_cache_lookup", dev);
    check(lib.hc_cache_lookup(idata(map), map.size(0), idata(ids), n, n1, offset, data<int64_t>(embed), data<int64_t>(feat),
                              stream_of(dev)), "hc_cache_lookup");
  }
  ++g_launches;
  return {embed, feat};
}

Tensor gather_rows(const Tensor& table_in, const Tensor& rows_in, bool zero_missing, const std::optional<at::ScalarType>& type) {
  const at::Device dev = require_cuda(table_in, rows_in);
  HC_ON(dev);
  at::NoGradGuard no_grad;
  const Tensor table = rows2d(table_in), rows = i64c(rows_in, "rows");
  const int64_t n = rows.size(0), F = table.size(1);
  Tensor out = new_cuda({n, F}, type ? *type : table.scalar_type(), dev);
  HC_SPAN("hc_gather_rows", dev);
  check(lib.hc_gather_rows(data(table), dtype_code(table), table.size(0), row_stride(table, F), (int32_t)F, idata(rows), n,
                           zero_missing ? 1 : 0, data(out), dtype_code(out), F, stream_of(dev)), "hc_gather_rows");
  ++g_launches;
  return out;
}

py::object load_rows(const Tensor& host_in, const OptTensor& cache_in, const Tensor& ids_in, const OptTensor& feat_in,
                     const OptTensor& used_in, const std::optional<at::ScalarType>& type, bool want_mask,
                     const OptTensor& stats, const OptTensor& out_in, const OptTensor& mask_out,
                     const std::optional<std::tuple<Tensor, Tensor>>& staged) {
  Where w;
  w.add(ids_in).add(feat_in).add(used_in).add(cache_in).add(out_in).add(mask_out);
  if (host_in.is_cuda()) w.add(host_in);
  TORCH_CHECK(w.any, "hiscache_backend: no CUDA tensor given");
  const at::Device dev = w.dev;
  HC_ON(dev);
  at::NoGradGuard no_grad;
  TORCH_CHECK(host_in.is_cuda() || host_in.is_pinned(), "load_rows: a host feature table must be pinned memory");
  const Tensor host = rows2d(host_in), ids = i64c(ids_in, "sub_to_full"), s2f = i64c(some(feat_in), "sub2feat");
  const int64_t n = ids.size(0), F = host.size(1);
  const at::ScalarType dt = type ? *type : host.scalar_type();
  Tensor x = some(out_in), mask = some(mask_out), used = some(used_in), cache = some(cache_in);
  if (x.defined()) {
    if (x.dim() != 2 || x.size(0) != n || x.size(1) != F || x.scalar_type() != dt || !x.is_contiguous())
      throw py::value_error("load_rows: out must be a contiguous [" + std::to_string(n) + ", " + std::to_string(F) +
                            "] tensor of the batch's type");
  } else {
    x = new_cuda({n, F}, dt, dev);
  }
  if (mask.defined()) {
    if (mask.scalar_type() != at::kByte || mask.size(0) != n || !mask.is_contiguous())
      throw py::value_error("load_rows: mask_out must be a contiguous uint8 tensor of " + std::to_string(n) + " entries");
  } else if (want_mask) {
    mask = new_cuda({n}, at::kByte, dev);
  }
  if (used.defined()) {
    used = used.contiguous();
    if (used.size(0) != n || used.element_size() != 1)
      throw py::value_error("load_rows: used must have " + std::to_string(n) + " one-byte entries");
  }
  int cd = HC_F32;
  int64_t cr = 0, cs = 0;
  if (cache.defined()) {
    cache = rows2d(cache);
    cd = dtype_code(cache);
    cr = cache.size(0);
    cs = row_stride(cache, F);
  }
  int64_t* st = stats ? data<int64_t>(*stats) : nullptr;
  {
    HC_SPAN("hc_load_rows", dev);
    if (!staged) {
      check(lib.hc_load_rows(data(host), dtype_code(host), host.size(0), row_stride(host, F), data(cache), cd, cr, cs,
                             (int32_t)F, idata(ids), idata(s2f), data<uint8_t>(used), n, data(x), dtype_code(x), F,
                             data<uint8_t>(mask), st, stream_of(dev)), "hc_load_rows");
    } else {
      const Tensor &sr = std::get<0>(*staged), &sm = std::get<1>(*staged);
      require_cuda(sr, sm);
      if (sr.dim() != 2 || sr.size(0) != n || sr.size(1) != F || sr.scalar_type() != x.scalar_type() ||
          !sr.is_contiguous() || sm.scalar_type() != at::kByte || sm.size(0) != n || !sm.is_contiguous())
        throw py::value_error("load_rows: staged must be ([" + std::to_string(n) + ", " + std::to_string(F) +
                              "] rows of the batch's type, [" + std::to_string(n) + "] uint8 mask)");
      if (stats && stats->numel() < 3) throw py::value_error("load_rows: stats needs three counters when rows are staged");
      check(lib.hc_load_rows_staged(data(host), dtype_code(host), host.size(0), row_stride(host, F), data(cache), cd, cr, cs,
                                    (int32_t)F, idata(ids), idata(s2f), data<uint8_t>(used), n, data(x), dtype_code(x), F,
                                    data<uint8_t>(mask), st, data(sr), data<uint8_t>(sm), stream_of(dev)),
            "hc_load_rows_staged");
    }
  }
  ++g_launches;
  if (want_mask) return py::make_tuple(x, mask.view(at::kBool));
  return py::cast(x);
}

void stage_host_rows(const Tensor& host_in, const Tensor& ids_in, const OptTensor& feat_in, const OptTensor& consider_in,
                     const Tensor& rows_out, const Tensor& mask_out, const OptTensor& stats, int64_t max_blocks) {
  Where w;
  w.add(ids_in).add(feat_in).add(consider_in).add(rows_out).add(mask_out);
  if (host_in.is_cuda()) w.add(host_in);
  TORCH_CHECK(w.any, "hiscache_backend: no CUDA tensor given");
  const at::Device dev = w.dev;
  HC_ON(dev);
  TORCH_CHECK(host_in.is_cuda() || host_in.is_pinned(), "stage_host_rows: a host feature table must be pinned memory");
  const Tensor host = rows2d(host_in), ids = i64c(ids_in, "ids"), s2f = i64c(some(feat_in), "sub2feat");
  const int64_t n = ids.size(0), F = host.size(1);
  if (s2f.defined() && s2f.size(0) != n)
    throw py::value_error("stage_host_rows: sub2feat must have " + std::to_string(n) + " entries");
  Tensor consider = some(consider_in);
  if (consider.defined()) {
    consider = consider.contiguous();
    if (consider.size(0) != n || consider.element_size() != 1)
      throw py::value_error("stage_host_rows: consider must have " + std::to_string(n) + " one-byte entries");
  }
  if (rows_out.dim() != 2 || rows_out.size(0) != n || rows_out.size(1) != F || rows_out.scalar_type() != host.scalar_type() ||
      !rows_out.is_contiguous() || mask_out.scalar_type() != at::kByte || mask_out.size(0) != n || !mask_out.is_contiguous())
    throw py::value_error("stage_host_rows: outputs must be [" + std::to_string(n) + ", " + std::to_string(F) +
                          "] rows of the table's type and [" + std::to_string(n) + "] uint8 mask");
  HC_SPAN("hc_stage_host_rows", dev);
  check(lib.hc_stage_host_rows(data(host), dtype_code(host), host.size(0), row_stride(host, F), (int32_t)F, idata(ids),
                               idata(s2f), data<uint8_t>(consider), n, data(rows_out), data<uint8_t>(mask_out),
                               stats ? data<int64_t>(*stats) : nullptr, (int32_t)max_blocks, stream_of(dev)),
        "hc_stage_host_rows");
  ++g_launches;
}

// ---------------------------------------------------------------------------
// sampling
// ---------------------------------------------------------------------------
void sample_batch(const Tensor& gptr, const Tensor& gidx, const Tensor& seeds_in, const Tensor& local_map, uint64_t seed,
                  const Tensor& batch_no, const std::vector<int64_t>& fanouts, const std::vector<int64_t>& caps,
                  int64_t edge_cap, const Tensor& ptr, const Tensor& idx, const Tensor& sub_to_full, const Tensor& mask,
                  const Tensor& counters, const OptTensor& labels, const OptTensor& y) {
  const at::Device dev = require_cuda(gptr, gidx, seeds_in, local_map, batch_no, ptr, idx, sub_to_full, mask, counters,
                                      labels, y);
  HC_ON(dev);
  const Tensor seeds = i64c(seeds_in, "seeds");
  hc_fixed_batch b{};
  b.struct_size = sizeof(hc_fixed_batch);
  const int64_t L = (int64_t)fanouts.size();
  b.num_hops = (int32_t)L;
  for (int64_t h = 0; h < L; ++h) b.fanout[h] = (int32_t)fanouts[h];
  for (int64_t k = 0; k <= L; ++k) b.caps[k] = caps[k];
  b.edge_cap = edge_cap;
  TORCH_CHECK(ptr.numel() >= caps[L - 1] + 1 && idx.numel() >= edge_cap && sub_to_full.numel() >= caps[L] &&
                  mask.numel() >= caps[L] && mask.element_size() == 1 && counters.numel() >= 4 &&
                  (!y || y->numel() >= caps[0]),
              "sample_fixed: an output is smaller than the batch's caps");
  b.ptr = data<int64_t>(ptr);
  b.idx = data<int64_t>(idx);
  b.sub_to_full = data<int64_t>(sub_to_full);
  b.mask = data<uint8_t>(mask);
  b.counters = data<int64_t>(counters);
  Tensor sc = new_scratch(lib.hc_sample_fixed_scratch_bytes(&b), dev);
  HC_SPAN("hc_sample_fixed", dev);
  check(lib.hc_sample_batch(idata(gptr), idata(gidx), idata(seeds), seeds.size(0), data<int32_t>(local_map), seed,
                            data<int64_t>(batch_no), labels ? idata(*labels) : nullptr, y ? data<int64_t>(*y) : nullptr, &b,
                            data(sc), stream_of(dev)),
        "hc_sample_fixed");
  ++g_launches;
}

py::tuple sample_hop(const Tensor& gptr, const Tensor& gidx, const Tensor& frontier_in, int64_t fanout, uint64_t seed,
                     int64_t base) {
  const at::Device dev = require_cuda(gptr, gidx, frontier_in);
  HC_ON(dev);
  const Tensor frontier = i64c(frontier_in, "frontier");
  const int64_t nf = frontier.size(0);
  Tensor out_ptr = at::zeros({nf + 1}, frontier.options());
  Tensor counts = out_ptr.slice(0, 1);
  {
    HC_SPAN("hc_sample_counts", dev);
    check(lib.hc_sample_counts(idata(gptr), idata(frontier), nf, (int32_t)fanout, data<int64_t>(counts), stream_of(dev)),
          "hc_sample_counts");
  }
  at::cumsum_out(counts, counts, 0);
  int64_t total = 0;
  if (nf > 0) {
    py::gil_scoped_release no_gil;
    total = out_ptr[nf].item<int64_t>();
  }
  Tensor nbr = new_i64({total}, dev);
  {
    HC_SPAN("hc_sample_picks", dev);
    check(lib.hc_sample_picks(idata(gptr), idata(gidx), idata(frontier), nf, (int32_t)fanout, idata(out_ptr), seed, base,
                              data<int64_t>(nbr), stream_of(dev)), "hc_sample_picks");
  }
  g_launches += 2;
  return py::make_tuple(out_ptr, nbr);
}

void relabel_seed(const Tensor& seeds_in, const Tensor& local_map) {
  const at::Device dev = require_cuda(seeds_in, local_map);
  HC_ON(dev);
  const Tensor seeds = i64c(seeds_in);
  check(lib.hc_relabel_seed(idata(seeds), seeds.size(0), data<int32_t>(local_map), stream_of(dev)), "hc_relabel_seed");
  ++g_launches;
}
void relabel_reset(const Tensor& nodes_in, const Tensor& local_map) {
  const at::Device dev = require_cuda(nodes_in, local_map);
  HC_ON(dev);
  const Tensor nodes = i64c(nodes_in);
  check(lib.hc_relabel_reset(idata(nodes), nodes.size(0), data<int32_t>(local_map), stream_of(dev)), "hc_relabel_reset");
  ++g_launches;
}
py::tuple relabel(const Tensor& nbr, const Tensor& local_map, int64_t n_total) {
  const at::Device dev = require_cuda(nbr, local_map);
  HC_ON(dev);
  const int64_t m = nbr.size(0);
  Tensor new_nodes = new_i64({std::max<int64_t>(m, 1)}, dev), n_new = at::zeros({1}, new_nodes.options());
  Tensor out_idx = new_i64({m}, dev), sc = new_scratch(lib.hc_relabel_scratch_bytes(m), dev);
  {
    HC_SPAN("hc_relabel", dev);
    check(lib.hc_relabel(idata(nbr), m, data<int32_t>(local_map), n_total, data<int64_t>(new_nodes), data<int64_t>(n_new),
                         data<int64_t>(out_idx), data(sc), stream_of(dev)), "hc_relabel");
  }
  g_launches += 6;
  int64_t n = 0;
  {
    py::gil_scoped_release no_gil;
    n = n_new.item<int64_t>();
  }
  return py::make_tuple(new_nodes.slice(0, 0, n), out_idx);
}

// ---------------------------------------------------------------------------
// heterogeneous layers
// ---------------------------------------------------------------------------
Tensor edge_types(const Tensor& ptr_in, const Tensor& idx_in, const Tensor& nodes_in, int64_t rows,
                  const std::vector<int64_t>& bounds, const std::vector<int64_t>& rel_table) {
  const at::Device dev = require_cuda(ptr_in, idx_in, nodes_in);
  HC_ON(dev);
  const int64_t T = (int64_t)bounds.size() - 1;
  if (T < 1 || T > 8 || (int64_t)rel_table.size() != T * T)
    throw py::value_error("edge_types: 1..8 node types, rel_table of n_types^2 entries");
  const Tensor ptr = i64c(ptr_in), idx = i64c(idx_in), nodes = i64c(nodes_in);
  Tensor out = new_i64({idx.size(0)}, dev);
  if (idx.size(0) && rows < ptr.size(0) - 1) out.fill_(0);     // edges behind the rows asked for
  const std::vector<int32_t> rel(rel_table.begin(), rel_table.end());
  HC_SPAN("hc_edge_types", dev);
  check(lib.hc_edge_types(idata(ptr), idata(idx), idata(nodes), rows, (int32_t)T, bounds.data(), rel.data(),
                          data<int64_t>(out), stream_of(dev)), "hc_edge_types");
  ++g_launches;
  return out;
}

py::tuple rgcn_group(const Tensor& ptr_in, const Tensor& idx_in, const Tensor& etype_in, int64_t num_node, int64_t num_rel,
                     const OptTensor& used_in, const OptTensor& hmap_in, bool want_perm, bool want_rel) {
  const at::Device dev = require_cuda(ptr_in, idx_in, etype_in, used_in, hmap_in);
  HC_ON(dev);
  const Tensor ptr = i64c(ptr_in, "ptr"), idx = i64c(idx_in, "idx"), etype = i64c(etype_in, "edge_type"),
               hmap = i64c(some(hmap_in));
  const int64_t E = std::min(idx.size(0), etype.size(0)), room = std::max<int64_t>(E, 1);
  TORCH_CHECK(ptr.size(0) >= num_node + 1, "rgcn_group: ptr shorter than num_node + 1");
  TORCH_CHECK(!hmap.defined() || hmap.size(0) >= num_node, "rgcn_group: history map shorter than num_node");
  Tensor used = some(used_in);
  if (used.defined()) {
    used = used.contiguous();
    if (used.scalar_type() != at::kBool && used.scalar_type() != at::kByte)
      throw py::type_error("rgcn_group: used mask must be bool");
  }
  Tensor ptr2 = new_i64({num_rel * num_node + 1}, dev), idx2 = new_i64({room}, dev), w2 = new_f32({room}, dev), perm, rel;
  if (want_perm) perm = new_i64({room}, dev);
  if (want_rel) rel = new_i64({room}, dev);
  Tensor sc = new_scratch(lib.hc_rgcn_group_scratch_bytes(E), dev);
  {
    HC_SPAN("hc_rgcn_group", dev);
    check(lib.hc_rgcn_group(idata(ptr), idata(idx), idata(etype), num_node, E, (int32_t)num_rel, data<uint8_t>(used),
                            idata(hmap), data<int64_t>(ptr2), data<int64_t>(idx2), fdata(w2), data<int64_t>(perm),
                            data<int64_t>(rel), data(sc), stream_of(dev)), "hc_rgcn_group");
  }
  g_launches += 7;
  auto cut = [&](const Tensor& t) -> py::object { return t.defined() ? py::cast(t.slice(0, 0, E)) : py::none(); };
  return py::make_tuple(ptr2, cut(idx2), cut(w2), cut(perm), cut(rel));
}

// A branch beside the current stream, joined at the end of the scope.  Only while a step is being captured:
// there the fork is two edges of the graph, while eager it would cost more host time than the overlap
// brings.  The stream is this thread's own: a pooled one may belong to somebody who is not being captured.
// What the branch writes is allocated before, on the main stream.
class Branch {
 public:
  explicit Branch(const at::Device& dev, bool wanted)
      : main_(c10::cuda::getCurrentCUDAStream(dev.index())), side_(main_) {
    if (!wanted || c10::cuda::currentStreamCaptureStatusMayInitCtx() == c10::cuda::CaptureStatus::None) return;
    thread_local std::array<cudaStream_t, 64> own{};
    TORCH_CHECK(dev.index() >= 0 && dev.index() < 64, "hiscache_backend: device index");
    cudaStream_t& st = own[dev.index()];
    if (!st && cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess) {
      st = nullptr;
      return;
    }
    side_ = c10::cuda::getStreamFromExternal(st, dev.index());
    fork_.record(main_);
    fork_.block(side_);
    open_ = true;
  }
  Branch(const Branch&) = delete;
  ~Branch() {
    if (!open_) return;
    try {
      join_.record(side_);
      join_.block(main_);
    } catch (const std::exception&) {      // the capture is lost, its end reports it
    }
  }
  c10::cuda::CUDAStream stream() const { return side_; }

 private:
  c10::cuda::CUDAStream main_, side_;
  at::cuda::CUDAEvent fork_, join_;
  bool open_ = false;
};

// g^T r for tall, narrow g [n, M] and r [n, N]: columns [0, split) of the result into left, the others into
// right; column sums of g into bias (undefined = not wanted).  Such a product has a very long reduction and a
// small output, which the library runs on a few dozen blocks: the rows are cut into slabs of at least 256, one
// batched product gives the slabs' results, and hc_slab_sums adds them up, takes the few rows that fill no
// slab along and finishes the bias.  The order of the additions is fixed.
constexpr int64_t kSlabRows = 256;
void tall_products(const Tensor& g, const Tensor& r, int64_t slabs, int64_t split, Tensor* left, Tensor* right, Tensor* bias,
                   const c10::cuda::CUDAStream& stream, variable_list& keep) {
  const at::Device dev = g.device();
  const int64_t n = g.size(0), M = g.size(1), N = r.size(1);
  int64_t s = std::max<int64_t>(slabs, 1);
  while (s > 1 && n / s < kSlabRows) s /= 2;
  const int64_t m = n / s, rest = n - m * s;
  Tensor parts, sc;
  const bool copied = s == 1 && split == N;      // the product is the result already
  if (left || right) {
    parts = s > 1 ? new_f32({s, M, N}, dev) : new_f32({M, N}, dev);
    if (left) *left = copied ? parts : new_f32({M, split}, dev);
    if (right) *right = new_f32({M, N - split}, dev);
  }
  if (bias) {
    *bias = new_f32({M}, dev);
    sc = new_scratch(lib.hc_slab_sums_scratch_bytes(M), dev);
  }
  keep = {parts, sc};      // the caller lets go of them behind the join
  c10::cuda::CUDAStreamGuard on(stream);
  if (parts.defined()) {
    if (s > 1)
      at::bmm_out(parts, g.narrow(0, 0, m * s).view({s, m, M}).transpose(1, 2), r.narrow(0, 0, m * s).view({s, m, N}));
    else
      at::mm_out(parts, g.t(), r);
  }
  if (!bias && copied) return;
  HC_SPAN("hc_slab_sums", dev);
  check(lib.hc_slab_sums(fdata(parts), (int32_t)s, M, (int32_t)N, rest ? fdata(g) + m * s * M : nullptr,
                         rest ? fdata(r) + m * s * N : nullptr, (int32_t)rest, (int32_t)split,
                         left && !copied ? fdata(*left) : nullptr, right ? fdata(*right) : nullptr, fdata(g), n,
                         bias ? fdata(*bias) : nullptr, data(sc), stream.stream()),
        "hc_slab_sums");
  g_launches += (bias ? 1 : 0) + 1;
}

// One RGCN layer (MyRGCNConvHistory2): relation-segmented rows by destination, their weighted sums as
// [num_node, num_rel * feat], one product with the stacked weights, history rows over it.  Destinations
// served from history have no edges here, so they add nothing to either gradient.
constexpr int64_t kRgcnSlabs = 16;
struct RgcnBackward : public torch::autograd::Node {
  SavedVariable x, weight;
  Tensor ptr2, idx2, w2, sums;
  int64_t num_node = 0, num_rel = 0;
  BwdRule rule;
  bool released = false;

  std::string name() const override { return "RgcnBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    x.reset_data();
    weight.reset_data();
    ptr2 = idx2 = w2 = sums = Tensor();
    released = true;
  }
  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    TORCH_CHECK(!released, torch::autograd::ERR_BACKWARD_TWICE);
    at::NoGradGuard no_grad;
    variable_list out(2);
    if (!grads[0].defined()) return out;
    const Tensor xt = x.unpack(), w = weight.unpack();
    const at::Device dev = xt.device();
    c10::cuda::CUDAGuard guard(dev);
    const int64_t F = xt.size(1), H = w.size(2);
    const Tensor g = grads[0].contiguous(), wide = sums.view({num_node, num_rel * F});
    variable_list keep;
    Branch beside(dev, task_should_compute_output(0) && task_should_compute_output(1));
    if (task_should_compute_output(1)) {
      Tensor gw;
      tall_products(wide, g, kRgcnSlabs, H, &gw, nullptr, nullptr, beside.stream(), keep);
      out[1] = gw.view({num_rel, F, H});
    }
    if (task_should_compute_output(0)) {
      const Tensor go = at::mm(g, w.reshape({num_rel * F, H}).t());      // [num_node, num_rel * F] = its rows
      Block b;
      b.inp = xt; b.ptr = ptr2; b.idx = idx2; b.ev = w2;
      b.num_node = num_node * num_rel;
      const hc_aggr_args a = aggr_args(b);
      Tensor gx = new_f32(xt.sizes(), dev);
      int64_t bytes = -1;
      if (!rule.deterministic && F >= rule.gather_min_feat && a.n_src * F * 4 >= rule.gather_min_bytes)
        bytes = lib.hc_aggr_bwd_source_scratch_bytes(&a, idx2.numel(), 0);
      if (bytes >= 0) {
        Tensor sc = new_scratch(bytes, dev);
        HC_SPAN_ROWS("hc_aggr_bwd_source", xt, dev);
        check(lib.hc_aggr_bwd_source(&a, idx2.numel(), fdata(go), fdata(gx), nullptr, data(sc), stream_of(dev)),
              "hc_aggr_bwd_source");
        g_launches += 5;
      } else {
        HC_SPAN_ROWS("hc_aggr_bwd", xt, dev);
        check(lib.hc_aggr_bwd(&a, fdata(go), fdata(gx), 1, nullptr, nullptr, nullptr, HC_SCORE_L2, stream_of(dev)),
              "hc_aggr_bwd");
        ++g_launches;
      }
      out[0] = xt.scalar_type() == at::kFloat ? gx : gx.to(xt.scalar_type());
    }
    return out;
  }
};

// (out [num_node, hidden], edges per relation)
py::tuple rgcn_layer(const Tensor& x_in, const Tensor& ptr_in, const Tensor& idx_in, const Tensor& etype_in,
                     int64_t num_node, const OptTensor& used_in, const OptTensor& hmap_in, const OptTensor& hbuf_in,
                     bool indexed, const Tensor& weight, bool deterministic, int64_t gather_min_bytes,
                     int64_t gather_min_feat) {
  const int64_t R = weight.size(0), F = weight.size(1), H = weight.size(2);
  const Tensor hm = i64c(some_nonempty(hmap_in), "history_map"), hbuf = rows2d(some_nonempty(hbuf_in));
  const at::Device dev = require_cuda(x_in, ptr_in, idx_in, etype_in, weight, hm, hbuf, used_in);
  std::shared_ptr<RgcnBackward> node;
  if (torch::autograd::compute_requires_grad(x_in, weight)) {
    node = std::shared_ptr<RgcnBackward>(new RgcnBackward(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(x_in, weight));
  }
  at::NoGradGuard no_grad;
  HC_ON(dev);
  const Tensor x = rows2d(x_in), ptr = i64c(ptr_in, "ptr"), idx = i64c(idx_in, "idx"), etype = i64c(etype_in, "edge_type");
  TORCH_CHECK(x.size(1) == F, "rgcn_layer: the weights take ", F, " columns, the rows have ", x.size(1));
  TORCH_CHECK(ptr.size(0) >= num_node + 1, "rgcn_layer: ptr shorter than num_node + 1");
  TORCH_CHECK(!hm.defined() || (hm.size(0) >= num_node && hbuf.defined() && (indexed || hbuf.size(0) >= num_node)),
              "rgcn_layer: history shorter than num_node");
  const int64_t E = std::min(idx.size(0), etype.size(0)), room = std::max<int64_t>(E, 1);
  const Tensor used = some(used_in).defined() ? some(used_in).contiguous() : Tensor();
  Tensor ptr2 = new_i64({num_node * R + 1}, dev), idx2 = new_i64({room}, dev), w2 = new_f32({room}, dev);
  Tensor count = new_cuda({R + 1}, at::kInt, dev), sc = new_scratch(lib.hc_rgcn_rows_scratch_bytes(), dev);
  {
    HC_SPAN("hc_rgcn_rows", dev);
    check(lib.hc_rgcn_rows(idata(ptr), idata(idx), idata(etype), num_node, E, (int32_t)R, data<uint8_t>(used), idata(hm),
                           data<int64_t>(ptr2), data<int64_t>(idx2), fdata(w2), data<int32_t>(count), data(sc),
                           stream_of(dev)), "hc_rgcn_rows");
  }
  Tensor sums = new_f32({num_node * R, F}, dev);
  Block b;
  b.inp = x; b.ptr = ptr2; b.idx = idx2; b.ev = w2;
  b.num_node = num_node * R;
  const hc_aggr_args a = aggr_args(b);
  {
    HC_SPAN_ROWS("hc_aggr_fwd", x, dev);
    check(lib.hc_aggr_fwd(&a, fdata(sums), stream_of(dev)), "hc_aggr_fwd");
  }
  g_launches += 2;
  Tensor out = at::mm(sums.view({num_node, R * F}), weight.reshape({R * F, H}));
  if (hm.defined()) {
    TORCH_CHECK(hbuf.size(-1) == H, "rgcn_layer: history rows have another width");
    HC_SPAN("hc_override_rows", dev);
    check(lib.hc_override_rows(idata(hm), num_node, data(hbuf), dtype_code(hbuf), row_stride(hbuf, H), indexed ? 1 : 0,
                               (int32_t)H, fdata(out), stream_of(dev)), "hc_override_rows");
    ++g_launches;
  }
  if (node) {
    node->x = SavedVariable(x, false);
    node->weight = SavedVariable(weight, false);
    node->ptr2 = ptr2; node->idx2 = idx2; node->w2 = w2; node->sums = sums;
    node->num_node = num_node;
    node->num_rel = R;
    node->rule = {deterministic, gather_min_bytes, gather_min_feat};
    torch::autograd::set_history(out, node);
  }
  return py::make_tuple(out, count);
}

// ---------------------------------------------------------------------------
// dense part of a SAGE layer: lin_l(aggregate) + lin_r(x[:num_node]) as one product over
// [aggregate | root].
// ---------------------------------------------------------------------------
struct SageLinearBackward : public torch::autograd::Node {
  SavedVariable weight;      // [wl | wr]
  Tensor rows;               // [aggregate | root]
  std::shared_ptr<RootGrad> root;
  int64_t K = 0, n_src = 0, slabs = 8;
  bool has_bias = false, released = false;
  at::ScalarType root_type = at::kFloat;

  std::string name() const override { return "SageLinearBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    weight.reset_data();
    rows = Tensor();
    released = true;
  }
  variable_list apply(variable_list&& grads) override {      // his, wl, bias, wr, x
    std::lock_guard<std::mutex> lock(mutex_);
    TORCH_CHECK(!released, torch::autograd::ERR_BACKWARD_TWICE);
    at::NoGradGuard no_grad;
    variable_list out(5);
    if (!grads[0].defined()) return out;
    c10::cuda::CUDAGuard guard(rows.device());
    const Tensor g = grads[0].contiguous(), w = weight.unpack();
    const int64_t n = rows.size(0);
    const bool want_x = task_should_compute_output(4);
    const bool want_l = task_should_compute_output(1), want_r = task_should_compute_output(3),
               want_b = has_bias && task_should_compute_output(2);
    const bool want_in = task_should_compute_output(0) || want_x || root;
    variable_list keep;
    Branch beside(rows.device(), want_in && (want_l || want_r || want_b));
    if (want_l || want_r || want_b)
      tall_products(g, rows, slabs, K, want_l ? &out[1] : nullptr, want_r ? &out[3] : nullptr, want_b ? &out[2] : nullptr,
                    beside.stream(), keep);
    if (want_in) {
      const Tensor g2 = at::mm(g, w);
      out[0] = g2.narrow(1, 0, K);
      if (root) root->rows = g2.narrow(1, K, K);
      if (want_x) {
        out[4] = at::zeros({n_src, K}, rows.options().dtype(root_type));
        out[4].slice(0, 0, n).copy_(g2.narrow(1, K, K));
      }
    }
    return out;
  }
};

Tensor sage_linear(const Tensor& his, const Tensor& x, int64_t num_node, const Tensor& wl, const OptTensor& bias_in,
                   const Tensor& wr, int64_t slabs) {
  const Tensor bias = some(bias_in);
  const at::Device dev = require_cuda(his, x, wl, bias, wr);
  const int64_t K = his.size(1);
  TORCH_CHECK(his.size(0) == num_node && x.size(0) >= num_node && x.size(1) == K && wl.size(1) == K && wr.sizes() == wl.sizes(),
              "sage_linear: shapes do not match");
  std::shared_ptr<SageLinearBackward> node;
  if (torch::autograd::compute_requires_grad(his, wl, bias, wr, x)) {
    node = std::shared_ptr<SageLinearBackward>(new SageLinearBackward(), torch::autograd::deleteNode);
    auto edges = torch::autograd::collect_next_edges(his, wl, bias, wr, x);
    // when `his` is the aggregation of this very x, its backward pass takes x's second gradient along
    auto* aggr = dynamic_cast<AggrBackward*>(his.grad_fn().get());
    if (aggr && aggr->source == x.unsafeGetTensorImpl() && x.requires_grad() && aggr->num_node == num_node && !aggr->root) {
      node->root = aggr->root = std::make_shared<RootGrad>();
      edges[4] = torch::autograd::Edge();
    }
    node->set_next_edges(std::move(edges));
  }
  at::NoGradGuard no_grad;
  HC_ON(dev);
  const Tensor left = f32_rows(his), right = rows2d(x), wlc = wl.contiguous(), wrc = wr.contiguous();
  const int64_t H = wl.size(0);
  Tensor rows = new_f32({num_node, 2 * K}, dev), w = new_f32({H, 2 * K}, dev), out = new_f32({num_node, H}, dev);
  const Tensor bc = bias.defined() ? bias.contiguous() : bias;
  {
    HC_SPAN("hc_sage_pack", dev);
    check(lib.hc_sage_pack(fdata(left), row_stride(left, K), data(right), dtype_code(right), row_stride(right, K), num_node,
                           (int32_t)K, fdata(rows), fdata(wlc), fdata(wrc), (int32_t)H, fdata(w), fdata(bc),
                           bias.defined() ? fdata(out) : nullptr, stream_of(dev)),
          "hc_sage_pack");
  }
  ++g_launches;
  if (bias.defined()) {
    out.addmm_(rows, w.t());
  } else {
    at::mm_out(out, rows, w.t());
  }
  if (node) {
    node->weight = SavedVariable(w, false);
    node->rows = rows;
    node->K = K;
    node->n_src = x.size(0);
    node->slabs = slabs;
    node->has_bias = bias.defined();
    node->root_type = x.scalar_type();
    torch::autograd::set_history(out, node);
  }
  return out;
}

// ---------------------------------------------------------------------------
// loss
// ---------------------------------------------------------------------------
struct NllBackward : public torch::autograd::Node {
  SavedVariable y;
  Tensor count;
  int64_t classes = 0, ignore = -100;
  bool released = false;

  std::string name() const override { return "NllBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    y.reset_data();
    count = Tensor();
    released = true;
  }
  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    TORCH_CHECK(!released, torch::autograd::ERR_BACKWARD_TWICE);
    at::NoGradGuard no_grad;
    variable_list out(1);
    if (!grads[0].defined() || !task_should_compute_output(0)) return out;
    const Tensor yt = y.unpack();
    const at::Device dev = yt.device();
    c10::cuda::CUDAGuard guard(dev);
    const Tensor g = grads[0].to(at::kFloat);
    out[0] = new_f32({yt.size(0), classes}, dev);
    HC_SPAN("hc_nll_bwd", dev);
    check(lib.hc_nll_bwd(fdata(g), idata(yt), ignore, fdata(count), yt.size(0), (int32_t)classes, fdata(out[0]),
                         stream_of(dev)), "hc_nll_bwd");
    ++g_launches;
    return out;
  }
};

Tensor nll_loss(const Tensor& logp_in, const Tensor& y_in, int64_t ignore) {
  const at::Device dev = require_cuda(logp_in, y_in);
  TORCH_CHECK(logp_in.dim() == 2 && y_in.dim() == 1 && y_in.size(0) == logp_in.size(0), "nll_loss: logp [n, classes], y [n]");
  if (logp_in.scalar_type() != at::kFloat) throw py::type_error("nll_loss: logp must be float32");
  std::shared_ptr<NllBackward> node;
  if (torch::autograd::compute_requires_grad(logp_in)) {
    node = std::shared_ptr<NllBackward>(new NllBackward(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(logp_in));
  }
  at::NoGradGuard no_grad;
  HC_ON(dev);
  const Tensor logp = rows2d(logp_in), y = i64c(y_in, "y");
  Tensor loss = new_f32({}, dev), count = new_f32({1}, dev);
  {
    HC_SPAN("hc_nll_fwd", dev);
    check(lib.hc_nll_fwd(fdata(logp), row_stride(logp, logp.size(1)), logp.size(0), (int32_t)logp.size(1), idata(y), ignore,
                         fdata(loss), fdata(count), stream_of(dev)), "hc_nll_fwd");
  }
  ++g_launches;
  if (node) {
    node->y = SavedVariable(y, false);
    node->count = count;
    node->classes = logp.size(1);
    node->ignore = ignore;
    torch::autograd::set_history(loss, node);
  }
  return loss;
}

// ---------------------------------------------------------------------------
// optimiser
// ---------------------------------------------------------------------------
// whether adam_step takes these tensors (device-side step counts, fp32, dense)
bool adam_fits(const std::vector<Tensor>& params, const std::vector<Tensor>& grads, const std::vector<Tensor>& avgs,
               const std::vector<Tensor>& avg_sqs, const std::vector<Tensor>& steps) {
  const size_t n = params.size();
  if (grads.size() != n || avgs.size() != n || avg_sqs.size() != n || steps.size() != n) return false;
  for (size_t k = 0; k < n; ++k) {
    const at::Device dev = params[0].device();
    for (const Tensor* t : {&params[k], &grads[k], &avgs[k], &avg_sqs[k], &steps[k]})
      if (!t->is_cuda() || t->device() != dev || t->scalar_type() != at::kFloat || t->layout() != at::kStrided) return false;
    for (const Tensor* t : {&params[k], &avgs[k], &avg_sqs[k]})
      if (!t->is_contiguous() || t->numel() != params[k].numel()) return false;
    if (params[k].numel() == 0 || grads[k].numel() != params[k].numel() || steps[k].numel() != 1) return false;
  }
  return true;
}

// false: not a case for the kernel, nothing done
bool adam_step(const std::vector<Tensor>& params, const std::vector<Tensor>& grads, const std::vector<Tensor>& avgs,
               const std::vector<Tensor>& avg_sqs, const std::vector<Tensor>& steps, double lr, double beta1, double beta2,
               double eps) {
  if (params.empty()) return true;
  if (!adam_fits(params, grads, avgs, avg_sqs, steps)) return false;
  at::NoGradGuard no_grad;
  const at::Device dev = params[0].device();
  HC_ON(dev);
  const size_t n = params.size();
  std::vector<void*> p(n), m(n), v(n), t(n);
  std::vector<const void*> g(n);
  std::vector<int64_t> numel(n);
  std::vector<Tensor> keep;
  for (size_t k = 0; k < n; ++k) {
    Tensor gr = grads[k];
    if (!gr.is_contiguous()) keep.push_back(gr = gr.contiguous());
    p[k] = params[k].data_ptr();
    g[k] = gr.data_ptr();
    m[k] = avgs[k].data_ptr();
    v[k] = avg_sqs[k].data_ptr();
    t[k] = steps[k].data_ptr();
    numel[k] = params[k].numel();
  }
  HC_SPAN("hc_adam_step", dev);
  check(lib.hc_adam_step(p.data(), g.data(), m.data(), v.data(), t.data(), numel.data(), (int32_t)n, lr, beta1, beta2, eps,
                         stream_of(dev)), "hc_adam_step");
  g_launches += 2;
  for (const auto* list : {&params, &avgs, &avg_sqs, &steps})
    for (const Tensor& x : *list) torch::autograd::impl::bump_version(x);
  return true;
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
  const py::object none = py::none();
  m.def("score_rows", &score_rows, py::arg("x"), py::arg("kind") = HC_SCORE_L2, py::arg("out") = none,
        "Per-row L2 / L1 norm in the library's fixed reduction order.");
  m.def("select_threshold", &select_threshold, py::arg("score"), py::arg("q"), py::arg("out") = none,
        py::arg("n_valid") = none, py::arg("valid") = none,
        "torch.quantile(score, q) (linear interpolation) without leaving the device.  With n_valid (device int64[1]) "
        "the quantile is over the n_valid smallest scores (padding rows carry +inf); with valid (one byte per row) "
        "over the rows whose byte is set.");
  m.def("record_history", &record_history, py::arg("buffer_new"), py::arg("buffer_all"), py::arg("used_mask"),
        py::arg("sub_to_full"), py::arg("sub_to_history"), py::arg("history_to_full"), py::arg("full_to_history"),
        py::arg("header"), py::arg("score"), py::arg("thres"), py::arg("checkin_iter"), py::arg("glb_iter"),
        py::arg("n_admitted") = none, py::arg("valid") = none,
        "src/cpp/src/grad_check.cu:48-68, same argument order; mutates buffer_all, both maps, header and checkin_iter "
        "in place.  `thres` is a 1-element tensor.  valid: rows whose byte is 0 are never admitted.");
  m.def("cache_admit", &cache_admit, py::arg("produced"), py::arg("buffer"), py::arg("hidden"), py::arg("in_feat"),
        py::arg("embed_capacity"), py::arg("sub_to_full"), py::arg("sub2embed"), py::arg("score"), py::arg("thres"),
        py::arg("full2embed"), py::arg("total_num_node"), py::arg("embed2full"), py::arg("feat2full"),
        py::arg("header"), py::arg("reset_header") = false, py::arg("n_admitted") = none, py::arg("valid") = none,
        "Device-side HistoryCache.update_history (hiscache/history_cache.py:211-254).");
  m.def("evict_stale", &evict_stale, py::arg("checkin_iter"), py::arg("history_to_full"), py::arg("full_to_history"),
        py::arg("glb_iter"), py::arg("limit"), "hiscache/history_table.py:189-200.");
  m.def("evict_stale_dev", &evict_stale_dev, py::arg("checkin_iter"), py::arg("history_to_full"),
        py::arg("full_to_history"), py::arg("iter_dev"), py::arg("limit"),
        "evict_stale with the iteration number read from a device int64[1].");
  m.def("stamp_checkin", &stamp_checkin, py::arg("checkin_iter"), py::arg("iter_dev"), py::arg("marker") = 1ll << 60,
        "checkin_iter[checkin_iter == marker] = iter_dev[0].");
  m.def("evict_by_score", &evict_by_score, py::arg("sub_to_history"), py::arg("score"), py::arg("thres"),
        py::arg("checkin_iter"), py::arg("history_to_full"), py::arg("full_to_history"),
        "hiscache/history_table.py:234-241.");
  m.def("evict_both", &evict_both);
  m.def("count_history_reconstruct", &used_masks, py::arg("ptr_t"), py::arg("idx_t"), py::arg("history_maps"),
        py::arg("num_node"), py::arg("num_seed"), py::arg("num_layer"),
        "src/cpp/src/grad_check.cu:103-130: list of num_layer+1 bool masks [num_node]; [num_layer] is the seed level, "
        "[0] gates raw-feature loading.");
  m.def("count_num", &count_num, py::arg("arr"), py::arg("mmax"),
        "src/cpp/src/grad_check.cu:174-182: int32 histogram [mmax+1]; value 0 is not counted.");
  m.def("map_lookup", &map_lookup, py::arg("map_t"), py::arg("ids"), py::arg("offset") = 0,
        py::arg("force_miss_below") = 0, py::arg("out") = none, py::arg("valid") = none,
        "out[i] = map[ids[i] + offset]; the first `force_miss_below` entries and rows whose byte of `valid` is 0 are -1.");
  m.def("cache_lookup", &cache_lookup);
  m.def("gather_rows", &gather_rows, py::arg("table"), py::arg("rows"), py::arg("zero_missing") = false,
        py::arg("out_dtype") = none,
        "table[rows] with torch's negative indexing (or zeros for -1 when zero_missing).");
  m.def("load_rows", &load_rows, py::arg("host_table"), py::arg("feat_cache"), py::arg("sub_to_full"),
        py::arg("sub2feat"), py::arg("used"), py::arg("out_dtype") = none, py::arg("want_mask") = false,
        py::arg("stats") = none, py::arg("out") = none, py::arg("mask_out") = none, py::arg("staged") = none,
        "One-pass batch.x assembly (hiscache/history_cache.py:327-350).  host_table may be a pinned host tensor (rows "
        "are then read over the host link by the kernel) or a CUDA tensor.  Returns x, or (x, load_mask) when "
        "want_mask.  out / mask_out: preallocated destinations ([n, F] rows, [n] uint8 mask).  staged = (rows [n, F], "
        "mask [n] uint8): host rows fetched ahead of the step by `stage_host_rows`; a row whose mask is set is read "
        "from there instead of host_table.  `stats` then needs three counters (host, cache, staged).");
  m.def("stage_host_rows", &stage_host_rows);
  m.def("sample_batch", &sample_batch);
  m.def("sample_hop", &sample_hop, py::arg("gptr"), py::arg("gidx"), py::arg("frontier"), py::arg("fanout"),
        py::arg("seed"), py::arg("base"),
        "One hop of uniform sampling with replacement: (out_ptr [nf+1], nbr [total]) with min(fanout, degree) draws per "
        "frontier node.  Reads one size back from the device.");
  m.def("relabel_seed", &relabel_seed, py::arg("seeds"), py::arg("local_map"));
  m.def("relabel_reset", &relabel_reset, py::arg("nodes"), py::arg("local_map"));
  m.def("relabel", &relabel, py::arg("nbr"), py::arg("local_map"), py::arg("n_total"),
        "(new_nodes [n_new], local ids of nbr): new nodes numbered from n_total in order of first occurrence.  Reads "
        "n_new back from the device.");
  m.def("edge_types", &edge_types, py::arg("ptr_t"), py::arg("idx_t"), py::arg("sub_to_full"), py::arg("rows"),
        py::arg("type_bounds"), py::arg("rel_table"),
        "etype[e] = rel_table[type(dst)][type(src)], node types being ranges of global ids: the counterpart of "
        "cxgnncomp_backend.gen_edge_type_mag240m (hiscache/history_model.py:354-357).");
  m.def("rgcn_group", &rgcn_group, py::arg("ptr_t"), py::arg("idx_t"), py::arg("etype"), py::arg("num_node"),
        py::arg("num_rel"), py::arg("used_src") = none, py::arg("hmap") = none, py::arg("want_perm") = false,
        py::arg("want_rel") = false,
        "The relation-segmented block of one RGCN layer (hc_rgcn_group): (ptr2 [num_rel*num_node+1], idx2 [E], w2 [E], "
        "perm or None, rel or None).");
  m.def("rgcn_layer", &rgcn_layer);
  m.def("sage_linear", &sage_linear);
  m.def("nll_loss", &nll_loss);
  m.def("adam_step", &adam_step);
  m.def("adam_fits", &adam_fits);
}
