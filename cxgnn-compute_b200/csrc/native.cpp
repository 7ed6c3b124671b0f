// Host path of the Python backend in C++: argument checks, scratch, descriptor, launch and autograd of the operators that
// are called often and on small inputs, where the interpreter cost more than the kernels (an aggregation of 11,000 edges:
// 32 us per call through ctypes and a Python autograd function, 20 us of it kernels).
//
// The kernels stay behind the C ABI of libcxgnn_b200.so: this module opens the library it is told to (init) and calls its
// entry points. No CUDA code, no other state than the scratch buffers per stream and the transposed graphs.
#include <ATen/TensorSubclassLikeUtils.h>
#include <ATen/autocast_mode.h>
#include <c10/core/Event.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <dlfcn.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/extension.h>

#include <algorithm>
#include <list>
#include <map>
#include <mutex>

#include "../../include/cxgnn_b200.h"

namespace {

using at::Tensor;
using c10::optional;
using torch::autograd::AutogradContext;
using torch::autograd::Variable;
using torch::autograd::variable_list;

// ---- the library -----------------------------------------------------------------------------------------------------
struct Lib {
  void *handle = nullptr;
#define CXG_FN(name) decltype(&::name) name = nullptr
  CXG_FN(cxg_last_error_string);
  CXG_FN(cxg_spmm_csr_workspace_size);
  CXG_FN(cxg_spmm_csr);
  CXG_FN(cxg_spmm_csr_rows_size);
  CXG_FN(cxg_spmm_csr_rows);
  CXG_FN(cxg_spmm_csr_backward);
  CXG_FN(cxg_csr_transpose_workspace_size);
  CXG_FN(cxg_csr_transpose);
  CXG_FN(cxg_gather_edges);
  CXG_FN(cxg_linear_f32_supported);
  CXG_FN(cxg_linear_f32);
  CXG_FN(cxg_dense_wgrad_f32_workspace_size);
  CXG_FN(cxg_dense_wgrad_f32);
  CXG_FN(cxg_column_sum_workspace_size);
  CXG_FN(cxg_column_sum);
  CXG_FN(cxg_gat_scores);
  CXG_FN(cxg_gat_fused_workspace_size);
  CXG_FN(cxg_gat_fused_forward);
  CXG_FN(cxg_gat_fused_backward_bias);
  CXG_FN(cxg_gat_att_grad_workspace_size);
  CXG_FN(cxg_gat_scores_backward_add);
  CXG_FN(cxg_head_mean_bias);
  CXG_FN(cxg_gat_pad_heads);
  CXG_FN(cxg_gat_unpad_heads);
  CXG_FN(cxg_gather_rows);
  CXG_FN(cxg_sample_batch_bounds);
  CXG_FN(cxg_sample_batch);
  CXG_FN(cxg_relation_pairs_workspace_size);
  CXG_FN(cxg_relation_pairs_count);
  CXG_FN(cxg_relation_pairs_fill);
#undef CXG_FN
} lib;

void init(const std::string &path) {
  lib.handle = dlopen(path.c_str(), RTLD_NOW | RTLD_LOCAL);
  if (lib.handle == nullptr) throw std::runtime_error(std::string("cannot open ") + path + ": " + dlerror());
#define CXG_FN(name)                                                                \
  lib.name = reinterpret_cast<decltype(&::name)>(dlsym(lib.handle, #name));         \
  if (lib.name == nullptr) throw std::runtime_error(std::string("no ") + #name + " in " + path)
  CXG_FN(cxg_last_error_string);
  CXG_FN(cxg_spmm_csr_workspace_size);
  CXG_FN(cxg_spmm_csr);
  CXG_FN(cxg_spmm_csr_rows_size);
  CXG_FN(cxg_spmm_csr_rows);
  CXG_FN(cxg_spmm_csr_backward);
  CXG_FN(cxg_csr_transpose_workspace_size);
  CXG_FN(cxg_csr_transpose);
  CXG_FN(cxg_gather_edges);
  CXG_FN(cxg_linear_f32_supported);
  CXG_FN(cxg_linear_f32);
  CXG_FN(cxg_dense_wgrad_f32_workspace_size);
  CXG_FN(cxg_dense_wgrad_f32);
  CXG_FN(cxg_column_sum_workspace_size);
  CXG_FN(cxg_column_sum);
  CXG_FN(cxg_gat_scores);
  CXG_FN(cxg_gat_fused_workspace_size);
  CXG_FN(cxg_gat_fused_forward);
  CXG_FN(cxg_gat_fused_backward_bias);
  CXG_FN(cxg_gat_att_grad_workspace_size);
  CXG_FN(cxg_gat_scores_backward_add);
  CXG_FN(cxg_head_mean_bias);
  CXG_FN(cxg_gat_pad_heads);
  CXG_FN(cxg_gat_unpad_heads);
  CXG_FN(cxg_gather_rows);
  CXG_FN(cxg_sample_batch_bounds);
  CXG_FN(cxg_sample_batch);
  CXG_FN(cxg_relation_pairs_workspace_size);
  CXG_FN(cxg_relation_pairs_count);
  CXG_FN(cxg_relation_pairs_fill);
#undef CXG_FN
}

[[noreturn]] void fail(const std::string &text) { throw std::runtime_error(text); }

void check(int rc, const char *what) {
  if (rc != 0) fail(std::string(what) + " failed with status " + std::to_string(rc) + ": " + lib.cxg_last_error_string());
}

const Tensor &cuda(const Tensor &t, const char *name) {
  if (!t.is_cuda()) fail(std::string(name) + " must be a CUDA tensor (this backend has no CPU path)");
  if (!t.is_contiguous()) fail(std::string(name) + " must be contiguous");
  return t;
}
const Tensor &of_type(const Tensor &t, const char *name, std::initializer_list<at::ScalarType> types) {
  cuda(t, name);
  for (auto s : types)
    if (t.scalar_type() == s) return t;
  fail(std::string(name) + " has dtype " + c10::toString(t.scalar_type()) + ", which this operator does not take");
}
const Tensor &feature(const Tensor &t, const char *name) { return of_type(t, name, {at::kFloat, at::kBFloat16}); }
const Tensor &index_of(const Tensor &t, const char *name) { return of_type(t, name, {at::kLong, at::kInt}); }
const Tensor &f32(const Tensor &t, const char *name) { return of_type(t, name, {at::kFloat}); }

// A tensor under forward-mode differentiation. The kernels know nothing of its tangent: torch's operators take it where
// there is one, and the operators of this module go through their autograd function, which refuses it.
bool has_tangent(const Tensor &t) { return t._fw_grad(/*level=*/0).defined(); }

// Whether the pass has to go through the autograd function.
bool recorded(const Tensor &t) { return (t.requires_grad() && at::GradMode::is_enabled()) || has_tangent(t); }
bool recorded(const optional<Tensor> &t) { return t && recorded(*t); }
template <typename A, typename... B>
bool recorded(const A &a, const B &...b) {
  return recorded(a) || recorded(b...);
}

// Whether torch's own operator has to be called: transforms (vmap, functionalisation, fake tensors and other subclasses),
// forward-mode differentiation, tracing.
bool foreign(const Tensor &t) { return at::isTensorSubclassLike(t) || has_tangent(t); }
bool foreign(const optional<Tensor> &t) { return t && foreign(*t); }
template <typename... T>
bool for_torch(const T &...t) {
  return torch::jit::tracer::isTracing() || (foreign(t) || ...);
}

void *stream_of(const Tensor &t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

// The capture that records what the stream is given, or none.
optional<unsigned long long> capture_of(cudaStream_t stream) {
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  unsigned long long id = 0;
  C10_CUDA_CHECK(cudaStreamGetCaptureInfo(stream, &status, &id));
  if (status == cudaStreamCaptureStatusNone) return c10::nullopt;
  return id;
}

// ---- scratch ---------------------------------------------------------------------------------------------------------
// One buffer per (device, stream), grown on demand; contents never carry over. `kind` names the entry point family that
// used it last (whose status word check_device_status can ask for). The launches of one call hand the buffer on to each
// other, so whoever uses it holds its lock until the last of them is issued: two threads may work on one stream (a backward
// runs on a thread of the autograd engine, without the interpreter's lock), and launches of another call in between would
// overwrite what the next kernel reads. A call that a graph capture records gets a buffer of its own out of the capture's
// memory: the graph runs it again when the stream's buffer has long been replaced, or is in use.
struct Scratch {
  std::mutex in_use;
  Tensor buf;
  std::string kind;
};
std::mutex scratch_lock;
std::map<std::pair<int, void *>, Scratch> scratch;

Scratch &scratch_of(int device, void *stream) {
  std::lock_guard<std::mutex> hold(scratch_lock);
  return scratch[{device, stream}];
}

// Takes the lock without keeping other threads from the interpreter meanwhile: the holder may be Python code.
std::unique_lock<std::mutex> lock_for_launches(std::mutex &m) {
  std::unique_lock<std::mutex> hold(m, std::try_to_lock);
  if (!hold.owns_lock()) {
    if (PyGILState_Check()) {
      py::gil_scoped_release others;
      hold.lock();
    } else {
      hold.lock();
    }
  }
  return hold;
}

// The stream's scratch buffer while this thread may use it.
struct Workspace {
  std::unique_lock<std::mutex> hold;
  Tensor buf;
  void *data() const { return buf.data_ptr(); }
  size_t bytes() const { return static_cast<size_t>(buf.numel()); }
};

Workspace workspace_on(int device, void *stream, int64_t bytes, const char *kind) {
  auto buffer = [&]() {
    return at::empty({std::max<int64_t>(bytes, 1 << 20)}, at::TensorOptions().dtype(at::kByte).device(at::kCUDA, device));
  };
  if (capture_of(static_cast<cudaStream_t>(stream))) {
    Workspace w;
    w.buf = buffer();
    return w;
  }
  Scratch &s = scratch_of(device, stream);
  Tensor grown;  // allocated without the lock
  for (;;) {
    Workspace w;
    w.hold = lock_for_launches(s.in_use);
    if (grown.defined() && (!s.buf.defined() || s.buf.numel() < grown.numel())) std::swap(s.buf, grown);
    if (s.buf.defined() && s.buf.numel() >= bytes) {
      if (s.kind != kind) s.kind = kind;
      w.buf = s.buf;
      return w;
    }
    w.hold.unlock();
    grown = buffer();
  }
}

// The same for Python: `with` the object, the buffer is the calling thread's until the block ends.
class HeldWorkspace {
 public:
  HeldWorkspace(int device, int64_t bytes, std::string kind) : device_(device), bytes_(bytes), kind_(std::move(kind)) {}
  Tensor enter() {
    w_ = workspace_on(device_, c10::cuda::getCurrentCUDAStream(device_).stream(), bytes_, kind_.c_str());
    return w_.buf;
  }
  void exit() { w_ = Workspace(); }

 private:
  int device_;
  int64_t bytes_;
  std::string kind_;
  Workspace w_;
};

// (buffer or None, kind) of the current stream
std::pair<optional<Tensor>, std::string> last_workspace(int device) {
  Scratch &s = scratch_of(device, c10::cuda::getCurrentCUDAStream(device).stream());
  const auto hold = lock_for_launches(s.in_use);
  return {s.buf.defined() ? optional<Tensor>(s.buf) : c10::nullopt, s.kind};
}

// ---- aggregation -----------------------------------------------------------------------------------------------------
int64_t rows_of(const Tensor &ptr, int64_t num_node) {
  const int64_t all = ptr.size(0) - 1;
  const int64_t n = num_node > 0 ? num_node : all;  // 0 means all rows
  if (n > all) fail("num_node " + std::to_string(n) + " exceeds the " + std::to_string(all) + " rows of ptr");
  return n;
}

cxg_spmm_desc describe(const Tensor &ptr, const Tensor &idx, int64_t n, int64_t heads, int64_t feat, at::ScalarType type,
                       int64_t reduce, int64_t flags, int64_t split) {
  cxg_spmm_desc d = {};
  d.ptr = ptr.data_ptr();
  d.idx = idx.data_ptr();
  d.n_dst = n;
  d.nnz = idx.size(0);
  d.feat = static_cast<int32_t>(feat);
  d.heads = static_cast<int32_t>(heads);
  d.dtype = type == at::kFloat ? CXG_F32 : CXG_BF16;
  d.ptr_bytes = static_cast<int32_t>(ptr.element_size());
  d.idx_bytes = static_cast<int32_t>(idx.element_size());
  d.reduce = static_cast<int32_t>(reduce);
  d.flags = static_cast<uint32_t>(flags);
  d.split_edges = static_cast<int32_t>(split);
  return d;
}

void run_spmm(cxg_spmm_desc &d, const Tensor &x) {
  size_t need = 0, copy = 0;
  check(lib.cxg_spmm_csr_workspace_size(d.n_dst, d.nnz, d.feat, d.heads, d.split_edges, &need), "cxg_spmm_csr_workspace_size");
  check(lib.cxg_spmm_csr_rows_size(&d, x.size(0), &copy), "cxg_spmm_csr_rows_size");
  Tensor rows;
  if (copy > 0) {
    try {
      rows = at::empty({static_cast<int64_t>(copy)}, x.options().dtype(at::kByte));
    } catch (const c10::OutOfMemoryError &) {  // x as it is, then
      copy = 0;
    }
  }
  void *st = stream_of(x);
  const Workspace ws = workspace_on(x.device().index(), st, static_cast<int64_t>(need), "spmm");
  check(lib.cxg_spmm_csr_rows(&d, x.size(0), copy > 0 ? rows.data_ptr() : nullptr, copy, ws.data(), ws.bytes(), st), "cxg_spmm_csr");
}

// y = A x for the first rows of the graph; x [N, F] or [N, H, F]
Tensor spmm(const Tensor &x, const Tensor &ptr, const Tensor &idx, int64_t num_node, const optional<Tensor> &edge_val,
            int64_t reduce, const optional<Tensor> &out, const optional<Tensor> &edge_mask, const optional<Tensor> &edge_rel,
            int64_t rel_stride, const optional<Tensor> &targets, int64_t flags, int64_t split) {
  feature(x, "x");
  index_of(ptr, "ptr");
  index_of(idx, "idx");
  const int64_t n = rows_of(ptr, num_node);
  if (x.dim() != 2 && x.dim() != 3) fail("x must be [N, F] or [N, H, F]");
  const int64_t heads = x.dim() == 3 ? x.size(1) : 1, feat = x.size(-1);
  if (edge_val) {
    f32(*edge_val, "edge_value");
    const int64_t vh = edge_val->dim() == 2 ? edge_val->size(1) : 1;
    if (vh != heads) fail("edge_value has " + std::to_string(vh) + " heads, x has " + std::to_string(heads));
  }
  if (x.size(0) > UINT32_MAX) flags |= CXG_SPMM_GENERIC_WALK;  // the default walk keeps source rows as 32-bit numbers
  c10::cuda::CUDAGuard guard(x.device());
  Tensor y = out ? *out : (x.dim() == 3 ? at::empty({n, heads, feat}, x.options()) : at::empty({n, feat}, x.options()));
  cxg_spmm_desc d = describe(ptr, idx, n, heads, feat, x.scalar_type(), reduce, flags, split);
  d.x = x.data_ptr();
  d.y = y.data_ptr();
  if (edge_val) d.edge_val = static_cast<const float *>(edge_val->data_ptr());
  if (edge_mask) d.edge_mask = static_cast<const uint8_t *>(edge_mask->data_ptr());
  if (edge_rel) d.edge_rel = static_cast<const int32_t *>(edge_rel->data_ptr());
  if (targets) d.targets = static_cast<const int64_t *>(targets->data_ptr());
  d.rel_stride = rel_stride;
  run_spmm(d, x);
  return y;
}

// ---- transposed graphs -----------------------------------------------------------------------------------------------
struct Transposed {
  Tensor t_ptr, t_idx, t_eid, inv_deg;
};

Transposed transpose(const Tensor &ptr, const Tensor &idx, int64_t num_node, int64_t n_src, bool want_eid) {
  index_of(ptr, "ptr");
  index_of(idx, "idx");
  const int64_t n = rows_of(ptr, num_node), nnz = idx.size(0);
  c10::cuda::CUDAGuard guard(ptr.device());
  Transposed t;
  t.t_ptr = at::empty({n_src + 1}, ptr.options().dtype(at::kLong));
  t.t_idx = at::empty({nnz}, idx.options());
  if (want_eid) t.t_eid = at::empty({nnz}, idx.options());
  t.inv_deg = at::empty({n}, ptr.options().dtype(at::kFloat));
  size_t need = 0;
  check(lib.cxg_csr_transpose_workspace_size(nnz, &need), "cxg_csr_transpose_workspace_size");
  void *st = stream_of(ptr);
  const Workspace ws = workspace_on(ptr.device().index(), st, static_cast<int64_t>(need), "");
  check(lib.cxg_csr_transpose(ptr.data_ptr(), idx.data_ptr(), static_cast<int>(ptr.element_size()),
                              static_cast<int>(idx.element_size()), n, n_src, nnz, t.t_ptr.data_ptr<int64_t>(),
                              t.t_idx.data_ptr(), want_eid ? t.t_eid.data_ptr() : nullptr, t.inv_deg.data_ptr<float>(),
                              ws.data(), ws.bytes(), st),
        "cxg_csr_transpose");
  return t;
}

// The stream that has built something for keeping, and an event behind that.
struct Built {
  c10::cuda::CUDAStream stream;
  std::shared_ptr<c10::Event> event;
  explicit Built(const c10::cuda::CUDAStream &s) : stream(s), event(std::make_shared<c10::Event>(c10::DeviceType::CUDA)) { event->record(s); }
  // Another stream waits for the build, and the memory for that stream. A stream under capture cannot wait for what lies in
  // front of the capture (`outside`): the host does.
  template <typename Tensors>
  void hand_to(const c10::cuda::CUDAStream &other, bool outside, const Tensors &tensors) const {
    if (outside) {
      c10::cuda::CUDAStreamCaptureModeGuard relaxed(cudaStreamCaptureModeRelaxed);
      event->synchronize();
    } else {
      event->block(other);
    }
    for (const Tensor &t : tensors) t.record_stream(other);
  }
};

// Tensors that the current stream has built and a cache of the Python side keeps.
class Kept {
 public:
  explicit Kept(std::vector<Tensor> tensors)
      : tensors_(std::move(tensors)), device_(tensors_.at(0).device().index()), built_(c10::cuda::getCurrentCUDAStream(device_)) {}
  // They are about to be used on the current stream. True: under a capture, whose replays use them again.
  bool take() const {
    const auto stream = c10::cuda::getCurrentCUDAStream(device_);
    const bool capturing = capture_of(stream.stream()).has_value();
    if (stream != built_.stream) built_.hand_to(stream, capturing, tensors_);
    return capturing;
  }

 private:
  std::vector<Tensor> tensors_;
  c10::DeviceIndex device_;
  Built built_;
};

// The last eight transposed graphs, by the tensors they came from. An entry keeps ptr and idx alive, so their addresses
// cannot be handed to another graph. What a graph capture has recorded is there for that capture alone.
struct CachedGraph {
  const void *ptr_data, *idx_data;
  int64_t n, n_src;
  uint32_t ptr_version, idx_version;
  int device;
  Tensor ptr, idx;
  Transposed t;
  Built built;
  optional<unsigned long long> capture;
  // 1 / in-degree of every transposed edge's destination, when a mean's gradient has asked for it
  Tensor weight;
  optional<Built> weight_built;
};
std::mutex graphs_lock;
std::list<CachedGraph> &graphs = *new std::list<CachedGraph>;  // not torn down at exit: events would outlive the driver
std::list<Transposed> &captured_graphs = *new std::list<Transposed>;  // those that captures have taken: replays read them
constexpr size_t kMostGraphs = 8;

Transposed transposed_graph(const Tensor &ptr, const Tensor &idx, int64_t n, int64_t n_src) {
  const uint32_t pv = ptr._version(), iv = idx._version();
  const auto stream = c10::cuda::getCurrentCUDAStream(ptr.device().index());
  const auto capture = capture_of(stream.stream());
  {
    std::lock_guard<std::mutex> hold(graphs_lock);
    for (const auto &g : graphs)
      if (g.ptr_data == ptr.data_ptr() && g.idx_data == idx.data_ptr() && g.n == n && g.n_src == n_src && g.ptr_version == pv &&
          g.idx_version == iv && g.device == ptr.device().index() && (!g.capture || g.capture == capture)) {
        const bool outside = capture && !g.capture;
        if (outside && std::none_of(captured_graphs.begin(), captured_graphs.end(), [&](const Transposed &c) { return c.t_idx.is_same(g.t.t_idx); }))
          captured_graphs.push_back(g.t);
        if (stream != g.built.stream)
          g.built.hand_to(stream, outside, std::initializer_list<Tensor>{g.t.t_ptr, g.t.t_idx, g.t.t_eid, g.t.inv_deg});
        return g.t;
      }
  }
  const Transposed t = transpose(ptr, idx, n, n_src, true);
  CachedGraph g{ptr.data_ptr(), idx.data_ptr(), n, n_src, pv, iv, ptr.device().index(), ptr, idx, t, Built(stream), capture,
                Tensor(), c10::nullopt};
  std::lock_guard<std::mutex> hold(graphs_lock);
  while (graphs.size() >= kMostGraphs) graphs.pop_front();
  graphs.push_back(std::move(g));
  return t;
}
void forget_graphs() {
  std::lock_guard<std::mutex> hold(graphs_lock);
  graphs.clear();
  captured_graphs.clear();
}
size_t count_graphs() {
  std::lock_guard<std::mutex> hold(graphs_lock);
  return graphs.size();
}

// The weights of a mean's gradient, per transposed edge: kept with the graph, on whichever stream they are wanted. All graphs'
// together take a gigabyte at most, like the plans of the relational layers: the weights of the oldest graphs make room, and
// those of a graph that alone has more are made for the call.
constexpr size_t kMostWeightBytes = size_t{1} << 30;

Tensor mean_weights(const Transposed &t) {
  auto make = [&]() {
    Tensor w = at::empty({t.t_idx.size(0)}, t.inv_deg.options());
    check(lib.cxg_gather_edges(t.inv_deg.data_ptr<float>(), t.t_idx.data_ptr(), static_cast<int>(t.t_idx.element_size()),
                               w.data_ptr<float>(), t.t_idx.size(0), 1, 1, stream_of(w)),
          "cxg_gather_edges");
    return w;
  };
  const auto stream = c10::cuda::getCurrentCUDAStream(t.t_idx.device().index());
  const size_t bytes = static_cast<size_t>(t.t_idx.size(0)) * sizeof(float);
  if (bytes > kMostWeightBytes || capture_of(stream.stream())) return make();  // what a graph capture records is not there for others
  std::lock_guard<std::mutex> hold(graphs_lock);
  for (auto &g : graphs)
    if (g.t.t_idx.is_same(t.t_idx)) {
      if (!g.weight.defined()) {
        size_t kept = 0;
        for (const auto &other : graphs) kept += other.weight.defined() ? other.weight.nbytes() : 0;
        for (auto &other : graphs)
          if (other.weight.defined() && kept + bytes > kMostWeightBytes) {
            kept -= other.weight.nbytes();
            other.weight = Tensor();
            other.weight_built.reset();
          }
        g.weight = make();
        g.weight_built.emplace(stream);
      } else if (stream != g.weight_built->stream) {
        g.weight_built->hand_to(stream, false, std::initializer_list<Tensor>{g.weight});
      }
      return g.weight;
    }
  return make();
}

// dX = A^T dY on the cached transposed graph, in dY's type
Tensor spmm_transposed(const Tensor &grad, const Tensor &ptr, const Tensor &idx, int64_t n, int64_t n_src,
                       const optional<Tensor> &edge_val, int64_t reduce, int64_t flags, int64_t split) {
  const Transposed t = transposed_graph(ptr, idx, n, n_src);
  Tensor dy = grad.size(0) == n ? grad : grad.narrow(0, 0, n);
  optional<Tensor> tv;
  // A mean's gradient: weights per edge instead of a pass over dY (two, and two more for bf16), except where the edges are many
  // more than the values (12.6 M edges, fp32: a weight costs 10 us at 18 columns and 29 at 128, the pass 8 and 45).
  const int64_t columns = dy.numel() / std::max<int64_t>(n, 1), passes = dy.scalar_type() == at::kFloat ? 2 : 5;
  if (reduce == CXG_MEAN && dy.dim() == 2 && !edge_val && 8 * t.t_idx.size(0) <= n * columns * passes) {
    tv = mean_weights(t);
  } else if (reduce == CXG_MEAN) {
    std::vector<int64_t> shape(dy.dim(), 1);
    shape[0] = n;
    const Tensor w = t.inv_deg.view(shape);
    dy = dy.scalar_type() == at::kFloat ? at::mul(dy, w) : at::mul(dy.to(at::kFloat), w).to(dy.scalar_type());
  }
  if (edge_val) {  // the edge values in transposed order
    const Tensor ev = edge_val->contiguous();
    tv = at::empty_like(ev);
    check(lib.cxg_gather_edges(ev.data_ptr<float>(), t.t_eid.data_ptr(), static_cast<int>(t.t_eid.element_size()),
                               tv->data_ptr<float>(), std::min(t.t_eid.size(0), ev.size(0)),
                               static_cast<int>(ev.dim() == 2 ? ev.size(1) : 1), 1, stream_of(ev)),
          "cxg_gather_edges");
  }
  return spmm(dy.contiguous(), t.t_ptr, t.t_idx, n_src, tv, CXG_SUM, c10::nullopt, c10::nullopt, c10::nullopt, 0, c10::nullopt,
              flags, split);
}

// Sum or mean aggregation with its gradients: x over the transposed graph (or, `scatter`, with atomics over the forward
// edges), the edge values by a second pass over the forward edges.
class SageFunction : public torch::autograd::Function<SageFunction> {
 public:
  static Tensor forward(AutogradContext *ctx, const Tensor &x, const Tensor &ptr, const Tensor &idx,
                        const optional<Tensor> &edge_val, int64_t num_node, int64_t reduce, int64_t flags, int64_t split,
                        bool scatter) {
    ctx->save_for_backward({x, ptr, idx, edge_val ? *edge_val : Tensor()});
    ctx->saved_data["n"] = num_node;
    ctx->saved_data["reduce"] = reduce;
    ctx->saved_data["flags"] = flags;
    ctx->saved_data["split"] = split;
    ctx->saved_data["scatter"] = scatter;
    return spmm(x, ptr, idx, num_node, edge_val, reduce, c10::nullopt, c10::nullopt, c10::nullopt, 0, c10::nullopt, flags, split);
  }
  static variable_list backward(AutogradContext *ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &ptr = saved[1], &idx = saved[2];
    optional<Tensor> edge_val;
    if (saved[3].defined()) edge_val = saved[3];
    const Tensor g = grads[0].contiguous();
    const int64_t n = rows_of(ptr, ctx->saved_data["n"].toInt()), reduce = ctx->saved_data["reduce"].toInt();
    const int64_t flags = ctx->saved_data["flags"].toInt(), split = ctx->saved_data["split"].toInt();
    c10::cuda::CUDAGuard guard(g.device());
    Tensor dx, dval;
    bool need_dx = ctx->needs_input_grad(0);
    const bool need_dval = edge_val && ctx->needs_input_grad(3);
    if (need_dx && !ctx->saved_data["scatter"].toBool() && n > 0 && idx.size(0) > 0) {
      dx = spmm_transposed(g, ptr, idx, n, x.size(0), edge_val, reduce, flags, split);
      need_dx = false;
    }
    if (need_dx || need_dval) {
      cxg_spmm_desc d = describe(ptr, idx, n, g.dim() == 3 ? g.size(1) : 1, g.size(-1), g.scalar_type(), reduce, flags, split);
      Tensor xs;
      if (edge_val) d.edge_val = static_cast<const float *>(edge_val->data_ptr());
      if (need_dx) dx = at::zeros(x.sizes(), x.options().dtype(at::kFloat));
      if (need_dval) {
        dval = at::zeros(edge_val->sizes(), edge_val->options());
        xs = x.scalar_type() == g.scalar_type() ? x : x.to(g.scalar_type());
        d.x = xs.data_ptr();
      }
      check(lib.cxg_spmm_csr_backward(&d, g.data_ptr(), need_dx ? dx.data_ptr<float>() : nullptr,
                                      need_dval ? dval.data_ptr<float>() : nullptr, stream_of(g)),
            "cxg_spmm_csr_backward");
    }
    if (dx.defined() && dx.scalar_type() != x.scalar_type()) dx = dx.to(x.scalar_type());
    return {dx, Tensor(), Tensor(), dval, Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

Tensor sage(const Tensor &x, const Tensor &ptr, const Tensor &idx, const optional<Tensor> &edge_val, int64_t num_node,
            int64_t reduce, int64_t flags, int64_t split, bool scatter) {
  if (recorded(x, edge_val))
    return SageFunction::apply(x, ptr, idx, edge_val, num_node, reduce, flags, split, scatter);
  return spmm(x, ptr, idx, num_node, edge_val, reduce, c10::nullopt, c10::nullopt, c10::nullopt, 0, c10::nullopt, flags, split);
}

Tensor gather_rows(const Tensor &x, const Tensor &rows) {
  if (for_torch(x, rows)) return x.index_select(0, rows);
  cuda(x, "x");
  of_type(rows, "rows", {at::kLong});
  c10::cuda::CUDAGuard guard(x.device());
  Tensor out = at::empty({rows.size(0), x.size(1)}, x.options());
  check(lib.cxg_gather_rows(x.data_ptr(), rows.data_ptr<int64_t>(), out.data_ptr(), rows.size(0),
                            x.size(1) * static_cast<int64_t>(x.element_size()), stream_of(x)),
        "cxg_gather_rows");
  return out;
}

// ---- linear transform ------------------------------------------------------------------------------------------------
bool aligned16(const Tensor &t) { return reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0; }

// fp32 matrices that the tensor-core kernel takes as they are
bool dense_rows(const Tensor &t) {
  return t.dim() == 2 && t.is_cuda() && t.scalar_type() == at::kFloat && t.is_contiguous() && t.numel() > 0 && aligned16(t);
}

// x [M, K] . w [N, K]^T (w_rows_k: w is [K, N]) + bias + add
Tensor linear_product(const Tensor &x, const Tensor &w, bool w_rows_k, const optional<Tensor> &bias, const optional<Tensor> &add) {
  const int64_t n = w_rows_k ? w.size(1) : w.size(0);
  Tensor y = at::empty({x.size(0), n}, x.options());
  check(lib.cxg_linear_f32(x.data_ptr<float>(), w.data_ptr<float>(), bias ? bias->data_ptr<float>() : nullptr,
                           add ? add->data_ptr<float>() : nullptr, y.data_ptr<float>(), x.size(0), static_cast<int>(x.size(1)),
                           static_cast<int>(n), w_rows_k ? 1 : 0, stream_of(x)),
        "cxg_linear_f32");
  return y;
}

// g [M, N]^T . x [M, K]
Tensor linear_weight_grad(const Tensor &g, const Tensor &x) {
  const int64_t m = x.size(0), n = g.size(1), k = x.size(1);
  if (!dense_rows(g) || !dense_rows(x) || n % 4 != 0 || k % 4 != 0) return at::mm(g.t(), x);
  Tensor dw = at::empty({n, k}, x.options());
  size_t need = 0;
  check(lib.cxg_dense_wgrad_f32_workspace_size(m, static_cast<int>(n), static_cast<int>(k), &need),
        "cxg_dense_wgrad_f32_workspace_size");
  void *st = stream_of(x);
  const Workspace ws = workspace_on(x.device().index(), st, static_cast<int64_t>(need), "");
  check(lib.cxg_dense_wgrad_f32(g.data_ptr<float>(), x.data_ptr<float>(), m, static_cast<int>(n), static_cast<int>(k),
                                dw.data_ptr<float>(), ws.data(), ws.bytes(), st),
        "cxg_dense_wgrad_f32");
  return dw;
}

Tensor rows_sum(const Tensor &g) {
  Tensor out = at::empty({g.size(1)}, g.options());
  size_t need = 0;
  check(lib.cxg_column_sum_workspace_size(static_cast<int>(g.size(1)), &need), "cxg_column_sum_workspace_size");
  void *st = stream_of(g);
  const Workspace ws = workspace_on(g.device().index(), st, static_cast<int64_t>(need), "");
  check(lib.cxg_column_sum(g.data_ptr(), CXG_F32, g.size(0), static_cast<int>(g.size(1)), out.data_ptr<float>(), ws.data(),
                           ws.bytes(), st),
        "cxg_column_sum");
  return out;
}

bool linear_fits(const Tensor &x, const Tensor &w) {
  return dense_rows(x) && dense_rows(w) && x.size(1) == w.size(1) && x.device() == w.device() &&
         lib.cxg_linear_f32_supported(x.size(0), static_cast<int>(x.size(1)), static_cast<int>(w.size(0))) == 1;
}

class LinearFunction : public torch::autograd::Function<LinearFunction> {
 public:
  static Tensor forward(AutogradContext *ctx, const Tensor &x, const Tensor &w, const optional<Tensor> &bias,
                        const optional<Tensor> &add, bool same_bits) {
    ctx->save_for_backward({x, w});
    ctx->saved_data["bias"] = bias.has_value();
    ctx->saved_data["add"] = add.has_value();
    if (!same_bits) return linear_product(x, w, false, bias, add);
    const Tensor y = at::linear(x, w, bias);
    return add ? *add + y : y;
  }
  static variable_list backward(AutogradContext *ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &w = saved[1];
    const Tensor g = grads[0].contiguous();
    c10::cuda::CUDAGuard guard(g.device());
    Tensor dx, dw, db;
    // the edges of the node are those of the tensors that were given
    const bool bias = ctx->saved_data["bias"].toBool(), need_db = bias && ctx->needs_input_grad(2);
    const bool need_add = ctx->saved_data["add"].toBool() && ctx->needs_input_grad(bias ? 3 : 2);
    if (at::GradMode::is_enabled()) {  // a graph of the backward itself is wanted
      if (ctx->needs_input_grad(0)) dx = at::mm(g, w);
      if (ctx->needs_input_grad(1)) dw = at::mm(g.t(), x);
      if (need_db) db = g.sum(0);
    } else {
      if (ctx->needs_input_grad(0))
        dx = dense_rows(g) && lib.cxg_linear_f32_supported(g.size(0), static_cast<int>(g.size(1)), static_cast<int>(w.size(1)))
                 ? linear_product(g, w, true, c10::nullopt, c10::nullopt)
                 : at::mm(g, w);
      if (ctx->needs_input_grad(1)) dw = linear_weight_grad(g, x);
      if (need_db) db = rows_sum(g);
    }
    return {dx, dw, db, need_add ? grads[0] : Tensor(), Tensor()};
  }
};

// x . w^T (+ bias) (+ add): the tensor-core kernel for fp32 matrices it takes, torch otherwise (CPU, other types, autocast,
// rows that are not whole 16-byte vectors). same_bits: where a gradient is recorded the product itself is torch's and only
// the gradients are the kernel's. In front of a ReLU (and of the LeakyReLU on a GAT layer's scores) another rounding, though
// a better one, puts the few values within rounding of zero on its other side, and each of them moves the gradients: those
// of a sampled batch by up to 3e-4 of their norm, those of a GAT layer by up to 2e-3.
Tensor linear(const Tensor &x, const Tensor &w, const optional<Tensor> &bias, const optional<Tensor> &add, bool same_bits) {
  const bool fits = !for_torch(x, w, bias, add) && linear_fits(x, w) && !at::autocast::is_autocast_enabled(at::kCUDA) &&
                    (!bias || (bias->scalar_type() == at::kFloat && bias->is_contiguous() && bias->device() == x.device() &&
                               bias->dim() == 1 && bias->size(0) == w.size(0)));
  const bool add_fits = add && dense_rows(*add) && add->size(0) == x.size(0) && add->size(1) == w.size(0) && add->device() == x.device();
  if (!fits || (add && !add_fits)) {
    const Tensor y = at::linear(x, w, bias);
    return add ? *add + y : y;
  }
  c10::cuda::CUDAGuard guard(x.device());
  if (recorded(x, w, bias, add)) return LinearFunction::apply(x, w, bias, add, same_bits);
  return linear_product(x, w, false, bias, add);
}

// ---- SAGE layer ------------------------------------------------------------------------------------------------------
// into += g . w, or g . w into a new matrix
Tensor linear_input_grad(const Tensor &g, const Tensor &w, const Tensor &into) {
  const int n = static_cast<int>(g.size(1)), k = static_cast<int>(w.size(1));
  if (dense_rows(g) && lib.cxg_linear_f32_supported(g.size(0), n, k) && (!into.defined() || aligned16(into))) {
    const Tensor out = into.defined() ? into : at::empty({g.size(0), k}, g.options());
    check(lib.cxg_linear_f32(g.data_ptr<float>(), w.data_ptr<float>(), nullptr, into.defined() ? into.data_ptr<float>() : nullptr,
                             out.data_ptr<float>(), g.size(0), n, k, 1, stream_of(g)),
          "cxg_linear_f32");
    return out;
  }
  return into.defined() ? into.addmm_(g, w) : at::mm(g, w);
}

// mean(x) . wl^T + x[:n] . wr^T + bl, the mean taken before (`first`) or behind the product with wl. As one operator the
// gradient of x[:n] is added to that of the aggregation in place; as separate ones it was a matrix of zeros, a copy and a sum.
class SageLayerFunction : public torch::autograd::Function<SageLayerFunction> {
 public:
  static Tensor run(const Tensor &x, const Tensor &ptr, const Tensor &idx, const Tensor &wl, const Tensor &wr,
                    const optional<Tensor> &bl, int64_t n, bool first, int64_t flags, int64_t split, Tensor *mean, bool record) {
    auto aggregate = [&](const Tensor &t) {
      return spmm(t, ptr, idx, n, c10::nullopt, CXG_MEAN, c10::nullopt, c10::nullopt, c10::nullopt, 0, c10::nullopt, flags, split);
    };
    // the products of a recorded pass keep torch's rounding, as in `linear`
    auto product = [&](const Tensor &t) { return record ? at::linear(t, wl, bl) : linear_product(t, wl, false, bl, c10::nullopt); };
    Tensor out;
    if (first) {
      const Tensor m = aggregate(x);
      if (mean != nullptr) *mean = m;
      out = product(m);
    } else {
      out = aggregate(product(x));
    }
    if (record) return out.add_(at::linear(x.narrow(0, 0, n), wr));
    check(lib.cxg_linear_f32(x.data_ptr<float>(), wr.data_ptr<float>(), nullptr, out.data_ptr<float>(), out.data_ptr<float>(), n,
                             static_cast<int>(x.size(1)), static_cast<int>(wr.size(0)), 0, stream_of(x)),
          "cxg_linear_f32");
    return out;
  }
  static Tensor forward(AutogradContext *ctx, const Tensor &x, const Tensor &ptr, const Tensor &idx, const Tensor &wl,
                        const Tensor &wr, const optional<Tensor> &bl, int64_t n, bool first, int64_t flags, int64_t split) {
    Tensor mean;
    const Tensor out = run(x, ptr, idx, wl, wr, bl, n, first, flags, split, &mean, true);
    ctx->save_for_backward({x, ptr, idx, wl, wr, mean});
    ctx->saved_data["bias"] = bl.has_value();
    ctx->saved_data["n"] = n;
    ctx->saved_data["first"] = first;
    ctx->saved_data["flags"] = flags;
    ctx->saved_data["split"] = split;
    return out;
  }
  static variable_list backward(AutogradContext *ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &ptr = saved[1], &idx = saved[2], &wl = saved[3], &wr = saved[4], &mean = saved[5];
    const int64_t n = ctx->saved_data["n"].toInt(), flags = ctx->saved_data["flags"].toInt(), split = ctx->saved_data["split"].toInt();
    const bool need_x = ctx->needs_input_grad(0), need_wl = ctx->needs_input_grad(3), need_wr = ctx->needs_input_grad(4);
    const bool need_bl = ctx->saved_data["bias"].toBool() && ctx->needs_input_grad(5);
    const Tensor g = grads[0].contiguous();
    c10::cuda::CUDAGuard guard(g.device());
    auto back = [&](const Tensor &t) { return spmm_transposed(t, ptr, idx, n, x.size(0), c10::nullopt, CXG_MEAN, flags, split); };
    Tensor dx, dwl, dwr, dbl;
    if (ctx->saved_data["first"].toBool()) {
      if (need_x) dx = back(linear_input_grad(g, wl, Tensor()));
      if (need_wl) dwl = linear_weight_grad(g, mean);
      if (need_bl) dbl = rows_sum(g);
    } else if (need_x || need_wl || need_bl) {
      const Tensor dh = back(g);
      if (need_x) dx = linear_input_grad(dh, wl, Tensor());
      if (need_wl) dwl = linear_weight_grad(dh, x);
      if (need_bl) dbl = rows_sum(dh);
    }
    if (need_x) linear_input_grad(g, wr, dx.narrow(0, 0, n));
    if (need_wr) dwr = linear_weight_grad(g, x.narrow(0, 0, n));
    return {dx, Tensor(), Tensor(), dwl, dwr, dbl, Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

// None when the operator does not cover the arguments.
optional<Tensor> sage_layer(const Tensor &x, const Tensor &ptr, const Tensor &idx, const Tensor &wl, const Tensor &wr,
                            const optional<Tensor> &bl, int64_t n, bool first, int64_t flags, int64_t split) {
  if (for_torch(x, wl, wr, bl) || n < 1 || !dense_rows(x) || x.size(0) < n || idx.size(0) < 1 || ptr.size(0) - 1 < n || wl.size(0) != wr.size(0) ||
      !linear_fits(x, wl) || !linear_fits(x, wr) ||
      !lib.cxg_linear_f32_supported(n, static_cast<int>(x.size(1)), static_cast<int>(wl.size(0))) ||
      at::autocast::is_autocast_enabled(at::kCUDA) ||
      (bl && (bl->scalar_type() != at::kFloat || !bl->is_contiguous() || bl->device() != x.device() || bl->numel() != wl.size(0))))
    return c10::nullopt;
  index_of(ptr, "ptr");
  index_of(idx, "idx");
  c10::cuda::CUDAGuard guard(x.device());
  if (recorded(x, wl, wr, bl)) return SageLayerFunction::apply(x, ptr, idx, wl, wr, bl, n, first, flags, split);
  return SageLayerFunction::run(x, ptr, idx, wl, wr, bl, n, first, flags, split, nullptr, false);
}

// ---- GAT layer -------------------------------------------------------------------------------------------------------
Tensor head_mean_bias(const Tensor &x, const optional<Tensor> &bias, int64_t heads, int64_t c) {
  Tensor out = at::empty({x.size(0), c}, x.options());
  check(lib.cxg_head_mean_bias(x.data_ptr<float>(), bias ? bias->data_ptr<float>() : nullptr, out.data_ptr<float>(), x.size(0),
                               static_cast<int>(heads), static_cast<int>(c), stream_of(x)),
        "cxg_head_mean_bias");
  return out;
}

// Attention scores, softmax, weighted neighbour sum, heads joined or averaged, bias: x [n_src, H, C] -> [n, H * C] or [n, C].
class GatFunction : public torch::autograd::Function<GatFunction> {
 public:
  static Tensor run(const Tensor &x, const Tensor &att_src, const Tensor &att_dst, const optional<Tensor> &bias, const Tensor &ptr,
                    const Tensor &idx, int64_t n, double slope, bool concat, variable_list *keep, Tensor *joined = nullptr) {
    const int64_t n_src = x.size(0), h = x.size(1), c = x.size(2);
    const int hi = static_cast<int>(h), ci = static_cast<int>(c);
    void *st = stream_of(x);
    const Tensor a_src = at::empty({n_src, h}, x.options()), a_dst = at::empty({n, h}, x.options());
    check(lib.cxg_gat_scores(x.data_ptr<float>(), att_src.data_ptr<float>(), att_dst.data_ptr<float>(), a_src.data_ptr<float>(),
                             a_dst.data_ptr<float>(), n_src, n, hi, ci, st),
          "cxg_gat_scores");
    const Tensor y = at::empty({n, h * c}, x.options()), top = at::empty({n, h}, x.options()), sum = at::empty({n, h}, x.options());
    size_t need = 0;
    check(lib.cxg_gat_fused_workspace_size(n, idx.size(0), hi, ci, &need), "cxg_gat_fused_workspace_size");
    {
      const Workspace ws = workspace_on(x.device().index(), st, static_cast<int64_t>(need), "");
      check(lib.cxg_gat_fused_forward(ptr.data_ptr(), idx.data_ptr(), static_cast<int>(ptr.element_size()),
                                      static_cast<int>(idx.element_size()), x.data_ptr<float>(), a_src.data_ptr<float>(),
                                      a_dst.data_ptr<float>(), y.data_ptr<float>(), top.data_ptr<float>(), sum.data_ptr<float>(), n,
                                      idx.size(0), hi, ci, static_cast<float>(slope), ws.data(),
                                      ws.bytes(), st),
            "cxg_gat_fused_forward");
    }
    if (keep != nullptr) *keep = {x, att_src, att_dst, ptr, idx, a_src, a_dst, y, top, sum};
    if (joined != nullptr) {
      *joined = y;
      return y;
    }
    if (concat) return bias ? head_mean_bias(y, bias, 1, h * c) : y;
    return head_mean_bias(y, bias, h, c);
  }
  static Tensor forward(AutogradContext *ctx, const Tensor &x, const Tensor &att_src, const Tensor &att_dst,
                        const optional<Tensor> &bias, const Tensor &ptr, const Tensor &idx, int64_t n, double slope, bool concat) {
    variable_list keep;
    Tensor out = run(x, att_src, att_dst, bias, ptr, idx, n, slope, concat, &keep);
    if (concat && !bias) out = out.view(out.sizes());  // y itself is kept for the backward
    ctx->save_for_backward(keep);
    ctx->saved_data["slope"] = slope;
    ctx->saved_data["concat"] = concat;
    ctx->saved_data["bias"] = bias.has_value();
    return out;
  }
  static variable_list backward(AutogradContext *ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &att_src = saved[1], &att_dst = saved[2], &ptr = saved[3], &idx = saved[4], &a_src = saved[5],
                 &a_dst = saved[6], &y = saved[7], &top = saved[8], &sum = saved[9];
    const int64_t n_src = x.size(0), h = x.size(1), c = x.size(2), n = y.size(0);
    const int hi = static_cast<int>(h), ci = static_cast<int>(c);
    c10::cuda::CUDAGuard guard(x.device());
    void *st = stream_of(x);
    const Tensor g = grads[0].contiguous();
    Tensor db;
    const bool concat = ctx->saved_data["concat"].toBool(), need_db = ctx->saved_data["bias"].toBool() && ctx->needs_input_grad(3);
    // heads side by side: the columns of dy are the bias's, and the backward reads them anyway
    if (need_db) db = concat && n > 0 && n_src > 0 ? at::empty({h * c}, x.options()) : rows_sum(g);
    const Tensor dy =
        concat ? g : g.mul(1.0 / static_cast<double>(h)).unsqueeze(1).expand({n, h, c}).contiguous();
    const Transposed t = transposed_graph(ptr, idx, n, n_src);
    const Tensor dx = at::empty_like(x), d_src = at::empty_like(a_src), d_dst = at::empty_like(a_dst);
    const Tensor g_as = at::empty_like(att_src), g_ad = at::empty_like(att_dst);
    size_t need = 0, need_att = 0;
    check(lib.cxg_gat_fused_workspace_size(n, idx.size(0), hi, ci, &need), "cxg_gat_fused_workspace_size");
    check(lib.cxg_gat_att_grad_workspace_size(hi, ci, &need_att), "cxg_gat_att_grad_workspace_size");
    const Workspace ws = workspace_on(x.device().index(), st, static_cast<int64_t>(std::max(need, need_att)), "");
    check(lib.cxg_gat_fused_backward_bias(t.t_ptr.data_ptr(), t.t_idx.data_ptr(), static_cast<int>(t.t_ptr.element_size()),
                                     static_cast<int>(t.t_idx.element_size()), dy.data_ptr<float>(), y.data_ptr<float>(),
                                     x.data_ptr<float>(), a_src.data_ptr<float>(), a_dst.data_ptr<float>(), top.data_ptr<float>(),
                                     sum.data_ptr<float>(), dx.data_ptr<float>(), d_src.data_ptr<float>(), d_dst.data_ptr<float>(),
                                     n_src, n, t.t_idx.size(0), hi, ci, static_cast<float>(ctx->saved_data["slope"].toDouble()),
                                     nullptr, nullptr, static_cast<int>(ptr.element_size()),
                                     need_db && concat && n > 0 && n_src > 0 ? db.data_ptr<float>() : nullptr, ws.data(), ws.bytes(), st),
          "cxg_gat_fused_backward");
    check(lib.cxg_gat_scores_backward_add(x.data_ptr<float>(), d_src.data_ptr<float>(), d_dst.data_ptr<float>(),
                                          att_src.data_ptr<float>(), att_dst.data_ptr<float>(), dx.data_ptr<float>(),
                                          g_as.data_ptr<float>(), g_ad.data_ptr<float>(), n_src, n, hi, ci, ws.data(),
                                          ws.bytes(), st),
          "cxg_gat_scores_backward_add");
    return {dx, g_as, g_ad, db, Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

Tensor gat_layer(const Tensor &x, const Tensor &att_src, const Tensor &att_dst, const optional<Tensor> &bias, const Tensor &ptr,
                 const Tensor &idx, int64_t num_dst, double slope, bool concat) {
  f32(x, "x");
  f32(att_src, "att_src");
  f32(att_dst, "att_dst");
  index_of(ptr, "ptr");
  index_of(idx, "idx");
  const int64_t n = rows_of(ptr, num_dst), h = x.size(1), c = x.size(2);
  if (x.dim() != 3 || att_src.numel() != h * c || att_dst.numel() != h * c || n > x.size(0))
    fail("gat_layer: x must be [n_src, H, C] with n_src >= num_dst, the attention vectors [H, C]");
  if (bias) {
    f32(*bias, "bias");
    if (bias->numel() != (concat ? h * c : c)) fail("gat_layer: the bias must have one value per output column");
  }
  c10::cuda::CUDAGuard guard(x.device());
  if (recorded(x, att_src, att_dst, bias))
    return GatFunction::apply(x, att_src, att_dst, bias, ptr, idx, n, slope, concat);
  return GatFunction::run(x, att_src, att_dst, bias, ptr, idx, n, slope, concat, nullptr);
}

// The whole layer in inference where its heads are not whole vectors (class counts): transformed with the heads padded, so that
// no vector lies across two of them (4 heads of 47, 2.3 M edges: 665 us without, see gat_weights for what the walk gains). None
// where it does not cover the arguments.
optional<Tensor> gat_layer_padded(const Tensor &x, const Tensor &w, const Tensor &att_src, const Tensor &att_dst,
                                  const optional<Tensor> &bias, const Tensor &ptr, const Tensor &idx, int64_t num_dst, int64_t heads,
                                  double slope, bool concat) {
  const int64_t c = w.dim() == 2 && heads > 0 ? w.size(0) / heads : 0, cp = (c + 3) / 4 * 4;
  // below eight columns the zeros are a third of a row and more
  if (c < 8 || cp == c || (heads & (heads - 1)) != 0 || heads > 8 || heads * cp > 512 || c * heads != w.size(0)) return c10::nullopt;
  if (for_torch(x, w, att_src, att_dst, bias) || recorded(x, w, att_src, att_dst, bias) || at::autocast::is_autocast_enabled(at::kCUDA) ||
      !linear_fits(x, w) || !lib.cxg_linear_f32_supported(x.size(0), static_cast<int>(x.size(1)), static_cast<int>(heads * cp)))
    return c10::nullopt;
  auto fits = [&](const Tensor &t, int64_t numel) {
    return t.is_cuda() && t.device() == x.device() && t.scalar_type() == at::kFloat && t.is_contiguous() && t.numel() == numel;
  };
  if (!fits(att_src, heads * c) || !fits(att_dst, heads * c) || (bias && !fits(*bias, concat ? heads * c : c))) return c10::nullopt;
  index_of(ptr, "ptr");
  index_of(idx, "idx");
  const int64_t n = rows_of(ptr, num_dst);
  if (n < 1 || n > x.size(0)) return c10::nullopt;
  c10::cuda::CUDAGuard guard(x.device());
  const int hi = static_cast<int>(heads), ci = static_cast<int>(c), cpi = static_cast<int>(cp);
  const Tensor wp = at::empty({heads * cp, x.size(1)}, x.options()), att = at::empty({2, heads, cp}, x.options());
  check(lib.cxg_gat_pad_heads(w.data_ptr<float>(), att_src.data_ptr<float>(), att_dst.data_ptr<float>(), wp.data_ptr<float>(),
                              att.data_ptr<float>(), att.data_ptr<float>() + heads * cp, hi, ci, cpi, static_cast<int>(x.size(1)),
                              stream_of(x)),
        "cxg_gat_pad_heads");
  const Tensor h = linear_product(x, wp, false, c10::nullopt, c10::nullopt).view({x.size(0), heads, cp});
  Tensor y;
  GatFunction::run(h, att.select(0, 0), att.select(0, 1), c10::nullopt, ptr, idx, n, slope, concat, nullptr, &y);
  Tensor out = at::empty({n, concat ? heads * c : c}, x.options());
  check(lib.cxg_gat_unpad_heads(y.data_ptr<float>(), bias ? bias->data_ptr<float>() : nullptr, out.data_ptr<float>(), n, hi, ci, cpi,
                                concat ? 1 : 0, stream_of(x)),
        "cxg_gat_unpad_heads");
  return out;
}

// ---- relational layer ------------------------------------------------------------------------------------------------
// (relation, source and number of every position, first position of every source's list, the lists, position of every edge)
std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor, Tensor> relation_pairs(const Tensor &idx, const Tensor &etype, int64_t n_src,
                                                                          int64_t num_rel) {
  index_of(idx, "idx");
  index_of(etype, "edge types");
  const int64_t nnz = std::min(idx.size(0), etype.size(0));
  const int ib = static_cast<int>(idx.element_size()), rb = static_cast<int>(etype.element_size()), r = static_cast<int>(num_rel);
  c10::cuda::CUDAGuard guard(idx.device());
  const auto i64 = idx.options().dtype(at::kLong), i32 = idx.options().dtype(at::kInt);
  size_t need = 0;
  check(lib.cxg_relation_pairs_workspace_size(n_src, r, &need), "cxg_relation_pairs_workspace_size");
  // a buffer of its own: the second call continues in it behind the read-back
  const Tensor ws = at::empty({static_cast<int64_t>(need)}, idx.options().dtype(at::kByte)), sizes = at::empty({3}, i64);
  void *st = stream_of(idx);
  check(lib.cxg_relation_pairs_count(idx.data_ptr(), ib, etype.data_ptr(), rb, nnz, n_src, r, sizes.data_ptr<int64_t>(),
                                     ws.data_ptr(), need, st),
        "cxg_relation_pairs_count");
  Tensor host;
  {
    py::gil_scoped_release other_threads;
    host = sizes.cpu();
  }
  const int64_t *h = host.data_ptr<int64_t>();
  if (h[2] != 0)
    fail("edge types must lie in [0, " + std::to_string(num_rel) + ") and sources in [0, " + std::to_string(n_src) + ")");
  Tensor rel = at::empty({h[0]}, i64), src = at::empty({h[0]}, i64), pos = at::empty({h[0]}, i64), src_ptr = at::empty({n_src + 1}, i64),
         src_pos = at::empty({h[1]}, i32), edge_pos = at::empty({nnz}, i32);
  check(lib.cxg_relation_pairs_fill(idx.data_ptr(), ib, etype.data_ptr(), rb, nnz, n_src, r, rel.data_ptr<int64_t>(),
                                    src.data_ptr<int64_t>(), pos.data_ptr<int64_t>(), src_ptr.data_ptr<int64_t>(),
                                    src_pos.data_ptr<int32_t>(), edge_pos.data_ptr<int32_t>(), ws.data_ptr(), need, st),
        "cxg_relation_pairs_fill");
  return {rel, src, pos, src_ptr, src_pos, edge_pos};
}

// ---- neighbour sampling ----------------------------------------------------------------------------------------------
// The most a call may reserve for the nodes and edges a batch can reach; above it the hops are run one by one.
constexpr int64_t kMostSampled = 1 << 27;

bool sample_batch_fits(int64_t n_seeds, std::vector<int> fanouts, int64_t n_nodes, int64_t nnz) {
  int64_t nodes = 0, rows = 0, edges = 0;
  size_t bytes = 0;
  if (n_seeds < 1 || lib.cxg_sample_batch_bounds(n_seeds, fanouts.data(), static_cast<int>(fanouts.size()), n_nodes, nnz, &nodes,
                                                 &rows, &edges, &bytes) != 0)
    return false;
  return nodes + edges <= kMostSampled;
}

// (nodes, ptr, idx, nodes after every hop, edges after every hop): one host synchronisation, at the end, for the sizes.
std::tuple<Tensor, Tensor, Tensor, std::vector<int64_t>, std::vector<int64_t>> sample_batch(
    const Tensor &gptr, const Tensor &gidx, const Tensor &seeds, std::vector<int> fanouts, std::vector<uint64_t> hop_seeds,
    const Tensor &local_of, const Tensor &bitmap, const Tensor &host_sizes) {
  index_of(gptr, "graph_ptr");
  index_of(gidx, "graph_idx");
  of_type(seeds, "seeds", {at::kLong});
  const int hops = static_cast<int>(fanouts.size());
  const int64_t n_nodes = gptr.size(0) - 1, nnz = gidx.size(0);
  int64_t max_nodes = 0, max_rows = 0, max_edges = 0;
  size_t bytes = 0;
  check(lib.cxg_sample_batch_bounds(seeds.size(0), fanouts.data(), hops, n_nodes, nnz, &max_nodes, &max_rows, &max_edges, &bytes),
        "cxg_sample_batch_bounds");
  c10::cuda::CUDAGuard guard(seeds.device());
  const auto opt = seeds.options();
  Tensor nodes = at::empty({max_nodes}, opt), ptr = at::empty({max_rows + 1}, opt), idx = at::empty({max_edges}, opt);
  Tensor sizes = at::empty({2 * (hops + 1)}, opt);
  void *st = stream_of(seeds);
  {
    const Workspace ws = workspace_on(seeds.device().index(), st, static_cast<int64_t>(bytes), "");
    check(lib.cxg_sample_batch(gptr.data_ptr(), gidx.data_ptr(), static_cast<int>(gptr.element_size()),
                               static_cast<int>(gidx.element_size()), n_nodes, nnz, seeds.data_ptr<int64_t>(), seeds.size(0),
                               fanouts.data(), hops, hop_seeds.data(), local_of.data_ptr<int64_t>(),
                               reinterpret_cast<uint32_t *>(bitmap.data_ptr()), nodes.data_ptr<int64_t>(), ptr.data_ptr<int64_t>(),
                               idx.data_ptr<int64_t>(), sizes.data_ptr<int64_t>(), ws.data(), ws.bytes(), st),
          "cxg_sample_batch");
  }
  host_sizes.narrow(0, 0, sizes.size(0)).copy_(sizes, /*non_blocking=*/true);
  {
    py::gil_scoped_release other_threads;
    c10::cuda::getCurrentCUDAStream(seeds.device().index()).synchronize();
  }
  const int64_t *h = host_sizes.data_ptr<int64_t>();
  if (h[0] < 0) fail("sample_batch: seeds must be node ids in [0, " + std::to_string(n_nodes) + ")");
  std::vector<int64_t> known(h, h + hops + 1), edges(h + hops + 2, h + 2 * (hops + 1));
  const int64_t rows = known[hops - 1];
  return {nodes.narrow(0, 0, known[hops]), ptr.narrow(0, 0, rows + 1), idx.narrow(0, 0, edges[hops - 1]), known, edges};
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.def("init", &init);
  py::class_<HeldWorkspace>(m, "Workspace")
      .def(py::init<int, int64_t, std::string>())
      .def("__enter__", &HeldWorkspace::enter)
      .def("__exit__", [](HeldWorkspace &w, const py::args &) { w.exit(); });
  m.def("last_workspace", &last_workspace);
  py::class_<Kept>(m, "Kept").def(py::init<std::vector<Tensor>>()).def("take", &Kept::take);
  m.def("capturing", [](int device) { return capture_of(c10::cuda::getCurrentCUDAStream(device).stream()).has_value(); });
  m.def("spmm", &spmm);
  m.def("sage", &sage);
  m.def("spmm_transposed", &spmm_transposed);
  m.def("transpose", [](const Tensor &ptr, const Tensor &idx, int64_t n, int64_t n_src, bool want_eid) {
    const Transposed t = transpose(ptr, idx, n, n_src, want_eid);
    return std::make_tuple(t.t_ptr, t.t_idx, want_eid ? optional<Tensor>(t.t_eid) : c10::nullopt, t.inv_deg);
  });
  m.def("transposed_graph", [](const Tensor &ptr, const Tensor &idx, int64_t n, int64_t n_src) {
    const Transposed t = transposed_graph(ptr, idx, n, n_src);
    return std::make_tuple(t.t_ptr, t.t_idx, t.t_eid, t.inv_deg);
  });
  m.def("forget_graphs", &forget_graphs);
  m.def("count_graphs", &count_graphs);
  m.def("gather_rows", &gather_rows);
  m.def("linear", &linear);
  m.def("gat_layer", &gat_layer);
  m.def("gat_layer_padded", &gat_layer_padded);
  m.def("sage_layer", &sage_layer);
  m.def("head_mean_bias", [](const Tensor &x, const optional<Tensor> &bias, int64_t heads, int64_t c) {
    f32(x, "x");
    c10::cuda::CUDAGuard guard(x.device());
    return head_mean_bias(x, bias, heads, c);
  });
  m.def("relation_pairs", &relation_pairs);
  m.def("sample_batch_fits", &sample_batch_fits);
  m.def("sample_batch", &sample_batch);
}
