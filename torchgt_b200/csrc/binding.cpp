// Python module torchgt_b200._native: edge layouts and the autograd node of the sparse attention.
#include "binding.h"

#include <ATen/cuda/CUDAContext.h>
#include <ATen/core/LegacyTypeDispatch.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <pybind11/stl.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/csrc/utils/pybind.h>

#include <sstream>

namespace py = pybind11;

namespace tgt_host {

namespace {
// torchgt_b200._cabi.TgtError; kept for the life of the process
PyObject* tgt_error(const TgtFailure& e, PyObject** type) {
  static py::object* error = new py::object(py::module_::import("torchgt_b200._cabi").attr("TgtError"));
  *type = error->ptr();
  return (*error)(e.code, e.message).release().ptr();
}
}  // namespace

void set_python_error(const TgtFailure& e) {
  PyObject* type = nullptr;
  PyObject* value = tgt_error(e, &type);
  PyErr_SetObject(type, value);
  Py_DECREF(value);
}

void throw_python_error(const TgtFailure& e) {
  const py::gil_scoped_acquire gil;
  set_python_error(e);
  python_error error;
  error.persist();
  throw error;
}

void* stream_of(const at::Tensor& t) { return at::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

namespace {

void check_cuda(cudaError_t e, const char* what) {
  if (e != cudaSuccess) throw TgtFailure(TGT_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

bool capturing(const at::Tensor& t) {
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  check_cuda(cudaStreamIsCapturing(static_cast<cudaStream_t>(stream_of(t)), &status), "cudaStreamIsCapturing");
  return status != cudaStreamCaptureStatusNone;
}

// Pinned words that receive the range-check results of layout builds, each with an event: at most kMost per
// process, allocated 64 at a time and handed out again once their copy has landed.  A layout that finds none free
// (a thousand builds outstanding) goes without and reads the device word when it is asked.
class CheckWords {
 public:
  struct Word { int32_t* host = nullptr; cudaEvent_t event = nullptr; int device = -1; };

  int take(int device) {
    std::lock_guard<std::mutex> lock(mutex_);
    for (size_t i = 0; i < returned_.size(); ++i) {
      const int slot = returned_[i];
      if (words_[slot].device == device && cudaEventQuery(words_[slot].event) == cudaSuccess) {
        returned_.erase(returned_.begin() + i);
        return slot;
      }
      if (i >= 3) break;        // the oldest ones are done first
    }
    cudaGetLastError();         // "not ready" is not an error
    if (fresh_ == 0) {
      if (words_.size() + kChunk > kMost) return -1;
      int32_t* p = nullptr;
      if (cudaHostAlloc(reinterpret_cast<void**>(&p), kChunk * sizeof(int32_t), cudaHostAllocPortable) != cudaSuccess) {
        cudaGetLastError();
        return -1;
      }
      for (int i = 0; i < kChunk; ++i) words_.push_back({p + i, nullptr, -1});
      fresh_ = kChunk;
    }
    const int slot = int(words_.size()) - fresh_;
    if (cudaEventCreateWithFlags(&words_[slot].event, cudaEventDisableTiming) != cudaSuccess) {
      cudaGetLastError();
      return -1;
    }
    words_[slot].device = device;
    --fresh_;
    return slot;
  }
  void give_back(int slot) {
    std::lock_guard<std::mutex> lock(mutex_);
    returned_.push_back(slot);
  }
  Word at(int slot) {
    std::lock_guard<std::mutex> lock(mutex_);
    return words_[slot];
  }

 private:
  static constexpr int kChunk = 64, kMost = 1024;
  std::mutex mutex_;
  std::vector<Word> words_;
  std::vector<int> returned_;
  int fresh_ = 0;
};

CheckWords& check_words() {
  static CheckWords* words = new CheckWords;   // outlives every layout, whatever the order of destruction
  return *words;
}

}  // namespace

// Edges from which on the first build of an int64 list keeps its endpoints for the second.  Shorter lists are bound by the host,
// which pays 3 us for the array (a list of 30,000 edges 104.9 -> 108.1 us), and save one or two.  They take the place of arrays of
// the build's workspace, but stay, 8 bytes per edge, until the second build or the graph's end: kept only where gradients are
// recorded, since nothing else asks for the second orientation.
constexpr int64_t kKeepFrom = int64_t(1) << 20;

// ---- layouts ------------------------------------------------------------------------------------------------
Layout::Layout(const at::Tensor& edge_index, int64_t n_rows, int group_by_, Kept* kept) : group_by(group_by_) {
  const c10::cuda::CUDAGuard guard(edge_index.device());
  const int64_t n_edges = edge_index.size(1);
  const bool wide = edge_index.scalar_type() == at::kLong, from_kept = kept != nullptr && kept->endpoints.defined();
  const bool keep = wide && kept != nullptr && !from_kept && n_edges >= kKeepFrom && at::GradMode::is_enabled() && !capturing(edge_index);
  size_t ws = 0;
  check((keep || from_kept ? tgt_edge_layout_sizes_kept : wide ? tgt_edge_layout_sizes : tgt_edge_layout_sizes_i32)(n_rows, n_edges, &ws));
  const auto i32 = edge_index.options().dtype(at::kInt);
  ptr = at::empty({n_rows + 1}, i32);
  other = at::empty({n_edges}, i32);
  perm = at::empty({n_edges}, i32);
  seg = at::empty({n_edges}, i32);
  bad_index = from_kept ? kept->bad_index : at::empty({1}, i32);
  at::Tensor workspace = at::empty({int64_t(ws < 16 ? 16 : ws)}, edge_index.options().dtype(at::kByte));
  auto words = [](const at::Tensor& t) { return static_cast<int32_t*>(tgt_host::ptr(t)); };
  const void* edges = tgt_host::ptr(edge_index);
  void* stream = stream_of(edge_index);
  if (from_kept) {
    check(tgt_edge_layout_build_kept(words(kept->endpoints), n_edges, n_rows, group_by, words(ptr), words(other), words(perm),
                                     words(seg), workspace.data_ptr(), workspace.numel(), stream));
  } else if (keep) {
    size_t kept_words = 0;
    check(tgt_edge_layout_kept_words(n_edges, &kept_words));
    at::Tensor endpoints = at::empty({int64_t(kept_words)}, i32);
    check(tgt_edge_layout_build_keep(static_cast<const int64_t*>(edges), n_edges, n_rows, group_by, words(ptr), words(other),
                                     words(perm), words(seg), workspace.data_ptr(), workspace.numel(), words(bad_index),
                                     words(endpoints), stream));
    kept->endpoints = std::move(endpoints);
    kept->bad_index = bad_index;
    kept->stream = stream;
  } else {
    check(wide ? tgt_edge_layout_build(static_cast<const int64_t*>(edges), n_edges, n_rows, group_by, words(ptr), words(other),
                                       words(perm), words(seg), workspace.data_ptr(), workspace.numel(), words(bad_index), stream)
               : tgt_edge_layout_build_i32(static_cast<const int32_t*>(edges), n_edges, n_rows, group_by, words(ptr),
                                           words(other), words(perm), words(seg), workspace.data_ptr(), workspace.numel(),
                                           words(bad_index), stream));
  }
  c.n_rows = n_rows;
  c.n_edges = n_edges;
  c.ptr = words(ptr);
  c.other = words(other);
  c.perm = words(perm);
  c.seg = words(seg);
  if (!capturing(edge_index)) {
    slot_ = check_words().take(edge_index.device().index());
    if (slot_ >= 0) {
      const auto w = check_words().at(slot_);
      cudaError_t e = cudaMemcpyAsync(w.host, bad_index.data_ptr(), 4, cudaMemcpyDeviceToHost,
                                      static_cast<cudaStream_t>(stream));
      if (e == cudaSuccess) e = cudaEventRecord(w.event, static_cast<cudaStream_t>(stream));
      if (e != cudaSuccess) check_words().give_back(slot_);   // no destructor runs after a throw
      check_cuda(e, "copy of the range check's result");
    }
  }
}

Layout::~Layout() {
  if (slot_ >= 0) check_words().give_back(slot_);
}

void Layout::settle(bool bad) {
  state_ = bad ? kBad : kGood;
  if (slot_ >= 0) {
    check_words().give_back(slot_);
    slot_ = -1;
  }
}

bool Layout::settled() const {
  if (state_ == kBad)
    throw TgtFailure(TGT_ERR_INDEX_RANGE, "edge_index holds a node id outside [0, " + std::to_string(c.n_rows) + ")");
  return state_ == kGood;
}

void Layout::poll() {
  if (state_.load(std::memory_order_acquire) == kGood) return;   // every call but a graph's first few
  std::lock_guard<std::mutex> lock(mutex_);
  if (settled() || slot_ < 0 || capturing(ptr)) return;
  const auto w = check_words().at(slot_);
  const cudaError_t e = cudaEventQuery(w.event);
  if (e == cudaSuccess) {
    settle(*static_cast<volatile int32_t*>(w.host) != 0);
    settled();
    return;
  }
  if (e != cudaErrorNotReady) check_cuda(e, "cudaEventQuery");
  cudaGetLastError();
}

void Layout::verify() {
  int slot;
  {
    std::lock_guard<std::mutex> lock(mutex_);
    if (settled()) return;
    slot = slot_;
  }
  // waits without the lock; while the state is pending the word and its event belong to this layout, and whoever
  // settles it first is believed
  bool bad = false;
  CheckWords::Word w;
  if (slot < 0) {
    bad = bad_index.item<int32_t>() != 0;
  } else {
    w = check_words().at(slot);
    check_cuda(cudaEventSynchronize(w.event), "cudaEventSynchronize");
  }
  std::lock_guard<std::mutex> lock(mutex_);
  if (state_ == kPending) settle(slot < 0 ? bad : *static_cast<volatile int32_t*>(w.host) != 0);
  settled();
}

Graph::Graph(const at::Tensor& edge_index, int64_t rows)
    : n_rows(rows), n_edges(edge_index.size(1)), edge_index_(edge_index),
      by_dst_(std::make_shared<Layout>(edge_index, rows, 1, &kept_)) {}

std::shared_ptr<Layout> Graph::by_src() {
  at::Tensor done;   // outlives the lock: a tensor that Python has seen takes the interpreter lock on its way out
  std::lock_guard<std::mutex> lock(mutex_);
  if (!by_src_) {
    // what the first build kept is complete, and its memory safe, on the stream of that build only; in a capture it would
    // tie the graph's replays to an array that is given back here
    const bool usable = kept_.endpoints.defined() && kept_.stream == stream_of(edge_index_) && !capturing(edge_index_);
    by_src_ = std::make_shared<Layout>(edge_index_, n_rows, 0, usable ? &kept_ : nullptr);
    built_.store(by_src_.get(), std::memory_order_release);
    kept_ = {};
    done = std::move(edge_index_);
  }
  return by_src_;
}

void Graph::poll() {
  by_dst_->poll();
  if (Layout* by_src = built_.load(std::memory_order_acquire)) by_src->poll();
}

size_t Graph::scratch_bytes(int heads, int head_dim, int dtype, int phase) {
  {
    std::lock_guard<std::mutex> lock(mutex_);
    for (const Need& n : needs_)
      if (n.heads == heads && n.head_dim == head_dim && n.dtype == dtype && n.phase == phase) return n.bytes;
  }
  size_t bytes = 0;
  check(tgt_sparse_attn_scratch_bytes(&by_dst_->c, phase == 1 ? &by_src()->c : nullptr, heads, head_dim, dtype, phase,
                                      &bytes));
  bytes = bytes < 16 ? 16 : bytes;
  std::lock_guard<std::mutex> lock(mutex_);
  needs_.push_back({heads, head_dim, dtype, phase, bytes});
  return bytes;
}

// ---- attention ----------------------------------------------------------------------------------------------
namespace {

int bias_heads(const at::Tensor& bias) {
  return bias.defined() ? (bias.dim() == 1 ? 1 : int(bias.size(1))) : 0;
}

int dtype_of(const at::Tensor& q) { return q.scalar_type() == at::kFloat ? TGT_F32 : TGT_BF16; }

// The kernels take bare pointers to n_rows rows of heads * head_dim values of one type and to one or `heads` bias values per edge,
// and the gradients are laid out like q, k, v and the bias: whoever calls them, anything else stops here.
void check_rows(const Graph& g, const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor& bias, int heads,
                int head_dim) {
  if (q.sizes() != k.sizes() || q.sizes() != v.sizes() || q.numel() != g.n_rows * heads * head_dim) {
    std::ostringstream what;
    what << "q, k, v must share the shape [N, H, D], here " << g.n_rows << " rows of " << heads << " x " << head_dim << "; got "
         << q.sizes() << ", " << k.sizes() << ", " << v.sizes();
    throw py::value_error(what.str());
  }
  if ((q.scalar_type() != at::kFloat && q.scalar_type() != at::kBFloat16) || k.scalar_type() != q.scalar_type() ||
      v.scalar_type() != q.scalar_type())
    throw py::type_error("q, k, v must all be float32 or all bfloat16");
  if (bias.defined() && (bias.scalar_type() != at::kFloat || bias.dim() < 1 || bias.dim() > 2 || bias.size(0) != g.n_edges ||
                         (bias.dim() == 2 && bias.size(1) != heads))) {
    std::ostringstream what;
    what << "bias must be float32 [E] or [E, H] with E=" << g.n_edges << ", H=" << heads << "; got " << bias.sizes();
    throw py::value_error(what.str());
  }
}

at::Tensor scratch(Graph& g, int heads, int head_dim, int dtype, int phase, const at::Tensor& like) {
  return at::empty({int64_t(g.scratch_bytes(heads, head_dim, dtype, phase))}, like.options().dtype(at::kByte));
}

}  // namespace

void attention_forward(Graph& g, const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor& bias,
                       const at::Tensor& out, const at::Tensor& z, int heads, int head_dim, int dtype) {
  at::Tensor tmp = scratch(g, heads, head_dim, dtype, 0, q);
  check(tgt_sparse_attn_fwd(ptr(q), ptr(k), ptr(v), fptr(bias), bias_heads(bias), &g.by_dst()->c, ptr(out), fptr(z),
                            heads, head_dim, dtype, tmp.data_ptr(), tmp.numel(), stream_of(q)));
}

void attention_backward(Graph& g, const at::Tensor& dout, const at::Tensor& q, const at::Tensor& k, const at::Tensor& v,
                        const at::Tensor& bias, const at::Tensor& out, const at::Tensor& z, const at::Tensor& dq,
                        const at::Tensor& dk, const at::Tensor& dv, const at::Tensor& dbias, int heads, int head_dim,
                        int dtype) {
  at::Tensor tmp = scratch(g, heads, head_dim, dtype, 1, q);
  check(tgt_sparse_attn_bwd(ptr(dout), ptr(q), ptr(k), ptr(v), fptr(bias), bias_heads(bias), ptr(out), fptr(z),
                            &g.by_dst()->c, &g.by_src()->c, ptr(dq), ptr(dk), ptr(dv), fptr(dbias), heads, head_dim,
                            dtype, tmp.data_ptr(), tmp.numel(), stream_of(q)));
}

namespace {

using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

struct SparseGraphAttentionBackward : public torch::autograd::Node {
  std::shared_ptr<Graph> graph;
  SavedVariable q, k, v, bias, out, z;
  int heads = 0, head_dim = 0, dtype = 0;
  bool with_dbias = false;
  bool reads_out() const { return with_dbias && dtype == TGT_F32; }   // tgt_sparse_attn_bwd: the output is kept only then

  variable_list apply(variable_list&& grads) override {
    return reporting([&] { return backward(grads); });
  }
  variable_list backward(const variable_list& grads) {
    if (!grads[0].defined()) return variable_list(4);
    const at::Tensor q_ = q.unpack(), k_ = k.unpack(), v_ = v.unpack(), bias_ = bias.unpack(), z_ = z.unpack();
    const bool want_dbias = with_dbias && task_should_compute_output(3);
    const at::Tensor out_ = want_dbias && reads_out() ? out.unpack(shared_from_this()) : at::Tensor();
    const at::AutoDispatchBelowADInplaceOrView below;
    const c10::cuda::CUDAGuard guard(q_.device());
    const at::Tensor dout = grads[0].contiguous();
    at::Tensor dq = at::empty_like(q_), dk = at::empty_like(k_), dv = at::empty_like(v_), dbias;
    if (want_dbias) dbias = at::empty_like(bias_);
    attention_backward(*graph, dout, q_, k_, v_, bias_, out_, z_, dq, dk, dv, dbias, heads, head_dim, dtype);
    return {dq, dk, dv, dbias};
  }
  std::string name() const override { return "SparseGraphAttentionBackward"; }
  void release_variables() override {
    q.reset_data(); k.reset_data(); v.reset_data(); bias.reset_data(); out.reset_data();
    z.reset_data();
  }
};

}  // namespace

at::Tensor attention_over_rows(const at::Tensor& q_in, const at::Tensor& k_in, const at::Tensor& v_in, const at::Tensor& bias,
                               const std::shared_ptr<Graph>& graph, int heads, int head_dim) {
  // the node has no forward-mode formula: refuse a dual tensor rather than drop its tangent
  for (const at::Tensor* t : {&q_in, &k_in, &v_in, &bias})
    TORCH_CHECK_NOT_IMPLEMENTED(!torch::autograd::isFwGradDefined(*t),
                                "sparse_graph_attention does not support forward-mode AD");
  check_rows(*graph, q_in, k_in, v_in, bias, heads, head_dim);
  const at::Tensor q = q_in.contiguous(), k = k_in.contiguous(), v = v_in.contiguous();
  const int dtype = dtype_of(q);
  const c10::cuda::CUDAGuard guard(q.device());
  at::Tensor out, z;
  {
    const at::AutoDispatchBelowADInplaceOrView below;
    out = at::empty_like(q);
    z = at::empty({graph->n_rows, heads}, q.options().dtype(at::kFloat));
    attention_forward(*graph, q, k, v, bias, out, z, heads, head_dim, dtype);
  }
  if (torch::autograd::compute_requires_grad(q, k, v, bias)) {
    auto node = std::shared_ptr<SparseGraphAttentionBackward>(new SparseGraphAttentionBackward(),
                                                             torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(q, k, v, bias));
    node->graph = graph;
    node->heads = heads;
    node->head_dim = head_dim;
    node->dtype = dtype;
    node->with_dbias = bias.defined() && bias.requires_grad();
    node->q = SavedVariable(q, false);
    node->k = SavedVariable(k, false);
    node->v = SavedVariable(v, false);
    node->bias = SavedVariable(bias, false);
    node->z = SavedVariable(z, false);
    torch::autograd::set_history(out, node);
    if (node->reads_out()) node->out = SavedVariable(out, true);
  }
  return out;
}

namespace {

at::Tensor attention(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const std::optional<at::Tensor>& bias,
                     const std::shared_ptr<Graph>& graph) {
  return attention_over_rows(q, k, v, bias.value_or(at::Tensor()), graph, int(q.size(1)), int(q.size(2)));
}

// The plain call of sparse_graph_attention: no bias, a prebuilt graph, nobody tracing.  Nothing where any of its checks is
// not clearly met: the caller goes through them one by one and words the errors.
std::optional<at::Tensor> plain_attention(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v,
                                          const std::shared_ptr<Graph>& graph) {
  const bool plain = q.is_cuda() && k.is_cuda() && v.is_cuda() && q.dim() == 3 && q.sizes() == k.sizes() && q.sizes() == v.sizes() &&
                     (q.scalar_type() == at::kFloat || q.scalar_type() == at::kBFloat16) && k.scalar_type() == q.scalar_type() &&
                     v.scalar_type() == q.scalar_type() && q.size(0) == graph->n_rows && !torch::jit::tracer::isTracing();
  if (!plain) return std::nullopt;
  graph->poll();
  return attention_over_rows(q, k, v, at::Tensor(), graph, int(q.size(1)), int(q.size(2)));
}

// The two passes without an autograd node, for callers that keep one of their own (torchgt_b200/sparse_attn.py).
std::pair<at::Tensor, at::Tensor> forward_pass(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v,
                                               const std::optional<at::Tensor>& bias, const std::shared_ptr<Graph>& graph) {
  const c10::cuda::CUDAGuard guard(q.device());
  const int heads = int(q.size(1)), head_dim = int(q.size(2));
  const at::Tensor bias_ = bias.value_or(at::Tensor());
  check_rows(*graph, q, k, v, bias_, heads, head_dim);
  at::Tensor out = at::empty_like(q), z = at::empty({q.size(0), heads}, q.options().dtype(at::kFloat));
  attention_forward(*graph, q, k, v, bias_, out, z, heads, head_dim, dtype_of(q));
  return {out, z};
}

std::vector<std::optional<at::Tensor>> backward_pass(const at::Tensor& dout, const at::Tensor& q, const at::Tensor& k,
                                                     const at::Tensor& v, const std::optional<at::Tensor>& bias,
                                                     const std::optional<at::Tensor>& out, const at::Tensor& z,
                                                     const std::shared_ptr<Graph>& graph, bool want_dbias) {
  const c10::cuda::CUDAGuard guard(q.device());
  const at::Tensor bias_ = bias.value_or(at::Tensor());
  at::Tensor dq = at::empty_like(q), dk = at::empty_like(k), dv = at::empty_like(v), dbias;
  if (want_dbias) dbias = at::empty_like(bias_);
  attention_backward(*graph, dout.contiguous(), q, k, v, bias_, out.value_or(at::Tensor()), z, dq, dk, dv, dbias, int(q.size(1)),
                     int(q.size(2)), dtype_of(q));
  return {dq, dk, dv, want_dbias ? std::optional<at::Tensor>(dbias) : std::nullopt};
}

// into[i] <- of[i] in one multi-tensor copy.  The caller drops the sources right away, so their memory, which may belong
// to another stream, is marked as in use on this one (for memory of this stream that is a comparison).
void take_gradients(const std::vector<at::Tensor>& into, const std::vector<at::Tensor>& of) {
  const at::NoGradGuard no_grad;
  at::_foreach_copy_(into, of);
  for (const at::Tensor& t : of)
    if (t.is_cuda())
      c10::cuda::CUDACachingAllocator::recordStream(t.storage().data_ptr(),
                                                    at::cuda::getCurrentCUDAStream(t.device().index()));
}

}  // namespace
}  // namespace tgt_host

PYBIND11_MODULE(_native, m) {
  using namespace tgt_host;
  py::register_exception_translator([](std::exception_ptr p) {
    try {
      if (p) std::rethrow_exception(p);
    } catch (const TgtFailure& e) {
      set_python_error(e);
    }
  });
  py::class_<Layout, std::shared_ptr<Layout>>(m, "Layout")
      .def(py::init([](const at::Tensor& edges, int64_t rows, int group_by) {
             return std::make_shared<Layout>(edges, rows, group_by);
           }), Unlocked())
      .def("poll", &Layout::poll)   // waits for nothing, and nobody waits for the interpreter under its mutex
      .def("verify", &Layout::verify, Unlocked())
      .def_property_readonly("verified", &Layout::verified)
      .def_readonly("ptr", &Layout::ptr)
      .def_readonly("other", &Layout::other)
      .def_readonly("perm", &Layout::perm)
      .def_readonly("seg", &Layout::seg)
      .def_readonly("bad_index", &Layout::bad_index)
      .def_readonly("group_by", &Layout::group_by);
  py::class_<Graph, std::shared_ptr<Graph>>(m, "Graph")
      .def(py::init<const at::Tensor&, int64_t>(), Unlocked())
      .def("by_dst", &Graph::by_dst)
      .def("by_src", &Graph::by_src, Unlocked())
      .def("has_by_src", &Graph::has_by_src)
      .def("poll", &Graph::poll);
  m.def("take_gradients", &take_gradients, Unlocked());
  m.def("attention", &attention, Unlocked());
  m.def("plain_attention", &plain_attention, Unlocked());
  m.def("attention_forward", &forward_pass, Unlocked());
  m.def("attention_backward", &backward_pass, Unlocked());
  bind_batching(m);
  bind_dense(m);
}
