// Host path between PyTorch and the C ABI (include/torchgt_b200.h): what the binding's translation units share.
// The Python modules keep their interfaces; argument checks, allocation, autograd bookkeeping and launches of the
// hot calls run here, because a small call is bound by exactly that: one attention forward + backward on 4,097
// rows and 45,056 edges took 132 us per call issued from Python through ctypes and takes 77 us from here (its
// kernels: 49 us).
#pragma once

#include <ATen/ATen.h>
#include <cuda_runtime_api.h>
#include <pybind11/pybind11.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/autograd/variable.h>

#include <atomic>
#include <cstdint>
#include <memory>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/torchgt_b200.h"

namespace tgt_host {

// A C-ABI call returned a non-zero code; Python sees torchgt_b200._cabi.TgtError.
struct TgtFailure : std::exception {
  int code;
  std::string message;
  TgtFailure(int c, std::string m) : code(c), message(std::move(m)) {}
  const char* what() const noexcept override { return message.c_str(); }
};

inline void check(int code) {
  if (code != TGT_OK) throw TgtFailure(code, tgt_last_error());
}

void set_python_error(const TgtFailure& e);                   // with the interpreter lock
[[noreturn]] void throw_python_error(const TgtFailure& e);    // without

// What a backward node runs in: an exception leaves it through PyTorch's engine, which hands on Python's exceptions as
// they are and makes a plain RuntimeError of anything else.
template <class F>
auto reporting(F&& f) -> decltype(f()) {
  try {
    return f();
  } catch (const TgtFailure& e) {
    throw_python_error(e);
  }
}

// Every entry that allocates, launches, waits or takes a mutex others allocate under runs without the interpreter lock: other Python threads
// (loaders, a prefetch) go on, and a thread that holds one of the mutexes never waits for one that holds the interpreter.
using Unlocked = pybind11::call_guard<pybind11::gil_scoped_release>;

void* stream_of(const at::Tensor& t);   // the current stream of t's device

inline void* ptr(const at::Tensor& t) { return t.defined() && t.numel() > 0 ? t.data_ptr() : nullptr; }
inline float* fptr(const at::Tensor& t) { return static_cast<float*>(ptr(t)); }

// One orientation of a graph (see torchgt_b200.graph.EdgeLayout).  The build enqueues kernels and does not wait;
// the result of its range check arrives in a pinned word behind an event.
class Layout {
 public:
  // What the build of one orientation of an int64 list keeps for the other's: both endpoints in 32 bits, checked
  // (tgt_edge_layout_build_keep), until that one is built or its graph goes.
  struct Kept {
    at::Tensor endpoints, bad_index;
    void* stream = nullptr;
  };
  Layout(const at::Tensor& edge_index, int64_t n_rows, int group_by, Kept* kept = nullptr);
  ~Layout();
  Layout(const Layout&) = delete;
  Layout& operator=(const Layout&) = delete;

  void poll();     // throws if the build is known to have seen a bad node id; never waits
  void verify();   // waits for the build first
  bool verified() const { return state_ == kGood; }

  tgt_layout c{};
  at::Tensor ptr, other, perm, seg, bad_index;
  int group_by;

 private:
  enum State { kPending, kGood, kBad };
  void settle(bool bad);
  bool settled() const;   // throws if the build saw a bad id
  std::mutex mutex_;      // of the two below: calls come from Python's threads and from autograd's
  std::atomic<State> state_{kPending};
  int slot_ = -1;   // pinned word and event of a pending check (-1: none, the device word is read instead)
};

// Both orientations of one batch graph; by_src is built on first use.
class Graph {
 public:
  Graph(const at::Tensor& edge_index, int64_t n_rows);
  std::shared_ptr<Layout> by_dst() const { return by_dst_; }
  std::shared_ptr<Layout> by_src();
  bool has_by_src() const { return built_ != nullptr; }
  void poll();
  // bytes of scratch the attention kernels need (asked from the library once per shape and phase)
  size_t scratch_bytes(int heads, int head_dim, int dtype, int phase);
  int64_t n_rows, n_edges;

 private:
  std::mutex mutex_;
  at::Tensor edge_index_;   // until by_src is built, as is what its build can use
  Layout::Kept kept_;
  std::shared_ptr<Layout> by_dst_, by_src_;
  std::atomic<Layout*> built_{nullptr};   // by_src_ once it is there, for whoever must not wait for its construction
  struct Need { int heads, head_dim, dtype, phase; size_t bytes; };
  std::vector<Need> needs_;
};

// z is the forward's sum of weights; forward on contiguous CUDA tensors, no autograd
void attention_forward(Graph& g, const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor& bias,
                       const at::Tensor& out, const at::Tensor& z, int heads, int head_dim, int dtype);
void attention_backward(Graph& g, const at::Tensor& dout, const at::Tensor& q, const at::Tensor& k, const at::Tensor& v,
                        const at::Tensor& bias, const at::Tensor& out, const at::Tensor& z, const at::Tensor& dq,
                        const at::Tensor& dk, const at::Tensor& dv, const at::Tensor& dbias, int heads, int head_dim,
                        int dtype);

// The attention as one autograd node: q, k and v of any one shape that is graph->n_rows rows of heads * head_dim values (a
// ValueError otherwise)
at::Tensor attention_over_rows(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor& bias,
                               const std::shared_ptr<Graph>& graph, int heads, int head_dim);

void bind_batching(pybind11::module_& m);   // binding_batch.cpp
void bind_dense(pybind11::module_& m);      // binding_dense.cpp

}  // namespace tgt_host
