// Batch construction for device tensors (csrc/batching.cu): allocations, the one wait each result's size needs, and
// the launches.
#include "binding.h"

#include <ATen/TensorSubclassLikeUtils.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/utils/pybind.h>

namespace tgt_host {
namespace {

const int64_t* ids(const at::Tensor& t) { return static_cast<const int64_t*>(ptr(t)); }

at::Tensor bytes_like(const at::Tensor& t, size_t n) {
  return at::empty({int64_t(n < 16 ? 16 : n)}, t.options().dtype(at::kByte));
}

// The first `n` result words of a pass, on the host (waits for the pass).
struct Words { int64_t v[4]; };
Words read_back(const int64_t* device, int n, const at::Tensor& like) {
  // from PyTorch's pool of pinned memory: nothing is pinned per call, nor kept by a thread that has ended
  const at::Tensor host = at::empty({4}, at::TensorOptions().dtype(at::kLong).pinned_memory(true));
  const int64_t* pinned = host.const_data_ptr<int64_t>();
  const auto stream = static_cast<cudaStream_t>(stream_of(like));
  cudaError_t e = cudaMemcpyAsync(host.data_ptr(), device, size_t(n) * 8, cudaMemcpyDeviceToHost, stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
  if (e != cudaSuccess) throw TgtFailure(TGT_ERR_CUDA, cudaGetErrorString(e));
  Words w{};
  for (int i = 0; i < n; ++i) w.v[i] = pinned[i];
  return w;
}

void bad_id(int64_t n) { throw pybind11::index_error("a node id is outside [0, " + std::to_string(n) + ")"); }

at::Tensor gather_rows(const at::Tensor& x, const at::Tensor& idx) {
  std::vector<int64_t> shape = x.sizes().vec();
  shape[0] = idx.numel();
  at::Tensor out = at::empty(shape, x.options());
  const int64_t row_bytes = x.size(0) > 0 ? int64_t(x.nbytes()) / x.size(0) : int64_t(x.element_size());
  if (out.numel() > 0)
    check(tgt_gather_rows(ptr(x), x.size(0), row_bytes, ids(idx), idx.numel(), ptr(out), stream_of(x)));
  return out;
}

// Rows `rows` (positions in idx) of every tensor of `xs`, and the batch's edges: {x[idx[lo:hi]]..., edges}.  The
// gathers are enqueued before the wait for the number of edges, so the GPU works meanwhile.
std::vector<at::Tensor> batch(const at::Tensor& edge_index, const at::Tensor& idx, int64_t n_nodes, bool add_token,
                              int64_t sub_seq_len, const std::vector<at::Tensor>& xs, int64_t lo, int64_t hi) {
  const c10::cuda::CUDAGuard guard(edge_index.device());
  const int64_t n_edges = edge_index.size(1), n_idx = idx.numel();
  size_t need = 0;
  check(tgt_subgraph_workspace_bytes(n_edges, n_nodes, &need));
  at::Tensor ws = bytes_like(edge_index, need);
  const int64_t* result = nullptr;
  check(tgt_subgraph_count(ids(edge_index), n_edges, n_nodes, ids(idx), n_idx, ws.data_ptr(), ws.numel(), &result,
                           stream_of(edge_index)));
  std::vector<at::Tensor> out;
  const at::Tensor mine = hi > lo || !xs.empty() ? idx.slice(0, lo, hi) : idx;
  for (const at::Tensor& x : xs) out.push_back(gather_rows(x, mine));
  const Words w = read_back(result, 2, edge_index);
  if (w.v[1] != 0) bad_id(n_nodes);
  const int64_t total = w.v[0] + (add_token ? 2 * n_idx : 0);
  at::Tensor edges = at::empty({2, total}, edge_index.options());
  check(tgt_subgraph_write(n_edges, n_nodes, n_idx, add_token, sub_seq_len, ws.data_ptr(),
                           static_cast<int64_t*>(ptr(edges)), total, stream_of(edge_index)));
  out.push_back(edges);
  return out;
}

// The block generator's edges, or None where the numpy formulation has to answer: some pair of partitions keeps its
// original edges, an id lies outside the nodes or the partitions (it counts from the end, has no edges, or is an
// error), or there are 2^31 blocks.
std::optional<at::Tensor> blocks(const at::Tensor& edge_index, int64_t n_nodes, const std::optional<at::Tensor>& partition,
                                 int k, double p, int64_t block, bool by_source, int64_t sub_seq_len) {
  const c10::cuda::CUDAGuard guard(edge_index.device());
  size_t need = 0;
  check(tgt_blocks_workspace_bytes(k, n_nodes, block, &need));
  at::Tensor ws = bytes_like(edge_index, need);
  const int64_t* result = nullptr;
  check(tgt_blocks_plan(ids(edge_index), edge_index.size(1), n_nodes, partition.has_value() ? ids(*partition) : nullptr, k,
                        p, block, ws.data_ptr(), ws.numel(), &result, stream_of(edge_index)));
  const Words w = read_back(result, 4, edge_index);
  if (w.v[2] != 0 || w.v[3] != 0 || w.v[0] >= (int64_t(1) << 31) - 1) return std::nullopt;
  at::Tensor out = at::empty({2, w.v[0] * block * block}, edge_index.options());
  check(tgt_blocks_list_bytes(w.v[0], &need));
  at::Tensor list = bytes_like(edge_index, need);
  check(tgt_blocks_write(n_nodes, k, block, ws.data_ptr(), list.data_ptr(), list.numel(), w.v[0], by_source, sub_seq_len,
                         static_cast<int64_t*>(ptr(out)), stream_of(edge_index)));
  return out;
}

}  // namespace

// strided tensors whose memory is theirs to read: no wrapper of a transform, no dispatch mode above, no pending
// conjugation or negation
bool plain(const std::vector<at::Tensor>& tensors) {
  for (const at::Tensor& t : tensors)
    if (at::isTensorSubclassLike(t) || t.layout() != at::kStrided || t.is_conj() || t.is_neg()) return false;
  return true;
}

void bind_batching(pybind11::module_& m) {
  m.def("plain", &plain);
  m.def("batch", &batch, Unlocked());
  m.def("blocks", &blocks, Unlocked());
  m.def("gather_rows", [](const at::Tensor& x, const at::Tensor& idx) {
    const c10::cuda::CUDAGuard guard(x.device());
    return gather_rows(x, idx);
  }, Unlocked());
}

}  // namespace tgt_host
