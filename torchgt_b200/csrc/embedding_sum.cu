// Sum of the embedding vectors of every node's integer features (models/gt_dist_graph_level.py:345,
// models/graphormer_dist_graph_level.py:60: embedding(x).sum(dim=-2) over padded batches of 10,000s of nodes) and its
// gradient with respect to the table.
//
// Forward: one pass, the vectors are read from the table (1.8 MB for 7,000 ids: L2) and only their sum is written; the
// gathered [rows, features, hidden] tensor, 410 MB for 320,000 rows of five features, never exists.
// Backward: every (row, feature) pair is an edge from the row's gradient to the table row it looked up, so the gradient is
// the attention's segmented reduction (attn_common.cuh) with nothing but the sum, over the same layout: no atomics, fixed
// order, hub ids (padding) cost the same per pair as any other.
#include "attn_common.cuh"

#include <assert.h>

namespace tgt {
namespace {

constexpr int kEmbThreads = 256;

__global__ void __launch_bounds__(kEmbThreads) embedding_sum_kernel(const float* __restrict__ table, int64_t n_table, int quads,
                                                                    const int64_t* __restrict__ ids, int64_t rows,
                                                                    int features, float* __restrict__ out) {
  const int64_t pieces = rows * quads;
  for (int64_t u = blockIdx.x * int64_t(kEmbThreads) + threadIdx.x; u < pieces; u += int64_t(gridDim.x) * kEmbThreads) {
    const int64_t row = u / quads;
    const int q = int(u - row * quads);
    const int64_t* id = ids + row * features;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 5
    for (int f = 0; f < features; ++f) {
      const int64_t i = __ldg(id + f);
      const bool known = i >= 0 && i < n_table;
      assert(known && "an id outside the embedding table");      // as torch.nn.Embedding on a GPU
      if (!known) continue;
      const float4 v = __ldg(reinterpret_cast<const float4*>(table) + i * quads + q);
      s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
    reinterpret_cast<float4*>(out)[u] = s;
  }
}

// The pairs as an edge list into the rows of the table.  Their other endpoint is the pair's position divided by `features`;
// the list has 0 in its place, for a layout takes endpoints of one range only.
__global__ void __launch_bounds__(kEmbThreads) embedding_pairs_kernel(const int64_t* __restrict__ ids, unsigned pairs,
                                                                      int64_t n_table, int32_t* __restrict__ edges) {
  for (unsigned i = blockIdx.x * kEmbThreads + threadIdx.x; i < pairs; i += gridDim.x * kEmbThreads) {
    const int64_t id = __ldg(ids + i);
    edges[i] = 0;
    edges[pairs + i] = id >= 0 && id < n_table ? int32_t(id) : 0;
  }
}

template <int G>
struct SumPolicy {
  static constexpr int VEC = 4, NACC = 4;
  static constexpr bool kPerm = true;
  static constexpr int kUnroll = 4;
  const float* __restrict__ grad;
  float* __restrict__ out;
  int skip;                    // a table row whose gradient is zero, or -1
  unsigned features, share;    // share = 2^32 / features, rounded up
  unsigned column;
  struct Operands {
    float4 v;
  };
  struct Scalars {};
  __device__ __forceinline__ void load(Operands& o, int, int, int pair) const {
    unsigned row = features > 1 ? __umulhi(unsigned(pair), share) : unsigned(pair);   // pair / features, or one more
    if (row * features > unsigned(pair)) --row;
    o.v = __ldg(reinterpret_cast<const float4*>(grad) + (row * G + column));
  }
  __device__ __forceinline__ void clear(Operands& o) const { o.v = make_float4(0.f, 0.f, 0.f, 0.f); }
  __device__ __forceinline__ Scalars prep(const Operands&, bool, int) const { return {}; }
  __device__ __forceinline__ void accumulate(float (&acc)[NACC], const Operands& o, const Scalars&) const {
    acc[0] += o.v.x; acc[1] += o.v.y; acc[2] += o.v.z; acc[3] += o.v.w;
  }
  __device__ __forceinline__ void finalize(int row, const float (&acc)[NACC]) const {
    reinterpret_cast<float4*>(out)[unsigned(row) * G + column] =
        row == skip ? make_float4(0.f, 0.f, 0.f, 0.f) : make_float4(acc[0], acc[1], acc[2], acc[3]);
  }
  __device__ __forceinline__ void zero_row(int row) const {
    reinterpret_cast<float4*>(out)[unsigned(row) * G + column] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
};

struct SumParams {
  const float* grad;
  float* out;
  int skip;
  unsigned features, share;
  SegWalk walk;
};

template <int G>
__global__ void TGT_WALK_BOUNDS embedding_grad_kernel(const SumParams p) {
  __shared__ TileSmem<G, SumPolicy<G>::NACC, true> sm;
  const SumPolicy<G> pol{p.grad, p.out, p.skip, p.features, p.share, threadIdx.x % G};
  walk_tile_in<G, SumPolicy<G>>(sm, p.walk, pol);
}

template <int G>
__global__ void __launch_bounds__(crossing_threads(G)) embedding_grad_crossing_kernel(const SumParams p) {
  const SumPolicy<G> pol{p.grad, p.out, p.skip, p.features, p.share, threadIdx.x % G};
  finish_crossing_rows<G, SumPolicy<G>>(p.walk, pol);
}

template <int G>
int launch_grad(const SumParams& p, unsigned ctas, cudaStream_t stream) {
  embedding_grad_kernel<G><<<ctas, kBlockThreads, 0, stream>>>(p);
  if (p.walk.n_tiles > 1)
    TGT_CHECK_CUDA(launch_chained(embedding_grad_crossing_kernel<G>, dim3(crossing_ctas(p.walk, G)), crossing_threads(G), stream,
                                  kLinkStitch, p));
  TGT_CHECK_CUDA(cudaGetLastError());
  return TGT_OK;
}

bool table_supported(int hidden) { return hidden == 32 || hidden == 64 || hidden == 128; }

struct GradPlan {
  HeadSplit hs;
  TilePlan tiles;
  size_t edges, ptr, other, perm, seg, status, layout, layout_bytes, walk, total;
};

template <int G>
int grad_ctas() {
  static int cache[kMaxDevices] = {};
  const int dev = current_device();
  return resident_ctas(embedding_grad_kernel<G>, &cache[dev < 0 ? 0 : dev]);
}

int plan_grad(int64_t pairs, int64_t n_table, int hidden, GradPlan* g) {
  if (!split_heads(1, hidden, TGT_F32, 16, &g->hs)) return set_error(TGT_ERR_UNSUPPORTED, "hidden=%d", hidden);
  const int ctas = hidden == 32 ? grad_ctas<8>() : hidden == 64 ? grad_ctas<16>() : grad_ctas<32>();
  g->tiles = plan_tiles(pairs, g->hs, SumPolicy<16>::kUnroll, 4, ctas);
  const int rc = tgt_edge_layout_sizes_i32(n_table, pairs, &g->layout_bytes);
  if (rc != TGT_OK) return rc;
  size_t off = 0;
  auto take = [&off](size_t bytes) {
    const size_t at = off;
    off += round_up(bytes, 256);
    return at;
  };
  g->edges = take(size_t(pairs) * 8);
  g->ptr = take(size_t(n_table + 1) * 4);
  g->other = take(size_t(pairs) * 4);
  g->perm = take(size_t(pairs) * 4);
  g->seg = take(size_t(pairs) * 4);
  g->status = take(4);
  g->layout = take(g->layout_bytes);
  g->walk = take(g->tiles.carry_bytes);
  g->total = off;
  return TGT_OK;
}

int check_table(int64_t n_table, int hidden, int64_t rows, int features) {
  TGT_CHECK_ARG(n_table >= 1 && rows >= 0 && features >= 1, "n_table and features must be >= 1, rows >= 0");
  if (!table_supported(hidden)) return set_error(TGT_ERR_UNSUPPORTED, "hidden=%d: 32, 64 or 128", hidden);
  if (n_table >= (int64_t(1) << 26) || rows >= (int64_t(1) << 26) || features > 1024 ||
      rows * features >= (int64_t(1) << 31) - 1)
    return set_error(TGT_ERR_UNSUPPORTED, "tables and batches from 2^26 rows or 2^31 pairs on are not covered");
  return TGT_OK;
}

}  // namespace
}  // namespace tgt

extern "C" int tgt_embedding_sum(const float* table, int64_t n_table, int hidden, const int64_t* ids, int64_t rows,
                                 int features, float* out, void* stream_) {
  using namespace tgt;
  const int rc = check_table(n_table, hidden, rows, features);
  if (rc != TGT_OK) return rc;
  if (rows == 0) return TGT_OK;
  TGT_CHECK_ARG(table && ids && out, "table, ids and out must not be null");
  TGT_CHECK_ARG(aligned16(table) && aligned16(out), "table and out must be 16-byte aligned");
  const int64_t blocks = (rows * (hidden / 4) + kEmbThreads - 1) / kEmbThreads, most = int64_t(sm_count()) * 32;
  embedding_sum_kernel<<<unsigned(blocks < most ? blocks : most), kEmbThreads, 0, static_cast<cudaStream_t>(stream_)>>>(
      table, n_table, hidden / 4, ids, rows, features, out);
  TGT_CHECK_CUDA(cudaGetLastError());
  return TGT_OK;
}

extern "C" int tgt_embedding_sum_grad_scratch_bytes(int64_t n_table, int hidden, int64_t rows, int features, size_t* bytes) {
  using namespace tgt;
  TGT_CHECK_ARG(bytes != nullptr, "bytes is null");
  int rc = check_table(n_table, hidden, rows, features);
  if (rc != TGT_OK) return rc;
  GradPlan g;
  rc = plan_grad(rows * features, n_table, hidden, &g);
  if (rc == TGT_OK) *bytes = g.total;
  return rc;
}

extern "C" int tgt_embedding_sum_grad(const float* dout, const int64_t* ids, int64_t rows, int features, int64_t n_table,
                                      int hidden, int64_t padding_idx, float* dtable, void* scratch, size_t scratch_bytes,
                                      void* stream_) {
  using namespace tgt;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  int rc = check_table(n_table, hidden, rows, features);
  if (rc != TGT_OK) return rc;
  TGT_CHECK_ARG(dtable && aligned16(dtable), "dtable must not be null and 16-byte aligned");
  if (rows == 0) {
    TGT_CHECK_CUDA(cudaMemsetAsync(dtable, 0, size_t(n_table) * hidden * sizeof(float), stream));
    return TGT_OK;
  }
  TGT_CHECK_ARG(dout && ids, "dout and ids must not be null");
  TGT_CHECK_ARG(aligned16(dout) && aligned16(scratch), "dout and scratch must be 16-byte aligned");
  const int64_t pairs = rows * features;
  GradPlan g;
  rc = plan_grad(pairs, n_table, hidden, &g);
  if (rc != TGT_OK) return rc;
  if (scratch == nullptr || scratch_bytes < g.total)
    return set_error(TGT_ERR_WORKSPACE, "scratch holds %zu bytes, %zu needed", scratch_bytes, g.total);
  char* const base = static_cast<char*>(scratch);
  auto words = [base](size_t at) { return reinterpret_cast<int32_t*>(base + at); };
  const int64_t blocks = (pairs + kEmbThreads - 1) / kEmbThreads, most = int64_t(sm_count()) * 16;
  embedding_pairs_kernel<<<unsigned(blocks < most ? blocks : most), kEmbThreads, 0, stream>>>(
      ids, unsigned(pairs), n_table, words(g.edges));
  TGT_CHECK_CUDA(cudaGetLastError());
  rc = tgt_edge_layout_build_i32(words(g.edges), pairs, n_table, 1, words(g.ptr), words(g.other), words(g.perm), words(g.seg),
                                 base + g.layout, g.layout_bytes, words(g.status), stream_);
  if (rc != TGT_OK) return rc;
  SumParams p;
  p.grad = dout;
  p.out = dtable;
  p.skip = padding_idx >= 0 && padding_idx < n_table ? int(padding_idx) : -1;
  p.features = unsigned(features);
  p.share = unsigned(((uint64_t(1) << 32) + p.features - 1) / p.features);     // features == 1 is not multiplied
  p.walk.ptr = words(g.ptr); p.walk.other = words(g.other); p.walk.perm = words(g.perm); p.walk.seg = words(g.seg);
  p.walk.n_rows = int(n_table); p.walk.n_edges = int(pairs);
  p.walk.ge = g.tiles.ge; p.walk.n_tiles = g.tiles.n_tiles; p.walk.gap_ctas = gap_ctas(n_table);
  p.walk.gcarry = reinterpret_cast<float*>(base + g.walk);
  const unsigned ctas = walk_ctas(g.tiles, n_table);
  return hidden == 32 ? launch_grad<8>(p, ctas, stream) : hidden == 64 ? launch_grad<16>(p, ctas, stream) : launch_grad<32>(p, ctas, stream);
}
