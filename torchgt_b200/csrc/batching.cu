// Batch construction of the node-level training loops on the device: the induced sub-graph of a batch
// (gt_sp/utils.py:202-215), its global-token and per-rank renumbering (gt_sp/utils.py:34-58), the cluster-sparse
// block generator (gt_sp/utils.py:218-359) and the gather of the batch's feature rows.  Integer work, bit for bit
// what the PyTorch / numpy formulation in gt_sp/batching.py gives (which host tensors still take).
//
// As single PyTorch operations a batch of 64,000 nodes of a graph with 1.17 M edges took 63 launches, four host
// synchronisations and 524 us with its layouts; the block generator sorted the edges on the host, drew the block
// coordinates in Python and uploaded 131 small pieces: 38.4 ms for 37,608 nodes.  They take 216 us and 285 us from
// here, two layout builds (about 90 us) included.  The sub-graph is two passes over
// the edge list with one synchronisation (the size of the result), and a block list is never sorted as edges: the
// generator's blocks are aligned to a grid, so sorting about a thousand BLOCKS by grid row sorts the edges by source.
#include "tgt_common.cuh"

namespace tgt {
namespace {

constexpr int kBatchThreads = 256;
constexpr int kChunk = 2048;   // candidate edges per CTA of the marking pass: eight per thread

inline unsigned blocks_for(int64_t n, int per_block, int per_sm = 32) {
  const int64_t b = (n + per_block - 1) / per_block, cap = int64_t(sm_count()) * per_sm;
  return unsigned(b < 1 ? 1 : (b > cap ? cap : b));
}

// ---- induced sub-graph ---------------------------------------------------------------------------------------
// workspace words, all -1 at the start: new_id[n_nodes], arrivals, bad; then counts, offsets, result, pairs
struct SubgraphWs {
  int32_t *new_id, *arrivals, *bad, *counts, *offsets;
  int64_t* result;   // {kept edges, a node id was out of range}
  int2* pairs;       // kept edges of chunk c, compacted, from position c * kChunk on
  int64_t chunks;
};

size_t subgraph_ws(char* base, int64_t n_edges, int64_t n_nodes, SubgraphWs* w) {
  const int64_t chunks = (n_edges + n_nodes + kChunk - 1) / kChunk;
  size_t off = 0;
  auto take = [&](size_t bytes) { char* p = base + off; off += round_up(bytes, 256); return p; };
  SubgraphWs s;
  s.new_id = reinterpret_cast<int32_t*>(take(size_t(n_nodes + 2) * 4));
  s.arrivals = s.new_id + n_nodes;
  s.bad = s.arrivals + 1;
  s.counts = reinterpret_cast<int32_t*>(take(size_t(chunks) * 4));
  s.offsets = reinterpret_cast<int32_t*>(take(size_t(chunks) * 4));
  s.result = reinterpret_cast<int64_t*>(take(16));
  s.pairs = reinterpret_cast<int2*>(take(size_t(chunks) * kChunk * sizeof(int2)));
  s.chunks = chunks;
  if (w != nullptr) *w = s;
  return off;
}

// new_id[node] = its position in idx (the last one where a node is listed twice); negative ids count from the end
__global__ void __launch_bounds__(kBatchThreads) number_nodes_kernel(const int64_t* __restrict__ idx, int64_t n_idx,
                                                                     int64_t n_nodes, int32_t* new_id, int32_t* bad) {
  for (int64_t j = blockIdx.x * int64_t(kBatchThreads) + threadIdx.x; j < n_idx; j += int64_t(gridDim.x) * kBatchThreads) {
    int64_t v = __ldg(idx + j);
    if (v < 0) v += n_nodes;
    if (v < 0 || v >= n_nodes) *bad = 1;
    else atomicMax(new_id + v, int32_t(j));
  }
}

// One chunk of candidates per CTA: the edges in their order, then one self loop per node in node order.  Kept are
// edges with two different endpoints inside the batch, and the self loops of its nodes.  The CTA that finishes last
// turns the chunks' counts into offsets.
__global__ void __launch_bounds__(kBatchThreads) mark_edges_kernel(const int64_t* __restrict__ edges, int64_t n_edges,
                                                                   int64_t n_nodes, const SubgraphWs w) {
  constexpr int kWarps = kBatchThreads / 32, kItems = kChunk / kBatchThreads;
  __shared__ int s_count[kItems * kWarps];
  __shared__ bool s_last;
  __shared__ int64_t s_sum[kWarps];
  const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
  const int64_t first = int64_t(blockIdx.x) * kChunk;
  int2 kept[kItems];
  unsigned votes[kItems];
  int64_t s[kItems], d[kItems];
#pragma unroll
  for (int j = 0; j < kItems; ++j) {
    const int64_t i = first + j * kBatchThreads + tid;
    s[j] = i < n_edges ? __ldg(edges + i) : i - n_edges;
    d[j] = i < n_edges ? __ldg(edges + n_edges + i) : i - n_edges;
  }
#pragma unroll
  for (int j = 0; j < kItems; ++j) {
    const int64_t i = first + j * kBatchThreads + tid;
    bool keep = i < n_edges + n_nodes && (i >= n_edges || s[j] != d[j]);
    if (s[j] < 0) s[j] += n_nodes;
    if (d[j] < 0) d[j] += n_nodes;
    const bool inside = s[j] >= 0 && s[j] < n_nodes && d[j] >= 0 && d[j] < n_nodes;
    if (keep && !inside) *w.bad = 1;
    kept[j] = make_int2(-1, -1);
    if (keep && inside) kept[j] = make_int2(__ldcg(w.new_id + s[j]), __ldcg(w.new_id + d[j]));
    votes[j] = __ballot_sync(0xffffffffu, kept[j].x >= 0 && kept[j].y >= 0);
    if (lane == 0) s_count[j * kWarps + warp] = __popc(votes[j]);
  }
  __syncthreads();
  if (warp == 0) {   // exclusive prefix sums of the 64 counts, two per lane
    static_assert(kItems * kWarps == 64, "two counts per lane");
    const int a = s_count[2 * lane], b = s_count[2 * lane + 1];
    int sum = a + b;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += t;
    }
    s_count[2 * lane] = sum - a - b;
    s_count[2 * lane + 1] = sum - b;
    if (lane == 31) w.counts[blockIdx.x] = sum;
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kItems; ++j)
    if (votes[j] >> lane & 1)
      w.pairs[first + s_count[j * kWarps + warp] + __popc(votes[j] & ((1u << lane) - 1))] = kept[j];
  __threadfence();
  __syncthreads();
  if (tid == 0) s_last = atomicAdd(w.arrivals, 1) == int(gridDim.x) - 2;   // the counter starts at -1
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  int64_t before = 0;
  for (int64_t c0 = 0; c0 < gridDim.x; c0 += kBatchThreads) {
    const int64_t c = c0 + tid;
    const int64_t v = c < gridDim.x ? int64_t(__ldcg(w.counts + c)) : 0;
    int64_t sum = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t t = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += t;
    }
    if (lane == 31) s_sum[warp] = sum;
    __syncthreads();
    int64_t add = before;
    for (int q = 0; q < warp; ++q) add += s_sum[q];
    if (c < gridDim.x) w.offsets[c] = int32_t(add + sum - v);
    for (int q = 0; q < kWarps; ++q) before += s_sum[q];
    __syncthreads();
  }
  if (tid == 0) {
    w.result[0] = before;
    w.result[1] = *static_cast<volatile int32_t*>(w.bad) == 1;
  }
}

__device__ __forceinline__ int64_t shifted(int64_t id, int64_t sub_seq_len) {   // adjust_edge_index_nomerge
  return sub_seq_len > 0 && id > 0 ? id + (id - 1) / sub_seq_len : id;
}

// Kept edges to their places (one CTA per chunk), then the global token's 2 * n_idx edges by the CTAs behind them.
__global__ void __launch_bounds__(kBatchThreads) write_edges_kernel(const SubgraphWs w, int64_t n_idx, int add_token,
                                                                    int64_t sub_seq_len, int64_t* __restrict__ out,
                                                                    int64_t out_total) {
  if (int64_t(blockIdx.x) < w.chunks) {
    const int count = __ldg(w.counts + blockIdx.x), at = __ldg(w.offsets + blockIdx.x);
    for (int i = threadIdx.x; i < count; i += kBatchThreads) {
      const int2 e = __ldg(w.pairs + int64_t(blockIdx.x) * kChunk + i);
      out[at + i] = shifted(int64_t(e.x) + add_token, sub_seq_len);
      out[out_total + at + i] = shifted(int64_t(e.y) + add_token, sub_seq_len);
    }
    return;
  }
  const int64_t kept = out_total - 2 * n_idx;
  for (int64_t i = (blockIdx.x - w.chunks) * kBatchThreads + threadIdx.x; i < n_idx;
       i += (gridDim.x - w.chunks) * kBatchThreads) {
    const int64_t id = shifted(i + 1, sub_seq_len);
    out[kept + i] = id;
    out[out_total + kept + i] = 0;
    out[kept + n_idx + i] = 0;
    out[out_total + kept + n_idx + i] = id;
  }
}

// ---- rows of a matrix by index -------------------------------------------------------------------------------
template <typename U>
__global__ void __launch_bounds__(kBatchThreads) gather_rows_kernel(const U* __restrict__ x, const int64_t* __restrict__ idx,
                                                                    int64_t n_rows, int64_t n_out, int units,
                                                                    U* __restrict__ out) {
  constexpr int kFlight = 4;   // units per thread whose loads are in flight together
  const int64_t total = n_out * units, stride = int64_t(gridDim.x) * kBatchThreads;
  for (int64_t u0 = blockIdx.x * int64_t(kBatchThreads) + threadIdx.x; u0 < total; u0 += stride * kFlight) {
    U v[kFlight];
    bool live[kFlight];
#pragma unroll
    for (int j = 0; j < kFlight; ++j) {
      const int64_t u = u0 + j * stride;
      live[j] = u < total;
      const int64_t r = !live[j] ? 0 : total >> 31 ? u / units : int64_t(unsigned(u) / unsigned(units));
      int64_t row = live[j] ? __ldg(idx + r) : 0;
      if (row < 0) row += n_rows;
      live[j] = live[j] && row >= 0 && row < n_rows;   // an id out of range is reported by the sub-graph's pass
      if (live[j]) v[j] = x[row * units + (u - r * units)];
    }
#pragma unroll
    for (int j = 0; j < kFlight; ++j)
      if (live[j]) out[u0 + j * stride] = v[j];
  }
}

// ---- cluster-sparse blocks -------------------------------------------------------------------------------------
struct BlockWs {
  int64_t *counts, *n_blocks, *first_block;    // [k * k] (first_block: k * k + 1)
  int64_t *nodes, *offset, *grid_base;         // [k]: nodes of a partition, its first new id, its first grid row
  int32_t *row_count, *row_start, *cursor;     // per grid row (at most n_nodes / block)
  int64_t* result;                             // {blocks, grid rows, original edges must be kept somewhere, bad id}
  size_t zero_bytes;                           // counts, nodes, row_count and result are cleared, in one piece
  void* zero;
};

size_t block_ws(char* base, int64_t k, int64_t n_nodes, int64_t block, BlockWs* out) {
  size_t off = 0;
  auto take = [&](size_t bytes) { char* p = base + off; off += round_up(bytes, 256); return p; };
  const size_t kk = size_t(k) * k, rows = size_t(n_nodes / block + 1);
  BlockWs w;
  w.zero = take(0);
  w.counts = reinterpret_cast<int64_t*>(take(kk * 8));
  w.nodes = reinterpret_cast<int64_t*>(take(size_t(k) * 8));
  w.row_count = reinterpret_cast<int32_t*>(take(rows * 4));
  w.result = reinterpret_cast<int64_t*>(take(32));
  w.zero_bytes = off;
  w.n_blocks = reinterpret_cast<int64_t*>(take(kk * 8));
  w.first_block = reinterpret_cast<int64_t*>(take((kk + 1) * 8));
  w.offset = reinterpret_cast<int64_t*>(take(size_t(k) * 8));
  w.grid_base = reinterpret_cast<int64_t*>(take(size_t(k) * 8));
  w.row_start = reinterpret_cast<int32_t*>(take(rows * 4));
  w.cursor = reinterpret_cast<int32_t*>(take(rows * 4));
  if (out != nullptr) *out = w;
  return off;
}

// partition of node v: part[v], or without a list k contiguous ranges
struct Partition {
  const int64_t* part;
  int64_t n_nodes;
  int k;
  __device__ __forceinline__ int64_t of(int64_t v) const { return part != nullptr ? __ldg(part + v) : v * k / n_nodes; }
};

constexpr int kPairBins = 4096;   // pair counts kept in shared memory up to k = 64

__global__ void __launch_bounds__(kBatchThreads) count_pairs_kernel(const int64_t* __restrict__ edges, int64_t n_edges,
                                                                    const Partition p, const BlockWs w) {
  __shared__ unsigned s_bin[kPairBins];
  const int kk = p.k * p.k;
  const bool shared = kk <= kPairBins;
  if (shared)
    for (int i = threadIdx.x; i < kk; i += kBatchThreads) s_bin[i] = 0;
  __syncthreads();
  const int64_t stride = int64_t(gridDim.x) * kBatchThreads;
  for (int64_t i = blockIdx.x * int64_t(kBatchThreads) + threadIdx.x; i < n_edges; i += stride) {
    const int64_t s = __ldg(edges + i), d = __ldg(edges + n_edges + i);
    int64_t ps = -1, pd = -1;
    if (s >= 0 && s < p.n_nodes && d >= 0 && d < p.n_nodes) { ps = p.of(s); pd = p.of(d); }
    if (ps < 0 || ps >= p.k || pd < 0 || pd >= p.k) { w.result[3] = 1; continue; }
    if (shared) atomicAdd(s_bin + ps * p.k + pd, 1u);
    else atomicAdd(reinterpret_cast<unsigned long long*>(w.counts) + ps * p.k + pd, 1ull);
  }
  // nodes per partition
  for (int64_t v = blockIdx.x * int64_t(kBatchThreads) + threadIdx.x; v < p.n_nodes; v += stride) {
    const int64_t q = p.of(v);
    if (q < 0 || q >= p.k) { w.result[3] = 1; continue; }
    if (p.part != nullptr) atomicAdd(reinterpret_cast<unsigned long long*>(w.nodes) + q, 1ull);
  }
  if (p.part == nullptr && blockIdx.x == 0)
    for (int q = threadIdx.x; q < p.k; q += kBatchThreads)
      w.nodes[q] = ((q + 1) * p.n_nodes + p.k - 1) / p.k - (q * p.n_nodes + p.k - 1) / p.k;
  __syncthreads();
  if (shared)
    for (int i = threadIdx.x; i < kk; i += kBatchThreads)
      if (s_bin[i] != 0) atomicAdd(reinterpret_cast<unsigned long long*>(w.counts) + i, s_bin[i]);
}

constexpr int kPlanThreads = 1024;

// Exclusive prefix sum over the block, plus `carry` (updated to the running total).
__device__ __forceinline__ int64_t block_exclusive(int64_t v, int64_t& carry, int64_t (&s_sum)[kPlanThreads / 32]) {
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  int64_t sum = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int64_t t = __shfl_up_sync(0xffffffffu, sum, o);
    if (lane >= o) sum += t;
  }
  if (lane == 31) s_sum[warp] = sum;
  __syncthreads();
  int64_t add = carry, all = 0;
  for (int q = 0; q < int(blockDim.x) / 32; ++q) {
    if (q < warp) add += s_sum[q];
    all += s_sum[q];
  }
  __syncthreads();
  carry += all;
  return add + sum - v;
}

// Blocks per partition pair, in double precision exactly as numpy's int64 / int64 gives them.  The counts of the
// non-empty pairs are read as a dense list by pair number, as the reference reads them.
__global__ void __launch_bounds__(kPlanThreads) plan_blocks_kernel(int k, int64_t block, double p, const BlockWs w) {
  __shared__ int64_t s_sum[kPlanThreads / 32];
  const int kk = k * k;
  int64_t offset = 0, rows = 0, ranks = 0, blocks = 0;
  for (int i0 = 0; i0 < k; i0 += kPlanThreads) {
    const int i = i0 + threadIdx.x;
    const int64_t n = i < k ? w.nodes[i] : 0;
    const int64_t at = block_exclusive(n, offset, s_sum), base = block_exclusive(n / block, rows, s_sum);
    if (i < k) { w.offset[i] = at; w.grid_base[i] = base; }
  }
  for (int i0 = 0; i0 < kk; i0 += kPlanThreads) {
    const int i = i0 + threadIdx.x;
    if (i < kk) w.n_blocks[i] = 0;
  }
  __syncthreads();
  for (int i0 = 0; i0 < kk; i0 += kPlanThreads) {
    const int i = i0 + threadIdx.x;
    const int64_t c = i < kk ? w.counts[i] : 0;
    const int64_t at = block_exclusive(c > 0 ? 1 : 0, ranks, s_sum);
    if (c > 0) w.n_blocks[at] = c;      // the dense list, turned into block counts below
  }
  __syncthreads();
  for (int i0 = 0; i0 < kk; i0 += kPlanThreads) {
    const int i = i0 + threadIdx.x;
    int64_t n = 0;
    if (i < kk) {
      const int64_t a = w.nodes[i / k], b = w.nodes[i % k], total = a * b;
      const double density = total > 0 ? __ddiv_rn(double(w.n_blocks[i]), double(total)) : 2.0 + p;
      if (density > p) w.result[2] = 1;
      else if (a >= block && b >= block)
        n = int64_t(__ddiv_rn(__dmul_rn(density, double(total)), double(block * block))) + 1;
    }
    const int64_t at = block_exclusive(n, blocks, s_sum);
    if (i < kk) { w.n_blocks[i] = n; w.first_block[i] = at; }
  }
  if (threadIdx.x == 0) {
    w.first_block[kk] = blocks;
    w.result[0] = blocks;
    w.result[1] = rows;
  }
}

// What draw_blocks_kernel and sort_blocks_kernel leave for the expansion.
struct BlockList {
  int32_t* row;       // grid row inside the source partition, in drawing order
  int32_t* col0;      // first destination id, in drawing order
  int32_t* row0;      // first source id, in drawing order
  int4* slot;         // in source order: {first source id, first slot of the grid row, blocks of the grid row, first destination id}
};

size_t block_list(char* base, int64_t blocks, BlockList* out) {
  size_t off = 0;
  auto take = [&](size_t bytes) { char* p = base + off; off += round_up(bytes, 256); return p; };
  BlockList l;
  l.row = reinterpret_cast<int32_t*>(take(size_t(blocks) * 4));
  l.col0 = reinterpret_cast<int32_t*>(take(size_t(blocks) * 4));
  l.row0 = reinterpret_cast<int32_t*>(take(size_t(blocks) * 4));
  l.slot = reinterpret_cast<int4*>(take(size_t(blocks) * 16));
  if (out != nullptr) *out = l;
  return off;
}

// One warp per partition pair draws its block coordinates with the 32-bit Mersenne Twister (Matsumoto and Nishimura,
// 1998) seeded by the number of blocks before it, row and column alternating, each below its bound by masked
// rejection: numpy's RandomState(seed).randint(0, bound), draw for draw.
__global__ void __launch_bounds__(32) draw_blocks_kernel(int k, int64_t block, const BlockWs w, const BlockList l) {
  constexpr int kN = 624, kM = 397;
  __shared__ uint32_t s_mt[kN], s_out[kN];
  const int pair = blockIdx.x, lane = threadIdx.x;
  const int64_t n = w.n_blocks[pair], first = w.first_block[pair];
  if (n == 0) return;
  const int i = pair / k, j = pair % k;
  const uint32_t bound[2] = {uint32_t(w.nodes[i] / block) - 1u, uint32_t(w.nodes[j] / block) - 1u};   // inclusive
  uint32_t mask[2];
#pragma unroll
  for (int a = 0; a < 2; ++a) mask[a] = bound[a] == 0 ? 0u : 0xffffffffu >> __clz(int(bound[a]));
  if (lane == 0) {
    uint32_t x = uint32_t(first);
    s_mt[0] = x;
    for (int q = 1; q < kN; ++q) s_mt[q] = x = 1812433253u * (x ^ (x >> 30)) + uint32_t(q);
  }
  __syncwarp();
  const int64_t row_off = w.offset[i], col_off = w.offset[j];
  int64_t drawn = 0;       // coordinates accepted so far (lane 0's copy counts)
  uint32_t row = 0;
  while (drawn < 2 * n) {
    for (int q0 = 0; q0 < kN; q0 += 32) {
      const int q = q0 + lane;
      uint32_t v = 0;
      if (q < kN) {
        const uint32_t y = (s_mt[q] & 0x80000000u) | (s_mt[(q + 1) % kN] & 0x7fffffffu);
        v = s_mt[(q + kM) % kN] ^ (y >> 1) ^ (y & 1u ? 0x9908b0dfu : 0u);
      }
      __syncwarp();
      if (q < kN) {
        s_mt[q] = v;
        v ^= v >> 11;
        v ^= (v << 7) & 0x9d2c5680u;
        v ^= (v << 15) & 0xefc60000u;
        s_out[q] = v ^ (v >> 18);
      }
      __syncwarp();
    }
    if (lane == 0) {
      for (int q = 0; q < kN && drawn < 2 * n;) {
        const int a = int(drawn & 1);
        uint32_t v = 0;
        if (bound[a] != 0) {           // a single choice takes no random number
          v = s_out[q++] & mask[a];
          if (v > bound[a]) continue;
        }
        if (a == 0) {
          row = v;
        } else {
          const int64_t b = first + (drawn >> 1);
          l.row[b] = int32_t(row);
          l.row0[b] = int32_t(row_off + int64_t(row) * block);
          l.col0[b] = int32_t(col_off + int64_t(v) * block);
        }
        ++drawn;
      }
    }
    drawn = __shfl_sync(0xffffffffu, drawn, 0);
  }
}

// Stable counting sort of one partition's blocks by grid row (one CTA per partition).
__global__ void __launch_bounds__(kPlanThreads) sort_blocks_kernel(int k, int64_t block, const BlockWs w, const BlockList l) {
  __shared__ int64_t s_sum[kPlanThreads / 32];
  const int i = blockIdx.x;
  const int64_t b0 = w.first_block[int64_t(i) * k], b1 = w.first_block[int64_t(i + 1) * k];
  if (b0 == b1) return;
  const int64_t base = w.grid_base[i], rows = w.nodes[i] / block;
  for (int64_t b = b0 + threadIdx.x; b < b1; b += kPlanThreads) atomicAdd(w.row_count + base + l.row[b], 1);
  __syncthreads();
  int64_t at = b0;
  for (int64_t r0 = 0; r0 < rows; r0 += kPlanThreads) {
    const int64_t r = r0 + threadIdx.x;
    const int64_t start = block_exclusive(r < rows ? __ldcg(w.row_count + base + r) : 0, at, s_sum);
    if (r < rows) w.row_start[base + r] = w.cursor[base + r] = int32_t(start);
  }
  __syncthreads();
  if (threadIdx.x >= 32) return;
  const int lane = threadIdx.x;
  for (int64_t c = b0; c < b1; c += 32) {
    const int64_t b = c + lane;
    const bool live = b < b1;
    const int row = live ? l.row[b] : -1;
    const unsigned same = __match_any_sync(0xffffffffu, row);
    int slot = 0;
    if (live) slot = w.cursor[base + row] + __popc(same & ((1u << lane) - 1));
    __syncwarp();
    if (live && (same >> lane) == 1u) w.cursor[base + row] = slot + 1;   // the last of its row in this chunk
    __syncwarp();
    if (live) l.slot[slot] = make_int4(l.row0[b], w.row_start[base + row], __ldcg(w.row_count + base + row), l.col0[b]);
  }
}

// I: unsigned when the edge count fits 32 bits
template <typename I, bool kBySource>
__global__ void __launch_bounds__(kBatchThreads) expand_blocks_kernel(I total, I block, const BlockList l, int64_t sub_seq_len,
                                                                      int64_t* __restrict__ out) {
  const I square = block * block;
  for (I e = I(blockIdx.x) * kBatchThreads + threadIdx.x; e < total; e += I(gridDim.x) * kBatchThreads) {
    const I b = e / square;
    int64_t s, d;
    if (kBySource) {
      const int4 slot = __ldg(l.slot + b);
      const I local = e - I(slot.y) * square, width = I(slot.z) * block;
      const I u = local / width, rest = local - u * width, t = rest / block;
      s = int64_t(slot.x) + int64_t(u);
      d = int64_t(__ldg(&l.slot[slot.y + int64_t(t)].w)) + int64_t(rest - t * block);
    } else {
      const I within = e - b * square, u = within / block;
      s = int64_t(__ldg(l.row0 + b)) + int64_t(u);
      d = int64_t(__ldg(l.col0 + b)) + int64_t(within - u * block);
    }
    out[e] = shifted(s, sub_seq_len);
    out[int64_t(total) + e] = shifted(d, sub_seq_len);
  }
}

}  // namespace
}  // namespace tgt

extern "C" int tgt_subgraph_workspace_bytes(int64_t n_edges, int64_t n_nodes, size_t* bytes) {
  using namespace tgt;
  TGT_CHECK_ARG(bytes != nullptr, "bytes is null");
  TGT_CHECK_ARG(n_edges >= 0 && n_nodes >= 0 && n_edges + n_nodes < (int64_t(1) << 31) - kChunk,
                "edges and nodes together must fit in int32");
  *bytes = subgraph_ws(nullptr, n_edges, n_nodes, nullptr);
  return TGT_OK;
}

extern "C" int tgt_subgraph_count(const int64_t* edge_index, int64_t n_edges, int64_t n_nodes, const int64_t* idx,
                                  int64_t n_idx, void* workspace, size_t workspace_bytes, const int64_t** result,
                                  void* stream_) {
  using namespace tgt;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  size_t need = 0;
  const int rc = tgt_subgraph_workspace_bytes(n_edges, n_nodes, &need);
  if (rc != TGT_OK) return rc;
  TGT_CHECK_ARG(n_nodes >= 1 && n_idx >= 0 && n_idx < (int64_t(1) << 30), "n_nodes must be >= 1, n_idx >= 0");
  TGT_CHECK_ARG((n_edges == 0 || edge_index) && (n_idx == 0 || idx) && workspace && result, "null pointer");
  if (workspace_bytes < need)
    return set_error(TGT_ERR_WORKSPACE, "workspace holds %zu bytes, %zu needed", workspace_bytes, need);
  SubgraphWs w;
  subgraph_ws(static_cast<char*>(workspace), n_edges, n_nodes, &w);
  TGT_CHECK_CUDA(cudaMemsetAsync(w.new_id, 0xff, size_t(n_nodes + 2) * 4, stream));
  if (n_idx > 0)
    number_nodes_kernel<<<blocks_for(n_idx, kBatchThreads), kBatchThreads, 0, stream>>>(idx, n_idx, n_nodes, w.new_id, w.bad);
  mark_edges_kernel<<<unsigned(w.chunks), kBatchThreads, 0, stream>>>(edge_index, n_edges, n_nodes, w);
  TGT_CHECK_CUDA(cudaGetLastError());
  *result = w.result;
  return TGT_OK;
}

extern "C" int tgt_subgraph_write(int64_t n_edges, int64_t n_nodes, int64_t n_idx, int add_global_token,
                                  int64_t sub_seq_len, const void* workspace, int64_t* out, int64_t out_total,
                                  void* stream_) {
  using namespace tgt;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  TGT_CHECK_ARG(add_global_token == 0 || add_global_token == 1, "add_global_token must be 0 or 1");
  TGT_CHECK_ARG(sub_seq_len >= 0 && out_total >= 0 && workspace && (out_total == 0 || out), "bad size or null pointer");
  if (out_total == 0) return TGT_OK;
  SubgraphWs w;
  subgraph_ws(static_cast<char*>(const_cast<void*>(workspace)), n_edges, n_nodes, &w);
  const unsigned token = add_global_token && n_idx > 0 ? blocks_for(n_idx, kBatchThreads) : 0;
  write_edges_kernel<<<unsigned(w.chunks) + token, kBatchThreads, 0, stream>>>(w, add_global_token ? n_idx : 0,
                                                                              add_global_token, sub_seq_len, out, out_total);
  TGT_CHECK_CUDA(cudaGetLastError());
  return TGT_OK;
}

extern "C" int tgt_gather_rows(const void* x, int64_t n_rows, int64_t row_bytes, const int64_t* idx, int64_t n_out,
                               void* out, void* stream_) {
  using namespace tgt;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  TGT_CHECK_ARG(n_rows >= 0 && row_bytes >= 1 && n_out >= 0, "sizes must not be negative");
  if (n_out == 0) return TGT_OK;
  TGT_CHECK_ARG(x && idx && out, "null pointer");
  const uintptr_t all = reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(out) | uintptr_t(row_bytes);
  auto launch = [&](auto unit) {
    using U = decltype(unit);
    const int64_t units = row_bytes / int64_t(sizeof(U));
    TGT_CHECK_ARG(units < (int64_t(1) << 31), "rows are too long");
    gather_rows_kernel<U><<<blocks_for(n_out * units, kBatchThreads * 4, 8), kBatchThreads, 0, stream>>>(
        static_cast<const U*>(x), idx, n_rows, n_out, int(units), static_cast<U*>(out));
    TGT_CHECK_CUDA(cudaGetLastError());
    return int(TGT_OK);
  };
  if (all % 16 == 0) return launch(uint4{});
  if (all % 8 == 0) return launch(uint2{});
  if (all % 4 == 0) return launch(uint32_t{});
  if (all % 2 == 0) return launch(uint16_t{});
  return launch(uint8_t{});
}

extern "C" int tgt_blocks_workspace_bytes(int k, int64_t n_nodes, int64_t block, size_t* bytes) {
  using namespace tgt;
  TGT_CHECK_ARG(bytes != nullptr, "bytes is null");
  TGT_CHECK_ARG(k >= 1 && k <= 8192 && n_nodes >= 1 && n_nodes < (int64_t(1) << 31) - 1 && block >= 1 && block <= 32768,
                "k, n_nodes or block is out of range");
  *bytes = block_ws(nullptr, k, n_nodes, block, nullptr);
  return TGT_OK;
}

extern "C" int tgt_blocks_plan(const int64_t* edge_index, int64_t n_edges, int64_t n_nodes, const int64_t* partition, int k,
                               double p, int64_t block, void* workspace, size_t workspace_bytes, const int64_t** result,
                               void* stream_) {
  using namespace tgt;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  size_t need = 0;
  const int rc = tgt_blocks_workspace_bytes(k, n_nodes, block, &need);
  if (rc != TGT_OK) return rc;
  TGT_CHECK_ARG(n_edges >= 0 && (n_edges == 0 || edge_index) && workspace && result, "bad size or null pointer");
  if (workspace_bytes < need)
    return set_error(TGT_ERR_WORKSPACE, "workspace holds %zu bytes, %zu needed", workspace_bytes, need);
  BlockWs w;
  block_ws(static_cast<char*>(workspace), k, n_nodes, block, &w);
  TGT_CHECK_CUDA(cudaMemsetAsync(w.zero, 0, w.zero_bytes, stream));
  const Partition part{partition, n_nodes, k};
  const int64_t most = n_edges > n_nodes ? n_edges : n_nodes;
  count_pairs_kernel<<<blocks_for(most, kBatchThreads * 4, 4), kBatchThreads, 0, stream>>>(edge_index, n_edges, part, w);
  plan_blocks_kernel<<<1, kPlanThreads, 0, stream>>>(k, block, p, w);
  TGT_CHECK_CUDA(cudaGetLastError());
  *result = w.result;
  return TGT_OK;
}

extern "C" int tgt_blocks_list_bytes(int64_t blocks, size_t* bytes) {
  using namespace tgt;
  TGT_CHECK_ARG(bytes != nullptr && blocks >= 0 && blocks < (int64_t(1) << 31) - 1, "bytes is null or blocks out of range");
  *bytes = block_list(nullptr, blocks, nullptr);
  return TGT_OK;
}

extern "C" int tgt_blocks_write(int64_t n_nodes, int k, int64_t block, const void* workspace, void* list, size_t list_bytes,
                                int64_t blocks, int by_source, int64_t sub_seq_len, int64_t* out, void* stream_) {
  using namespace tgt;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  size_t need = 0;
  int rc = tgt_blocks_list_bytes(blocks, &need);
  if (rc == TGT_OK) rc = tgt_blocks_workspace_bytes(k, n_nodes, block, &need);
  if (rc != TGT_OK) return rc;
  if (blocks == 0) return TGT_OK;
  TGT_CHECK_ARG(workspace && list && out && sub_seq_len >= 0, "null pointer or negative sub_seq_len");
  if (list_bytes < block_list(nullptr, blocks, nullptr)) return set_error(TGT_ERR_WORKSPACE, "the block list is too small");
  BlockWs w;
  block_ws(static_cast<char*>(const_cast<void*>(workspace)), k, n_nodes, block, &w);
  BlockList l;
  block_list(static_cast<char*>(list), blocks, &l);
  draw_blocks_kernel<<<unsigned(k) * unsigned(k), 32, 0, stream>>>(k, block, w, l);
  if (by_source) sort_blocks_kernel<<<unsigned(k), kPlanThreads, 0, stream>>>(k, block, w, l);
  const int64_t total = blocks * block * block;
  const unsigned grid = blocks_for(total, kBatchThreads * 2);
  auto expand = [&](auto tag) {
    using I = decltype(tag);
    if (by_source) expand_blocks_kernel<I, true><<<grid, kBatchThreads, 0, stream>>>(I(total), I(block), l, sub_seq_len, out);
    else expand_blocks_kernel<I, false><<<grid, kBatchThreads, 0, stream>>>(I(total), I(block), l, sub_seq_len, out);
  };
  if (total < (int64_t(1) << 31)) expand(uint32_t{});
  else expand(uint64_t{});
  TGT_CHECK_CUDA(cudaGetLastError());
  return TGT_OK;
}
