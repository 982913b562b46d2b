// fp32 products of long matrices with small ones on the tensor cores, for the forward and the input gradient of narrow
// linear layers over many rows (models/graphormer_dist_node_level.py:241-245,281-286,
// models/gt_dist_node_level.py:189-193,232-236: 64 x 64 to 128 x 64 over 8,000 to 870,000 rows).
//
// A tile is 128 rows x 64 columns.  A CTA keeps its columns' weights as bf16 pieces in shared memory (tensor_core.cuh) and
// walks row tiles: 256 threads split the rows' values on their way from registers into shared memory, a ninth warp issues
// the products, and while they run the next rows are on their way in and the tile before is finished from the other half
// of the tensor memory.  CTAs of the same rows are neighbours in the grid, so a second column tile or a second layer finds
// the rows in the L2.
//
// Tensor cores round a running sum towards zero at every step, so an error of one sign grows with the sum's length.  One
// running sum of the large products therefore takes at most two chunks of 64; a tile has up to three of them side by side,
// added in fp32 on the way out, and longer reductions are several launches, each adding to what the one before has written.
//
// us back to back, here | FMA kernel that was here | library's input gradient: 320,000 rows of 64 x 64 42 | 75 | 87 (a copy of
// the same bytes: 25), 64 x 128 69 | 139 | 132, 128 x 64 70 | 144 | 127, three layers of 64 x 64 99 forward and 106 back; 64,001
// rows 12 | 19 | 18.  Sums stored row by row straight from tensor memory, without the blocks in shared memory, and without
// the second half: + 11 us; with a worker issuing the products and a general finish for every call: + 4 us.  Issue slots are
// 42 % busy; what is left is the wait for the rows, with the 17 warps per SM that the registers allow.
// Relative error against 64 bits, normal operands: 64 long 7e-8 (FMA 1.1e-7, library 1.5e-7), 128 long 1.2e-7 (1.5e-7, 2.0e-7),
// 1024 long 1.2e-7 (4.1e-7, 5.7e-7; with one running sum 1.0e-6), three gradients 64 long 7.6e-8 (library 1.5e-7, one running
// sum 1.7e-7); operands of one sign, 128 long 1.8e-7 (9e-8, 1.7e-7), 1024 long 1.6e-7 (2.5e-7, 4.9e-7; 2.2e-6).  Six chunks at
// most are one launch because their weights fit shared memory; 1024 x 1024 over 8,192 rows in three launches 282 us.
#include "linear_rows.cuh"
#include "tensor_core.cuh"

namespace tgt {
namespace {

constexpr int kWarps = 8, kWorkers = 32 * kWarps;   // split, load and finish; one warp more issues the products
constexpr int kThreads = kWorkers + 32;
constexpr int kRows = 128, kCols = 64;     // of a tile: M and N of one product
constexpr int kChunk = 64;                 // reduction elements staged at a time
constexpr int kPieceA = kRows * 128;       // bytes of one piece of a tile of A
constexpr int kPieceW = kCols * 128;
constexpr int kMostSums = 3;               // running sums of large products per tile, of at most two chunks each
constexpr int kMostChunks = 2 * kMostSums; // of one launch; the weights' pieces of all of them are kept

struct SplitGemm : LinearRows {
  int col_tiles;                    // per output
  int first, chunks;                // the part of the reduction this launch sums, in chunks (sources one after the other)
  int big_sums;                     // of two chunks each, the last perhaps of one
  int ahead;                        // tiles between the one whose products run and the one that is brought into the L2, or 0
  int* expired;                     // expired_wait_word
};
// Tensor memory of a CTA: for each of two tiles the first sum of large products, the sum of small ones, more sums of large ones
constexpr int tile_columns(bool more) { return (more ? 1 + kMostSums : 2) * kCols; }

// Finished sums on their way out: 32 rows x 16 columns per warp, 16-byte pieces in an order that keeps rows' equal pieces
// in different banks.
constexpr int kBlockCols = 16, kBlockBytes = 32 * kBlockCols * 4;
__device__ __forceinline__ int block_offset(int row, int piece) { return row * 64 + ((piece ^ (row / 2)) & 3) * 16; }

// An infinity or NaN among the operands, or a sum past the range of fp32: the pieces' sum says no more than that.  The values
// of such rows (bits of `rows`, counted from row0) that are not finite are summed again from the operands themselves, a row at a
// time by the whole warp: a lane has one of the 16 columns of the warp's block and every other reduction element.  (320,000 rows
// of 64 x 64, one row not finite: 43 us, with a thread per row and column after column 200; all rows 2.5 ms and 4.9.)
template <int UNROLL>
__device__ __forceinline__ void sum_rows_again(const SplitGemm& p, int out, int64_t row0, uint32_t rows, int col, uint8_t* block) {
  const int src_chunks = (p.red + kChunk - 1) / kChunk, lane = threadIdx.x % 32;
  col += lane % 16;
  __syncwarp();                                             // the block is complete
  for (; rows != 0; rows &= rows - 1) {
    const int r = __ffs(rows) - 1;
    float s = 0.f;
    if (row0 + r < p.rows && col < p.cols)
#pragma unroll 1
      for (int chunk = p.first; chunk < p.first + p.chunks; ++chunk) {
        const int src = chunk / src_chunks, k0 = chunk % src_chunks * kChunk, k1 = min(k0 + kChunk, p.red);
        const float* a = p.a[src] + (row0 + r) * p.red;
        const float* w = p.w[p.sources > 1 ? src : out] + (p.transposed ? col : int64_t(col) * p.red);
        const int step = p.transposed ? p.cols : 1;
#pragma unroll UNROLL
        for (int k = k0 + lane / 16; k < k1; k += 2) s = fmaf(__ldg(a + k), __ldg(w + k * step), s);
      }
    s += __shfl_xor_sync(~0u, s, 16);
    float* const v = reinterpret_cast<float*>(block + block_offset(r, lane % 16 / 4)) + lane % 4;
    if (lane < 16 && !(fabsf(*v) < __int_as_float(0x7f800000)) && row0 + r < p.rows && col < p.cols) *v = s;
  }
}

// as a call, which costs fewer registers where the finish has need of them itself
__device__ __noinline__ void sum_rows_again_called(const SplitGemm& p, int out, int64_t row0, uint32_t rows, int col, uint8_t* block) {
  sum_rows_again<2>(p, out, row0, rows, col, block);
}

// A wait for the products has run out: this CTA's results from `tile` on become NaN.
__device__ __noinline__ void give_up(const SplitGemm& p, int out, int c0, int64_t tile, int walkers) {
  if (threadIdx.x == 0) tc::report_expired_wait(p.expired);
  const float nan = __int_as_float(0x7fffffff);
  const int col = c0 + 4 * (threadIdx.x % 16);
  if (col >= p.cols) return;
  for (; tile * kRows < p.rows; tile += walkers)
    for (int64_t row = tile * kRows + threadIdx.x / 16; row < min((tile + 1) * kRows, p.rows); row += kWorkers / 16) {
      *reinterpret_cast<float4*>(p.c[out] + row * p.cols + col) = make_float4(nan, nan, nan, nan);
      if (p.pre != nullptr) *reinterpret_cast<float4*>(p.pre + row * p.cols + col) = make_float4(nan, nan, nan, nan);
    }
}

// Shared memory of a CTA, from a 1,024-byte boundary on: pieces of a chunk of A, pieces of the chunks of the weights, one block
// of finished sums per warp, the barrier and the tensor memory's address.
__host__ __device__ inline int split_gemm_smem(int chunks) {
  return 3 * kPieceA + chunks * 3 * kPieceW + kWarps * kBlockBytes + 16;
}
static_assert(3 * kPieceA + kMostChunks * 3 * kPieceW + kWarps * kBlockBytes + 16 <= 227 * 1024, "one CTA per SM");
static_assert(2 * (3 * kPieceA + 2 * 3 * kPieceW + kWarps * kBlockBytes + 16 + 1024) <= 228 * 1024, "two with two chunks");

template <bool PLAIN, bool LONG>   // nothing but a bias is added to the sums; more than two chunks
__global__ void __launch_bounds__(kThreads, LONG ? 1 : 2) split_gemm_kernel(const __grid_constant__ SplitGemm p) {
  extern __shared__ __align__(1024) uint8_t s_raw[];
  const int src_chunks = (p.red + kChunk - 1) / kChunk;
  const uint32_t s_a = tc::smem_address(s_raw);
  const uint32_t s_w = s_a + 3 * kPieceA;
  uint8_t* const s_block = s_raw + 3 * kPieceA + p.chunks * 3 * kPieceW + threadIdx.x / 32 * kBlockBytes;
  uint64_t* const s_done = reinterpret_cast<uint64_t*>(s_raw + split_gemm_smem(p.chunks) - 16);
  uint32_t* const s_tmem = reinterpret_cast<uint32_t*>(s_done + 1);
  const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
  const int across = p.col_tiles * p.outputs;               // neighbours in the grid read the same rows of A
  const int tile_col = blockIdx.x % across;
  const int out = tile_col / p.col_tiles, c0 = tile_col % p.col_tiles * kCols;
  const int walkers = gridDim.x / across;
  const int64_t tiles = (p.rows + kRows - 1) / kRows;

  constexpr int kHalf = tile_columns(LONG);                 // of the tensor memory: a tile's sums
  if (warp == 0) tc::allocate<2 * kHalf>(s_tmem);
  if (tid == 32) tc::barrier_init(s_done);

  const int q = 4 * (tid % 16), r0 = tid / 16;              // a worker's four reduction elements and first row
  float4 next[kRows / 16];
  auto load = [&](int64_t tile, int chunk) {
    chunk += p.first;
    const int src = src_chunks == 1 ? chunk : chunk / src_chunks;
    const int k = (src_chunks == 1 ? 0 : chunk % src_chunks * kChunk) + q;
    const int64_t row = tile * kRows + r0;
    const float* a = p.a[src] + row * p.red + k;
    const int64_t step = int64_t(16) * p.red;
    if (tile * kRows + kRows <= p.rows && k < p.red) {
#pragma unroll
      for (int i = 0; i < kRows / 16; ++i, a += step) next[i] = __ldg(reinterpret_cast<const float4*>(a));
    } else {
#pragma unroll
      for (int i = 0; i < kRows / 16; ++i, a += step)
        next[i] = row + 16 * i < p.rows && k < p.red ? __ldg(reinterpret_cast<const float4*>(a))
                                                     : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  int64_t tile = blockIdx.x / across;
  if (warp < kWarps) load(tile, 0);
  auto stage_weights = [&](int slot) {
    const int src = (p.first + slot) / src_chunks, k0 = (p.first + slot) % src_chunks * kChunk;
    const float* w = p.w[p.sources > 1 ? src : out];
#pragma unroll 4
    for (int u = tid; u < kCols * 16; u += kWorkers) {
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      int n, k;
      if (!p.transposed) {
        n = u / 16; k = 4 * (u % 16);
        if (c0 + n < p.cols && k0 + k < p.red)
          v = __ldg(reinterpret_cast<const float4*>(w + int64_t(c0 + n) * p.red + k0 + k));
      } else {
        n = u % kCols; k = 4 * (u / kCols);
        if (c0 + n < p.cols && k0 + k < p.red) {
          const float* f = w + int64_t(k0 + k) * p.cols + c0 + n;
          v = make_float4(__ldg(f), __ldg(f + p.cols), __ldg(f + 2 * p.cols), __ldg(f + 3 * p.cols));
        }
      }
      tc::store4(s_w + slot * (3 * kPieceW), kPieceW, tc::tile_offset(n, k), tc::split4(v));
    }
  };
  if (warp < kWarps)
    for (int chunk = 0; chunk < p.chunks; ++chunk) stage_weights(chunk);
  if (warp < kWarps) tc::publish_operands();
  tc::fence_before_barrier();
  __syncthreads();
  tc::fence_after_barrier();
  const uint32_t tmem = *s_tmem;
  uint32_t phase = 0;
  bool ok = true;                      // no wait of this thread has run out
  int64_t failed = -1;                 // the first tile of whose products one has

  // sums of a tile -> C: a warp finishes 32 rows x 32 columns, 16 columns at a time through its block of shared memory, so
  // that the stores are runs of 64 bytes per row
  auto finish = [&](int64_t of, uint32_t sums) {
    const int64_t row0 = of * kRows + warp % 4 * 32;
    sums += (uint32_t(warp % 4 * 32) << 16) + warp / 4 * 32;
#pragma unroll 1
    for (int j = 0; j < 32; j += kBlockCols) {
      uint32_t big[16], small[16];
      tc::read16(sums + j, big);
      tc::read16(sums + kCols + j, small);
      tc::reads_done();
      const int col = c0 + warp / 4 * 32 + j;
      float v[16], size = 0.f;
#pragma unroll
      for (int x = 0; x < 16; ++x) v[x] = __uint_as_float(big[x]) + __uint_as_float(small[x]);
#pragma unroll 1
      for (int more = 1; LONG && more < p.big_sums; ++more) {
        tc::read16(sums + (1 + more) * kCols + j, big);
        tc::reads_done();
#pragma unroll
        for (int x = 0; x < 16; ++x) v[x] += __uint_as_float(big[x]);
      }
#pragma unroll
      for (int x = 0; x < 16; x += 4) {
        size += (fabsf(v[x]) + fabsf(v[x + 1])) + (fabsf(v[x + 2]) + fabsf(v[x + 3]));
        *reinterpret_cast<float4*>(s_block + block_offset(lane, x / 4)) = make_float4(v[x], v[x + 1], v[x + 2], v[x + 3]);
      }
      const uint32_t odd = __ballot_sync(~0u, !(size < __int_as_float(0x7f800000)));
      if (odd != 0) {
        if (PLAIN) sum_rows_again<4>(p, out, row0, odd, col, s_block);
        else sum_rows_again_called(p, out, row0, odd, col, s_block);
      }
      __syncwarp();
      const int my_col = col + 4 * (lane % 4);
      if (my_col < p.cols) {
        float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
        if (PLAIN && p.bias[out] != nullptr) b = __ldg(reinterpret_cast<const float4*>(p.bias[out] + my_col));
        float* c = p.c[out] + (row0 + lane / 4) * p.cols + my_col;
        const int left = int(min(p.rows - row0, int64_t(32)));        // of the warp's rows
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int r = lane / 4 + 8 * i;
          const float4 v = *reinterpret_cast<const float4*>(s_block + block_offset(r, lane % 4));
          if (r >= left) continue;
          if (PLAIN) {
            *reinterpret_cast<float4*>(c + int64_t(8 * i) * p.cols) = make_float4(v.x + b.x, v.y + b.y, v.z + b.z, v.w + b.w);
          } else {
            finish_values(p, out, row0 + r, my_col, v);
          }
        }
      }
      __syncwarp();
    }
  };

  // A tile's products run under the finishing of the tile before, whose sums lie in the other half of the tensor memory.
  uint32_t sums = tmem;
  if (warp == kWarps) {
    for (; tile < tiles; tile += walkers) {
      for (int chunk = 0; chunk < p.chunks; ++chunk) {
        if (!__syncthreads_and(true)) goto finished;        // the workers' pieces are in place
        if (lane == 0) {
          tc::fence_after_barrier();
          const uint32_t w = s_w + chunk * (3 * kPieceW);
#pragma unroll
          for (int k = 0; k < kChunk / 16; ++k) {
            const uint64_t a1 = tc::k_major(s_a + 32 * k), a2 = tc::k_major(s_a + kPieceA + 32 * k),
                           a3 = tc::k_major(s_a + 2 * kPieceA + 32 * k);
            const uint64_t w1 = tc::k_major(w + 32 * k), w2 = tc::k_major(w + kPieceW + 32 * k),
                           w3 = tc::k_major(w + 2 * kPieceW + 32 * k);
            constexpr uint32_t both = tc::instruction(kRows, 2 * kCols, false, false),
                               one = tc::instruction(kRows, kCols, false, false);
            if (!LONG || chunk < 2) {
              tc::multiply(sums, a1, w1, both, chunk + k > 0);   // a1 w1 | a1 w2
            } else {
              tc::multiply(sums + (1 + chunk / 2) * kCols, a1, w1, one, chunk % 2 + k > 0);
              tc::multiply(sums + kCols, a1, w2, one, true);
            }
            tc::multiply(sums + kCols, a2, w1, one, true);
            tc::multiply(sums + kCols, a2, w2, one, true);
            tc::multiply(sums + kCols, a1, w3, one, true);
            tc::multiply(sums + kCols, a3, w1, one, true);
          }
          tc::commit(s_done);
        }
        __syncwarp();
      }
      sums = tmem + (sums == tmem ? kHalf : 0);
    }
    __syncthreads_and(true);
  } else {
    int64_t before = -1;
    for (; tile < tiles; tile += walkers) {
      for (int chunk = 0; chunk < p.chunks; ++chunk) {
#pragma unroll
        for (int i = 0; i < kRows / 16; ++i)
          tc::store4(s_a, kPieceA, tc::tile_offset(r0 + 16 * i, q), tc::split4(next[i]));
        tc::publish_operands();
        tc::fence_before_barrier();                         // everybody has read the sums of two tiles ago
        ok = __syncthreads_and(ok);
        if (!ok) {
          failed = chunk > 0 ? tile : before;
          goto last;
        }
        // the next step's rows arrive under the products and the stores
        const bool last = chunk + 1 == p.chunks;
        const int64_t next_tile = last ? tile + walkers : tile;
        if (next_tile < tiles) load(next_tile, last ? 0 : chunk + 1);
        if (p.ahead > 0 && tid == 0 && chunk == 0 && tile_col == 0)        // the neighbours read the same rows
          for (int src = 0; src < p.sources; ++src)
            tc::prefetch_rows(p.a[src], (tile + p.ahead * walkers) * kRows, kRows, p.rows, p.red);
        if (chunk == 0 && before >= 0) finish(before, tmem + (sums == tmem ? kHalf : 0));
        ok = tc::wait(s_done, phase);
        phase ^= 1;
      }
      tc::fence_after_barrier();
      before = tile;
      sums = tmem + (sums == tmem ? kHalf : 0);
    }
    if (!__syncthreads_and(ok)) failed = before;
  last:
    if (failed >= 0) give_up(p, out, c0, failed, walkers);
    else if (before >= 0) finish(before, tmem + (sums == tmem ? kHalf : 0));
  }
finished:
  tc::fence_before_barrier();
  __syncthreads();
  if (warp == 0) {
    if (failed >= 0) tc::wait(s_done, phase ^ 1);           // products that still run write to the memory given back
    tc::release<2 * kHalf>(tmem);
  }
}

template <bool PLAIN, bool LONG>
int launch_part(SplitGemm& p, cudaStream_t stream) {
  const int rc = allow_shared_memory<split_gemm_kernel<PLAIN, LONG>>(split_gemm_smem(LONG ? kMostChunks : 2));
  if (rc != TGT_OK) return rc;
  p.big_sums = (p.chunks + 1) / 2;
  p.col_tiles = (p.cols + kCols - 1) / kCols;
  const int64_t tiles = (p.rows + kRows - 1) / kRows;
  const int resident = LONG ? 1 : 2;               // by shared memory, and tensor memory has 512 columns
  const int across = p.col_tiles * p.outputs;
  int64_t walkers = int64_t(sm_count()) * resident / across;
  if (walkers < 1) walkers = 1;
  if (walkers > tiles) walkers = tiles;
  split_gemm_kernel<PLAIN, LONG><<<unsigned(walkers * across), kThreads, split_gemm_smem(p.chunks), stream>>>(p);
  TGT_CHECK_CUDA(cudaGetLastError());
  return TGT_OK;
}

int launch_split_gemm(const LinearRows& of, int* expired, cudaStream_t stream) {
  const int chunks = (of.red + kChunk - 1) / kChunk * of.sources, parts = (chunks + kMostChunks - 1) / kMostChunks;
  for (int part = 0; part < parts; ++part) {
    SplitGemm p{};
    static_cast<LinearRows&>(p) = of;
    p.first = chunks * part / parts;
    p.chunks = chunks * (part + 1) / parts - p.first;
    p.onto = part > 0;
    p.expired = expired;
    // Two tiles, past the one on its way into registers.  64 x 64 at 320,000 rows 40.4 -> 38.4 us, 128 x 128 119 -> 106, its three
    // gradients (one tile: six chunks take long enough) 429 -> 368
    if (of.rows * of.red * 4 * of.sources >= tc::kPrefetchFrom) p.ahead = p.chunks > 2 ? 1 : 2;
    if (part + 1 < parts) {            // what follows the sum is for the last part
      for (const float*& b : p.bias) b = nullptr;
      p.act = p.gate_act = TGT_ACT_NONE;
      p.pre = nullptr;
      p.gate = p.add = nullptr;
    }
    const bool plain = is_plain(p);
    const int rc = p.chunks > 2 ? (plain ? launch_part<true, true>(p, stream) : launch_part<false, true>(p, stream))
                                : (plain ? launch_part<true, false>(p, stream) : launch_part<false, false>(p, stream));
    if (rc != TGT_OK) return rc;
  }
  return TGT_OK;
}

bool shape_supported(int reduce, int cols) {
  return reduce >= 4 && reduce % 4 == 0 && reduce <= 1024 && cols >= 4 && cols % 4 == 0 && cols <= 1024;
}

}  // namespace
}  // namespace tgt

extern "C" int tgt_linear_rows(const float* a, const float* w, const float* bias, int64_t rows, int reduce, int cols,
                               float* c, void* stream) {
  return tgt_linear_rows_multi(a, &w, &bias, 1, rows, reduce, cols, TGT_ACT_NONE, nullptr, nullptr, &c, stream);
}

extern "C" int tgt_linear_rows_multi(const float* a, const float* const* w, const float* const* bias, int count, int64_t rows,
                                     int reduce, int cols, int act, float* pre, const float* add, float* const* c,
                                     void* stream_) {
  using namespace tgt;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  TGT_CHECK_ARG(rows >= 0, "rows must be >= 0");
  TGT_CHECK_ARG(count >= 1 && count <= kMostProducts, "count must be 1 to %d", kMostProducts);
  TGT_CHECK_ARG(act == TGT_ACT_NONE || act == TGT_ACT_RELU || act == TGT_ACT_GELU, "act is none of TGT_ACT_*");
  TGT_CHECK_ARG(count == 1 || (act == TGT_ACT_NONE && !pre && !add), "act, pre and add are for one product");
  if (!shape_supported(reduce, cols))
    return set_error(TGT_ERR_UNSUPPORTED, "reduce=%d cols=%d: both must be multiples of 4, at most 1024", reduce, cols);
  if (rows == 0) return TGT_OK;
  int* expired = nullptr;
  const int rc = expired_wait_word(&expired);
  if (rc != TGT_OK) return rc;
  TGT_CHECK_ARG(a && w && bias && c, "a, w, bias and c must not be null");
  TGT_CHECK_ARG(aligned16(a) && aligned16(pre) && aligned16(add), "tensors must be 16-byte aligned");
  LinearRows p{};
  p.a[0] = a;
  for (int i = 0; i < count; ++i) {
    TGT_CHECK_ARG(w[i] && c[i], "a, w and c must not be null");
    TGT_CHECK_ARG(aligned16(w[i]) && aligned16(bias[i]) && aligned16(c[i]), "tensors must be 16-byte aligned");
    p.w[i] = w[i]; p.bias[i] = bias[i]; p.c[i] = c[i];
  }
  p.rows = rows; p.red = reduce; p.cols = cols; p.sources = 1; p.outputs = count;
  p.act = act; p.pre = pre; p.add = add;
  return few_rows(rows, cols * count) ? linear_few_rows(p, stream) : launch_split_gemm(p, expired, stream);
}

extern "C" int tgt_linear_input_grad(const float* dy, const float* w, int64_t rows, int out_features, int in_features,
                                     float* dx, void* stream) {
  return tgt_linear_input_grad_multi(&dy, &w, 1, rows, out_features, in_features, TGT_ACT_NONE, nullptr, dx, stream);
}

extern "C" int tgt_linear_input_grad_multi(const float* const* dy, const float* const* w, int count, int64_t rows,
                                           int out_features, int in_features, int act, const float* gate, float* dx,
                                           void* stream_) {
  using namespace tgt;
  TGT_CHECK_ARG(rows >= 0, "rows must be >= 0");
  TGT_CHECK_ARG(count >= 1 && count <= kMostProducts, "count must be 1 to %d", kMostProducts);
  TGT_CHECK_ARG(act == TGT_ACT_NONE || act == TGT_ACT_RELU || act == TGT_ACT_GELU, "act is none of TGT_ACT_*");
  TGT_CHECK_ARG((act == TGT_ACT_NONE) == (gate == nullptr) || rows == 0, "act and gate disagree");
  if (!shape_supported(out_features, in_features))
    return set_error(TGT_ERR_UNSUPPORTED, "out_features=%d in_features=%d: both must be multiples of 4, at most 1024",
                     out_features, in_features);
  if (rows == 0) return TGT_OK;
  int* expired = nullptr;
  const int rc = expired_wait_word(&expired);
  if (rc != TGT_OK) return rc;
  TGT_CHECK_ARG(dy && w && dx, "dy, w and dx must not be null");
  TGT_CHECK_ARG(aligned16(dx) && aligned16(gate), "tensors must be 16-byte aligned");
  LinearRows p{};
  for (int i = 0; i < count; ++i) {
    TGT_CHECK_ARG(dy[i] && w[i], "dy, w and dx must not be null");
    TGT_CHECK_ARG(aligned16(dy[i]) && aligned16(w[i]), "tensors must be 16-byte aligned");
    p.a[i] = dy[i]; p.w[i] = w[i];
  }
  p.c[0] = dx;
  p.rows = rows; p.red = out_features; p.cols = in_features; p.sources = count; p.outputs = 1; p.transposed = true;
  p.gate_act = act; p.gate = gate;
  return launch_split_gemm(p, expired, static_cast<cudaStream_t>(stream_));
}

namespace tgt {
namespace {

// A wait as the products' kernels have it, for an arrival that never comes.
__global__ void expire_wait_kernel(int* expired) {
  __shared__ uint64_t s_bar;
  tc::barrier_init(&s_bar);
  if (!tc::wait(&s_bar, 0)) tc::report_expired_wait(expired);
}

}  // namespace
}  // namespace tgt

extern "C" int tgt_debug_expire_wait(void* stream) {
  using namespace tgt;
  int* expired = nullptr;
  const int rc = expired_wait_word(&expired);
  if (rc != TGT_OK) return rc;
  expire_wait_kernel<<<1, 1, 0, static_cast<cudaStream_t>(stream)>>>(expired);
  TGT_CHECK_CUDA(cudaGetLastError());
  return TGT_OK;
}
