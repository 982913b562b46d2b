// Narrow fp32 nn.Linear over a few thousand rows: Y[r][c] = sum_k X[r][k] W[c][k] + b[c], full fp32 products and sums
// (models/graphormer_dist_node_level.py:241-245,281-286 and models/gt_dist_node_level.py:189-193,232-236).  More rows go
// to the tensor cores (linear_mma.cu); down here a call is a few microseconds of latency, which tiles of 32 rows on four
// CTAs per SM keep short.
//
// One CTA keeps the 64 weight rows of its column tile in shared memory and walks row tiles, the next tile's rows
// arriving by asynchronous copies under the arithmetic.  A thread owns 2 rows x 8 columns and walks k four at a time:
// the two halves of a 16-byte shared-memory read are the operand pairs of the packed FMA (fma.rn.f32x2: even and odd k
// in separate sums), so no operand is ever moved or duplicated.  Rows are 68 floats apart in shared memory (eight rows'
// pieces fall into different banks) and weight rows are permuted so that a thread's columns are two runs of four, stored
// 16 bytes at a time.  4,097 rows of 64 x 64 in 4.2 us (the library's product and its pass that adds the bias: 6.4 us).
#include "linear_rows.cuh"

namespace tgt {
namespace {

constexpr int kLrThreads = 128;
constexpr int kLrRows = 32;     // rows of a tile
constexpr int kLrTile = 64;     // columns of a tile, and reduction elements staged at a time
constexpr int kLrPitch = 68;    // floats between rows in shared memory

__device__ __forceinline__ void lr_copy_async(float* smem_dst, const float* src, bool live) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(uint32_t(__cvta_generic_to_shared(smem_dst))),
               "l"(src), "r"(live ? 16 : 0)
               : "memory");
}

// a pair of fp32 sums advanced by a pair of products, each rounded as fmaf rounds
__device__ __forceinline__ void fma_pair(uint64_t& acc, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ float pair_sum(uint64_t v) {
  return __uint_as_float(uint32_t(v)) + __uint_as_float(uint32_t(v >> 32));
}

// weight row c of a tile lives in slot(c): thread column tx reads slots tx + 8 j (j = 0..7) and owns columns
// 4 tx .. 4 tx + 3 and 32 + 4 tx .. 32 + 4 tx + 3
__device__ __forceinline__ int lr_slot(int c) { return (c % 32) / 4 + 8 * (4 * (c / 32) + c % 4); }

template <bool PLAIN>   // nothing but a bias is added to the sums
__global__ void __launch_bounds__(kLrThreads, 4) linear_rows_kernel(const __grid_constant__ LinearRows p) {
  constexpr int TM = kLrRows / 16, BM = kLrRows;
  extern __shared__ __align__(16) float s_mem[];
  float* const s_x = s_mem;                          // [2][BM][kLrPitch]
  float* const s_w = s_mem + 2 * BM * kLrPitch;      // [1 or 2][64][kLrPitch]
  const int tid = threadIdx.x, tx = tid % 8, ty = tid / 8;
  const int out = blockIdx.z, c0 = blockIdx.y * kLrTile;
  const float* const a = p.a[0];
  const float* const weight = p.w[out];
  const int chunks = (p.red + kLrTile - 1) / kLrTile;
  const int64_t tiles = (p.rows + BM - 1) / BM;

  auto stage = [&](int64_t tile, int chunk, int buf, bool weights) {
    const int k0 = chunk * kLrTile;
    float* x = s_x + buf * (BM * kLrPitch);
#pragma unroll
    for (int u = tid; u < BM * 16; u += kLrThreads) {
      const int r = u / 16, q = 4 * (u % 16);
      const int64_t row = tile * BM + r;
      const bool live = row < p.rows && k0 + q < p.red;     // what is not there is zero in both operands
      lr_copy_async(x + r * kLrPitch + q, live ? a + row * p.red + k0 + q : a, live);
    }
    if (!weights) return;
    float* w = s_w + (chunks > 1 ? buf * (kLrTile * kLrPitch) : 0);
    for (int u = tid; u < kLrTile * 16; u += kLrThreads) {
      const int r = u / 16, q = 4 * (u % 16);
      const bool live = c0 + r < p.cols && k0 + q < p.red;
      lr_copy_async(w + lr_slot(r) * kLrPitch + q, live ? weight + int64_t(c0 + r) * p.red + k0 + q : weight, live);
    }
  };

  float4 b[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int col = c0 + 32 * h + 4 * tx;
    b[h] = p.bias[out] != nullptr && col < p.cols ? __ldg(reinterpret_cast<const float4*>(p.bias[out] + col))
                                                  : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  float* const c = p.c[out];
  auto finish = [&](int64_t row, int col, const float4& v) {
    if (PLAIN) {
      const float4& add = col < c0 + 32 ? b[0] : b[1];
      *reinterpret_cast<float4*>(c + row * p.cols + col) = make_float4(v.x + add.x, v.y + add.y, v.z + add.z, v.w + add.w);
    } else {
      finish_values(p, out, row, col, v);
    }
  };
  uint64_t acc[TM][8];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0;

  int64_t tile = blockIdx.x;
  int chunk = 0, buf = 0;
  if (tile < tiles) stage(tile, 0, 0, true);
  asm volatile("cp.async.commit_group;" ::: "memory");
  while (tile < tiles) {                             // the same for every thread of the CTA
    const int next_chunk = chunk + 1 == chunks ? 0 : chunk + 1;
    const int64_t next_tile = next_chunk == 0 ? tile + gridDim.x : tile;
    if (next_tile < tiles) stage(next_tile, next_chunk, buf ^ 1, chunks > 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 1;" ::: "memory");   // this step's copies have landed
    __syncthreads();
    const float* x = s_x + buf * (BM * kLrPitch) + ty * kLrPitch;
    const float* w = s_w + (chunks > 1 ? buf * (kLrTile * kLrPitch) : 0) + tx * kLrPitch;
#pragma unroll 2
    for (int k = 0; k < kLrTile; k += 4) {
      ulonglong2 wv[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) wv[j] = *reinterpret_cast<const ulonglong2*>(w + 8 * j * kLrPitch + k);
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const ulonglong2 xv = *reinterpret_cast<const ulonglong2*>(x + 16 * i * kLrPitch + k);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          fma_pair(acc[i][j], xv.x, wv[j].x);
          fma_pair(acc[i][j], xv.y, wv[j].y);
        }
      }
    }
    if (next_chunk == 0) {
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const int64_t row = tile * BM + ty + 16 * i;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int col = c0 + 32 * h + 4 * tx;
          if (row < p.rows && col < p.cols)
            finish(row, col, make_float4(pair_sum(acc[i][4 * h]), pair_sum(acc[i][4 * h + 1]),
                                         pair_sum(acc[i][4 * h + 2]), pair_sum(acc[i][4 * h + 3])));
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0;
      }
    }
    __syncthreads();                                 // the next step's copies overwrite this buffer
    tile = next_tile;
    chunk = next_chunk;
    buf ^= 1;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

}  // namespace

int linear_few_rows(const LinearRows& p, cudaStream_t stream) {
  const int col_tiles = (p.cols + kLrTile - 1) / kLrTile, chunks = (p.red + kLrTile - 1) / kLrTile;
  const int smem = (2 * kLrRows + kLrTile * (chunks > 1 ? 2 : 1)) * kLrPitch * int(sizeof(float));
  constexpr int kMost = (2 * kLrRows + 2 * kLrTile) * kLrPitch * int(sizeof(float));
  const bool plain = is_plain(p);
  const int rc = plain ? allow_shared_memory<linear_rows_kernel<true>>(kMost) : allow_shared_memory<linear_rows_kernel<false>>(kMost);
  if (rc != TGT_OK) return rc;
  const int64_t tiles = (p.rows + kLrRows - 1) / kLrRows;
  int64_t ctas = int64_t(sm_count()) * 4 / (col_tiles * p.outputs);
  if (ctas < 1) ctas = 1;
  if (ctas > tiles) ctas = tiles;
  const dim3 grid(unsigned(ctas), col_tiles, p.outputs);
  if (plain) linear_rows_kernel<true><<<grid, kLrThreads, smem, stream>>>(p);
  else linear_rows_kernel<false><<<grid, kLrThreads, smem, stream>>>(p);
  TGT_CHECK_CUDA(cudaGetLastError());
  return TGT_OK;
}

}  // namespace tgt
