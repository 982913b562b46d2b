// Narrow fp32 nn.Linear over many rows: Y[r][c] = sum_k X[r][k] W[c][k] + b[c], full fp32 products and sums
// (models/graphormer_dist_node_level.py:241-245,281-286 and models/gt_dist_node_level.py:189-193,232-236: 64 x 64 and
// 64 x 128 layers over 4,000 to 870,000 rows).
//
// Bound by the fp32 FMA pipe (64 MACs per 8 bytes moved: 37 us of FMAs against 25 us of traffic at 320,000 rows of
// 64 x 64).  One CTA keeps the 64 weight rows of its column tile in shared memory and walks row tiles, the next
// tile's rows arriving by asynchronous copies under the arithmetic.  A thread owns TM rows x 8 columns and walks k
// four at a time: the two halves of a 16-byte shared-memory read are the operand pairs of the packed FMA
// (fma.rn.f32x2: even and odd k in separate sums), so no operand is ever moved or duplicated.  Rows are 68 floats
// apart in shared memory (eight rows' pieces fall into different banks) and weight rows are permuted so that a
// thread's columns are two runs of four, stored 16 bytes at a time.
//
// 320,000 rows: 64 x 64 in 78 us, 64 x 128 in 140 us (34 and 37 TFLOP/s; the library's product and its pass that adds
// the bias: 195 and about 300 us), relative error against 64 bits 1.1e-7 (the library's 1.4e-7); 4,097 rows of 64 x 64
// in 4.0 us (6.8 us).  The FMA pipe is then 64 % busy with 8 warps per SM; tiles of 64 rows with 4 x 8 values a thread
// and 16 warps per SM take 81 and 149 us, so what is left is not latency.  The input gradient is the library's: the
// same kernel with the weights transposed on their way in took 79 us at 64 x 64 but 142 and 168 us at the 128-wide
// layers, where the library's takes 128 and 135 us.
#include "tgt_common.cuh"

namespace tgt {
namespace {

constexpr int kLrThreads = 128;
constexpr int kLrTile = 64;     // columns of a tile, and reduction elements staged at a time
constexpr int kLrPitch = 68;    // floats between rows in shared memory

struct LinearRowsParams {
  const float* a;      // [rows, red]
  const float* w;      // [cols, red]
  const float* bias;   // [cols] or null
  float* c;            // [rows, cols]
  int64_t rows;
  int red, cols;
};

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

template <int TM>
__global__ void __launch_bounds__(kLrThreads, TM == 8 ? 2 : 4) linear_rows_kernel(const LinearRowsParams p) {
  constexpr int BM = 16 * TM;
  extern __shared__ __align__(16) float s_mem[];
  float* const s_x = s_mem;                          // [2][BM][kLrPitch]
  float* const s_w = s_mem + 2 * BM * kLrPitch;      // [1 or 2][64][kLrPitch]
  const int tid = threadIdx.x, tx = tid % 8, ty = tid / 8;
  const int c0 = blockIdx.y * kLrTile;
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
      lr_copy_async(x + r * kLrPitch + q, live ? p.a + row * p.red + k0 + q : p.a, live);
    }
    if (!weights) return;
    float* w = s_w + (chunks > 1 ? buf * (kLrTile * kLrPitch) : 0);
    for (int u = tid; u < kLrTile * 16; u += kLrThreads) {
      const int r = u / 16, q = 4 * (u % 16);
      const bool live = c0 + r < p.cols && k0 + q < p.red;
      lr_copy_async(w + lr_slot(r) * kLrPitch + q, live ? p.w + int64_t(c0 + r) * p.red + k0 + q : p.w, live);
    }
  };

  float4 b[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int col = c0 + 32 * h + 4 * tx;
    b[h] = p.bias != nullptr && col < p.cols ? __ldg(reinterpret_cast<const float4*>(p.bias + col))
                                             : make_float4(0.f, 0.f, 0.f, 0.f);
  }
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
            *reinterpret_cast<float4*>(p.c + row * p.cols + col) =
                make_float4(pair_sum(acc[i][4 * h]) + b[h].x, pair_sum(acc[i][4 * h + 1]) + b[h].y,
                            pair_sum(acc[i][4 * h + 2]) + b[h].z, pair_sum(acc[i][4 * h + 3]) + b[h].w);
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

template <int TM>
int launch_linear_rows(const LinearRowsParams& p, cudaStream_t stream) {
  constexpr int BM = 16 * TM;
  const int col_tiles = (p.cols + kLrTile - 1) / kLrTile, chunks = (p.red + kLrTile - 1) / kLrTile;
  const int smem = (2 * BM + kLrTile * (chunks > 1 ? 2 : 1)) * kLrPitch * int(sizeof(float));
  static bool raised[kMaxDevices] = {};   // the function's limit is a property of the device; setting it twice is harmless
  const int dev = current_device();
  if (dev < 0) return TGT_ERR_CUDA;
  if (!__atomic_load_n(&raised[dev], __ATOMIC_ACQUIRE)) {
    TGT_CHECK_CUDA(cudaFuncSetAttribute(linear_rows_kernel<TM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (2 * BM + 2 * kLrTile) * kLrPitch * int(sizeof(float))));
    __atomic_store_n(&raised[dev], true, __ATOMIC_RELEASE);
  }
  const int64_t tiles = (p.rows + BM - 1) / BM;
  int64_t ctas = int64_t(sm_count()) * (TM == 8 ? 2 : 4) / col_tiles;
  if (ctas < 1) ctas = 1;
  if (ctas > tiles) ctas = tiles;
  linear_rows_kernel<TM><<<dim3(unsigned(ctas), col_tiles), kLrThreads, smem, stream>>>(p);
  TGT_CHECK_CUDA(cudaGetLastError());
  return TGT_OK;
}

}  // namespace
}  // namespace tgt

extern "C" int tgt_linear_rows(const float* a, const float* w, const float* bias, int64_t rows, int reduce, int cols,
                               float* c, void* stream_) {
  using namespace tgt;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  TGT_CHECK_ARG(rows >= 0, "rows must be >= 0");
  if (reduce < 4 || reduce % 4 != 0 || reduce > 1024 || cols < 4 || cols % 4 != 0 || cols > 1024)
    return set_error(TGT_ERR_UNSUPPORTED, "reduce=%d cols=%d: both must be multiples of 4, at most 1024", reduce, cols);
  if (rows == 0) return TGT_OK;
  TGT_CHECK_ARG(a && w && c, "a, w and c must not be null");
  TGT_CHECK_ARG(aligned16(a) && aligned16(w) && aligned16(bias) && aligned16(c), "tensors must be 16-byte aligned");
  const LinearRowsParams p{a, w, bias, c, rows, reduce, cols};
  // tiles of 128 rows reuse every weight read eight times; with fewer of them than the chip holds at once, tiles of
  // 32 rows occupy it better (4,097 rows of 64 x 64: 33 CTAs of 128 rows, 129 of 32)
  const bool small = (rows + 127) / 128 * ((cols + kLrTile - 1) / kLrTile) < 2 * int64_t(sm_count());
  return small ? launch_linear_rows<2>(p, stream) : launch_linear_rows<8>(p, stream);
}
