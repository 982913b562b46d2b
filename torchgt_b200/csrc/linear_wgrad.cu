// Weight and bias gradient of a narrow nn.Linear over many rows: dW[o][i] = sum_r dY[r][o] X[r][i],
// db[o] = sum_r dY[r][o], fp32.  The graph transformers' projections are 64 x 64 (128 x 64 for the node
// encoder) over 64,000 to 870,000 rows (models/graphormer_dist_node_level.py:241-245,281-286,343: linear_q/k/v,
// output_layer, the two FFN layers, node_encoder): a product with a tiny result and a very long reduction.
//
// Every CTA walks its share of the rows in chunks of 64, splits both operands into three bf16 pieces on their way into
// shared memory (tensor_core.cuh) and keeps a 64 x 64 tile of dW in tensor memory; dY and X are both read as they lie,
// rows being the reduction.  Tensor cores round a running sum towards zero at every step, so the large products are
// drained after every chunk and added in fp32 registers; the small ones, 2^-8 of them, stay till the end.  The CTAs'
// tiles are then added in a fixed order by a second kernel.  No atomics: results are bitwise reproducible.
//
// us back to back with the sums, here | FMA kernel that was here: 320,000 rows of 64 x 64 50 | 66 (a copy of the same bytes:
// 25), 64 x 128 and 128 x 64 80 | 121, three gradients of one input 110; 64,001 rows 18 | 19, three 29.  Relative error against
// 64 bits at 320,000 rows 1.5e-7, the FMA kernel's 4.4e-7.
#include "tensor_core.cuh"

namespace tgt {
namespace {

constexpr int kMostGrads = 3;                   // products that share x
constexpr int kWgTile = 64;                     // outputs and inputs per tile
constexpr int kWgThreads = 256;
constexpr int kWgChunk = 64;                    // rows staged at a time
constexpr int kWgPiece = kWgChunk * 128;        // bytes of one piece of a chunk, 64 columns wide
constexpr int kWgTmemCols = 256;

struct WgradParams {
  const float* dy[kMostGrads];   // [rows, out]
  const float* x;                // [rows, in]
  float* partial;                // [gridDim.x][count][out * in + out]
  int64_t rows;
  int in, out, count;
  int* expired;                  // expired_wait_word
};

// Where a sum of pieces is not finite (an operand is not, or a sum passes the range of fp32) it says no more than that.  The
// CTA sums its tile again over its rows with FMAs, four outputs x four inputs a thread, and replaces those elements.  (320,000
// rows of 64 x 64 with one NaN 180 us, with a thread per element 7.1 ms; 64,001 of 1024 x 1024 12 ms and 0.98 s.)
__device__ __noinline__ void sum_again(const WgradParams& p, const float* dy, int o0, int i0, float* out) {
  const int o = o0 + 4 * (threadIdx.x / 16), i = i0 + 4 * (threadIdx.x % 16);
  if (o >= p.out || i >= p.in) return;
  float s[4][4] = {};
  const int64_t chunks = (p.rows + kWgChunk - 1) / kWgChunk;
  for (int64_t chunk = blockIdx.x; chunk < chunks; chunk += gridDim.x) {
    const int64_t row = chunk * kWgChunk;
    const int n = int(min(p.rows - row, int64_t(kWgChunk)));
    const float *a = dy + row * p.out + o, *b = p.x + row * p.in + i;
#pragma unroll 4
    for (int r = 0; r < n; ++r, a += p.out, b += p.in) {
      const float4 y = __ldg(reinterpret_cast<const float4*>(a)), x = __ldg(reinterpret_cast<const float4*>(b));
      const float yv[4] = {y.x, y.y, y.z, y.w}, xv[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int l = 0; l < 4; ++l) s[j][l] = fmaf(yv[j], xv[l], s[j][l]);
    }
  }
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      float* at = out + int64_t(o + j) * p.in + i + l;
      if (!(fabsf(*at) < __int_as_float(0x7f800000))) *at = s[j][l];
    }
}

__global__ void __launch_bounds__(kWgThreads, 2) linear_wgrad_kernel(const __grid_constant__ WgradParams p) {
  extern __shared__ __align__(1024) uint8_t s_base[];
  const uint32_t s_dy = tc::smem_address(s_base);            // [2][dy's pieces, x's pieces]
  uint64_t* const s_done = reinterpret_cast<uint64_t*>(s_base + 12 * kWgPiece);
  uint32_t* const s_tmem = reinterpret_cast<uint32_t*>(s_done + 2);
  const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
  const int tiles_in = (p.in + 63) / 64;
  const int tile = blockIdx.y / p.count, which = blockIdx.y % p.count;    // neighbours read the same rows of x
  const int o0 = tile / tiles_in * 64, i0 = tile % tiles_in * 64;
  const float* const from = p.dy[which];
  const int64_t chunks = (p.rows + kWgChunk - 1) / kWgChunk;
  if (warp == 0) tc::allocate<kWgTmemCols>(s_tmem);
  if (tid == 32) {
    tc::barrier_init(s_done);
    tc::barrier_init(s_done + 1);
  }

  const int q = 4 * (tid % 16), r0 = tid / 16;
  float4 dy[kWgChunk / 16], x[kWgChunk / 16];
  const bool has_dy = o0 + q < p.out, has_x = i0 + q < p.in;
  auto load = [&](int64_t chunk) {
    const int64_t row = chunk * kWgChunk + r0;
    const float *a = from + row * p.out + o0 + q, *b = p.x + row * p.in + i0 + q;
    const int64_t step_a = int64_t(16) * p.out, step_b = int64_t(16) * p.in;
    const bool whole = (chunk + 1) * kWgChunk <= p.rows;
#pragma unroll
    for (int i = 0; i < kWgChunk / 16; ++i, a += step_a, b += step_b) {
      const bool live = whole || row + 16 * i < p.rows;
      const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
      dy[i] = live && has_dy ? __ldg(reinterpret_cast<const float4*>(a)) : zero;
      x[i] = live && has_x ? __ldg(reinterpret_cast<const float4*>(b)) : zero;
    }
  };
  float4 bias = make_float4(0.f, 0.f, 0.f, 0.f);
  float main_sum[32];     // of warps 0, 1, 4 and 5: row 32 (warp % 4) + lane, columns 32 (warp / 4) ..
#pragma unroll
  for (int j = 0; j < 32; ++j) main_sum[j] = 0.f;
  int64_t chunk = blockIdx.x;
  if (chunk < chunks) load(chunk);
  tc::fence_before_barrier();
  __syncthreads();
  tc::fence_after_barrier();
  const uint32_t tmem = *s_tmem;
  const uint32_t mine = tmem + (uint32_t(warp % 4 * 32) << 16) + warp / 4 * 32;
  bool ok = true;
  // A chunk's products run under the split of the next one (two buffers) and under the draining of the last one's large
  // products (two places in tensor memory).  Waits alternate over two barriers.
  auto drain = [&](int n) {                        // large products of this CTA's n-th chunk, counted from 0
    ok = tc::wait(s_done + n % 2, n / 2 % 2) && ok;
    tc::fence_after_barrier();
    if (warp % 4 < 2) {
#pragma unroll
      for (int j = 0; j < 32; j += 16) {
        uint32_t v[16];
        tc::read16(mine + n % 2 * 64 + j, v);
        tc::reads_done();
#pragma unroll
        for (int a = 0; a < 16; ++a) main_sum[j + a] += __uint_as_float(v[a]);
      }
    }
  };
  int n = 0;
  for (; chunk < chunks; chunk += gridDim.x, ++n) {
    const uint32_t b_dy = s_dy + n % 2 * (6 * kWgPiece), b_x = b_dy + 3 * kWgPiece;
#pragma unroll
    for (int i = 0; i < kWgChunk / 16; ++i) {
      tc::store4(b_dy, kWgPiece, tc::tile_offset(r0 + 16 * i, q), tc::split4(dy[i]));
      tc::store4(b_x, kWgPiece, tc::tile_offset(r0 + 16 * i, q), tc::split4(x[i]));
      bias.x += dy[i].x; bias.y += dy[i].y; bias.z += dy[i].z; bias.w += dy[i].w;
    }
    tc::publish_operands();
    tc::fence_before_barrier();
    ok = __syncthreads_and(ok);
    if (!ok) break;
    if (tid == 64) {                                 // of a warp that does not drain
      tc::fence_after_barrier();
      constexpr uint32_t one = tc::instruction(128, 64, true, true);
#pragma unroll
      for (int k = 0; k < kWgChunk / 16; ++k) {
        const uint64_t dy12 = tc::mn_major(b_dy + 2048 * k, kWgPiece), dy23 = tc::mn_major(b_dy + kWgPiece + 2048 * k, kWgPiece);
        const uint64_t x1 = tc::mn_major(b_x + 2048 * k, kWgPiece), x2 = tc::mn_major(b_x + kWgPiece + 2048 * k, kWgPiece),
                       x3 = tc::mn_major(b_x + 2 * kWgPiece + 2048 * k, kWgPiece);
        // lanes 0..63 | 64..127 of columns 0..63 or 64..127: dy1 x1 | dy2 x1 (not used), afresh in every chunk, of columns
        // 128..191: dy1 x2 + dy1 x3 + dy2 x1 | dy2 x2 + dy2 x3 + dy3 x1
        tc::multiply(tmem + n % 2 * 64, dy12, x1, one, k > 0);
        tc::multiply(tmem + 128, dy12, x2, one, n + k > 0);
        tc::multiply(tmem + 128, dy12, x3, one, true);
        tc::multiply(tmem + 128, dy23, x1, one, true);
      }
      tc::commit(s_done + n % 2);
    }
    if (chunk + gridDim.x < chunks) load(chunk + gridDim.x);
    // 64 x 64 at 320,000 rows 48.5 -> 44.1 us, with the sums; of the CTAs that read the same rows one each
    if (tid == 0 && p.rows * (p.in + int64_t(p.count) * p.out) * 4 >= tc::kPrefetchFrom) {
      const int64_t ahead = (chunk + 2 * int64_t(gridDim.x)) * kWgChunk;
      if (tile == 0) tc::prefetch_rows(from, ahead, kWgChunk, p.rows, p.out);
      if (blockIdx.y == 0) tc::prefetch_rows(p.x, ahead, kWgChunk, p.rows, p.in);
    }
    if (n > 0) drain(n - 1);
  }
  if (n > 0) drain(n - 1);
  // the small products of lanes 64..127 go to the warps that hold the same rows of the large ones
  ok = __syncthreads_and(ok);
  if (!ok && tid == 0) tc::report_expired_wait(p.expired);
  float* const s_small = reinterpret_cast<float*>(s_base);       // [64][65]
  float4* const s_bias = reinterpret_cast<float4*>(s_base + 64 * 65 * 4);   // [16][16]
  if (warp % 4 >= 2) {                                           // every CTA has a chunk: wgrad_grid
#pragma unroll
    for (int j = 0; j < 32; j += 16) {
      uint32_t v[16];
      tc::read16(mine + 128 + j, v);
      tc::reads_done();
#pragma unroll
      for (int a = 0; a < 16; ++a) s_small[(warp % 4 * 32 - 64 + lane) * 65 + warp / 4 * 32 + j + a] = __uint_as_float(v[a]);
    }
  }
  s_bias[r0 * 16 + tid % 16] = bias;
  __syncthreads();
  float* out = p.partial + (int64_t(blockIdx.x) * p.count + which) * (int64_t(p.out) * p.in + p.out);
  bool again = false;
  if (warp % 4 < 2) {
    const int row = warp % 4 * 32 + lane;
#pragma unroll
    for (int j = 0; j < 32; j += 16) {
      uint32_t v[16];
      tc::read16(mine + 128 + j, v);
      tc::reads_done();
#pragma unroll
      for (int a = 0; a < 16; a += 4) {
        const int col = warp / 4 * 32 + j + a;
        if (o0 + row >= p.out || i0 + col >= p.in) continue;
        float f[4];
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          f[b] = main_sum[j + a + b] + (__uint_as_float(v[a + b]) + s_small[row * 65 + col + b]);
          if (!ok) f[b] = __int_as_float(0x7fffffff);
          again = again || (ok && !(fabsf(f[b]) < __int_as_float(0x7f800000)));
        }
        *reinterpret_cast<float4*>(out + int64_t(o0 + row) * p.in + i0 + col) = make_float4(f[0], f[1], f[2], f[3]);
      }
      __syncwarp();
    }
  }
  if (i0 == 0 && tid < 64 && o0 + tid < p.out) {
    float s = 0.f;
    for (int r = 0; r < 16; ++r) s += reinterpret_cast<const float*>(s_bias)[r * 64 + tid];
    if (!ok) s = __int_as_float(0x7fffffff);
    out[int64_t(p.out) * p.in + o0 + tid] = s;
  }
  tc::fence_before_barrier();
  again = __syncthreads_or(again);                   // all reads of tensor memory are done, the tile is written
  if (warp == 0) tc::release<kWgTmemCols>(tmem);
  if (again) sum_again(p, from, o0, i0, out);
}

struct WgradSumParams {
  const float* partial;
  float* dw[kMostGrads];
  float* db[kMostGrads];         // may be null
  int ctas, count, n_w, n_b;
};

// dw[j] = sum over CTAs of partial[cta][j], db likewise; sum_partials: fixed association.
__global__ void __launch_bounds__(kPartialSumThreads) linear_wgrad_sum_kernel(const __grid_constant__ WgradSumParams p) {
  __shared__ float s_part[16][32];
  const int i = blockIdx.x * 32 + threadIdx.x % 32, each = p.n_w + p.n_b;
  const bool live = i < p.count * each;
  const float s = sum_partials(p.partial, p.ctas, int64_t(p.count) * each, i, live, s_part);
  if (threadIdx.x < 32 && live) {
    const int which = i / each, j = i % each;
    if (j < p.n_w) p.dw[which][j] = s;
    else if (p.db[which] != nullptr) p.db[which][j - p.n_w] = s;
  }
}

// inputs in whole tiles of 64; outputs any multiple of 4 (a classifier head of 40 classes, say): the last tile
// of outputs is padded with zero columns that are never stored
bool wgrad_supported(int in, int out) {
  return in >= kWgTile && in % kWgTile == 0 && in <= 1024 && out >= 4 && out % 4 == 0 && out <= 1024;
}
int wgrad_out_tiles(int out) { return (out + kWgTile - 1) / kWgTile; }
constexpr int kWgSmem = 12 * kWgPiece + 32;     // two buffers, two barriers and the tensor memory's address

int wgrad_grid(int64_t rows, int in, int out, int count) {
  const int tiles = (in / kWgTile) * wgrad_out_tiles(out) * count;
  const int64_t chunks = (rows + kWgChunk - 1) / kWgChunk;
  // The two CTAs an SM holds, over all tiles; one where that leaves them a chunk or two each, so that the sums have half as
  // many tiles to read (16,384 rows of 64 x 64: 12.7 us, with 256 CTAs 14.8)
  int64_t g = int64_t(sm_count()) * (chunks * tiles > 4 * int64_t(sm_count()) ? 2 : 1) / tiles;
  if (g < 1) g = 1;
  if (g > chunks) g = chunks < 1 ? 1 : chunks;
  return int(g);
}

}  // namespace
}  // namespace tgt

extern "C" int tgt_linear_wgrad_scratch_bytes(int64_t rows, int in_features, int out_features, size_t* bytes) {
  return tgt_linear_wgrad_multi_scratch_bytes(1, rows, in_features, out_features, bytes);
}

extern "C" int tgt_linear_wgrad_multi_scratch_bytes(int count, int64_t rows, int in_features, int out_features, size_t* bytes) {
  using namespace tgt;
  TGT_CHECK_ARG(bytes != nullptr, "bytes is null");
  TGT_CHECK_ARG(rows >= 0, "rows must be >= 0");
  TGT_CHECK_ARG(count >= 1 && count <= kMostGrads, "count must be 1 to %d", kMostGrads);
  if (!wgrad_supported(in_features, out_features))
    return set_error(TGT_ERR_UNSUPPORTED, "in_features=%d out_features=%d: in_features must be a multiple of 64, out_features of 4, both at most 1024",
                     in_features, out_features);
  *bytes = size_t(wgrad_grid(rows, in_features, out_features, count)) * count *
           (size_t(in_features) * out_features + out_features) * sizeof(float);
  return TGT_OK;
}

extern "C" int tgt_linear_wgrad(const float* dy, const float* x, int64_t rows, int in_features, int out_features,
                                float* dw, float* db, void* scratch, size_t scratch_bytes, void* stream) {
  return tgt_linear_wgrad_multi(&dy, x, 1, rows, in_features, out_features, &dw, &db, scratch, scratch_bytes, stream);
}

extern "C" int tgt_linear_wgrad_multi(const float* const* dy, const float* x, int count, int64_t rows, int in_features,
                                      int out_features, float* const* dw, float* const* db, void* scratch,
                                      size_t scratch_bytes, void* stream_) {
  using namespace tgt;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  TGT_CHECK_ARG(rows >= 0, "rows must be >= 0");
  TGT_CHECK_ARG(count >= 1 && count <= kMostGrads, "count must be 1 to %d", kMostGrads);
  if (!wgrad_supported(in_features, out_features))
    return set_error(TGT_ERR_UNSUPPORTED, "in_features=%d out_features=%d: in_features must be a multiple of 64, out_features of 4, both at most 1024",
                     in_features, out_features);
  TGT_CHECK_ARG(dy && dw && db, "dy, dw and db must not be null");
  const size_t n_w = size_t(in_features) * out_features;
  WgradParams p{};
  WgradSumParams q{};
  for (int i = 0; i < count; ++i) {
    TGT_CHECK_ARG(dw[i] != nullptr, "dw must not be null");
    TGT_CHECK_ARG(rows == 0 || (dy[i] && x), "dy and x must not be null");
    TGT_CHECK_ARG(aligned16(dy[i]) && aligned16(dw[i]), "tensors must be 16-byte aligned");
    p.dy[i] = dy[i];
    q.dw[i] = dw[i]; q.db[i] = db[i];
  }
  if (rows == 0) {
    for (int i = 0; i < count; ++i) {
      TGT_CHECK_CUDA(cudaMemsetAsync(dw[i], 0, n_w * sizeof(float), stream));
      if (db[i] != nullptr) TGT_CHECK_CUDA(cudaMemsetAsync(db[i], 0, size_t(out_features) * sizeof(float), stream));
    }
    return TGT_OK;
  }
  int rc = expired_wait_word(&p.expired);
  if (rc != TGT_OK) return rc;
  TGT_CHECK_ARG(aligned16(x) && aligned16(scratch), "tensors must be 16-byte aligned");
  const int grid = wgrad_grid(rows, in_features, out_features, count);
  const size_t need = size_t(grid) * count * (n_w + out_features) * sizeof(float);
  if (scratch == nullptr || scratch_bytes < need)
    return set_error(TGT_ERR_WORKSPACE, "scratch holds %zu bytes, %zu needed", scratch_bytes, need);
  rc = allow_shared_memory<linear_wgrad_kernel>(kWgSmem);
  if (rc != TGT_OK) return rc;
  p.x = x; p.partial = static_cast<float*>(scratch); p.rows = rows; p.in = in_features; p.out = out_features; p.count = count;
  const dim3 g(grid, (in_features / kWgTile) * wgrad_out_tiles(out_features) * count);
  linear_wgrad_kernel<<<g, kWgThreads, kWgSmem, stream>>>(p);
  q.partial = p.partial; q.ctas = grid; q.count = count; q.n_w = int(n_w); q.n_b = out_features;
  const int n = count * (q.n_w + q.n_b);
  linear_wgrad_sum_kernel<<<(n + 31) / 32, kPartialSumThreads, 0, stream>>>(q);
  TGT_CHECK_CUDA(cudaGetLastError());
  return TGT_OK;
}
