// The two kernels behind the products of narrow linear layers and the line between them.
#pragma once

#include "tgt_common.cuh"

namespace tgt {

constexpr int kMostProducts = 3;

// torch's relu and (exact) gelu and the latter's derivative; NaN stays NaN
__device__ __forceinline__ float relu(float x) { return x < 0.f ? 0.f : x; }
__device__ __forceinline__ float normal_cdf(float x) { return 0.5f * (1.f + erff(x * 0.70710678118654752440f)); }
__device__ __forceinline__ float gelu(float x) { return x * normal_cdf(x); }
__device__ __forceinline__ float gelu_slope(float x) {
  return normal_cdf(x) + x * (0.39894228040143267794f * expf(-0.5f * x * x));
}

// C_j[r][c] = f(sum_s sum_k A_s[r][k] B_sj[c][k] + bias_j[c]); one of `sources` (s) and `outputs` (j) is 1.
struct LinearRows {
  const float* a[kMostProducts];      // [rows, red]
  const float* w[kMostProducts];      // [cols, red], or [red, cols] when transposed
  const float* bias[kMostProducts];   // [cols] or null
  float* c[kMostProducts];            // [rows, cols]
  int64_t rows;
  int red, cols;
  int sources, outputs;
  bool transposed;
  bool onto;                          // c holds part of the sums already, they are added to it
  // what is done to a sum on its way out, all of it for a single output only (null / 0: nothing):
  int act;                            // TGT_ACT_*: c = act(sum + bias); pre (may be null) receives sum + bias
  float* pre;
  int gate_act;                       // c = sum * act'(at gate[r][c]); for TGT_ACT_RELU gate is the activation's result
  const float* gate;
  const float* add;                   // c = ... + add[r][c]
};

// nothing but a bias is added to the sums
inline bool is_plain(const LinearRows& p) {
  return !p.onto && p.act == TGT_ACT_NONE && p.pre == nullptr && p.gate_act == TGT_ACT_NONE && p.add == nullptr;
}

// four values of a row
__device__ __forceinline__ void finish_values(const LinearRows& p, int out, int64_t row, int col, float4 v) {
  const int64_t at = row * p.cols + col;
  if (p.onto) {
    const float4 c = *reinterpret_cast<const float4*>(p.c[out] + at);
    v.x += c.x; v.y += c.y; v.z += c.z; v.w += c.w;
  }
  if (p.bias[out] != nullptr) {
    const float4 b = __ldg(reinterpret_cast<const float4*>(p.bias[out] + col));
    v.x += b.x; v.y += b.y; v.z += b.z; v.w += b.w;
  }
  if (p.pre != nullptr) *reinterpret_cast<float4*>(p.pre + at) = v;
  if (p.act == TGT_ACT_RELU) {
    v.x = relu(v.x); v.y = relu(v.y); v.z = relu(v.z); v.w = relu(v.w);
  } else if (p.act == TGT_ACT_GELU) {
    v.x = gelu(v.x); v.y = gelu(v.y); v.z = gelu(v.z); v.w = gelu(v.w);
  }
  if (p.gate_act != 0) {
    const float4 g = __ldg(reinterpret_cast<const float4*>(p.gate + at));
    if (p.gate_act == TGT_ACT_RELU) {
      v.x = g.x <= 0.f ? 0.f : v.x; v.y = g.y <= 0.f ? 0.f : v.y;
      v.z = g.z <= 0.f ? 0.f : v.z; v.w = g.w <= 0.f ? 0.f : v.w;
    } else {
      v.x *= gelu_slope(g.x); v.y *= gelu_slope(g.y); v.z *= gelu_slope(g.z); v.w *= gelu_slope(g.w);
    }
  }
  if (p.add != nullptr) {
    const float4 a = __ldg(reinterpret_cast<const float4*>(p.add + at));
    v.x += a.x; v.y += a.y; v.z += a.z; v.w += a.w;
  }
  *reinterpret_cast<float4*>(p.c[out] + at) = v;
}

// Full fp32 FMAs on tiles of 32 rows (linear_rows.cu): sources == 1, not transposed, not onto.
int linear_few_rows(const LinearRows& p, cudaStream_t stream);

// Tiles of 128 rows x 64 columns that the tensor cores would get; with fewer, the FMA kernel's smaller tiles occupy the
// chip better (us back to back, FMA / tensor cores, 64 x 64: 4,097 rows 4.2 / 6.3, 8,192 rows 6.0 / 6.5, 16,384 rows 10.7 / 6.5;
// 64 x 128 at 8,192 rows, 128 tiles, 8.9 / 6.6).
inline bool few_rows(int64_t rows, int cols) { return (rows + 127) / 128 * ((cols + 63) / 64) < 80; }

}  // namespace tgt
