// Backward of the sparse graph attention, pass B: dK and dV (see sparse_attn_bwd.cuh).
#include "sparse_attn_bwd.cuh"

namespace tgt {
namespace bwd {
namespace {

// ---- pass B: dK and dV --------------------------------------------------------------------------
template <typename T, int W, int LPH, int G, int BIAS>
struct DkvPolicy {
  static constexpr int VEC = Lane<T, W>::kElems;
  static constexpr int NACC = 2 * VEC;  // dK then dV
  static constexpr bool kPairs = sizeof(T) == 2;
  static constexpr bool kPerm = BIAS != kNoBias;
  static constexpr int kUnroll = walk_unroll<T, W, G>();

  const T* __restrict__ q;
  const T* __restrict__ k;
  const T* __restrict__ v;
  const T* __restrict__ dout;
  const float2* __restrict__ stats;
  const float* __restrict__ bias;
  T* __restrict__ dk;
  T* __restrict__ dv;
  float* __restrict__ dbias;   // original edge order, null unless this pass writes it
  int bias_stride, bias_off;
  unsigned row_vecs, cvec, q_vecs, kv_vecs, g_vecs;
  int heads, head;
  bool head_leader, group_leader;
  float inv_scale;

  using Raw = typename Lane<T, W>::Raw;
  struct Operands {
    Raw q, g, k, v;  // packed 16-byte pieces, unpacked where they are used
    float2 st;
    float b;
  };
  struct Scalars {
    float da, wi;
  };

  // `row` is the source (K/V row), `dst` the destination whose Q, dO and statistics are gathered
  __device__ __forceinline__ void load(Operands& o, int row, int dst, int pe) const {
    const unsigned ro = unsigned(row) * kv_vecs + cvec;
    o.q = Lane<T, W>::raw_at(q, unsigned(dst) * q_vecs + cvec);
    o.g = Lane<T, W>::raw_at(dout, unsigned(dst) * g_vecs + cvec);
    o.k = Lane<T, W>::raw_at(k, ro);
    o.v = Lane<T, W>::raw_at(v, ro);
    o.st = __ldg(stats + int64_t(dst) * heads + head);
    o.b = BIAS != kNoBias ? __ldg(bias + int64_t(pe) * bias_stride + bias_off) : 0.f;
  }
  __device__ __forceinline__ void clear(Operands& o) const {
    o.k = o.v = o.q = o.g = Lane<T, W>::raw_zero();
    o.st = make_float2(0.f, 0.f);
    o.b = 0.f;
  }
  __device__ __forceinline__ Scalars prep(const Operands& o, bool valid, int pe) const {
    float a[VEC], b[VEC];
    Lane<T, W>::unpack(o.q, a);
    Lane<T, W>::unpack(o.k, b);
    const float raw = group_sum<LPH>(dot<kPairs>(a, b)) * inv_scale;
    Lane<T, W>::unpack(o.g, a);
    Lane<T, W>::unpack(o.v, b);
    const float gv = group_sum<LPH>(dot<kPairs>(a, b));
    const float wgt = valid ? fast_exp(clamp_score(raw) + o.b) : 0.f;
    const float dt = (gv - o.st.y) * o.st.x * wgt;
    if (BIAS == kBiasGrad) {
      if (bias_stride == 1) {
        const float sum = sum_over_heads<LPH, G>(dt);   // every head's dt sits on all LPH lanes of the head
        if (valid && group_leader) dbias[pe] = sum;
      } else if (valid && head_leader) {
        dbias[int64_t(pe) * bias_stride + head] = dt;
      }
    }
    Scalars s;
    s.da = clamp_passes_grad(raw) ? dt : 0.f;
    s.wi = wgt * o.st.x;
    return s;
  }
  __device__ __forceinline__ void accumulate(float (&acc)[NACC], const Operands& o,
                                             const Scalars& s) const {
    float qf[VEC], gf[VEC];
    Lane<T, W>::unpack(o.q, qf);
    Lane<T, W>::unpack(o.g, gf);
    add_scaled<kPairs, 0>(acc, s.da, qf);
    add_scaled<kPairs, VEC>(acc, s.wi, gf);
  }
  __device__ __forceinline__ void finalize(int row, const float (&acc)[NACC]) const {
    float a[VEC], b[VEC];
#pragma unroll
    for (int j = 0; j < VEC; ++j) {
      a[j] = acc[j] * inv_scale;
      b[j] = acc[VEC + j];
    }
    const unsigned off = unsigned(row) * row_vecs + cvec;
    Lane<T, W>::store_at(dk, off, a);
    Lane<T, W>::store_at(dv, off, b);
  }
  __device__ __forceinline__ void zero_row(int row) const {
    float o[VEC];
#pragma unroll
    for (int j = 0; j < VEC; ++j) o[j] = 0.f;
    const unsigned off = unsigned(row) * row_vecs + cvec;
    Lane<T, W>::store_at(dk, off, o);
    Lane<T, W>::store_at(dv, off, o);
  }
};

template <typename T, int W, int LPH, int G, int BIAS>
__device__ __forceinline__ DkvPolicy<T, W, LPH, G, BIAS> make_dkv_policy(const BwdParams& p) {
  constexpr int VEC = Lane<T, W>::kElems;
  const int c = threadIdx.x % G;
  DkvPolicy<T, W, LPH, G, BIAS> pol;
  pol.q = static_cast<const T*>(p.q);
  pol.k = static_cast<const T*>(p.k);
  pol.v = static_cast<const T*>(p.v);
  pol.dout = static_cast<const T*>(p.dout);
  pol.stats = p.stats;
  pol.bias = p.bias;
  pol.dk = static_cast<T*>(p.dk);
  pol.dv = static_cast<T*>(p.dv);
  pol.dbias = p.dbias_in_dkv ? p.dbias : nullptr;
  pol.head_leader = c % LPH == 0;
  pol.group_leader = c == 0;
  pol.head = blockIdx.y * (G / LPH) + c / LPH;
  pol.bias_stride = p.bias_heads;
  pol.bias_off = p.bias_heads > 1 ? pol.head : 0;
  pol.row_vecs = unsigned(p.row_elems / VEC);
  pol.q_vecs = unsigned(p.q_row_bytes / W);
  pol.kv_vecs = unsigned(p.kv_row_bytes / W);
  pol.g_vecs = unsigned(p.g_row_bytes / W);
  pol.heads = p.heads;
  pol.cvec = blockIdx.y * G + c;
  pol.inv_scale = p.inv_scale;
  return pol;
}

// The bias gradient's sum takes the bf16 kernels to 144 registers and three CTAs per SM; held to 128 there are four (64,000
// nodes 8 x 8 with a bias gradient, backward 92.1 -> 86.4 us; 16 x 8 163 -> 154).
template <typename T, int W, int LPH, int G, int BIAS>
__global__ void __launch_bounds__(kBlockThreads, sizeof(T) == 2 && BIAS == kBiasGrad ? 4 : 0) bwd_dkv_kernel(const BwdParams p) {
  using Policy = DkvPolicy<T, W, LPH, G, BIAS>;
  __shared__ TileSmem<G, Policy::NACC, Policy::kPerm> sm;
  const Policy pol = make_dkv_policy<T, W, LPH, G, BIAS>(p);
  walk_tile_in<G, Policy>(sm, p.walk, pol);
}

template <typename T, int W, int LPH, int G, int BIAS>
__global__ void __launch_bounds__(crossing_threads(G)) bwd_dkv_stitch_kernel(const BwdParams p) {
  using Policy = DkvPolicy<T, W, LPH, G, BIAS>;
  const Policy pol = make_dkv_policy<T, W, LPH, G, BIAS>(p);
  finish_crossing_rows<G, Policy>(p.walk, pol);
}


}  // namespace

bool launch_dkv(const BwdParams& p, int dtype, const HeadSplit& hs, dim3 grid, int link,
                cudaStream_t stream) {
  return dispatch_shape(dtype, hs.w, hs.lph, hs.g, [&](auto sh) {
    using S = decltype(sh);
    dispatch_bias<kBiasGrad>(bias_use(p), [&](auto use) {
      launch_chained(bwd_dkv_kernel<typename S::T, S::W, S::LPH, S::G, decltype(use)::value>, grid, kBlockThreads, stream, link, p);
    });
    if (p.walk.n_tiles > 1)
      launch_chained(bwd_dkv_stitch_kernel<typename S::T, S::W, S::LPH, S::G, kNoBias>, dim3(crossing_ctas(p.walk, S::G), grid.y), crossing_threads(S::G), stream, kLinkStitch, p);
  });
}

int occupancy_dkv(int dtype, const HeadSplit& hs, int use, int* cache_slot) {
  int result = 4;
  dispatch_shape(dtype, hs.w, hs.lph, hs.g, [&](auto sh) {
    using S = decltype(sh);
    dispatch_bias<kBiasGrad>(use, [&](auto u) {
      result = resident_ctas(bwd_dkv_kernel<typename S::T, S::W, S::LPH, S::G, decltype(u)::value>, cache_slot);
    });
  });
  return result;
}

}  // namespace bwd
}  // namespace tgt
