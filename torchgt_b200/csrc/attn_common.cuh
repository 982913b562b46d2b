// Edge-balanced segmented reduction shared by the three sparse-attention kernels.
//
// Lanes move 16 bytes of a row each (VEC values): LPH = head_dim / VEC lanes cover one head and
// G = LPH * heads_per_group lanes ("lane group") cover the heads one CTA column handles; heads that
// do not fit 32 lanes are walked by blockIdx.y.
//
// The edges, sorted by the grouping endpoint ("row"), are cut into tiles of NG * ge consecutive
// edges, one CTA per tile, NG = 128 / G lane groups per CTA.  Lane group g walks ge consecutive
// edges, kUnroll at a time: all gathers of a batch are issued before any arithmetic.  Edge
// positions, not rows, are what is divided, so a row with 100,000 edges and a row with one edge
// cost the same per edge and every lane group does the same amount of work.
//
// A row whose edges lie inside one lane group's range is finished by that group and written once.
// A row that crosses a range boundary leaves partial sums in shared memory ("head" = the range
// starts inside the row, "tail" = the row starts here and runs past the range); after a barrier
// the group that holds the tail adds the heads of the following groups in order.  If the row
// also crosses the tile boundary the CTA writes its sum to a per-tile carry in global memory, and a second
// kernel adds the carries and finishes the row (finish_crossing_rows).  Every sum has a fixed order: no
// floating-point atomics, bitwise reproducible results.
//
// Rows without edges are zero-filled.  The few between two rows of a range are filled by the group that walks over
// them; aligned blocks of kGapRows rows that are empty as a whole are looked for by the first CTAs, 4,096 rows each, two
// words of ptr[] per block, between the walk and the stitching.  Left to the walking group, the padding behind the graphs of a
// padded batch is one serial chain of stores: 16 graphs of 2,000 to 18,000 nodes padded to 20,000 rows (2.5 edges per node, 8
// heads of 8) take 467 us forward, 217 dQ and 274 dK/dV that way and 84, 101 and 118 this way.  Batches without empty rows pay
// nothing that shows: with the search taken out the 64K step takes 126.5 us against 126.5, one head at 512K rows 263.9 against
// 264.4.
#pragma once

#include <type_traits>

#include "tgt_common.cuh"

namespace tgt {

// Build-time tuning knobs (defaults are what the measurements in the repository use).
#ifndef TGT_UNROLL
#define TGT_UNROLL 4
#endif
// Which walks use 32-byte lanes when nobody forces a lane width (see lane_bytes()).  Measured on B200, 64,000 nodes, us with
// 16- | 32-byte lanes: rows of 512 bytes (8 heads x 16) forward 68.0 | 59.8, backward 187 | 166, 16 heads x 8 with a bias per head
// 78.6 | 64.5 and 217 | 205, of 384 (12 x 8) 59.1 | 56.3 and 178 | 165: half the lane groups and no exchange between the lanes of a
// head.  Rows of 128 bytes 21.9 | 21.7 forward, dQ 3 us less, but not the dK/dV pass, which has twice the accumulators per lane.
// Rows of 256 bytes 31.7 | 33.5 and 89.6 | 96.2 (870,000 nodes 797 | 849 and 2440 | 2556), where two lane groups per warp at 56 to
// 72 registers count for more; 64 bytes 15.7 | 19.8 and 39.7 | 56.5; 32 bytes 73 | 137 and 194 | 239.
// Wide rows in groups of two lanes (10 heads x 8) 61.1 | 70.5 and 184 | 214.  Short lists wait for the lanes' longer chains
// (8 x 16: 45,000 edges 9.8 | 10.6 and 26.4 | 35.1, 197,000 26.3 | 24.3 and 75.7 | 75.5, 263,000 35.3 | 31.9 and 92.3 | 91.1).
// Groups of four lanes pay without a bias only (12 x 8 with a bias per head 69.8 | 115 and 214 | 229).
constexpr int64_t kWideFrom = 250000;   // edges
#ifndef TGT_WIDE_DEFAULT
#define TGT_WIDE_DEFAULT(pass, row_bytes, lanes, n_edges, biased) \
  ((row_bytes) > 256 ? (lanes) >= ((biased) ? 8 : 4) && (n_edges) >= kWideFrom : ((pass) != kPassDkv && (row_bytes) == 128))
#endif
// Edges per batch of the walk with 32-byte lanes (their operands take twice the registers).
#ifndef TGT_WIDE_UNROLL
#define TGT_WIDE_UNROLL 2
#endif
#ifdef TGT_MIN_CTAS
#define TGT_WALK_BOUNDS __launch_bounds__(128, TGT_MIN_CTAS)
#else
#define TGT_WALK_BOUNDS __launch_bounds__(128)
#endif

constexpr int kBlockThreads = 128;
constexpr int kUnroll = TGT_UNROLL;  // edges per lane group whose gathers are in flight together
constexpr int kGeStep = 4;           // a forced ge is a multiple of this (and of every batch size below)
// Fewest edges per lane group: with 16, 1,000 nodes take 10.0 + 23.7 us forward and backward, with 8 7.5 + 16.2, with 4
// 6.9 + 16.2; 4,096 nodes take 9.3 + 22.6, 9.4 + 25.4, 9.4 + 25.4.
constexpr int kLeastEdges = 8;

// Batch size of the walk for element type T and lane-group width G.  Measured on B200 (fp32, 8-byte to
// 256-byte rows; bf16 128-byte rows): batches of 4 edges are best everywhere except for fp32 rows of
// 16 lanes (the 8 heads x 8 case, two lane groups per warp), where batches of 2 are 9-10 % faster
// (64K benchmark step 176 -> 158 us, 870K step 5.11 -> 4.67 ms); narrower groups lose 20-70 % with 2.
constexpr int walk_batch(bool fp32, int w, int g) {
  if (w == 32) return TGT_WIDE_UNROLL;
  return (fp32 && g == 16 && TGT_UNROLL == 4) ? 2 : TGT_UNROLL;
}
template <typename T, int W, int G>
constexpr int walk_unroll() { return walk_batch(std::is_same<T, float>::value, W, G); }
static_assert(kGeStep % TGT_WIDE_UNROLL == 0, "ge must stay a multiple of the batch size");
static_assert(kGeStep % TGT_UNROLL == 0, "ge must stay a multiple of the batch size");

template <int G>
struct TileGeom {
  static constexpr int NG = kBlockThreads / G;  // lane groups per CTA
  static constexpr int GE_MAX = (2048 / NG) > 128 ? 128 : ((2048 / NG) < 8 ? 8 : (2048 / NG));
  static constexpr int TE_MAX = NG * GE_MAX;    // most edges a tile can hold
};

// What every kernel needs to walk the edges.
struct SegWalk {
  const int32_t* ptr;
  const int32_t* other;
  const int32_t* perm;
  const int32_t* seg;
  int n_rows;
  int n_edges;
  int ge;          // edges per lane group per tile (a multiple of the walk's batch, <= GE_MAX; of kGeStep where forced)
  int n_tiles;
  int gap_ctas;    // CTAs that look for rows without edges (fill_gaps)
  float* gcarry;   // [n_tiles][2][gridDim.y * G * NACC] cross-tile partial sums
};

inline int host_ge_max(int g) {
  const int ng = kBlockThreads / g;
  int m = 2048 / ng;
  return m > 128 ? 128 : (m < 8 ? 8 : m);
}

// Edges per lane group: one balanced wave over the GPU when the graph is small enough, else the
// largest tile.  `ctas_per_sm` is the occupancy the caller expects, `step` the walk's batch.
int forced_ge();  // 0 unless tgt_debug_set_tile_edges() overrides the choice

inline int choose_ge(int64_t n_edges, int g, int step, int ctas_per_sm) {
  const int ng = kBlockThreads / g;
  const int ge_max = host_ge_max(g);
  if (forced_ge() > 0) {
    int f = (forced_ge() + kGeStep - 1) / kGeStep * kGeStep;
    return f > ge_max ? ge_max : f;
  }
  // Time is roughly (number of CTA waves) x (work of one tile); a tile costs its ge edges per lane
  // group plus a fixed part (index staging, barriers, stitching) worth about 8 edges.  Few, full
  // waves win; with many waves the tail does not matter and larger tiles amortise the fixed part.  Of the tiles that
  // need the same number of waves the smallest is best.
  const int64_t capacity = int64_t(sm_count()) * ctas_per_sm;
  const int least = ge_max < kLeastEdges ? ge_max : kLeastEdges;
  int best = ge_max;
  double best_cost = 1e300;
  const int64_t fewest = (n_edges + capacity * ng * ge_max - 1) / (capacity * ng * ge_max);
  for (int64_t waves = fewest < 1 ? 1 : fewest; waves <= fewest + 15; ++waves) {
    const int64_t lanes = capacity * ng * waves;
    int ge = int((n_edges + lanes - 1) / lanes + step - 1) / step * step;   // the smallest tile that needs no more waves
    if (ge < least) ge = least;
    if (ge > ge_max) continue;
    const double cost = double(waves) * (ge + 8);
    if (cost < best_cost) {
      best_cost = cost;
      best = ge;
    }
    if (ge == least) break;
  }
  return best;
}

// Multiply-adds of a lane.  PAIRS takes two neighbouring values with one instruction (fma.rn.f32x2, sm_100; each value is
// rounded as by fmaf) where that pays: everywhere in bf16 (16 heads x 8 at 64K nodes, forward 48.0 -> 45.5 us, backward
// 144 -> 140) and in the fp32 forward (870K nodes 839 -> 781 us).  The fp32 gradient passes keep single ones: operands in
// even register pairs cost them a resident CTA per SM (64K step with 8 heads x 8, backward 89.7 against 93.3 us).
// Either way the even and the odd positions are summed apart: a score has the same bits in every pass, and what rounds it
// cancels between an edge's weight and the sum of its row's weights.  With one running sum in the gradient passes and two in the
// forward rows of one edge had dQ off by 3.5e-7 (2-norm, relative) and dV by 8.9e-8, not 2.3e-7 and 5.6e-8.  It costs the
// backward at 870K nodes 2 % (2.56 -> 2.62 ms); one running sum in the forward would cost 5 % of that (796 -> 838 us).
template <bool PAIRS, int VEC>
__device__ __forceinline__ float dot(const float (&a)[VEC], const float (&b)[VEC]) {
  if constexpr (PAIRS) {
    float2 s = make_float2(0.f, 0.f);
#pragma unroll
    for (int j = 0; j < VEC; j += 2) s = __ffma2_rn(make_float2(a[j], a[j + 1]), make_float2(b[j], b[j + 1]), s);
    return s.x + s.y;
  }
  float even = 0.f, odd = 0.f;
#pragma unroll
  for (int j = 0; j < VEC; j += 2) {
    even = fmaf(a[j], b[j], even);
    odd = fmaf(a[j + 1], b[j + 1], odd);
  }
  return even + odd;
}

// acc[AT + j] += w * x[j]
template <bool PAIRS, int AT, int VEC, int NACC>
__device__ __forceinline__ void add_scaled(float (&acc)[NACC], float w, const float (&x)[VEC]) {
#pragma unroll
  for (int j = 0; j < VEC; j += PAIRS ? 2 : 1) {
    if constexpr (PAIRS) {
      const float2 r = __ffma2_rn(make_float2(w, w), make_float2(x[j], x[j + 1]), make_float2(acc[AT + j], acc[AT + j + 1]));
      acc[AT + j] = r.x;
      acc[AT + j + 1] = r.y;
    } else {
      acc[AT + j] = fmaf(w, x[j], acc[AT + j]);
    }
  }
}

__device__ __forceinline__ float clamp_score(float raw) {
  return fminf(fmaxf(raw, kClampLo), kClampHi);
}

// torch.clamp passes the gradient where the input lies inside [lo, hi], bounds included
__device__ __forceinline__ bool clamp_passes_grad(float raw) {
  return raw >= kClampLo && raw <= kClampHi;
}

// Sum of a per-head value (replicated on the LPH lanes of each head) over the heads of a lane group.
template <int LPH, int G>
__device__ __forceinline__ float sum_over_heads(float x) {
#pragma unroll
  for (int off = LPH; off < G; off <<= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
  return x;
}

// exp(x) for |x| < 80: ex2.approx on the rounded product x*log2(e), corrected for the rounding error
// of that product with one fma (relative error about 2^-22, like expf).  Building with
// -DTGT_EXP_CORRECT=0 drops the correction: four instructions per edge and lane fewer (the 64K
// benchmark step goes from 176 to 170 us), relative error |x| * 1.44 * 2^-24 * ln 2 + 2^-22, i.e. below
// 6e-7 for clamped scores and 5e-6 at |x| = 80; the op-level parity tests still pass with it, but
// gradients that cancel heavily (key-bias gradients of a whole model) move by more than 1e-4.
#ifndef TGT_EXP_CORRECT
#define TGT_EXP_CORRECT 1
#endif
__device__ __forceinline__ float fast_exp(float x) {
  constexpr float kLog2eHi = 1.4426950216293335f;   // log2(e) rounded to fp32
  const float t = x * kLog2eHi;
  float e;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(t));
#if TGT_EXP_CORRECT
  constexpr float kLog2eLo = 1.9259629911e-8f;      // log2(e) - kLog2eHi
  constexpr float kLn2 = 0.6931471805599453f;
  const float r = fmaf(x, kLog2eHi, -t) + x * kLog2eLo;  // what the product lost
  e = fmaf(e, r * kLn2, e);
#endif
  return e;
}

constexpr int kGapRows = 8;   // rows of an aligned block that fill_gaps fills when it is empty as a whole

// Zero-fills the rows strictly between `before` and `after`, which have no edges, except the whole aligned blocks.
template <class Policy>
__device__ __forceinline__ void zero_gap(const Policy& pol, int before, int after) {
  for (int r = before + 1; r < after; ++r) {
    if (r % kGapRows == 0 && after - r >= kGapRows) r = after / kGapRows * kGapRows;   // behind the last whole block
    if (r < after) pol.zero_row(r);
  }
}

// The first CTAs of the grid test kGapShare rows each, whole blocks of kGapRows, and zero-fill the empty ones.
constexpr int kGapShare = 4096;
template <int G, class Policy>
__device__ __forceinline__ void fill_gaps(const SegWalk& w, const Policy& pol) {
  const int lane = threadIdx.x % 32;
  constexpr int kRounds = kGapShare / (kBlockThreads * kGapRows);   // of 32 blocks per warp
  const int64_t row0 = int64_t(blockIdx.x) * kGapShare + threadIdx.x / 32 * (kRounds * 32 * kGapRows);
  bool empty[kRounds];
#pragma unroll
  for (int i = 0; i < kRounds; ++i) {
    const int64_t row = row0 + (32 * i + lane) * kGapRows;
    empty[i] = row + kGapRows <= w.n_rows && __ldg(w.ptr + row) == __ldg(w.ptr + row + kGapRows);
  }
#pragma unroll
  for (int i = 0; i < kRounds; ++i) {
    const unsigned mask = __ballot_sync(0xffffffffu, empty[i]);
    if (mask == 0) continue;
    for (int r = lane / G; r < 32 * kGapRows; r += 32 / G)
      if (mask >> (r / kGapRows) & 1) pol.zero_row(int(row0) + 32 * i * kGapRows + r);
  }
}

// The walk.  Policy supplies:
//   static constexpr int NACC;                     accumulators per lane
//   static constexpr bool kPerm;                   whether it reads perm[] (bias in original edge order)
//   static constexpr int kUnroll;                  edges per batch (walk_unroll<T, G>())
//   struct Operands;                               what one edge loads
//   void load(Operands&, int row, int other, int perm_e) const;      issue the gathers of one edge
//   void clear(Operands&) const;                                     operands of a padding slot
//   Scalars prep(const Operands&, bool valid, int perm_e) const;     warp-uniform part (shuffles)
//   void accumulate(float (&acc)[NACC], const Operands&, const Scalars&) const;
//   void finalize(int row, const float (&acc)[NACC]) const;          write the finished row
//   void zero_row(int row) const;                                    row without edges
template <int G, class Policy>
__device__ __forceinline__ void walk_tile(const SegWalk& w, const Policy& pol, int32_t* s_other,
                                          int32_t* s_seg, int32_t* s_perm, float* s_carry,
                                          int32_t* s_carry_row) {
  constexpr int NG = TileGeom<G>::NG;
  constexpr int NACC = Policy::NACC;
  constexpr int kUnroll = Policy::kUnroll;   // edges per batch (shadows the default)
  const int tid = threadIdx.x;
  const int g = tid / G;        // lane group inside the CTA
  const int c = tid % G;        // 16-byte column inside the group
  const int te = NG * w.ge;
  const int64_t t0 = int64_t(blockIdx.x) * te;
  const int n = int(min(int64_t(te), int64_t(w.n_edges) - t0));  // edges in this tile (>= 1)

  // ---- stage the tile's indices.  Tile edge i lives at position i + i / ge: one pad word per
  // lane-group range, so the groups of a warp (which read ranges ge apart) hit different banks.
  // The rows of the edge before and after the tile go to the two words behind the padded array.
  const int ge = w.ge;
  auto pos = [ge](int i) { return i + i / ge; };
  int32_t* s_halo = s_seg + TileGeom<G>::TE_MAX + NG;   // [0] = row before the tile, [1] = row after
  for (int i = tid; i < n; i += kBlockThreads) {
    const int p = pos(i);
    s_seg[p] = __ldg(w.seg + t0 + i);
    s_other[p] = __ldg(w.other + t0 + i);
    if (Policy::kPerm) s_perm[p] = __ldg(w.perm + t0 + i);
  }
  if (tid == 0) {
    s_halo[0] = t0 == 0 ? -1 : __ldg(w.seg + t0 - 1);
    s_halo[1] = t0 + n >= w.n_edges ? -2 : __ldg(w.seg + t0 + n);
  }
  for (int i = tid; i < 2 * NG; i += kBlockThreads) s_carry_row[i] = -3;  // [g][0] head row, [g][1] tail row
  // the indices are the layout's, complete long before this call; everything below reads or overwrites what
  // the previous kernel of the call works on
  dependent_wait();
  __syncthreads();

  // ---- walk this group's range [gb, ge) of the tile
  const int gb = min(g * w.ge, n);
  const int gend = min(gb + w.ge, n);
  float acc[NACC];
#pragma unroll
  for (int a = 0; a < NACC; ++a) acc[a] = 0.f;
  // row of tile edge i, for i in [-1, n]
  auto row_of = [&](int i) { return i < 0 ? s_halo[0] : (i >= n ? s_halo[1] : s_seg[pos(i)]); };
  int cur = row_of(gb - 1);                          // row of the edge just before the range
  bool own = gb < gend && row_of(gb) == cur;         // the range starts inside row `cur`
  const int gb_pos = pos(gb);                        // the range is contiguous in padded positions
  bool head_pending = own;
  float* my_head = s_carry + (g * 2 + 0) * (G * NACC) + c * NACC;
  float* my_tail = s_carry + (g * 2 + 1) * (G * NACC) + c * NACC;

  // State of the segmented walk, advanced one batch of kUnroll edges at a time.  FULL = every
  // slot of the batch holds an edge of this group's range (all tiles but the last one).
  auto batch = [&](int first, auto full_tag) {
    constexpr bool FULL = decltype(full_tag)::value;
    typename Policy::Operands ops[kUnroll];
    int row[kUnroll], pe[kUnroll];
    bool valid[kUnroll];
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      const int i = first + u;
      valid[u] = FULL || i < gend;
      const int ii = valid[u] ? gb_pos + (i - gb) : 0;
      row[u] = s_seg[ii];
      pe[u] = Policy::kPerm ? s_perm[ii] : 0;
      if (valid[u]) pol.load(ops[u], row[u], s_other[ii], pe[u]);
      else pol.clear(ops[u]);
    }
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      const typename Policy::Scalars sc = pol.prep(ops[u], valid[u], pe[u]);
      if (valid[u]) {
        if (row[u] != cur) {
          if (own) {
            if (head_pending) {
#pragma unroll
              for (int a = 0; a < NACC; ++a) my_head[a] = acc[a];
              if (c == 0) s_carry_row[g * 2 + 0] = cur;
            } else {
              pol.finalize(cur, acc);
            }
          }
          head_pending = false;
          zero_gap(pol, cur, row[u]);
          cur = row[u];
          own = true;
#pragma unroll
          for (int a = 0; a < NACC; ++a) acc[a] = 0.f;
        }
        pol.accumulate(acc, ops[u], sc);
      }
    }
  };
  if (n == te) {
    // ge is a multiple of the batch size, so every batch of every group is full
    for (int first = gb; first < gend; first += kUnroll) batch(first, std::true_type{});
  } else {
    // last tile: all groups of a warp run the same number of batches (the shuffles inside need
    // the full warp), slots past the group's range are padding
    const int warp_first_group = (tid / 32) * (32 / G);
    const int warp_gb = min(warp_first_group * w.ge, n);
    const int batches = (min(w.ge, n - warp_gb) + kUnroll - 1) / kUnroll;
    for (int b = 0; b < batches; ++b) batch(gb + b * kUnroll, std::false_type{});
  }
  if (gb < gend) {  // close the last row of the range
    const bool cont_out = row_of(gend) == cur;
    if (head_pending) {
#pragma unroll
      for (int a = 0; a < NACC; ++a) my_head[a] = acc[a];
      if (c == 0) s_carry_row[g * 2 + 0] = cur;
    } else if (cont_out) {
#pragma unroll
      for (int a = 0; a < NACC; ++a) my_tail[a] = acc[a];
      if (c == 0) s_carry_row[g * 2 + 1] = cur;
    } else {
      pol.finalize(cur, acc);
    }
    if (t0 + gend == w.n_edges) zero_gap(pol, cur, w.n_rows);  // this group owns the last edge
  }
  if (blockIdx.x < w.gap_ctas) fill_gaps<G, Policy>(w, pol);
  release_dependents();   // the next kernel of the call may take this SM's slots as they free up
  __syncthreads();

  // ---- stitch rows that cross group boundaries, in group order
  const int last_row = row_of(n - 1);       // row of the tile's last edge
  const bool tile_cont_out = s_halo[1] == last_row;
  const int lanes_all = gridDim.y * G;
  float* tile_carry = w.gcarry + (int64_t(blockIdx.x) * 2) * (int64_t(lanes_all) * NACC) +
                      int64_t(blockIdx.y * G + c) * NACC;
  if (g == 0 && s_halo[0] == row_of(0)) {
    // the tile starts inside a row that began in an earlier tile: sum its heads into the tile's
    // head carry
    const int r = row_of(0);
#pragma unroll
    for (int a = 0; a < NACC; ++a) acc[a] = 0.f;
    for (int j = 0; j < NG && s_carry_row[j * 2] == r; ++j) {
      const float* h = s_carry + (j * 2) * (G * NACC) + c * NACC;
#pragma unroll
      for (int a = 0; a < NACC; ++a) acc[a] += h[a];
    }
#pragma unroll
    for (int a = 0; a < NACC; ++a) tile_carry[a] = acc[a];
  }
  const int r = s_carry_row[g * 2 + 1];
  if (r >= 0) {
    // this group holds the start of row r: add the heads of the groups the row runs through
#pragma unroll
    for (int a = 0; a < NACC; ++a) acc[a] = my_tail[a];
    for (int j = g + 1; j < NG && s_carry_row[j * 2] == r; ++j) {
      const float* h = s_carry + (j * 2) * (G * NACC) + c * NACC;
#pragma unroll
      for (int a = 0; a < NACC; ++a) acc[a] += h[a];
    }
    if (r == last_row && tile_cont_out) {
      float* t = tile_carry + int64_t(lanes_all) * NACC;  // the tile's tail carry
#pragma unroll
      for (int a = 0; a < NACC; ++a) t[a] = acc[a];
    } else {
      pol.finalize(r, acc);
    }
  }
}

// ---- rows that cross tiles ---------------------------------------------------------------------------------------
// A second kernel, one lane group per tile: that of the tile in which a row that runs past the tile's end STARTS adds
// up what the row's tiles have left (the tail carry of that tile, the head carries of the following ones) and finishes
// it; rows of more than kGroupTiles further tiles are taken by the whole CTA.  Every sum has a fixed order.  Launched as
// the dependent of the walk, and what does not depend on the walk is read before it has ended.
constexpr int kGroupTiles = 8;
// Threads of its CTAs.  A row of every eighth edge has over a hundred carries at 64,000 nodes, which wide groups need many
// slots for; narrow ones have enough of them, and CTAs of 512 threads would hold hundreds of tiles each (64,000 nodes backward, 512 |
// 128 threads: one bf16 head of 8 58.1 | 46.1 us, two with a bias gradient 52.1 | 44.1, four fp32 heads 63.7 | 61.3).
constexpr int crossing_threads(int g) { return g <= 4 ? 128 : 512; }
template <int G, class Policy>
__device__ __forceinline__ void finish_crossing_rows(const SegWalk& w, const Policy& pol) {
  constexpr int kCrossingThreads = crossing_threads(G);
  constexpr int NG = kCrossingThreads / G, NACC = Policy::NACC;
  __shared__ float s_part[kCrossingThreads * NACC];
  __shared__ int s_many[NG][3], s_n;   // rows of many tiles: first tile, further tiles, row
  const int g = threadIdx.x / G, c = threadIdx.x % G;
  const int te = TileGeom<G>::NG * w.ge;
  const int tile = blockIdx.x * NG + g;
  const int64_t t1 = int64_t(tile + 1) * te;
  if (threadIdx.x == 0) s_n = 0;
  __syncthreads();
  int row = -1, further = 0;
  if (t1 < w.n_edges) {
    const int r = __ldg(w.seg + t1 - 1), behind = __ldg(w.seg + t1);
    const int begin = __ldg(w.ptr + r), end = __ldg(w.ptr + r + 1);
    if (r == behind && begin >= t1 - te) {
      row = r;
      further = (end - 1) / te - tile;
    }
  }
  if (row >= 0 && further > kGroupTiles && c == 0) {
    const int at = atomicAdd(&s_n, 1);
    s_many[at][0] = tile;
    s_many[at][1] = further;
    s_many[at][2] = row;
  }
  release_dependents();
  dependent_wait();   // the walk's carries; every CTA waits, also those that have nothing to finish
  const int64_t stride = int64_t(gridDim.y) * G * NACC;
  const float* base = w.gcarry + int64_t(blockIdx.y * G + c) * NACC;
  float acc[NACC];
  auto carry = [&](int t, int which) { return base + (int64_t(t) * 2 + which) * stride; };   // 0 = head, 1 = tail
  if (row >= 0 && further <= kGroupTiles) {
    const float *tail = carry(tile, 1), *head = carry(tile + 1, 0);
#pragma unroll
    for (int a = 0; a < NACC; ++a) acc[a] = __ldcg(tail + a) + __ldcg(head + a);
    for (int i = 2; i <= further; ++i) {
      const float* p = carry(tile + i, 0);
#pragma unroll
      for (int a = 0; a < NACC; ++a) acc[a] += __ldcg(p + a);
    }
    pol.finalize(row, acc);
  }
  __syncthreads();
  for (int j = 0; j < s_n; ++j) {
    const int start = s_many[j][0], n = s_many[j][1];
#pragma unroll
    for (int a = 0; a < NACC; ++a) acc[a] = 0.f;
#pragma unroll 4
    for (int i = g; i <= n; i += NG) {
      const float* p = carry(start + i, i == 0 ? 1 : 0);
#pragma unroll
      for (int a = 0; a < NACC; ++a) acc[a] += __ldcg(p + a);
    }
#pragma unroll
    for (int a = 0; a < NACC; ++a) s_part[a * kCrossingThreads + threadIdx.x] = acc[a];
    __syncthreads();
    int half = NG / 2;
    while (half > n) half >>= 1;     // the groups behind the row's n + 1 carries have nothing
    for (; half >= 1; half >>= 1) {  // halving tree
      if (g < half) {
#pragma unroll
        for (int a = 0; a < NACC; ++a)
          s_part[a * kCrossingThreads + threadIdx.x] += s_part[a * kCrossingThreads + threadIdx.x + half * G];
      }
      __syncthreads();
    }
    if (g == 0) {
#pragma unroll
      for (int a = 0; a < NACC; ++a) acc[a] = s_part[a * kCrossingThreads + c];
      pol.finalize(s_many[j][2], acc);
    }
    __syncthreads();
  }
}
// CTAs of that kernel in x for lane groups of g lanes.
inline unsigned crossing_ctas(const SegWalk& w, int g) {
  const int ng = crossing_threads(g) / g;
  return unsigned((w.n_tiles + ng - 1) / ng);
}

struct HeadSplit {
  int w;       // bytes one lane moves: 16 or 32
  int lph;     // lanes per head
  int hpg;     // heads per lane group
  int g;       // lanes per group
  int groups;  // number of head groups (gridDim.y)
};

enum { kPassFwd = 0, kPassDq = 1, kPassDkv = 2 };
// What a walk does with the edge bias; a kernel of its own for each, since the registers of the code that is not run count.
enum BiasUse { kNoBias = 0, kReadBias = 1, kBiasGrad = 2 };

// Lane width of the walk kernels: 0 = chosen by the library, 1 = 16-byte lanes, 2 = 32-byte lanes
// wherever the head size allows.  Set by tgt_debug_set_lane_mode().
int lane_mode();

// Bytes per lane for heads of head_dim elements.  32-byte lanes need heads that are whole multiples of
// 32 bytes and 32-byte aligned tensors and strides (`can32`).
inline int lane_bytes(int heads, int head_dim, int dtype, bool can32, int pass, int64_t n_edges, bool biased) {
  const int head_bytes = head_dim * (dtype == TGT_F32 ? 4 : 2);
  if (!can32 || dtype != TGT_F32 || head_bytes % 32 != 0 || head_bytes > 128) return 16;
  const int mode = lane_mode();
  if (mode == 1) return 16;
  if (mode == 2) return 32;
  int group = head_bytes / 32;   // lanes of a group of 32-byte lanes, as split_heads makes them
  for (int hpg = 1; hpg * 2 * (head_bytes / 32) <= 32 && heads % (hpg * 2) == 0; hpg *= 2) group *= 2;
  return TGT_WIDE_DEFAULT(pass, heads * head_bytes, group, n_edges, biased) ? 32 : 16;
}

// Returns false when (heads, head_dim, dtype) cannot be mapped onto lanes of w bytes.
inline bool split_heads(int heads, int head_dim, int dtype, int w, HeadSplit* hs) {
  const int vec = w / (dtype == TGT_F32 ? 4 : 2);
  if (heads < 1 || head_dim < vec || head_dim % vec != 0) return false;
  const int lph = head_dim / vec;
  if (lph > 32 || (lph & (lph - 1)) != 0) return false;
  int hpg = 1;
  while (hpg * 2 * lph <= 32 && heads % (hpg * 2) == 0) hpg *= 2;
  hs->w = w;
  hs->lph = lph;
  hs->hpg = hpg;
  hs->g = lph * hpg;
  hs->groups = heads / hpg;
  return true;
}

// Compile-time shape of one kernel instantiation: element type, bytes per lane, lanes per head, lanes
// per group.
template <typename T_, int W_, int LPH_, int G_>
struct LaneShape {
  using T = T_;
  static constexpr int W = W_, LPH = LPH_, G = G_;
};

// Calls f(LaneShape<...>{}) for the run-time (dtype, w, lph, g); only shapes that can occur are
// instantiated (a group holds whole heads: LPH <= G; 32-byte lanes are built for fp32 heads of up to
// 128 bytes).  Returns false when the combination is not built.
template <typename T, int W, int LPH, class F>
inline bool dispatch_group(int g, F&& f) {
  switch (g) {
    case 1: if constexpr (LPH <= 1) { f(LaneShape<T, W, LPH, 1>{}); return true; } break;
    case 2: if constexpr (LPH <= 2) { f(LaneShape<T, W, LPH, 2>{}); return true; } break;
    case 4: if constexpr (LPH <= 4) { f(LaneShape<T, W, LPH, 4>{}); return true; } break;
    case 8: if constexpr (LPH <= 8) { f(LaneShape<T, W, LPH, 8>{}); return true; } break;
    case 16: if constexpr (LPH <= 16) { f(LaneShape<T, W, LPH, 16>{}); return true; } break;
    case 32: if constexpr (LPH <= 32) { f(LaneShape<T, W, LPH, 32>{}); return true; } break;
    default: break;
  }
  return false;
}

template <typename T, int W, class F>
inline bool dispatch_head(int lph, int g, F&& f) {
  switch (lph) {
    case 1: return dispatch_group<T, W, 1>(g, f);
    case 2: return dispatch_group<T, W, 2>(g, f);
    case 4: return dispatch_group<T, W, 4>(g, f);
    case 8: if constexpr (W == 16) return dispatch_group<T, W, 8>(g, f); else break;
    case 16: if constexpr (W == 16) return dispatch_group<T, W, 16>(g, f); else break;
    case 32: if constexpr (W == 16) return dispatch_group<T, W, 32>(g, f); else break;
    default: break;
  }
  return false;
}

template <class F>
inline bool dispatch_shape(int dtype, int w, int lph, int g, F&& f) {
  if (dtype == TGT_F32) return w == 32 ? dispatch_head<float, 32>(lph, g, f) : dispatch_head<float, 16>(lph, g, f);
  return w == 16 ? dispatch_head<__nv_bfloat16, 16>(lph, g, f) : false;
}

// Calls f with the bias use as a compile-time constant; a walk whose MOST is kReadBias only reads.
template <int MOST, class F>
inline void dispatch_bias(int use, F&& f) {
  if constexpr (MOST >= kBiasGrad) {
    if (use == kBiasGrad) return f(std::integral_constant<int, kBiasGrad>{});
  }
  if (use != kNoBias) return f(std::integral_constant<int, kReadBias>{});
  f(std::integral_constant<int, kNoBias>{});
}

int check_layout(const tgt_layout* L, const char* name);

// Resident CTAs per SM of a walk kernel on the current device (asked from the runtime once per
// instantiation): the tile size is chosen so that one wave of CTAs covers the graph.
template <typename Kernel>
inline int resident_ctas(Kernel kernel, int* cache) {
  if (*cache <= 0) {
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, kBlockThreads, 0) != cudaSuccess || n < 1) {
      cudaGetLastError();
      n = 4;
    }
    *cache = n;
  }
  return *cache;
}

// Tiling of one pass: edges per lane group, number of tiles, bytes of cross-tile carry.
struct TilePlan {
  int ge;
  int n_tiles;
  size_t carry_bytes;
};
TilePlan plan_tiles(int64_t n_edges, const HeadSplit& hs, int step, int nacc, int ctas_per_sm);

// CTAs of a walk kernel in x: one per tile, and more where there are over kGapShare rows per tile.
inline int gap_ctas(int64_t n_rows) { return int((n_rows + kGapShare - 1) / kGapShare); }
inline unsigned walk_ctas(const TilePlan& tp, int64_t n_rows) {
  const int gaps = gap_ctas(n_rows);
  return unsigned(gaps > tp.n_tiles ? gaps : tp.n_tiles);
}

// Shared-memory bytes walk_tile needs (indices + carries), as the kernels declare them.
template <int G, int NACC, bool PERM>
struct TileSmem {
  static constexpr int TE = TileGeom<G>::TE_MAX;
  static constexpr int NG = TileGeom<G>::NG;
  struct Indices {
    int32_t other[TE + NG];
    int32_t seg[TE + NG + 2];   // padded rows + the two halo words
    int32_t perm[PERM ? TE + NG : 1];
  };
  Indices idx;
  float carry[NG * 2 * G * NACC];
  int32_t carry_row[NG * 2];
};

// The call every walk kernel makes.
template <int G, class Policy>
__device__ __forceinline__ void walk_tile_in(TileSmem<G, Policy::NACC, Policy::kPerm>& sm, const SegWalk& w, const Policy& pol) {
  if (blockIdx.x >= w.n_tiles) {     // launched for its share of the empty rows only
    release_dependents();
    dependent_wait();                // the rows may be what the previous kernel of the call works on
    fill_gaps<G, Policy>(w, pol);
    return;
  }
  walk_tile<G, Policy>(w, pol, sm.idx.other, sm.idx.seg, sm.idx.perm, sm.carry, sm.carry_row);
}

}  // namespace tgt
