// Fifth-generation tensor cores (tcgen05): allocation, descriptors, issue and read-back, and the split of an fp32 value
// into three bf16 pieces that gives them fp32 products.
//
// x = x1 + x2 + x3 with x1 = bf16(x), x2 = bf16(x - x1), x3 = bf16(x - x1 - x2): 3 x 8 significant bits hold all 24 of
// x (both subtractions are exact).  Of the nine products of two such values the six of order 2^-16 and above are kept;
// what is dropped is below 2^-23 of the product.  The leading products are summed apart from the others, so the small ones
// are not rounded away against the large, and the two sums are added in fp32 at the end.  (Below 2^-110 the last piece runs
// into bf16's smallest numbers: such values keep an absolute error of 2^-133 instead.)
#pragma once

#include "tgt_common.cuh"

namespace tgt {
namespace tc {

__device__ __forceinline__ uint32_t smem_address(const void* p) { return uint32_t(__cvta_generic_to_shared(p)); }

// ---- tensor memory ----------------------------------------------------------------------------------------------
// Called by one whole warp; the address appears in *slot (shared memory) for everybody after a barrier.
template <int COLS>
__device__ __forceinline__ void allocate(uint32_t* slot) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_address(slot)), "n"(COLS)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
template <int COLS>
__device__ __forceinline__ void release(uint32_t address) {   // by the warp that allocated
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(address), "n"(COLS));
}

// 16 consecutive fp32 columns of the calling warp's 32 lanes (warp w of a CTA reaches lanes 32 (w % 4) and up)
__device__ __forceinline__ void read16(uint32_t address, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(address));
}
__device__ __forceinline__ void reads_done() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void fence_before_barrier() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after_barrier() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// this thread's writes to shared memory become visible to the tensor cores (in front of the barrier)
__device__ __forceinline__ void publish_operands() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// ---- operands and products ----------------------------------------------------------------------------------------
// Operand tiles are rows of 128 bytes (64 bf16) whose eight 16-byte pieces are permuted by the row's number modulo 8
// (the 128-byte swizzle); tiles start on 1,024 bytes.
__device__ __forceinline__ uint32_t tile_offset(int row, int element) {   // element: a multiple of 4
  return uint32_t(row * 128 + ((((element >> 3) ^ row) & 7) << 4) + ((element & 7) << 1));
}
constexpr uint64_t kDescriptorBase = (uint64_t(1) << 46) | (uint64_t(2) << 61) | (uint64_t(1024 >> 4) << 32);
// Rows are M or N, the 64 elements of a row are K: step 16 of K is 32 bytes further on.
__device__ __forceinline__ uint64_t k_major(uint32_t address) {
  return kDescriptorBase | (uint64_t(1) << 16) | ((address & 0x3ffff) >> 4);
}
// Rows are K, the 64 elements of a row are M or N; the next 64 of M or N lie `next` bytes further on.
__device__ __forceinline__ uint64_t mn_major(uint32_t address, uint32_t next) {
  return kDescriptorBase | (uint64_t(next >> 4) << 16) | ((address & 0x3ffff) >> 4);
}
constexpr uint32_t instruction(int m, int n, bool a_mn_major, bool b_mn_major) {   // bf16 x bf16 -> fp32
  return (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(a_mn_major) << 15) | (uint32_t(b_mn_major) << 16) |
         (uint32_t(n >> 3) << 17) | (uint32_t(m >> 4) << 24);
}
// D[m][n] (+)= sum over 16 k; one thread issues it
__device__ __forceinline__ void multiply(uint32_t d, uint64_t a, uint64_t b, uint32_t instr, bool add) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d), "l"(a), "l"(b), "r"(instr), "r"(uint32_t(add)) : "memory");
}

// Brings n of `rows` rows from `row` on into the L2 (rows of `width` values, a multiple of 4, from a 16-byte boundary on): the
// kernels hold one step's rows in registers, which is not far enough ahead of memory.
__device__ __forceinline__ void prefetch_rows(const float* from, int64_t row, int64_t n, int64_t rows, int width) {
  const int64_t left = rows - row;
  if (left <= 0) return;
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(from + row * width),
               "r"(uint32_t((left < n ? left : n) * width * 4)) : "memory");
}

// Bytes of rows from which on they are taken not to be in the L2 (126 MB, shared with what was written meanwhile).  Shorter lists
// lose by the prefetch: 64,001 rows of 64 x 64 12.0 -> 12.3 us.
constexpr int64_t kPrefetchFrom = int64_t(64) << 20;

// ---- completion ------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void barrier_init(uint64_t* bar) {   // by one thread
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_address(bar)) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
// bar completes a phase when all products this thread has issued are done
__device__ __forceinline__ void commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_address(bar))
               : "memory");
}
// False when the phase has not completed after about a second, far beyond any product's time.  The last look comes after the
// clock: a CTA that was switched out in between sees what has been done meanwhile.
__device__ __forceinline__ bool wait(uint64_t* bar, uint32_t phase) {
  const uint32_t address = smem_address(bar);
  const long long start = clock64();
  bool late = false;
  while (true) {
    uint32_t done;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.b32 %0, 1, 0, p;\n\t}"
                 : "=r"(done) : "r"(address), "r"(phase) : "memory");
    if (done) return true;
    if (late) return false;
    late = clock64() - start >= (1ll << 31);
  }
}
// What a kernel does whose wait ran out, besides making its results NaN: the host finds it out at its next call
// (expired_wait_word).
__device__ __forceinline__ void report_expired_wait(int* word) {
  *reinterpret_cast<volatile int*>(word) = 1;
  __threadfence_system();
}

// ---- the split ----------------------------------------------------------------------------------------------------
struct Pieces {
  uint2 p[3];   // four values each, two per word
};
__device__ __forceinline__ Pieces split4(const float4& v) {
  Pieces out;
  float r[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    out.p[i] = make_uint2(f32_to_bf16x2(r[0], r[1]), f32_to_bf16x2(r[2], r[3]));
    if (i == 2) break;
    float f[4];
    bf16x2_to_f32(out.p[i].x, f[0], f[1]);
    bf16x2_to_f32(out.p[i].y, f[2], f[3]);
#pragma unroll
    for (int j = 0; j < 4; ++j) r[j] -= f[j];
  }
  return out;
}
// pieces lie `piece_bytes` apart
__device__ __forceinline__ void store4(uint32_t tile, uint32_t piece_bytes, uint32_t offset, const Pieces& s) {
#pragma unroll
  for (int i = 0; i < 3; ++i)
    asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(tile + i * piece_bytes + offset), "r"(s.p[i].x), "r"(s.p[i].y)
                 : "memory");
}

}  // namespace tc
}  // namespace tgt
