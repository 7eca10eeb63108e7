// tc05.cuh -- thin inline-PTX wrappers for Blackwell tensor-core MMAs
// (tcgen05.*), tensor memory (TMEM) and mbarriers, as used by the guiding
// MLP kernels (mlp.cu).
//
// Shared-memory operands use the no-swizzle K-major "core matrix" layout:
// a core matrix is 8 rows x 16 bytes (8 fp16 along K) stored as 128
// contiguous bytes; the matrix descriptor's leading byte offset (LBO) is the
// distance between core matrices adjacent along K and its stride byte offset
// (SBO) the distance between core matrices adjacent along M (or N). Here
// core matrices along K are contiguous (LBO = 128) and 8-row groups follow
// each other (SBO = K / 8 * 128).
#pragma once

#include <cuda_fp16.h>
#include <stdint.h>

namespace trg {
namespace tc05 {

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// Byte offset of element (row, k) of a [rows x K] fp16 operand in the
// core-matrix layout.
__host__ __device__ __forceinline__ uint32_t core_off(uint32_t row, uint32_t k, uint32_t K) {
  return (row >> 3) * (K >> 3) * 128u + (k >> 3) * 128u + (row & 7u) * 16u + (k & 7u) * 2u;
}

// The same bytes also serve as an operand whose K runs over the tile's rows
// (an MN-major operand, the tile transposed): 16 bytes then hold 8 values
// along M (or N) for one k, 8 such for consecutive k are contiguous, SBO is
// the distance between neighbouring 8-value groups along M or N (128) and LBO
// that between 8-row groups along K (columns / 8 * 128). kTransA and kTransB
// in the instruction descriptor select that reading.

// Instruction descriptor of kind::f16: fp16 A and B, both K-major, fp32
// accumulator, dense; N >> 3 at bit 17, M >> 4 at bit 24.
__host__ __device__ constexpr uint32_t idesc_f16_f32(uint32_t M, uint32_t N) {
  return (1u << 4) | ((N >> 3) << 17) | ((M >> 4) << 24);
}

constexpr uint32_t kTransA = 1u << 15, kTransB = 1u << 16;

// TMEM allocation by one whole warp; the address lands in *slot (shared).
__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// D[tmem] (+)= A[smem] * B[smem]^T, issued by one thread. A and B are
// shared-memory matrix descriptors: start address, LBO and SBO (each >> 4),
// descriptor version 1 (bit 46), no swizzle.
//
// A descriptor in two words. Stepping through a tile adds a multiple of 16
// bytes to its start address, the low word's low 14 bits (shared memory ends
// below 2^18, so nothing carries): one add per MMA. The MMAs of a step are
// issued by a single thread, one instruction after another; building the
// descriptors anew for each took it longer than the products themselves.
struct Desc {
  uint32_t lo, hi;
};
__device__ __forceinline__ Desc desc_of(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  return Desc{(saddr >> 4) | (lbo >> 4) << 16, (sbo >> 4) | 1u << 14};
}
__device__ __forceinline__ Desc step(Desc d, uint32_t bytes) { return Desc{d.lo + (bytes >> 4), d.hi}; }
__device__ __forceinline__ void mma_f16(uint32_t tmem_d, Desc a, Desc b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\tmov.b64 a, {%1, %2};\n\tmov.b64 b, {%3, %4};\n\t"
      "setp.ne.b32 p, %6, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %5, p;\n\t}\n" ::"r"(tmem_d),
      "r"(a.lo), "r"(a.hi), "r"(b.lo), "r"(b.hi), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Arrive on the mbarrier once every tcgen05 operation issued so far by this
// thread has completed.
__device__ __forceinline__ void commit(uint64_t* mbar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(mbar))
               : "memory");
}

__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// Generic-proxy shared-memory writes become visible to the tensor cores.
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void mbar_init(uint64_t* mbar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(mbar)), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* mbar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(mbar)) : "memory");
}

// Waits for the given phase parity with a bounded number of polls, each
// suspended for at most a microsecond (a second or so in all); returns false
// when it gave up.
__device__ __forceinline__ bool mbar_wait(uint64_t* mbar, uint32_t parity, uint32_t max_polls = 1u << 20) {
  const uint32_t a = smem_u32(mbar);
  for (uint32_t i = 0; i < max_polls; ++i) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(a), "r"(parity), "r"(1000u)
        : "memory");
    if (done) return true;
  }
  return false;
}

// Meets the other threads that use named barrier `id`, `threads` in all (whole
// warps). Unbounded: every one of them has to come.
__device__ __forceinline__ void bar_sync(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
// The same, and whether `mine` holds for all of them.
__device__ __forceinline__ bool bar_all(int id, int threads, bool mine) {
  uint32_t all;
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %3, 0;\n\tbar.red.and.pred p, %1, %2, p;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(all)
      : "r"(id), "r"(threads), "r"(mine ? 1u : 0u)
      : "memory");
  return all != 0u;
}

// 32 lanes x 32 consecutive 32-bit columns; the values are there after
// tmem_wait.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_wait(uint32_t (&r)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) asm volatile("" : "+r"(r[i]));  // no use of r moves above the wait
}

// 32 lanes x 16 consecutive 32-bit columns: thread i of the warp receives
// row (lane base + i), columns col..col+15.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

}  // namespace tc05
}  // namespace trg
