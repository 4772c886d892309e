// Small helpers for 5th-generation tensor-core kernels (sm_100a): shared-memory matrix descriptors,
// tcgen05.mma with BF16 operands and FP32 accumulation in tensor memory, bounded mbarrier waits,
// tensor-memory loads, and the proxy fences around a CTA barrier.
#pragma once
#include <cstdint>

namespace feb {
namespace tc {

constexpr int kWaitPolls = 1 << 22;     // bounded mbarrier polling: a wait that runs out reports an error

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor, K-major, no swizzle: core matrices of 8 rows x 16 bytes; `lbo` = byte
// offset between the two 8-element K halves of a K16 step, `sbo` = byte offset between 8-row groups along
// M (or N).  Fields are byte offsets >> 4; descriptor version 1 at bits 46-47.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)((lbo >> 4) & 0x3FFF) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFF) << 32) | (1ull << 46);
}

// The two words of a descriptor, for loops that move its start address: the low word grows by one per 16 bytes.
__device__ __forceinline__ uint64_t desc_join(uint32_t lo, uint32_t hi) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(lo), "r"(hi));
  return d;
}

// K-major operand in rows of 64 or 128 bytes in the swizzle of that width (16-byte chunk c of row r at chunk
// c ^ ((r >> 1) & 3) or c ^ (r & 7)), 8-row groups contiguous.  The swizzle is a function of the address, so a matrix may
// start at any row of a region that is aligned to 8 rows, and a multiple of 32 bytes into it for the next K16 step.
template <int ROW>
struct DescSwz {
  static_assert(ROW == 64 || ROW == 128, "rows of 32 or 64 BF16 values");
  static constexpr uint32_t kHi = (8 * ROW >> 4) | (1u << 14) | (ROW == 64 ? 4u << 29 : 2u << 29);
  static __device__ __forceinline__ uint32_t lo(uint32_t addr) { return ((addr >> 4) & 0x3FFF) | (1u << 16); }
};

// Operand in rows of 64 bytes read along its rows (MN-major): M or N runs over 32 channels of a row, then over blocks of
// 32 whose rows lie `lbo` bytes apart (any multiple of a row: blocks may overlap); K runs over the rows.  Goes with
// kIdescMnMajor.
struct DescSwz64Mn {
  static constexpr uint32_t kHi = DescSwz<64>::kHi;
  static __device__ __forceinline__ uint32_t lo(uint32_t addr, uint32_t lbo) { return ((addr >> 4) & 0x3FFF) | ((lbo >> 4) << 16); }
};
constexpr uint32_t kIdescMnMajor = (1u << 15) | (1u << 16);    // A and B both MN-major

// Instruction descriptor of kind::f16 with BF16 A and B (both K-major), FP32 D, tile M x N.
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void mma_bf16(uint32_t dtmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, int acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n" ::"r"(dtmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc), "r"(0), "r"(0), "r"(0), "r"(0));
}

// completion of every tcgen05 operation this thread issued so far -> one arrival on the mbarrier
__device__ __forceinline__ void commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(bar))
               : "memory");
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count));
}

__device__ __forceinline__ void mbar_fence_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}

// one arrival that also announces `bytes` of asynchronous copies into the barrier's phase
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}

// TMA tile load into shared memory, completion counted on the mbarrier; `map` is a CUtensorMap in kernel parameter space
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const void* map, int x, int y, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
               "l"(map), "r"(smem_addr(bar)), "r"(x), "r"(y)
               : "memory");
}

__device__ __forceinline__ void tma_load_3d(uint32_t dst, const void* map, int x, int y, int z, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(
                   dst),
               "l"(map), "r"(smem_addr(bar)), "r"(x), "r"(y), "r"(z)
               : "memory");
}

// named barrier over `threads` threads with the AND of `ok`
__device__ __forceinline__ bool barrier_and(int id, int threads, bool ok) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %3, 0;\n\tbarrier.cta.red.and.pred q, %1, %2, p;\n\tselp.b32 %0, 1, 0, q;\n\t}\n"
      : "=r"(r)
      : "r"(id), "r"(threads), "r"((uint32_t)ok)
      : "memory");
  return r != 0;
}

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  for (int i = 0; i < kWaitPolls; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred P;\n\tmbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\n\tselp.b32 %0, 1, 0, P;\n\t}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}

// tensor memory: `ncols` columns (a power of two >= 32) for the CTA; warp 0 allocates and frees
__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(slot)), "r"(ncols));
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}

__device__ __forceinline__ void tmem_free(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols));
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&d)[32]) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,"
      "%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
#pragma unroll
  for (int q = 0; q < 32; ++q) d[q] = __uint_as_float(r[q]);
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&d)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
#pragma unroll
  for (int q = 0; q < 16; ++q) d[q] = __uint_as_float(r[q]);
}

__device__ __forceinline__ void wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// shared-memory writes of every thread made visible to the tensor cores, then a CTA barrier
__device__ __forceinline__ void sync_for_tensor_core() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// the same, and the AND over the CTA of `ok`
__device__ __forceinline__ bool sync_for_tensor_core_and(bool ok) {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  const int all = __syncthreads_and(ok ? 1 : 0);
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  return all != 0;
}

}  // namespace tc
}  // namespace feb
