// tcgen05 building blocks of the tensor-core kernels (sm_100a): 8-bit unsigned integer
// matrix products with 32-bit accumulators in tensor memory, mbarriers, bulk copies.
//
// Every wait is bounded: after kWaitPolls unsuccessful polls or kWaitNs the wait gives up, the
// block's `fail` word is set and later waits return at once, so a block always reaches its
// end (settle), frees its tensor memory and reports through the engine's error flag.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace cpoly {
namespace umma {

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_init_fence() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

constexpr uint32_t kWaitPolls = 1u << 20;         // each poll suspends for the hardware's own time limit
constexpr uint64_t kWaitNs = 2000000000ull;       // and no wait lasts much longer than 2 s, by a clock that is
constexpr uint32_t kWaitLook = 1u << 8;           // looked at after so many polls: it runs on while the context is
                                                  // switched out, the copies and products waited for do not

__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// Waits until the phase of the given parity has completed; see the file comment for the bound.
__device__ __forceinline__ void mbar_wait(uint32_t bar, uint32_t parity, volatile int* fail) {
  if (mbar_try(bar, parity)) return;
  uint64_t t0 = 0;
  for (uint32_t i = 0; i < kWaitPolls; ++i) {
    if (mbar_try(bar, parity)) return;
    if (i % kWaitLook == kWaitLook - 1) {
      uint64_t t;
      asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
      if (t0 == 0) t0 = t;
      if (*fail || t - t0 > kWaitNs) break;
    }
  }
  *fail = 1;
}
// At a block's end, after a barrier of its threads and before its memory passes on: copies and
// products may still be in flight if a wait ran out, and get 0.1 s to land.
static __device__ __noinline__ void settle_slow() {
  for (int i = 0; i < 100; ++i) __nanosleep(1000000);
}
__device__ __forceinline__ void settle(const volatile int* fail) {
  if (*fail) settle_slow();
}

// Tensor memory: `ncols` (a power of two >= 32) 32-bit columns of 128 lanes, by one whole warp.
__device__ __forceinline__ void tmem_alloc(uint32_t slot_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot_smem), "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t tmem, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ncols));
}
__device__ __forceinline__ void fence_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// Shared-memory writes of this thread become visible to the tensor core and bulk copies.
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// Shared-memory matrix descriptor of a K-major 8-bit operand.  No swizzle: 8-row groups of
// 16-byte rows (128 contiguous bytes), `sbo` between groups, `lbo` between 16-byte K chunks.
// Swizzled: rows of 32 / 64 / 128 bytes, `sbo` = 8 rows; the 16-byte chunk index is xored with
// address bits 7.. (1, 2 or 3 bits).
enum : uint32_t { kSwzNone = 0, kSwz128 = 2, kSwz64 = 4, kSwz32 = 6 };
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo, uint32_t swz) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46) | ((uint64_t)swz << 61);
}
// Instruction descriptor: D s32 (M x N) = A u8 (M x K) B u8 (N x K)^T, both K-major.
__host__ __device__ constexpr uint32_t idesc_u8(int m, int n) {
  return (2u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
// One K = 32 step, issued by one thread.
__device__ __forceinline__ void mma_u8(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// The mbarrier receives one arrival when every product issued so far by this thread is done.
__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// 16 consecutive columns of this warp's 32 lanes.
__device__ __forceinline__ void tmem_ld16(uint32_t (&r)[16], uint32_t taddr) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, "
      "[%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
// 32 consecutive columns of 16 lanes, spread over the warp: thread T gets columns
// 8 b + 2 (T % 4) + {0, 1}, b = 0 .. 3, of lane T / 4 in r[4 b + {0, 1}] and of lane T / 4 + 8 in
// r[4 b + {2, 3}].
__device__ __forceinline__ void tmem_ld_quad(uint32_t (&r)[16], uint32_t taddr) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, "
      "[%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
// Two times 8 consecutive columns.
__device__ __forceinline__ void tmem_ld8x2(uint32_t (&r)[16], uint32_t taddr0, uint32_t taddr1) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr0));
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
               : "r"(taddr1));
}
// Waits for this thread's loads; the registers pass through it, so that no use moves above it.
__device__ __forceinline__ void tmem_ld_wait(uint32_t (&r)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                 "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
               :
               : "memory");
}

// `bytes` (a multiple of 16) from global to shared memory, both 16-byte aligned, counted on the mbarrier.
__device__ __forceinline__ void bulk_load(uint32_t dst_smem, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst_smem),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

// A box of a tensor of 3 dimensions (coordinates x, y, z) to shared memory, counted on the mbarrier.
__device__ __forceinline__ void tensor_load3(uint32_t dst_smem, const void* map, int x, int y, int z, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
          dst_smem),
      "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar)
      : "memory");
}

}  // namespace umma
}  // namespace cpoly
