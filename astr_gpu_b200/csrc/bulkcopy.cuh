// Bulk copies of contiguous rows into shared memory, completing on an mbarrier.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace astr {

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, unsigned bytes) {
  asm volatile("{\n .reg .b64 st;\n mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n}\n" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}
// Both addresses and the size are multiples of 16 bytes.
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, unsigned bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
// Poll the barrier's first phase at most `limit` times; false when it did not complete.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, int limit) {
  for (int it = 0; it < limit; ++it) {
    unsigned done;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0;\n selp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(done)
                 : "r"(smem_u32(bar))
                 : "memory");
    if (done) return true;
  }
  return false;
}
constexpr int kBarrierPolls = 1 << 22;   // bounded wait (far beyond any copy's duration)

// A wait that does not complete sets bit 1 of the error word and waits once more, so that the copies do
// not land after the CTA has gone; the kernel then runs to its end on whatever the tile holds.
__device__ __forceinline__ void mbar_wait_or_flag(uint64_t* bar, int* err) {
  if (mbar_wait(bar, kBarrierPolls)) return;
  atomicOr(err, 2);
  mbar_wait(bar, kBarrierPolls);
}

}  // namespace astr
