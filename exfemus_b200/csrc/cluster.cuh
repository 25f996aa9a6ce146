// cluster.cuh -- thread-block cluster primitives of the one-launch level smoothers.
//
// A cluster's CTAs run on the SMs of one GPC, so a barrier over them costs a few hundred
// nanoseconds instead of the 1.3 us of a kernel boundary, and each CTA writes the others'
// shared memory directly.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace exf {

__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned cluster_size() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
// every thread of the cluster arrives and waits; writes before the arrival (shared memory
// of any CTA, global memory) are visible to the cluster after the wait
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }

// the address of `p` (this CTA's shared memory) in the shared memory of CTA `rank`
__device__ __forceinline__ unsigned cluster_addr(const void *p, unsigned rank) {
  unsigned a = (unsigned)__cvta_generic_to_shared(p), r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
// mbarriers; every wait is bounded
#ifndef EXF_WAIT_TRIES
#define EXF_WAIT_TRIES (1 << 22)
#endif

__device__ __forceinline__ unsigned smem_addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t *b, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive_tx(uint64_t *b, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(b)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(b)) : "memory");
}
// true once the phase of parity `par` has completed; false after `tries` tries
__device__ __forceinline__ bool mbar_wait(uint64_t *b, unsigned par, int tries = EXF_WAIT_TRIES) {
  for (int t = 0; t < tries; t++) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_addr(b)), "r"(par)
        : "memory");
    if (ok) return true;
  }
  return false;
}

// bulk copy into this CTA's shared memory, completing on its mbarrier (16-byte aligned)
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, unsigned bytes, uint64_t *bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_addr(dst)),
               "l"(src), "r"(bytes), "r"(smem_addr(bar))
               : "memory");
}

// asynchronous store of two or four consecutive values into the shared memory of a CTA of the
// cluster, completing on an mbarrier of the same CTA: the receiver waits for the data
// themselves, no barrier or fence is needed.  `addr` is aligned to the stored vector.
__device__ __forceinline__ void cluster_send2(unsigned addr, double a, double b, unsigned bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(addr),
               "l"(__double_as_longlong(a)), "l"(__double_as_longlong(b)), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void cluster_send2(unsigned addr, float a, float b, unsigned bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b32 [%0], {%1, %2}, [%3];" ::"r"(addr),
               "r"(__float_as_uint(a)), "r"(__float_as_uint(b)), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void cluster_send4(unsigned addr, float a, float b, float c, float d, unsigned bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(
                   addr),
               "r"(__float_as_uint(a)), "r"(__float_as_uint(b)), "r"(__float_as_uint(c)), "r"(__float_as_uint(d)),
               "r"(bar)
               : "memory");
}

}  // namespace exf
