// tma.cuh -- TMA copies and mbarrier waits of the forward projectors (inline PTX).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace mexct {

// ---------------------------------------------------------------------------
// TMA / mbarrier helpers (inline PTX).
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
               : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int c0, int c1,
                                            int c2, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(smem_u32(dst)),
      "l"((uint64_t)map), "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Non-blocking test of a phase (try_wait may suspend the thread for a while).
__device__ __forceinline__ bool mbar_test_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Cluster barrier (every thread of every CTA), and a float of another CTA's
// shared memory at the address that `p` has in this one.
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::
                   : "memory");
}
__device__ __forceinline__ float cluster_ld(const float* p, uint32_t rank) {
  float v;
  asm volatile(
      "{\n .reg .b32 a;\n mapa.shared::cluster.u32 a, %1, %2;\n ld.shared::cluster.f32 %0, [a];\n}"
      : "=f"(v)
      : "r"(smem_u32(p)), "r"(rank)
      : "memory");
  return v;
}

// After a CTA gave up waiting: copies issued before still land in its
// buffers, so wait (at most 2 s each) until the last copy issued into each
// buffer has completed.  Copies into one buffer complete in order, so the
// last one's phase parity is (count - 1) & 1.  issued: 16-bit counts per
// buffer of up to four.  Kept out of line: it only runs after a failure.
static __device__ __noinline__ void slab_drain(uint64_t* bar, uint64_t issued, unsigned* err) {
  for (int b = 0; b < 4; ++b) {
    const uint32_t n = (uint32_t)(issued >> (16 * b)) & 0xffffu;
    if (n == 0) continue;
    const uint64_t t0 = global_ns();
    bool done = false;
    do {
      done = mbar_try_wait(&bar[b], (n - 1u) & 1u);
    } while (!done && global_ns() - t0 < 2000000000ull);
    if (!done && err) atomicOr(err, 2u);
  }
}

// Bounded wait: after one attempt, keeps trying for at most wait_us
// microseconds of wall time (default 2 s; < 0: one non-blocking test only), then records the
// failure in err and in the CTA's abort flag and reports it to the caller,
// which samples the slab from global memory instead (the result is the same).
// Once a CTA has given up, its later waits return at once and no further
// copies are issued, so a broken pipeline costs one time-out per CTA.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, unsigned* err,
                                                  volatile int* abort, int wait_us) {
  if (*abort) return false;
  if (wait_us < 0) {
    if (mbar_test_wait(bar, parity)) return true;
  } else {
    // the usual short waits end here, without reading the clock
    for (int i = 0; i < 64; ++i)
      if (mbar_try_wait(bar, parity)) return true;
    const uint64_t limit = wait_us > 0 ? (uint64_t)wait_us * 1000ull : 2000000000ull;
    const uint64_t t0 = global_ns();
    while (global_ns() - t0 < limit)
      if (mbar_try_wait(bar, parity)) return true;
  }
  *abort = 1;
  if (err) atomicOr(err, 1u);
  return false;
}

}  // namespace mexct
