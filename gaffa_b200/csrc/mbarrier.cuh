// Barriers in shared memory, bulk copies that complete on them, and bounded
// waits (PTX ISA 8.x: mbarrier, cp.async.bulk).
#pragma once

#include <cstdint>

#include "gaffa_b200.h"

namespace gf {
namespace {

constexpr unsigned kFull = 0xffffffffu;
// A stage whose copies have not landed after this many SM cycles (~2 s) is
// given up: the CTA sets GF_STATUS_PIPELINE in the program's status word
// (read by gf_dedisp_check) and returns, after waiting as long for its own
// copies and steps in flight.  (A test of the wait shortens the first limit.)
#ifndef GF_WAIT_CYCLES
#define GF_WAIT_CYCLES 4000000000ll
#endif
constexpr long long kWaitCycles = GF_WAIT_CYCLES;
constexpr long long kDrainCycles = 4000000000ll;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile(
      "{\n\t.reg .b64 state;\n\t"
      "mbarrier.arrive.release.cta.shared::cta.b64 state, [%0];\n}\n" ::"r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(done)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return done != 0;
}
// Global -> shared copy of `bytes` (a multiple of 16, both addresses 16-byte
// aligned) completing on `bar`.  No multicast: the source is this GPU's memory.
__device__ __forceinline__ void bulk_copy(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
}

// Waits for phase `parity` of `bar`, whole warp; false when this CTA (`failed`,
// shared memory) or another one of the launch (`status`) gave up, or after
// kWaitCycles.  The answer is the warp's, voted at every poll: full-mask
// operations and the CTA's barriers follow, so no lane may leave by itself (and
// lanes that poll apart cost up to 15 % of the tensor-core kernel's rate).
__device__ __forceinline__ bool wait_warp(uint64_t* bar, uint32_t parity, uint32_t* failed, uint32_t* status) {
  if (__all_sync(kFull, mbar_try_wait(bar, parity))) return true;
  const long long start = clock64();
  for (uint32_t i = 0;; ++i) {
    if (__all_sync(kFull, mbar_try_wait(bar, parity))) return true;
    bool stop = *reinterpret_cast<const volatile uint32_t*>(failed) != 0;
    if ((i & 255u) == 255u) stop |= (*reinterpret_cast<const volatile uint32_t*>(status) & GF_STATUS_PIPELINE) != 0;
    stop |= clock64() - start > kWaitCycles;
    if (__any_sync(kFull, stop)) {
      if ((threadIdx.x & 31) == 0) {
        *reinterpret_cast<volatile uint32_t*>(failed) = 1u;
        atomicOr(status, GF_STATUS_PIPELINE);
      }
      return false;
    }
  }
}

}  // namespace
}  // namespace gf
