// Shared-memory barriers (mbarrier) of the kernels whose warps hand work to one another.
#pragma once

#include <stdint.h>

namespace mq {

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// whether the phase of this parity has completed (the hardware waits a moment before it says no)
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

__device__ __forceinline__ uint64_t global_ns() {
  uint64_t now;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
  return now;
}

// The limit of a wait: call expired() now and then while waiting.  After about a second, or as soon as any wait on
// this device has run out, it records `code` in *fault (an earlier code stays) and says so; every later wait on the device
// then gives up at once.
struct WaitLimit {
  uint64_t t0 = 0;
  __device__ __forceinline__ bool expired(int* fault, int code) {
    if (*reinterpret_cast<volatile int*>(fault) != 0) return true;
    const uint64_t now = global_ns();
    if (t0 == 0) t0 = now;
    else if (now - t0 > 1000000000ull) {
      atomicCAS(fault, 0, code);
      return true;
    }
    return false;
  }
};

// By one lane, or where nothing that the warp does together depends on the answer.
__device__ __forceinline__ bool mbar_wait_lane(uint32_t bar, uint32_t parity, int* fault, int code) {
  WaitLimit limit;
  for (uint32_t it = 0;; ++it) {
    if (mbar_try(bar, parity)) return true;
    if ((it & 255u) == 255u && limit.expired(fault, code)) return false;
  }
}
// By a whole warp.  Its lanes poll one by one, and a barrier may complete between the poll of one that gives up and that of the next:
// they agree, so that what follows (shuffles, tensor memory loads) is entered by all of them or by none.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int* fault, int code) {
  return __all_sync(0xffffffffu, mbar_wait_lane(bar, parity, fault, code));
}

// The word on the current device that a wait records its code in (defined beside the tensor-core kernels).
int engine_fault_word(int** out);

}  // namespace mq
