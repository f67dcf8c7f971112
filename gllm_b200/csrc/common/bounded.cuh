// Bounded mbarrier waits. A wait that never ends would hang the GPU for everyone on it, so after a limit the kernel records
// that it gave up, every later wait of the CTA returns at once, the roles run their loops out without issuing copies or
// products, wait (again bounded) for what is in flight and return. The count is read by `gllm_waits_given_up_*`.
#pragma once

#include "ptx.cuh"

namespace b200 {

// each translation unit has its own counter (no relocatable device code)
static __device__ unsigned int g_waits_given_up;

struct WaitGuard {
  volatile uint32_t* dead;       // shared memory, zero at the start of the CTA

  __device__ __forceinline__ bool gave_up() const { return *dead != 0; }

  // true: the phase completed. try_wait suspends the thread for a while in hardware, so 2^22 tries are well over a second's
  // worth of polling only when something is stuck
  __device__ __forceinline__ bool wait(uint64_t* bar, uint32_t parity) const {
    if (mbar_try_wait(bar, parity)) return true;
    for (uint32_t n = 1; n < (1u << 22); ++n) {
      if (mbar_try_wait(bar, parity)) return true;
      if ((n & 1023u) == 0u && *dead != 0) return false;
    }
    if (*dead == 0) {
      *dead = 1;
      atomicAdd(&g_waits_given_up, 1u);
    }
    return false;
  }
};

inline int read_waits_given_up() {
  unsigned int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_waits_given_up, sizeof v) != cudaSuccess) return -1;
  return static_cast<int>(v);
}

}  // namespace b200
