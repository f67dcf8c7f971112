// Bounded mbarrier waits. A wait that never ends would hang the GPU for everyone on it, so after a limit the kernel records
// that it gave up, every later wait of the CTA returns at once, the roles run their loops out without issuing copies or
// products, what is in flight lands and the kernel returns. Its results are wrong then: the record is one word of pinned host
// memory, which the engine reads before it uses a step's tokens (ops/lib.py) and fails on.
#pragma once

#include "host_utils.h"
#include "ptx.cuh"

namespace b200 {

struct WaitConfig {              // part of a kernel's parameters
  uint32_t* word;                // set to 1 when a wait gives up (null: nobody reads it)
  uint32_t limit_ns;             // at most 2^32 - 1; 0 (tests): what is not there at the first look is given up
};

// one per process, set when the library is loaded
inline WaitConfig g_wait_config{nullptr, 2000000000u};

__device__ __forceinline__ uint32_t global_ns() {        // wraps every 4.3 s
  uint32_t t;
  asm volatile("mov.u32 %0, %%globaltimer_lo;" : "=r"(t));
  return t;
}

struct WaitGuard {
  volatile uint32_t* dead;       // shared memory, zero at the start of the CTA
  WaitConfig cfg;

  __device__ __forceinline__ bool gave_up() const { return *dead != 0; }

  // true: the phase completed. try_wait suspends the thread in hardware, so the clock is read rarely. SOON: it polls
  template <bool SOON = false>
  __device__ __forceinline__ bool wait(uint64_t* bar, uint32_t parity) const {
    if (look<SOON>(bar, parity)) return true;
    return wait_on<SOON>(bar, parity);
  }

  // a role's first wait, looked at once: with a limit of 0 (tests) it is given up unless the phase has completed already
  __device__ __forceinline__ bool first(uint64_t* bar) const {
    if (cfg.limit_ns != 0 || mbar_test_wait(bar, 0)) return true;
    give_up();
    return false;
  }

  // copies and products in flight: they end by themselves, whatever the limit of the waits
  __device__ __forceinline__ static void land(uint64_t* bar, uint32_t parity) {
    if (mbar_try_wait(bar, parity)) return;
    const uint32_t t0 = global_ns();
    do {
#pragma unroll 1
      for (int n = 0; n < 64; ++n)
        if (mbar_try_wait(bar, parity)) return;
    } while (global_ns() - t0 < 2000000000u);
  }

 private:
  template <bool SOON>
  __device__ __forceinline__ static bool look(uint64_t* bar, uint32_t parity) {
    return SOON ? mbar_try_wait_soon(bar, parity) : mbar_try_wait(bar, parity);
  }
  __device__ __forceinline__ void give_up() const {
    *dead = 1;
    if (cfg.word != nullptr) {
      st_relaxed_sys(cfg.word, 1u);
      __threadfence_system();
    }
  }
  // the clock and the flag are looked at every 64 tries: in front of each, they cost the fp8 GEMM of one or two rows 3 %
  template <bool SOON>
  __device__ __forceinline__ bool wait_on(uint64_t* bar, uint32_t parity) const {
    if (cfg.limit_ns == 0) {
      give_up();
      return false;
    }
    uint32_t t0 = 0;
    for (bool again = false;; again = true) {
#pragma unroll 1
      for (int n = 0; n < 64; ++n)
        if (look<SOON>(bar, parity)) return true;
      if (*dead != 0) return false;
      const uint32_t now = global_ns();
      if (!again) t0 = now;
      else if (now - t0 >= cfg.limit_ns) {
        give_up();
        return false;
      }
    }
  }
};

}  // namespace b200

// word: 4 bytes of pinned host memory, kept for the process's life
extern "C" __attribute__((visibility("default"), weak)) int gllm_set_waits(void* word, unsigned int limit_ns) {
  b200::g_wait_config = b200::WaitConfig{reinterpret_cast<uint32_t*>(word), limit_ns};
  return 0;
}
