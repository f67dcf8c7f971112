// Bounded mbarrier waits. A wait that never ends would hang the GPU for everyone on it, so after a limit the kernel records
// that it gave up, every later wait of the CTA ends within a suspension (0.1 ms; polled ones within a microsecond or two), the
// roles run or leave their loops without issuing copies or products, what is in flight lands and the kernel returns. Its results
// are wrong then: the record is one word of pinned host memory, which the engine reads before it uses a step's tokens (ops/lib.py)
// and fails on.
#pragma once

#include "host_utils.h"
#include "ptx.cuh"

namespace b200 {

struct WaitConfig {              // part of a kernel's parameters
  uint32_t* word;                // set to 1 when a wait gives up (null: nobody reads it)
  uint32_t limit_ns;             // at most 2^32 - 1; 0 (tests): what is not there at the first look is given up
  uint32_t suspend_ns;           // how long a waiting thread may stay suspended before it looks again: no longer than the limit
};
inline WaitConfig wait_config(uint32_t* word, uint32_t limit_ns) {
  return WaitConfig{word, limit_ns, limit_ns < kSuspendNs ? limit_ns : kSuspendNs};
}

// one per process, set when the library is loaded
inline WaitConfig g_wait_config = wait_config(nullptr, 2000000000u);

__device__ __forceinline__ uint32_t global_ns() {        // wraps every 4.3 s
  uint32_t t;
  asm volatile("mov.u32 %0, %%globaltimer_lo;" : "=r"(t));
  return t;
}

struct WaitGuard {
  volatile uint32_t* dead;       // shared memory, zero at the start of the CTA
  WaitConfig cfg;

  __device__ __forceinline__ bool gave_up() const { return *dead != 0; }

  // true: the phase completed. The thread is suspended in hardware until it does; SOON: it polls
  template <bool SOON = false>
  __device__ __forceinline__ bool wait(uint64_t* bar, uint32_t parity) const {
    if constexpr (SOON) return mbar_try_wait_soon(bar, parity) || poll_on(bar, parity);
    else return mbar_try_wait(bar, parity, cfg.suspend_ns) || wait_on(bar, parity);
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
    while (!mbar_try_wait(bar, parity) && global_ns() - t0 < 2000000000u) {
    }
  }

 private:
  __device__ __forceinline__ void give_up() const {
    *dead = 1;
    if (cfg.word != nullptr) {
      st_relaxed_sys(cfg.word, 1u);
      __threadfence_system();
    }
  }
  // A try is long: the flag and the clock are looked at behind each. So a wait ends within two suspensions of its limit, and within one of
  // another role's giving up. (Looked at before the first try, they cost the block-scaled fp8 feed-forward of 4096 rows 1913 -> 2004 us.)
  __device__ __forceinline__ bool wait_on(uint64_t* bar, uint32_t parity) const {
    if (cfg.limit_ns == 0) {
      give_up();
      return false;
    }
    const uint32_t t0 = global_ns();
    for (;;) {
      if (*dead != 0) return false;
      if (mbar_try_wait(bar, parity, cfg.suspend_ns)) return true;
      if (global_ns() - t0 >= cfg.limit_ns) {
        give_up();
        return false;
      }
    }
  }
  // a try is short: the clock and the flag are looked at every 64
  __device__ __forceinline__ bool poll_on(uint64_t* bar, uint32_t parity) const {
    if (cfg.limit_ns == 0) {
      give_up();
      return false;
    }
    uint32_t t0 = 0;
    for (bool again = false;; again = true) {
#pragma unroll 1
      for (int n = 0; n < 64; ++n)
        if (mbar_try_wait_soon(bar, parity)) return true;
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
  b200::g_wait_config = b200::wait_config(reinterpret_cast<uint32_t*>(word), limit_ns);
  return 0;
}
