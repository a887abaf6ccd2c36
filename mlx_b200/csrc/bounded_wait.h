// A wait that always ends, for the roles of a persistent thread block.  Also compiled by the host compiler, for tests.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define B200Q_WAIT_FN __device__ __forceinline__
#else
#define B200Q_WAIT_FN inline
#endif

namespace b200q {

// Looks until look() says yes (true), another role has raised the abort flag, or `looks` looks are over (false); nap() between
// two looks.  `beat` is a word of the block that roles change while they work or wait longer than others may wait for them (a peer's
// flag with a limit of its own); the looks are counted from its last change, so such a role must end by itself.  Whoever's wait runs out raises the flag and stores `code` in the status word itself: a role that reads the flag for
// others may have ended before it goes up.  `status` may be null.
template <class Look, class Nap>
B200Q_WAIT_FN bool bounded_wait(Look look, Nap nap, uint32_t looks, volatile int* abort_flag, const volatile uint32_t* beat, uint32_t* status,
                                uint32_t code) {
  uint32_t seen = 0;
  for (uint32_t i = 0; i < looks; ++i) {
    if (look()) return true;
    if ((i & 255u) == 255u) {
      if (*abort_flag) return false;
      const uint32_t now = *beat;
      if (now != seen) {
        seen = now;
        i = 0;
      }
    }
    nap();
  }
  *abort_flag = 1;
  if (status) {
#ifdef __CUDA_ARCH__
    atomicMax(status, code);
#else
    if (*status < code) *status = code;
#endif
  }
  return false;
}

}  // namespace b200q
