// Waits that always end, and the end of the roles that wait, for a persistent thread block.  Also compiled by the host compiler, for
// tests.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define B200Q_WAIT_FN __device__ __forceinline__
#else
#define B200Q_WAIT_FN inline
#endif

namespace b200q {

// Looks until look() says yes (true), another role has raised the abort flag, or `looks` looks are over (false, the flag raised);
// nap() between two looks.  Looks do not count while held_up(): others are still waiting for something outside the block, which may
// take longer than a role may wait for them and must end by itself.  (Nothing else belongs here: a store to the status word where the
// looks are over cost decode of 16 rows 5 %, a second loop around this one, which moved registers of x out to memory, 25 %.)
template <class Look, class Nap, class HeldUp>
B200Q_WAIT_FN bool bounded_wait(Look look, Nap nap, HeldUp held_up, uint32_t looks, volatile int* abort_flag) {
  for (uint32_t i = 0; i < looks; ++i) {
    if (look()) return true;
    if ((i & 255u) == 255u) {
      if (*abort_flag) return false;
      if (held_up()) i = 0;
    }
    nap();
  }
  *abort_flag = 1;
  return false;
}

// The end of a role that stores results: last(), then a look at the flag.  Every such role looks for itself, after its own last wait:
// one that looked for all could be done before another's wait runs out.  `status` may be null.
template <class Last>
B200Q_WAIT_FN void end_of_role(Last last, const volatile int* abort_flag, uint32_t* status, uint32_t code) {
  last();
  if (*abort_flag && status) {
#ifdef __CUDA_ARCH__
    atomicMax(status, code);
#else
    if (*status < code) *status = code;
#endif
  }
}

}  // namespace b200q
