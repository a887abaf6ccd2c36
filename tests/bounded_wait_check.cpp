// CPU check of csrc/bounded_wait.h: what a role does whose wait runs out.  Prints WAIT-OK on success.
#include <cstdio>

#include "bounded_wait.h"

using b200q::bounded_wait;

static int bad = 0;
static void expect(const char* what, bool ok) {
  if (!ok) {
    std::printf("%s\n", what);
    bad = 1;
  }
}

int main() {
  auto never = [] { return false; };
  auto idle = [] {};
  volatile uint32_t beat = 0;
  {
    // the role that ends the block has gone by the flag before the last role's wait runs out: that one reports
    volatile int abort_flag = 0;
    uint32_t status = 0;
    expect("a role that is done goes on", bounded_wait([] { return true; }, idle, 1000, &abort_flag, &beat, &status, 7));
    expect("nothing to report yet", abort_flag == 0 && status == 0);
    expect("the last wait runs out", !bounded_wait(never, idle, 1000, &abort_flag, &beat, &status, 7));
    expect("its expiry is in the status word", status == 7);
    expect("the others are told", abort_flag == 1);
  }
  {
    // one that follows another's flag leaves within 256 looks; a larger code stays
    volatile int abort_flag = 1;
    uint32_t status = 9;
    int naps = 0;
    expect("the flag ends a wait", !bounded_wait(never, [&] { ++naps; }, 1u << 20, &abort_flag, &beat, &status, 7));
    expect("soon", naps < 256);
    abort_flag = 0;
    bounded_wait(never, idle, 10, &abort_flag, &beat, &status, 7);
    expect("a larger code stays", status == 9);
    expect("without a status word", !bounded_wait(never, idle, 10, &abort_flag, &beat, (uint32_t*)nullptr, 7));
  }
  {
    // while another role waits for a peer, with a limit of its own, those that wait for it go on; then the count starts again
    volatile int abort_flag = 0;
    uint32_t status = 0;
    int naps = 0;
    auto peer = [&] {
      if (++naps < 100000) beat = naps;
    };
    expect("landed at last", bounded_wait([&] { return naps >= 100200; }, peer, 1000, &abort_flag, &beat, &status, 7));
    naps = 0;
    expect("no beat, no end", !bounded_wait(never, peer, 1000, &abort_flag, &beat, &status, 7));
    expect("the looks count from the last beat", naps > 100000 && naps < 102000 && status == 7);
  }
  if (!bad) std::printf("WAIT-OK\n");
  return bad;
}
