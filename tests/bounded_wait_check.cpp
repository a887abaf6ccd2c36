// CPU check of csrc/bounded_wait.h: what becomes of a wait that runs out.  Prints WAIT-OK on success.
#include <cstdio>

#include "bounded_wait.h"

static int bad = 0;
static void expect(const char* what, bool ok) {
  if (!ok) {
    std::printf("%s\n", what);
    bad = 1;
  }
}

int main() {
  auto never = [] { return false; };
  {
    // one that follows another's flag leaves within 256 looks
    volatile int abort_flag = 1;
    int naps = 0;
    expect("the flag ends a wait", !b200q::bounded_wait(never, [&] { ++naps; }, never, 1u << 20, &abort_flag) && naps < 256);
    abort_flag = 0;
    expect("landed", b200q::bounded_wait([&] { return ++naps > 300; }, [] {}, never, 1u << 20, &abort_flag) && abort_flag == 0);
  }
  {
    // a role that starts early does not count the time for which those it waits for are held up by a late peer
    volatile int abort_flag = 0;
    int naps = 0;
    auto nap = [&] { ++naps; };
    auto late = [&] { return naps < 100000; };
    expect("landed at last", b200q::bounded_wait([&] { return naps >= 100200; }, nap, late, 1000, &abort_flag) && abort_flag == 0);
    naps = 0;
    expect("then it does", !b200q::bounded_wait(never, nap, late, 1000, &abort_flag) && naps > 100000 && naps < 102000 && abort_flag == 1);
  }
  // Two roles that store results; one is done long before the other's wait runs out.
  {
    volatile int abort_flag = 0;
    uint32_t status = 0;
    auto end = [&] { b200q::end_of_role([] {}, &abort_flag, &status, 7); };
    end();
    expect("nothing to report yet", status == 0);
    b200q::bounded_wait(never, [] {}, never, 1000, &abort_flag);
    end();
    expect("a wait that ran out is in the status word", status == 7);
  }
  {
    volatile int abort_flag = 1;
    uint32_t status = 9;
    b200q::end_of_role([] {}, &abort_flag, &status, 7);
    expect("a larger code stays", status == 9);
    b200q::end_of_role([] {}, &abort_flag, (uint32_t*)nullptr, 7);
  }
  if (!bad) std::printf("WAIT-OK\n");
  return bad;
}
