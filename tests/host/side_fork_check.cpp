// Host check of SideFork (csrc/side_fork.h): which runtime calls it makes when the work
// between fork and join ends well, ends in an error, or one of its own calls fails.
#include <cstdio>

#include "side_fork.h"

static const int side[3] = {11, 12, 13}, join_ev[3] = {21, 22, 23};
static void show(const char* name, cudaError_t e) {
  std::printf("%s %d", name, (int)e);
  for (const auto& s : fake_log) std::printf("; %s", s.c_str());
  std::printf("\n");
  fake_log.clear();
  fake_fail_at = 0;
}

int main() {
  using gbhf::SideFork;
  cudaError_t e;
  {
    SideFork f(1, 5, side, join_ev, 3);
    e = f.fork();
    fake_call("work");
    if (e == cudaSuccess) e = f.join();
  }
  show("good", e);
  {
    SideFork f(1, 5, side, join_ev, 3);
    e = f.fork();
    fake_call("work");   // and an error: the scope is left without a join
  }
  show("error_in_work", e);
  { SideFork f(1, 5, side, join_ev, 3); }
  show("not_forked", cudaSuccess);
  for (int at = 1; at <= 10; ++at) {
    fake_fail_at = at;
    {
      SideFork f(1, 5, side, join_ev, 3);
      e = f.fork();
      if (e == cudaSuccess) e = f.join();
    }
    char name[16];
    std::snprintf(name, sizeof name, "fails_%d", at);
    show(name, e);
  }
  return 0;
}
