// C entry to the round loop (round_loop.h) over a script in the GPU's place, for
// tests/test_round_loop.py.
#include <cstring>
#include <string>

#include "round_loop.h"

namespace {
struct Script {
  const long long* left;  // live cells after each launch
  int n, at = 0;
  int fail_capture, fail_launch;  // class whose graph cannot be made, launch that fails (-1: none)
  bool running = false;
  std::string log;
  int capture(int cls) {
    log += "c" + std::to_string(cls) + " ";
    return cls == fail_capture ? -7 : 0;
  }
  int launch(int cls) {
    log += "l" + std::to_string(cls) + " ";
    running = true;  // a failing launch may have enqueued some of its rounds
    return at == fail_launch ? -8 : 0;
  }
  int wait(long long* live) {
    log += "w ";
    running = false;
    *live = at < n ? left[at] : 0;
    ++at;
    return 0;
  }
  int timed_out() { return -9; }
};
}  // namespace

extern "C" int round_loop(long long live, long long warp_cells, long long max_rounds, int graph, const long long* left,
                          int n, int fail_capture, int fail_launch, char* log, int* running) {
  Script s{left, n, 0, fail_capture, fail_launch};
  const int err = b200::run_rounds(s, live, warp_cells, max_rounds, 4, graph != 0);
  strcpy(log, s.log.c_str());
  *running = s.running;
  return err;
}
