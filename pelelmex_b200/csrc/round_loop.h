// round_loop.h -- the host side of a chunk's rounds: which launch shape they take,
// and the loop that launches them until no cell is live.
#pragma once

namespace b200 {

// Launch shapes of a round by how many cells are live: many (kernels in a row,
// right-hand sides by thread), fewer (setup kernels on a branch), few
// (right-hand sides by warp as well), and so few that the grids shrink to them.
// With the branch against without it, ms a react: 32^3 H2 4.56 and 5.03, 61x43x37
// CH4 44.3 and 45.8; above the line 64^3 H2 23.2 and 26.2, 64^3 CH4 54.2 and 55.8,
// 80^3 CH4 96.7 and 99.4, 80^3 dodecane 391 and 392, 96^3 H2 72.9 and 74.1, 96^3
// CH4 160.6 and 163.1; 128^3 CH4 445 and 408, where the kernels contend for L2.  So
// the two cross between one and two million cells, and the line lies at the
// largest size that was measured when it was drawn.
constexpr int kRoundClasses = 4;
constexpr int kForkCells = 131072;
constexpr int kTinyCells = 1024;

// Shape of a round with `live` cells; warp_cells: most cells that take the warp
// form of the right-hand sides.
inline int round_class(long long live, long long warp_cells) {
  return live <= kTinyCells ? 3 : live <= warp_cells ? 2 : live <= kForkCells ? 1 : 0;
}

// The shape after cls that a call comes to next, or kRoundClasses: a mechanism
// without a warp form (warp_cells 0) has no class 2.
inline int next_round_class(int cls, long long warp_cells) {
  for (++cls; cls < kRoundClasses; ++cls)
    if (cls == 1 ? warp_cells < kForkCells : cls == 2 ? warp_cells > kTinyCells : true) break;
  return cls;
}

// Launches per_check rounds at a time until none of the `live` cells is left.
// Ops: capture(cls) makes the graph of a shape, launch(cls) enqueues per_check
// rounds of it and the read of the live count, wait(&live) waits for both;
// timed_out() reports max_rounds.  All but timed_out return 0 or an error.
// The next shape's graph is made while the rounds of this one run.  Should that
// fail it is tried again when the shape is needed and nothing is running: the
// loop never returns while the GPU still works on the caller's arrays.
template <class Ops>
int run_rounds(Ops& ops, long long live, long long warp_cells, long long max_rounds, int per_check, bool graph) {
  bool captured[kRoundClasses] = {};
  for (long long round = 0; live > 0; round += per_check) {
    if (round >= max_rounds) return ops.timed_out();
    const int cls = round_class(live, warp_cells);
    int err = 0;
    if (graph && !captured[cls]) {
      err = ops.capture(cls);
      captured[cls] = err == 0;
    }
    if (!err) err = ops.launch(cls);
    const int next = next_round_class(cls, warp_cells);
    if (!err && graph && next < kRoundClasses && !captured[next]) captured[next] = ops.capture(next) == 0;
    long long left = 0;
    const int werr = ops.wait(&left);
    if (err || werr) return err ? err : werr;
    live = left;
  }
  return 0;
}

}  // namespace b200
