// warp_host.h -- a warp on the CPU.  The 32 lanes are coroutines: each runs alone
// from one warp-wide operation to the next, in the order asked for, which is one
// of the schedules that independent threads of a warp may take.  A store that
// another lane's earlier load does not have to wait for is then seen by that load.
// Warp-wide operations order memory here, so what passes may still rely on more
// than the GPU promises; what fails is wrong there.
#pragma once
#include <ucontext.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <functional>
#include <random>
#include <type_traits>
#include <vector>

#define __host__
#define __device__
#define __forceinline__ inline
#define __align__(n) alignas(n)

using std::fabs;
using std::isnan;

struct alignas(16) uint4 { uint32_t x, y, z, w; };
struct alignas(16) float4 { float x, y, z, w; };
struct alignas(16) double2 { double x, y; };
inline double2 make_double2(double x, double y) { return {x, y}; }
inline unsigned __float_as_uint(float v) { unsigned u; memcpy(&u, &v, 4); return u; }
inline int __double2hiint(double v) { uint64_t u; memcpy(&u, &v, 8); return (int)(u >> 32); }

namespace warp_host {
struct Warp {
  ucontext_t sched, lane[32];
  bool done[32];
  int cur;
  uint64_t slot[32];
  std::function<void(int)> body;
};
inline Warp W;

inline void yield() { swapcontext(&W.lane[W.cur], &W.sched); }
inline void entry() {
  const int me = W.cur;
  W.body(me);
  W.done[me] = true;
  swapcontext(&W.lane[me], &W.sched);
}

// order 0: lanes upwards, 1: downwards, 2 and above: shuffled anew each time
// around (the number is the seed).
inline void run(std::function<void(int)> body, int order) {
  constexpr size_t kStack = 1 << 18;
  std::vector<char> stacks(32 * kStack);
  W.body = std::move(body);
  for (int l = 0; l < 32; ++l) {
    W.done[l] = false;
    getcontext(&W.lane[l]);
    W.lane[l].uc_stack.ss_sp = stacks.data() + l * kStack;
    W.lane[l].uc_stack.ss_size = kStack;
    W.lane[l].uc_link = nullptr;
    makecontext(&W.lane[l], entry, 0);
  }
  std::vector<int> idx(32);
  for (int l = 0; l < 32; ++l) idx[l] = order == 1 ? 31 - l : l;
  std::mt19937 rng((unsigned)order);
  for (bool any = true; any;) {
    any = false;
    if (order >= 2) std::shuffle(idx.begin(), idx.end(), rng);
    for (int l : idx) {
      if (W.done[l]) continue;
      any = true;
      W.cur = l;
      swapcontext(&W.sched, &W.lane[l]);
    }
  }
}

template <typename T>
T exchange(T v, int src) {
  const int me = W.cur;
  W.slot[me] = 0;
  memcpy(&W.slot[me], &v, sizeof(T));
  yield();
  T r;
  memcpy(&r, &W.slot[src], sizeof(T));
  yield();
  return r;
}
}  // namespace warp_host

inline void __syncwarp(unsigned = 0xffffffffu) { warp_host::yield(); }
template <typename T>
T __shfl_sync(unsigned, T v, int src, int width = 32) {
  return warp_host::exchange(v, warp_host::W.cur / width * width + src % width);
}
template <typename T>
T __shfl_xor_sync(unsigned, T v, int o, int = 32) { return warp_host::exchange(v, warp_host::W.cur ^ o); }
inline unsigned __reduce_max_sync(unsigned, unsigned v) {
  for (int o = 16; o > 0; o >>= 1) v = std::max(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
