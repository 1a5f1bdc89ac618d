// step_graphs.h -- how many steps of a run are captured into one CUDA graph
// (plain C++, so that the tests run it without the library).
#pragma once
#include <algorithm>

namespace lbx {

// Steps of level 0 after which every level's buffers are back in their roles.
// A level's two buffers are swapped by each of its steps, and a finer level takes
// an even number of them.  The faithful cycle rotates three buffers on each level
// but the finest, which swaps two of its three once a cycle of the level below.
inline int role_period(int finest, bool faithful) {
  if (finest > 0 && faithful) return finest == 1 ? 6 : 3;
  return 2;
}

// launches of a step, about
inline int step_launches(int finest) { return finest == 0 ? 1 : 4 << std::min(finest - 1, 8); }

// Steps of the graph that `left` steps are to be taken in, a multiple of the role
// period and at most `left`; 0: launch them directly.  Between the kernels of one
// graph there is no gap (chained, launch.cuh), between two replays there is:
// graphs of 32 launches, and of 8 for what is left (10x10x50 FP64, 60 steps: 4.1 us
// a step in graphs of two).  The faithful cycle's kernels are not chained: graphs
// of one period, so that runs of any length find theirs again (of at least eight
// steps, a run of nine was captured at each call).
inline int graph_steps(int finest, bool faithful, int left) {
  const int period = role_period(finest, faithful);
  if (finest > 0 && faithful) return left >= period ? period : 0;
  const int per_step = step_launches(finest);
  for (const int launches : {32, 8}) {
    const int steps = (std::max(1, launches / per_step) + period - 1) / period * period;
    if (left >= steps) return steps;
  }
  return 0;
}

// Whether a run of `left` steps is launched directly where no graph of it is at
// hand: as long as a handle has made fewer than kDirectLaunches this way, and no
// long run.  A graph of 32 launches takes about 100 us to make, and its replay
// little less than the direct launches, which are chained too.  us for the first
// 9 / 40 / 100 steps of a handle, graphs of two | graphs of 32 and 8 at once |
// this: 10x10x50 FP32 61 / 157 / 341 | 68 / 166 / 256 | 33 / 89 / 194, FP64 128 /
// 476 / 1,153 | 78 / 199 / 335 | 39 / 118 / 278; repeated calls alike.  The
// faithful cycle's launches are more and not chained: its graph pays at once
// (24^3, first 20 steps: 1,660 us, 1,885 with the first 128 launches direct).
constexpr long long kDirectLaunches = 128;
inline bool run_directly(int finest, bool faithful, int left, long long made) {
  return !(finest > 0 && faithful) && made < kDirectLaunches &&
         (long long)left * step_launches(finest) < 2 * kDirectLaunches;
}

}  // namespace lbx
