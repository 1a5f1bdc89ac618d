// Host build of the choice of step graphs (csrc/step_graphs.h) for
// tests/test_step_graphs.py: for every line "finest faithful left" the role
// period, the steps of the graph and whether a handle's first run is direct.
#include <cstdio>

#include "step_graphs.h"

int main() {
  int finest, faithful, left;
  while (std::scanf("%d %d %d", &finest, &faithful, &left) == 3)
    std::printf("%d %d %d\n", lbx::role_period(finest, faithful != 0),
                lbx::graph_steps(finest, faithful != 0, left),
                (int)lbx::run_directly(finest, faithful != 0, left, 0));
  return 0;
}
