// Host build of the choice of step graphs (csrc/step_graphs.h) for
// tests/test_step_graphs.py: for every line "finest faithful left" the role
// period and the steps of the graph.
#include <cstdio>

#include "step_graphs.h"

int main() {
  int finest, faithful, left;
  while (std::scanf("%d %d %d", &finest, &faithful, &left) == 3)
    std::printf("%d %d\n", lbx::role_period(finest, faithful != 0),
                lbx::graph_steps(finest, faithful != 0, left));
  return 0;
}
