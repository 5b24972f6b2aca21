// Test driver (CPU): plans the model in argv[1] (A-form, two-point scheme) and prints, for
// argv[2] columns, the column groups that each level of the many-column solves takes.
#include <cstdio>
#include <cstdlib>
#include <string>

#include "driver.h"
using namespace tdem;

int main(int argc, char** argv) {
  if (argc < 3) return 2;
  TransientSolve ts;
  RunOptions opt;
  opt.scheme = 2;
  opt.formulation = 0;
  const std::string e = ts.plan(argv[1], opt);
  if (!e.empty() || !ts.planned_symbolic()) {
    printf("%s\n", e.c_str());
    return 1;
  }
  printf("ok");
  for (const LevelPlan& lp : ts.planned_symbolic()->levels) printf(" %d", solve_column_groups(lp, std::atoi(argv[2])));
  printf("\n");
  return 0;
}
