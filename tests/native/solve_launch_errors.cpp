// Test driver (CPU, no device): a solve whose CUDA calls fail says so.  Prints "ok <message>".
#include <cstdio>
#include <string>

#include "gpu_cholesky.h"
using namespace tdem;

int main() {
  GpuCholesky chol;
  std::string msg;
  for (int nrhs : {1, 2, 5, 40}) {  // streaming, block and one-unit-per-CTA solves
    msg = chol.solve(nullptr, nullptr, 0, nrhs, nullptr);
    if (msg.empty()) {
      printf("%d columns: no error\n", nrhs);
      return 1;
    }
    if (msg.find("CUDA") == std::string::npos) return 1;
    if (chol.solve_graph(nullptr, nullptr, 0, nrhs, nullptr).empty()) return 1;
  }
  printf("ok %s\n", msg.c_str());
  return 0;
}
