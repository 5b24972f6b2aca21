// Test driver (CPU): what only set-up reads (the child-to-parent row maps) is not part of the
// device memory that a factorization holds.  Prints "ok <bytes held> <bytes of the maps>".
#include <cstdio>
#include <string>
#include <vector>

#include "gpu_cholesky.h"
using namespace tdem;

int main() {
  // lower triangle of a 12 x 12 x 12 grid's 7-point matrix
  const int k = 12, n = k * k * k;
  std::vector<int64_t> ptr{0};
  std::vector<int> col;
  for (int z = 0; z < k; ++z)
    for (int y = 0; y < k; ++y)
      for (int x = 0; x < k; ++x) {
        const int i = (z * k + y) * k + x;
        if (z) col.push_back(i - k * k);
        if (y) col.push_back(i - k);
        if (x) col.push_back(i - 1);
        col.push_back(i);
        ptr.push_back((int64_t)col.size());
      }
  Symbolic sy;
  const std::string e = analyse(n, ptr.data(), col.data(), nullptr, sy);
  if (!e.empty() || sy.rel.empty()) {
    printf("%s\n", e.c_str());
    return 1;
  }
  const int64_t maps = 4 * (int64_t)(sy.rel.size() + sy.front_parent.size()) + 8 * (int64_t)sy.rel_off.size();
  for (int elem : {4, 8}) {
    const int64_t held = GpuCholesky::bytes_needed(sy, 1, elem);
    Symbolic without = sy;
    without.rel.clear();
    without.rel_off.clear();
    without.front_parent.clear();
    const int64_t bare = GpuCholesky::bytes_needed(without, 1, elem);
    if (held != bare) {
      printf("%d-byte factor: %lld bytes with the maps, %lld without\n", elem, (long long)held, (long long)bare);
      return 1;
    }
    if (elem == 8) printf("ok %lld %lld\n", (long long)held, (long long)maps);
  }
  return 0;
}
