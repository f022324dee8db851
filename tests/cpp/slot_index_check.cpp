// SlotIndex on the CPU: for dense and closed sets (up to the widest and the
// deepest that one key holds, and one wider) every carried multi-index, its
// neighbours along unit steps and multi-indices outside the range are found or
// refused as TableSet::find does.  Built and run by tests/test_slot_index.py.
#include <cstdio>
#include <vector>

#include "tables.hpp"
using namespace dnnf90;

static int check(int d0, int k, int nseed, const int *seeds) {
  TableSet t;
  const std::string err = build_tables(d0, k, nseed, seeds, t);
  if (!err.empty()) { printf("tables: %s\n", err.c_str()); return 1; }
  const SlotIndex at(t);
  std::vector<int> b(d0);
  for (int ia = 0; ia < t.na; ++ia) {
    const int *a = &t.alpha[(size_t)ia * d0];
    if (at.find(a) != ia) { printf("slot %d\n", ia); return 1; }
    for (int i = 0; i < d0; ++i)
      for (int step : {-1, 1, 15}) {
        b.assign(a, a + d0);
        b[i] += step;
        if (at.find(b.data()) != t.find(b.data())) { printf("slot %d, step %d\n", ia, step); return 1; }
      }
  }
  printf("d0=%d k=%d na=%d ok\n", d0, k, t.na);
  return 0;
}

int main() {
  const int s2[] = {0, 1, 1, 0, 3, 0}, s3[] = {2, 1, 0, 0, 0, 15};
  std::vector<int> s16(16, 0), s17(17, 0);
  s16[0] = 2; s16[15] = 3; s17[16] = 2; s17[1] = 1;
  return check(1, 15, 0, nullptr) | check(4, 7, 0, nullptr) | check(2, 8, 0, nullptr) |
         check(2, 3, 3, s2) | check(3, 15, 2, s3) | check(16, 5, 1, s16.data()) |
         check(17, 3, 1, s17.data());
}
