/* How lanes share the members of a reduction (lanes_within_int, lane_leaf,
 * csrc/reduce_core.cuh), on the host: for every count of lanes asked for, the
 * shares of those it gets lie end to end over [0, n), each within one member
 * of n / lanes, and no product leaves an int. */
#include <cstdio>

#include "b200shm.h"
#include "reduce_core.cuh"

int main() {
  const int sizes[] = {1,       2,           15,          16,      1 << 20, (1 << 27) - 1, 1 << 27,
                       (1 << 28) + 3, 1 << 30, 0x7fffff00, b200::kMaxMembers, 0x7fffffff};
  for (int n : sizes)
    for (int ask = 0; ask <= 5; ask++) {
      const int lg = b200::lanes_within_int(ask, n);
      if ((long long)n << lg > 0x7fffffffll || (ask && n <= 1 << 25 && lg != ask)) {
        printf("n %d lanes %d: got %d\n", n, 1 << ask, 1 << lg);
        return 1;
      }
      long long at = 0;
      for (int g = 0; g < 1 << lg; g++) {
        const long long lo = b200::lane_leaf(g, n, lg), hi = b200::lane_leaf(g + 1, n, lg);
        const long long even = n >> lg;
        if (lo != at || hi < lo || hi - lo < even || hi - lo > even + 1) {
          printf("n %d lanes %d: lane %d has [%lld, %lld), expected from %lld\n", n, 1 << lg, g, lo,
                 hi, at);
          return 1;
        }
        at = hi;
      }
      if (at != n) {
        printf("n %d lanes %d: the last lane ends at %lld\n", n, 1 << lg, at);
        return 1;
      }
    }
  puts("ok");
  return 0;
}
