// The walk of the adjoint's list kernels at list lengths near 32 bits, on the host: prints one line per
// check, <name> <items visited> <last item>.
#define GP_HD inline
#include <stdio.h>

#include "gp_adjoint_cell.cuh"

static void walk(const char* name, int cells, int per, long long first, long long step) {
  long long n = 0, last = -1;
  for (gpadj::ListWalk w(cells, per, first, step); w.more(); w.next()) {
    if (w.at <= last) {  // wrapped
      printf("%s -1 %lld\n", name, (long long)w.at);
      return;
    }
    n++;
    last = w.at;
  }
  printf("%s %lld %lld\n", name, n, last);
}

int main() {
  const int top = 2147483647;
  walk("empty", 0, 4, 0, 75776);
  walk("one", 1, 4, 3, 75776);
  walk("faces_below", 536870911, 4, 5, 75776);  // 4 n still fits 32 bits
  walk("faces_at", 536870912, 4, 5, 75776);     // 4 n = 2^31
  walk("faces_top", top, 4, 75775, 75776);
  walk("cells_top", top, 1, 9468, 9472);        // the last stride passes 2^31
  return 0;
}
