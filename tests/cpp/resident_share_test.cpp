// Host check of the cut of narrow closed grids (csrc/resident_layout.h): bands of one or two whole
// rows that leave at least half the SMs to other solvers. Exit status 0 when all hold.
#include <cstdio>
#include <initializer_list>

#include "resident_layout.h"

int main() {
  using namespace lbm_b200;
  long bad = 0, n = 0;
  for (int nx = 1; nx <= 128; ++nx)
    for (int ny = 1; ny <= 126; ++ny)
      for (int elem : {4, 2}) {
        const ResLayout L = elem == 4 ? resident_layout<4>(nx, ny, 152, 32, false) : resident_layout<2>(nx, ny, 152, 28, false);
        const bool ok = L.tx == 1 && L.w == nx && L.hs <= 2 && 2 * L.ty <= 152 && L.ty <= ny;
        if (!ok && bad++ < 5) std::printf("%d x %d, %d bytes: %d x %d tiles of %d x %d\n", nx, ny, elem, L.tx, L.ty, L.w, L.hs);
        ++n;
      }
  std::printf("%ld cuts, %ld wrong\n", n, bad);
  return bad == 0 ? 0 : 1;
}
