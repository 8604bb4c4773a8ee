// csrc/kernels/tile_walk.cuh on the host.  A line "walk mt nt group_m extra" on standard input answers with the
// coordinates of tiles 0 to mt * nt + extra; "parts pairs tiles kt split_tiles split_pairs" with the parts of each pair's
// work, a line a pair.
#include <cstdio>
#include <cstring>

#define __device__
#define __forceinline__ inline
#include "kernels/tile_walk.cuh"

using namespace ft::gemm;

int main() {
  char what[16];
  int a, b, c, d, e;
  while (scanf("%15s", what) == 1) {
    if (!strcmp(what, "walk")) {
      if (scanf("%d %d %d %d", &a, &b, &c, &d) != 4) return 1;
      for (int t = 0; t <= a * b + d; ++t) {
        int mb = -1, nb = -1;
        tile_coords(t, a, b, mb, nb, c);
        printf("%d,%d ", mb, nb);
      }
      puts("");
    } else {
      if (scanf("%d %d %d %d %d", &a, &b, &c, &d, &e) != 5) return 1;
      for (int p = 0; p < a; ++p) {
        const PairWork work(p, a, b, c, d, e);
        WorkPart w;
        for (int i = 0; work.part(i, w); ++i) printf("%d,%d,%d ", w.tile, w.kb0, w.kb1);
        puts("");
      }
    }
  }
  return 0;
}
