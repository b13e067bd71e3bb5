// Prints the dataflow factorization's layouts for the (nt, mixed, sms) triples
// on standard input: a line "grid rows helpers max_own", then a line of
// "i,j" pairs per CTA.
#include <cstdio>

#include "gba_factor_layout.h"

int main() {
  int nt, mixed, sms;
  while (std::scanf("%d %d %d", &nt, &mixed, &sms) == 3) {
    const gba::DfLayout l = gba::df_layout(nt, mixed != 0, sms);
    std::printf("%d %d %d %d\n", l.grid, l.rows, l.helpers, l.max_own);
    for (const auto& o : l.own) {
      for (const gba::DfTile& t : o) std::printf("%d,%d ", t.i, t.j);
      std::printf("\n");
    }
  }
  return 0;
}
