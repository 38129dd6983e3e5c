// Prints the plane range of a single-patch launch (drnum_b200/csrc/dn_range.h)
// for each patch "precision ni nj nk" read from standard input, and behind it the
// ranges that the autotuner measures.
#include <cstdio>

#include "dn_range.h"

int main()
{
  int prec, ni, nj, nk;
  while (std::scanf("%d %d %d %d", &prec, &ni, &nj, &nk) == 4) {
    const int tj = prec == 32 ? 16 : 4;
    const dn::RangeCost& c = prec == 32 ? dn::kRangeFx32 : dn::kRangeF64;
    std::printf("%d", dn::best_ranges(ni, nj, nk, tj, 32, 148, c, 1)[0]);
    for (int r : dn::best_ranges(ni, nj, nk, tj, 32, 148, c, prec == 32 ? 6 : 4, true)) std::printf(" %d", r);
    std::printf("\n");
  }
}
