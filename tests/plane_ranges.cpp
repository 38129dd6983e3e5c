// Prints the plane range of a single-patch launch (drnum_b200/csrc/dn_range.h)
// for each patch "precision ni nj nk" read from standard input.
#include <cstdio>

#include "dn_range.h"

int main()
{
  int prec, ni, nj, nk;
  while (std::scanf("%d %d %d %d", &prec, &ni, &nj, &nk) == 4)
    std::printf("%d\n", dn::best_ranges(ni, nj, nk, prec == 32 ? 16 : 4, 32, 148,
                                        prec == 32 ? dn::kRangeFx32 : dn::kRangeF64, 1)[0]);
}
