// Prints, for each sample count given, the largest distance of the library's
// fixed-point lgamma table (bdeu_table_into, eddy_host.cpp) from lgammal, in
// steps of the table.
#include <math.h>
#include <stdio.h>
#include <stdlib.h>

#include <vector>

#include "eddy_host.h"

int main(int argc, char **argv) {
  static const int D[eddy::kDivisors] = {1, 2, 3, 4, 6, 8, 9, 12, 16, 18, 24, 27, 36, 54, 81};
  for (int k = 1; k < argc; k++) {
    const int n = atoi(argv[k]);
    std::vector<int64_t> lg;
    int shift = 0;
    int8_t dmap[82];
    eddy::bdeu_table(n, lg, shift, dmap);
    long double worst = 0;
    for (int i = 0; i < eddy::kDivisors; i++) {
      const long double a = 4.0L / D[i], la = lgammal(a), scale = ldexpl(1.0L, shift);
      for (int m = 0; m <= n; m++)
        worst = fmaxl(worst, fabsl((lgammal(m + a) - la) * scale -
                                   (long double)lg[(size_t)dmap[D[i]] * (n + 1) + m]));
    }
    printf("%.6Lf\n", worst);
  }
}
