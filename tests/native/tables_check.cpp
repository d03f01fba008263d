// Checks the pair stage's derived tables against the per-site contributions they stand for, over every mode and every
// pair of codes: the operand image's class weights (their outer product is a site's whole contribution in the modes
// without resolution), and the event kernel's byte-lane tables and group length.
#include <stdio.h>
#include <string.h>

#include "tables.h"

using namespace tn93;

int main()
{
  static Tables T;
  int bad = 0;
  auto fail = [&](const char *what, int mode, int a, int b) {
    if (bad++ < 10) printf("%s: mode %d codes %d %d\n", what, mode, a, b);
  };
  for (int mode = 0; mode < 5; mode++) {
    unsigned char subset[kCodes] = {0};
    subset[5] = subset[6] = subset[kN] = 1;
    build_tables(&T, mode, subset);
    uint32_t w[kCodes];
    class_weights(mode, mode == 1 || mode == 2 || mode == 3, w);
    // the contribution (sixteenths: T, D, AG, CT, nfA, nfC, nfG) of a site, from the site table in the first sequence's
    // orientation; clean sites count one
    for (int a = 0; a < kCodes; a++)
      for (int b = 0; b < kCodes; b++) {
        double cell[16];
        const SiteEntry &S = T.site[0][a * kCodes + b];
        for (int q = 0; q < 16; q++) cell[q] = a < 4 && b < 4 ? (q == a * 4 + b) : S.fc[q] + (q % 5 ? 0 : S.icd[q / 5]);
        bool dyadic = true;
        for (int q = 0; q < 16; q++) dyadic &= cell[q] * 16 == (double)(long)(cell[q] * 16);
        double product[16];
        for (int q = 0; q < 16; q++)
          product[q] = (double)(w[a] >> 8 * (q >> 2) & 255u) * (double)(w[b] >> 8 * (q & 3) & 255u);
        if (mode >= 1 && mode <= 3) {
          const double gg = mode == 3 && a == kGap && b == kGap ? 1. : 0.;  // taken off again (counted as N against N)
          for (int q = 0; q < 16; q++)
            if (product[q] != (dyadic ? 16 * cell[q] + gg : 0.)) fail("weights", mode, a, b);
          if (!dyadic && !((a >= 11 && a <= 14) || (b >= 11 && b <= 14))) fail("not three-fold", mode, a, b);
        } else {
          for (int q = 0; q < 16; q++)
            if (product[q] != (a < 4 && b < 4 && q == a * 4 + b ? 1. : 0.)) fail("one-hot", mode, a, b);
        }
      }
    for (int wp = 0; wp < 2; wp++) {
      static EventTables E;
      event_tables(T, wp, &E);
      if (E.group < 4 || E.group % 4) fail("group", mode, E.group, wp);
      for (int c = kSparse0; c <= kGap; c++)
        for (int o = 0; o < kCodes; o++) {
          const int k = (c - kSparse0) * kCodes + o;
          const int32_t *v = T.ev[k].v;
          for (int side = 0; side < 2; side++) {
            const uint32_t *x = side ? E.col[k] : E.row[k];
            const bool zero = side && is_sparse_code(o, wp);
            // lanes as the kernel widens them: T | D, AG | CT, nfA | nfC, nfG | ambiguities
            const uint32_t p[4] = {x[0] & 0x00FF00FFu, x[0] >> 8 & 0x00FF00FFu, x[1] & 0x00FF00FFu, x[1] >> 8 & 0x00FF00FFu};
            for (int q = 0; q < 8; q++) {
              const uint32_t lane = q & 1 ? p[q / 2] >> 16 : p[q / 2] & 0xFFFFu;
              if (lane * (uint32_t)E.group > 255) fail("overflow", mode, c, o);
              if ((q < 7 ? lane << E.shift : lane) != (zero ? 0u : (uint32_t)v[q])) fail("lane", mode, c, o);
            }
          }
          if (E.flag[k] != v[8]) fail("flag", mode, c, o);
        }
    }
  }
  printf("bad %d\n", bad);
  return bad != 0;
}
