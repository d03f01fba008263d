// Checks chain_sum.cuh on the host: sums of random non-negative terms, taken in groups as the kernels take them (all at
// once in a shuffled order when the group allows it, else one by one), against the sequential sum, bit for bit.
#include <math.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <random>
#include <vector>

#include "chain_sum.cuh"

using namespace tn93;

int main()
{
  std::mt19937_64 rng(7);
  auto u = [&] { return (double)(rng() >> 11) * 0x1p-53; };
  long bad = 0, grouped = 0, single = 0;
  for (int trial = 0; trial < 4000; trial++) {
    const int kind = trial % 8, n = 1 + (int)(rng() % 3000), group = 1 << (rng() % 11);
    double s = kind == 6 ? 0x1p-950 * u() : kind == 7 ? 0x1p52 : 0.;
    std::vector<double> x(n);
    for (double &t : x) {
      if (kind == 0) t = 0.06 + 0.05 * u();                             // distances
      else if (kind == 1) t = rng() % 3 ? 0. : 0.001 * u();             // many identical pairs
      else if (kind == 2) t = ldexp(u(), (int)(rng() % 80) - 60);       // widely spread
      else if (kind == 3) t = ldexp((double)(rng() % 64), -(int)(rng() % 54));  // half-way cases
      else if (kind == 4) t = rng() % 500 ? u() : 1000. * (1 + rng() % 9);      // the maximum distance, weights
      else if (kind == 5) t = rng() % 700 ? u() : rng() % 2 ? INFINITY : NAN;
      else if (kind == 6) t = ldexp(u(), -900 - (int)(rng() % 170));
      else t = (double)(rng() % 5) / 2;
    }
    double want = s;
    for (double t : x) want += t;
    for (int a = 0; a < n; a += group) {
      const int m = std::min(group, n - a);
      ChainBinade c;
      bool ok = chain_binade(s, c);
      std::vector<double> r(m);
      for (int k = 0; k < m; k++) r[k] = chain_round(c, x[a + k], ok);
      std::shuffle(r.begin(), r.end(), rng);
      double tot = 0.;
      for (double t : r) tot += t;
      if (ok && s + tot < c.end) {
        s += tot;
        grouped++;
      } else {
        for (int k = 0; k < m; k++) s += x[a + k];
        single++;
      }
    }
    if (memcmp(&s, &want, 8) && !(s != s && want != want)) {
      if (bad++ < 5) printf("kind %d n %d group %d: %a, want %a\n", kind, n, group, s, want);
    }
  }
  printf("%ld groups at once, %ld one by one, %ld wrong\n", grouped, single, bad);
  return bad != 0 || grouped < 10000;
}
