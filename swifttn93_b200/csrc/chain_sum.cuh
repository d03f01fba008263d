// chain_sum.cuh -- sums of non-negative doubles "in order" (s = s + t one term at a time, each sum rounded to nearest),
// evaluated in parallel with the same bits.
//
// While the running sum s stays in one binade [B, 2B), every rounded sum is a multiple of that binade's unit
// u = B 2^-52, so s + t rounds to s + r(t), where r(t) is t rounded to a multiple of u: the term's rounding does not
// depend on s, except when t lies exactly half way between two multiples (there the even result is taken, and which one
// is even depends on s). The r(t) are multiples of u whose sum stays below 2^53 u, so they add without error in any
// order. A group of terms is therefore added at once when it holds no half-way term and its total stays below 2B;
// otherwise a smaller group is tried, and 32 terms at the last are added one by one. Of a row of n like terms the groups
// that double the sum fail (about log2 n of them) and those with a half-way term: a term k bits below the sum is half way
// once in 2^k, so about ln n groups of 32.
#pragma once
#include "tn93_math.cuh"

namespace tn93 {

struct ChainBinade {
  double B, half, end;  // the binade [B, end) and half its unit
};

// the binade of s; false where the scheme does not apply (zero, tiny, infinite, negative or NaN)
TN_HD bool chain_binade(double s, ChainBinade &c)
{
  c.B = TDBL(TBITS(s) & 0x7FF0000000000000ull);
  c.half = TMUL(c.B, 0x1p-53);
  c.end = TMUL(c.B, 2.0);
  return s >= 0x1p-900 && s < 0x1p1000;
}

// t rounded to a multiple of the binade's unit; ok is cleared when t is half way between two of them or not a
// non-negative number (a term past the binade rounds coarser, and the total then lies past the binade too)
TN_HD double chain_round(const ChainBinade &c, double t, bool &ok)
{
  const double r = TSUB(TADD(c.B, t), c.B), e = TSUB(t, r);
  ok &= t >= 0. && e != c.half && e != -c.half;
  return r;
}

}  // namespace tn93
