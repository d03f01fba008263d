// split_pair.cuh -- the pair stage behind the tensor-core counts, as two kernels over the pairs' records:
//   event_kernel    adds the sparse ambiguity events (and N-plane cross terms) to each pair's clean-site record and takes
//                   tn93's -l, -g and site-order decisions; integers, 495 instructions per 32 pairs;
//   formula_kernel  the FP64 formula, its logarithms and the certificate; 807 instructions per 32 pairs, the FP64 pipe
//                   busy for half of its time (0.47 ms per 22.4 M pairs).
// One fused kernel (pair_kernel) holds the formula's registers through the event loads, whose latency then shows: it took
// 1,871 instructions per 32 pairs (a third more for the certificate, which ran for one ambiguous lane in six) and issued
// half of the time. Pair stage without the count kernel, per 22.4 M pairs of the 6,700 x 1,500 benchmark set: fused
// 2.10 ms, split 1.36 ms under resolve; serving 38 M pairs, counts included, 6.2 -> 5.0 ms.
// The fused kernel stays for the popcount path, for sequences with more than 1,023 events, for the N plane where its words
// are not listed (batches and servers), and where there is no room for the event offsets (pair_split).
// Under average, gapmm and skip the records hold whole pairs and formula_kernel runs alone.
//
// Included by engine.cu inside its unnamed namespace.

// Adds the table entries of the events [e0, e1) of one sequence (a multiple of 4 of them) against two partners, whose
// codes stand side by side at ccp (an even column of the position-major matrix): one 16-bit load serves both. An event
// is {offset of its column's codes, offset of its code's table row}, two to a 16-byte load, so that an event costs one
// address, one load and, per partner, one table address, one 8-byte shared load and two adds. Entries are 8 bytes of
// 8-bit lanes (EventTables), summed `group` events at a time before they could overflow and then widened to the 16-bit
// lanes of A and B: {T | D, AG | CT, nfA | nfC, nfG | ambiguities}. Four code loads (mostly L2) are in flight together.
// !PAIRED: one partner.
template <bool PAIRED>
__device__ __forceinline__ void add_events2(uint32_t (&A)[4], uint32_t (&B)[4], const unsigned char *tab, uint32_t group,
                                            const uint2 *ev2, const uint8_t *ccp, uint32_t e0, uint32_t e1)
{
  const uint4 *ep = reinterpret_cast<const uint4 *>(ev2 + e0);
  auto code = [&](uint32_t off) -> uint32_t {
    return PAIRED ? (uint32_t)__ldg(reinterpret_cast<const unsigned short *>(ccp + off)) : (uint32_t)__ldg(ccp + off);
  };
  uint2 s, t;
  auto add = [&](uint32_t row, uint32_t c) {
    const uint2 u = *reinterpret_cast<const uint2 *>(tab + (row + (PAIRED ? (c & 255u) : c) * 8));
    s.x += u.x;
    s.y += u.y;
    if (PAIRED) {
      const uint2 w = *reinterpret_cast<const uint2 *>(tab + (row + (c >> 8) * 8));
      t.x += w.x;
      t.y += w.y;
    }
  };
  for (int n = (int)(e1 - e0); n > 0;) {
    int g = min(n, (int)group);
    n -= g;
    s = t = make_uint2(0u, 0u);
    for (; g >= 8; g -= 8, ep += 4) {
      const uint4 x = __ldg(ep), y = __ldg(ep + 1), z = __ldg(ep + 2), w = __ldg(ep + 3);
      const uint32_t c0 = code(x.x), c1 = code(x.z), c2 = code(y.x), c3 = code(y.z);
      const uint32_t c4 = code(z.x), c5 = code(z.z), c6 = code(w.x), c7 = code(w.z);
      add(x.y, c0);
      add(x.w, c1);
      add(y.y, c2);
      add(y.w, c3);
      add(z.y, c4);
      add(z.w, c5);
      add(w.y, c6);
      add(w.w, c7);
    }
    if (g > 0) {
      const uint4 x = __ldg(ep), y = __ldg(ep + 1);
      ep += 2;
      const uint32_t c0 = code(x.x), c1 = code(x.z), c2 = code(y.x), c3 = code(y.z);
      add(x.y, c0);
      add(x.w, c1);
      add(y.y, c2);
      add(y.w, c3);
    }
    A[0] += s.x & 0x00FF00FFu;
    A[1] += (s.x >> 8) & 0x00FF00FFu;
    A[2] += s.y & 0x00FF00FFu;
    A[3] += (s.y >> 8) & 0x00FF00FFu;
    if (PAIRED) {
      B[0] += t.x & 0x00FF00FFu;
      B[1] += (t.x >> 8) & 0x00FF00FFu;
      B[2] += t.y & 0x00FF00FFu;
      B[3] += (t.y >> 8) & 0x00FF00FFu;
    }
  }
}

// The flags (EventTables::flag, in bits 30 and 31) of the three-fold events of one sequence against one partner: the
// only contributions that are not multiples of 1/16 involve a three-fold code, and few sequences have one.
__device__ __forceinline__ uint32_t three_flags(const uint8_t *flag, const uint32_t *ev, const uint8_t *ccp, uint32_t Np,
                                                uint32_t e0, uint32_t e1)
{
  uint32_t f = 0;
  for (uint32_t e = e0; e < e1; e++) {
    const uint32_t v = __ldg(ev + e), c = v & 31;
    if (c < 11 || c > 14) continue;
    f |= flag[(c - 4) * kCodes + __ldg(ccp + (size_t)(v >> 5) * Np)];
  }
  return f << 30;
}

// N-plane cross counts of one ordered pair: the N words of sequence s against the clean bases of p (sites with any base,
// with the hi bit, the lo bit, both)
struct WCross {
  int c, h, l, t;
};
__device__ __forceinline__ WCross w_cross(const uint64_t *planes, int NP, long Np, const uint32_t *wl, uint32_t q0,
                                          uint32_t q1, long s, long p)
{
  WCross x = {0, 0, 0, 0};
  for (uint32_t q = q0; q < q1; q++) {
    const uint64_t *P = planes + (size_t)__ldg(wl + q) * NP * Np;
    const uint64_t n = __ldg(P + 3 * Np + s);
    const uint64_t hi = __ldg(P + p), lo = __ldg(P + Np + p), cl = __ldg(P + 2 * Np + p);
    x.c += popc(n & cl);
    x.h += popc(n & hi);
    x.l += popc(n & lo);
    x.t += popc(n & hi & lo);
  }
  return x;
}

// What AVERAGE mode adds to the event sums of pair (i, j) past the -g test (PackedTables::avg words): the events of i
// against the codes of j, then those of j where i is not a sparse code itself (such a site is counted once, from i's
// side). Two forms: with few such pairs in a warp (high-ambiguity sequences that meet) the whole warp sums one pair, its
// lanes over the events, because one lane walking two lists of 60 events alone held its tile for 50 us; with many (a low
// -g, N runs) every lane sums its own pair, four events at a time.
__device__ __forceinline__ void avg_add(uint4 &s, const unsigned char *avg, uint2 e, uint32_t pc, bool skip)
{
  const uint4 t = *reinterpret_cast<const uint4 *>(avg + e.y * 2 + (skip ? 0u : pc) * 16);
  s.x += skip ? 0u : t.x;
  s.y += skip ? 0u : t.y;
  s.z += skip ? 0u : t.z;
  s.w += skip ? 0u : t.w;
}

__device__ __noinline__ uint4 avg_warp(const unsigned char *avg, bool wplane, const uint2 *ev2, const uint8_t *ccT,
                                       uint32_t ei0, uint32_t ei1, uint32_t ej0, uint32_t ej1, int i, int j)
{
  const uint32_t lane = threadIdx.x & 31;
  uint4 s = make_uint4(0u, 0u, 0u, 0u);
  for (uint32_t e = ei0 + lane; e < ei1; e += 32) {
    const uint2 v = __ldg(ev2 + e);
    avg_add(s, avg, v, __ldg(ccT + v.x + (uint32_t)j), false);
  }
  for (uint32_t e = ej0 + lane; e < ej1; e += 32) {
    const uint2 v = __ldg(ev2 + e);
    const uint32_t pc = __ldg(ccT + v.x + (uint32_t)i);
    avg_add(s, avg, v, pc, sparse_code((int)pc, wplane));
  }
  for (int o = 16; o; o >>= 1) {
    s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
    s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
    s.z += __shfl_xor_sync(0xffffffffu, s.z, o);
    s.w += __shfl_xor_sync(0xffffffffu, s.w, o);
  }
  return s;
}

__device__ __noinline__ uint4 avg_lane(const unsigned char *avg, bool wplane, const uint2 *ev2, const uint8_t *ccT,
                                       uint32_t ei0, uint32_t ei1, uint32_t ej0, uint32_t ej1, int i, int j)
{
  uint4 s = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll 1
  for (int side = 0; side < 2; side++) {
    const uint32_t e1 = side ? ej1 : ei1;
    const uint8_t *cp = ccT + (side ? i : j);
    for (uint32_t e = side ? ej0 : ei0; e < e1; e += 4) {
      const uint4 *q = reinterpret_cast<const uint4 *>(ev2 + e);
      const uint4 x = __ldg(q), y = __ldg(q + 1);
      const uint32_t c0 = __ldg(cp + x.x), c1 = __ldg(cp + x.z), c2 = __ldg(cp + y.x), c3 = __ldg(cp + y.z);
      avg_add(s, avg, make_uint2(x.x, x.y), c0, side && sparse_code((int)c0, wplane));
      avg_add(s, avg, make_uint2(x.z, x.w), c1, side && sparse_code((int)c1, wplane));
      avg_add(s, avg, make_uint2(y.x, y.y), c2, side && sparse_code((int)c2, wplane));
      avg_add(s, avg, make_uint2(y.z, y.w), c3, side && sparse_code((int)c3, wplane));
    }
  }
  return s;
}
constexpr int kAvgLanes = 6;  // pairs of a warp past the -g test from which each lane sums its own

// Tile of a block: rows x 64 columns, 16 warps. Column phase: lanes over the tile's rows, a warp-uniform column's events
// (and N words) into the shared accumulator; row phase: lanes over pairs of columns, a warp-uniform row's events, the
// records and the decisions. With 64 rows both phases take two partners per lane from one load; with the N plane the
// accumulator also holds the column's four cross counts and the tile has 32 rows. Two blocks of 16 warps a SM (64
// registers, no spills) beat three (40 registers; 6,700 x 1,500 pair stage 1.98 against 2.11 ms). Rows and columns are kept at slots
// (x & 1) * 32 + x / 2 (64 of them) so that the two partners of a lane stand 32 slots apart: 16-byte accesses without
// bank conflicts.
constexpr int kEvThreads = 512;
constexpr int kEvCols = 64;
template <bool WPLANE>
struct EvTile {
  static constexpr int rows = WPLANE ? 32 : 64;
  static constexpr int words = WPLANE ? 8 : 4;                 // accumulator words of a pair
  static constexpr int stride = kEvCols * words + 4;           // words of a row (+4: conflict-free column phase)
  static constexpr size_t tab = (sizeof(EventTables) + sizeof(((PackedTables *)0)->avg) + 5 * sizeof(AggEntry) + 15) / 16 * 16;
  static constexpr size_t off = tab + (size_t)rows * stride * 4;  // event offsets of the tile's rows, then its columns
  static constexpr size_t smem = off + (size_t)(rows + 1 + kEvCols + 1) * 4;
};

// the -l limit in sixteenths of a site (a pair's total is below 2^29)
__device__ __forceinline__ int overlap16(const RunConsts &rc) { return 16 * (int)max(-1l, min(rc.min_overlap, 1l << 26)); }

__device__ __forceinline__ int next_item(int *counter)
{
  int x = 0;
  if ((threadIdx.x & 31) == 0) x = atomicAdd(counter, 1);
  return __shfl_sync(0xffffffffu, x, 0);
}

__device__ __forceinline__ int ev_slot(int x) { return (x & 1) * 32 + (x >> 1); }

// tile (bx, by) of the columns from a.cstart and the rows from a.r0, by all threads of the block
template <bool WPLANE, bool PACK>
__device__ __forceinline__ void event_tile(const PairArgs &a, int bx, int by)
{
  using T = EvTile<WPLANE>;
  extern __shared__ __align__(16) unsigned char smem[];
  const RunConsts &rc = a.rc;
  __shared__ int items[2];  // next column, next row: warps take them one by one, as list lengths differ
  const int lane = threadIdx.x & 31;
  if (threadIdx.x < 2) items[threadIdx.x] = 0;
  // tiles start on even rows and columns (two codes per load); rows before r0 and columns before colbase are skipped
  const int i0 = (int)(a.r0 & ~1l) + by * T::rows, j0 = (int)(a.cstart & ~1l) + bx * kEvCols;
  const int N = (int)rc.N, r1 = (int)a.r1, cend = (int)a.cend;
  if (i0 >= r1 || j0 >= cend || (!rc.cross && j0 + kEvCols - 1 <= i0)) return;
  const EventTables &ET = *reinterpret_cast<const EventTables *>(smem);
  const unsigned char *avg = smem + sizeof(EventTables);
  const AggEntry *EW = reinterpret_cast<const AggEntry *>(smem + sizeof(EventTables) + sizeof(a.tab->packed.avg));
  uint32_t *acc = reinterpret_cast<uint32_t *>(smem + T::tab);
  uint32_t *soff = reinterpret_cast<uint32_t *>(smem + T::off);
  {
    const int n0 = (int)(sizeof(EventTables) / 16);
    const int n1 = rc.fallback_avg ? (int)(sizeof(a.tab->packed.avg) / 16) : 0;
    const int n2 = WPLANE ? (int)(5 * sizeof(AggEntry) / 16) : 0;
    const uint4 *s0 = reinterpret_cast<const uint4 *>(&a.tab->events);
    const uint4 *s1 = reinterpret_cast<const uint4 *>(a.tab->packed.avg);
    const uint4 *s2 = reinterpret_cast<const uint4 *>(&a.tab->agg[kEvEntries]);
    uint4 *d0 = reinterpret_cast<uint4 *>(smem);
    uint4 *d1 = reinterpret_cast<uint4 *>(smem + sizeof(EventTables));
    uint4 *d2 = d1 + sizeof(a.tab->packed.avg) / 16;
    for (int t = threadIdx.x; t < T::rows + 1 + kEvCols + 1; t += kEvThreads)
      soff[t] = a.ev_off[min(t <= T::rows ? i0 + t : j0 + t - T::rows - 1, N)];
    for (int t = threadIdx.x; t < n0; t += kEvThreads) d0[t] = s0[t];
    for (int t = threadIdx.x; t < n1; t += kEvThreads) d1[t] = s1[t];
    for (int t = threadIdx.x; t < n2; t += kEvThreads) d2[t] = s2[t];
  }
  __syncthreads();
  const uint32_t Np = (uint32_t)rc.Npad;
  const uint32_t group = (uint32_t)ET.group;
  const int shift = ET.shift;
  const bool three = a.three != nullptr;
  {
    const int ib = WPLANE ? min(i0 + lane, (int)Np - 1) : min(i0 + 2 * lane, (int)Np - 2);
    const int iw = min(i0 + lane, N - 1);
    for (int cl = next_item(&items[0]); cl < kEvCols; cl = next_item(&items[0])) {
      const int j = j0 + cl;
      if (j >= cend || (!rc.cross && j <= i0)) continue;  // no pair of the tile reads this column
      uint32_t A[4] = {0u, 0u, 0u, 0u}, B[4] = {0u, 0u, 0u, 0u};
      const uint32_t e0 = soff[T::rows + 1 + cl], e1 = soff[T::rows + 2 + cl];
      add_events2<!WPLANE>(A, B, smem + sizeof ET.row, group, a.ev2, a.ccT + ib, e0, e1);
      if (three && a.three[j]) {
        A[3] |= three_flags(ET.flag, a.ev, a.ccT + ib, Np, e0, e1);
        if (!WPLANE) B[3] |= three_flags(ET.flag, a.ev, a.ccT + ib + 1, Np, e0, e1);
      }
      uint32_t *dst = acc + lane * T::stride + ev_slot(cl) * T::words;
      *reinterpret_cast<uint4 *>(dst) = make_uint4(A[0], A[1], A[2], A[3]);
      if (WPLANE) {
        const WCross x = w_cross(a.planes, rc.NP, rc.Npad, a.wl, a.wl_off[j], a.wl_off[j + 1], j, iw);
        *reinterpret_cast<int4 *>(dst + 4) = make_int4(x.c, x.h, x.l, x.t);
      } else {
        *reinterpret_cast<uint4 *>(dst + 32 * T::stride) = make_uint4(B[0], B[1], B[2], B[3]);
      }
    }
  }
  __syncthreads();
  const long tn = a.tcncols ? a.tcncols : a.ncols, tb = a.tcncols ? a.tccolbase : a.colbase;
  // the constant columns' share of packed words
  const uint32_t cw[3] = {16u * (uint32_t)rc.constT * 0x10001u,
                          16u * ((uint32_t)rc.constNf[0] + ((uint32_t)rc.constNf[1] << 16)), 16u * (uint32_t)rc.constNf[2]};
  const int jmin = (int)tb, jmax = (int)min(a.cend, tb + tn);
  // below this share of the sites (less a margin over single precision) the -g test cannot fire
  const float gfloor = (float)(rc.resolve_fraction / 16.0) * 0.9999f;
  const int l16 = overlap16(rc);
  const int jp = min(j0 + 2 * lane, (int)Np - 2);
  for (int r = next_item(&items[1]); r < T::rows; r = next_item(&items[1])) {
    const int i = i0 + r;
    if (i >= r1) break;
    const int lb = rc.cross ? (int)rc.n1 : i + 1;
    if (i < a.r0 || j0 + kEvCols <= lb) continue;
    const size_t at0 = (size_t)(i - a.r0) * tn + (j0 - tb);
    uint32_t P[2][4];
    WCross wc[2];
    const uint32_t *src = acc + (WPLANE ? r : ev_slot(r)) * T::stride;
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const uint32_t *s = src + (h * 32 + lane) * T::words;
      const uint4 x = *reinterpret_cast<const uint4 *>(s);
      P[h][0] = x.x;
      P[h][1] = x.y;
      P[h][2] = x.z;
      P[h][3] = x.w;
      if (WPLANE) {
        const int4 y = *reinterpret_cast<const int4 *>(s + 4);
        wc[h] = WCross{y.x, y.y, y.z, y.w};
      }
    }
    // slots of columns outside the tile's valid range were not written: their pairs are not stored below
    const uint32_t e0 = soff[r], e1 = soff[r + 1];
    // the packed records are read before the events, whose loads then hide theirs
    uint4 g2[2];
    if (PACK) {
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int j = j0 + 2 * lane + h;
        g2[h] = (j < max(lb, jmin) || j >= jmax) ? make_uint4(0u, 0u, 0u, 0u)
                                                 : reinterpret_cast<const uint4 *>(a.tcagg)[at0 + 2 * lane + h];
      }
    }
    add_events2<true>(P[0], P[1], smem, group, a.ev2, a.ccT + jp, e0, e1);
    if (three && a.three[i]) {
      P[0][3] |= three_flags(ET.flag, a.ev, a.ccT + jp, Np, e0, e1);
      P[1][3] |= three_flags(ET.flag, a.ev, a.ccT + jp + 1, Np, e0, e1);
    }
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int j = j0 + 2 * lane + h;
      const bool valid = j >= max(lb, jmin) && j < jmax;
      const size_t at = at0 + 2 * lane + h;
      const uint32_t flags = P[h][3] >> 30;
      int amb = (int)(P[h][3] >> 16 & 0x3FFFu);
      int ag[7];
      uint32_t w[4] = {P[h][0] << shift, P[h][1] << shift, P[h][2] << shift, (P[h][3] & 0xFFFFu) << shift};
      if (PACK) {
        // no lane of the sum passes 65,535 (32 L < 65,536), so the packed words add as they are
        const uint4 g = g2[h];
        w[0] += (g.x << 4) + cw[0];
        w[1] += g.y << 4;
        w[2] += (g.z << 4) + cw[1];
        w[3] += (g.w << 4) + cw[2];
        ag[0] = (int)(w[0] & 0xFFFFu);
      } else {
        int cl[7] = {0, 0, 0, 0, 0, 0, 0};
        if (!valid) {
        } else if (a.tc16) {
          const uint4 g = reinterpret_cast<const uint4 *>(a.tcagg)[at];
          cl[0] = (int)(g.x & 0xFFFFu);
          cl[1] = (int)(g.x >> 16);
          cl[2] = (int)(g.y & 0xFFFFu);
          cl[3] = (int)(g.y >> 16);
          cl[4] = (int)(g.z & 0xFFFFu);
          cl[5] = (int)(g.z >> 16);
          cl[6] = (int)(g.w & 0xFFFFu);
        } else {
          const uint4 *g = reinterpret_cast<const uint4 *>(a.tcagg) + 2 * at;
          const uint4 g0 = g[0], g1 = g[1];
          cl[0] = (int)g0.x;
          cl[1] = (int)g0.y;
          cl[2] = (int)g0.z;
          cl[3] = (int)g0.w;
          cl[4] = (int)g1.x;
          cl[5] = (int)g1.y;
          cl[6] = (int)g1.z;
        }
        ag[0] = 16 * (cl[0] + (int)rc.constT) + (int)(w[0] & 0xFFFFu);
        ag[1] = 16 * (cl[1] + (int)rc.constT) + (int)(w[0] >> 16);
        ag[2] = 16 * cl[2] + (int)(w[1] & 0xFFFFu);
        ag[3] = 16 * cl[3] + (int)(w[1] >> 16);
        ag[4] = 16 * (cl[4] + (int)rc.constNf[0]) + (int)(w[2] & 0xFFFFu);
        ag[5] = 16 * (cl[5] + (int)rc.constNf[1]) + (int)(w[2] >> 16);
        ag[6] = 16 * (cl[6] + (int)rc.constNf[2]) + (int)w[3];
      }
      int wb[5] = {0, 0, 0, 0, 0};
      if (WPLANE && valid) {
        // the row's N words against the column's clean bases and N sites, plus the column's share
        const uint32_t q0 = a.wl_off[i], q1 = a.wl_off[i + 1];
        int nWW = 0;
        for (uint32_t q = q0; q < q1; q++) {
          const uint64_t *Pw = a.planes + (size_t)__ldg(a.wl + q) * rc.NP * Np;
          const uint64_t ni = __ldg(Pw + 3 * (size_t)Np + i);
          const uint64_t hj = __ldg(Pw + j), lj = __ldg(Pw + Np + j), cj = __ldg(Pw + 2 * (size_t)Np + j);
          wc[h].c += popc(ni & cj);
          wc[h].h += popc(ni & hj);
          wc[h].l += popc(ni & lj);
          wc[h].t += popc(ni & hj & lj);
          nWW += popc(ni & __ldg(Pw + 3 * (size_t)Np + j));
        }
        wb[3] = wc[h].t;
        wb[1] = wc[h].h - wc[h].t;
        wb[2] = wc[h].l - wc[h].t;
        wb[0] = wc[h].c - wb[1] - wb[2] - wb[3];
        wb[4] = nWW;
#pragma unroll
        for (int b = 0; b < 5; b++) {
#pragma unroll
          for (int q = 0; q < 7; q++) ag[q] += wb[b] * EW[b].v[q];
          amb += wb[b] * EW[b].v[7];
        }
      }
      // tn93's decisions: a pair with a contribution that is not a multiple of 1/16 takes the site-order walk; past the
      // -g test it is recomputed with -a average (refkernel.cpp:742-750), here by adding the differences of its events
      // and N-plane counts (or by the walk when those are not multiples of 1/16); at or below the overlap it is skipped
      uint32_t state = flags & 1u;
      if (rc.fallback_avg) {
        bool avgs = false;
        if (valid && !state && !((float)ag[0] * gfloor > (float)amb)) {
          const double tng = (double)ag[0] / 16.0;
          avgs = tng > (double)rc.min_overlap && tng * rc.resolve_fraction <= (double)amb;
          if (avgs && (flags & 2u)) {
            state = 1 | 4;
            avgs = false;
          }
        }
        unsigned m = __ballot_sync(0xffffffffu, avgs);
        if (m) {
          uint4 d = make_uint4(0u, 0u, 0u, 0u);
          const uint32_t *co = soff + T::rows + 1;
          if (__popc(m) >= kAvgLanes) {
            if (avgs) d = avg_lane(avg, rc.wplane, a.ev2, a.ccT, e0, e1, co[j - j0], co[j - j0 + 1], i, j);
          } else {
            for (; m; m &= m - 1) {
              const int from = __ffs(m) - 1, jc = 2 * from + h;
              const uint4 x = avg_warp(avg, rc.wplane, a.ev2, a.ccT, e0, e1, co[jc], co[jc + 1], i, j0 + jc);
              if (lane == from) d = x;
            }
          }
          if (avgs) {
            if (PACK) {
              // the differences' words are low + high * 65536 of signed lanes, so they add to packed words too
              w[0] += d.x;
              w[1] += d.y;
              w[2] += d.z;
              w[3] += d.w;
              ag[0] = (int)(w[0] & 0xFFFFu);
            } else {
              ag[0] += lane_lo(d.x);
              ag[1] += lane_hi(d.x);
              ag[2] += lane_lo(d.y);
              ag[3] += lane_hi(d.y);
              ag[4] += lane_lo(d.z);
              ag[5] += lane_hi(d.z);
              ag[6] += (int)d.w;
            }
            if (WPLANE) {
#pragma unroll
              for (int b = 0; b < 5; b++)
#pragma unroll
                for (int q = 0; q < 7; q++) ag[q] += wb[b] * (EW[b].v[9 + q] - EW[b].v[q]);
            }
          }
        }
      }
      if (!valid) continue;
      if (state) {
        const unsigned idx = atomicAdd(a.replay_n, 1u);
        if (idx < a.replay_cap)
          a.replay_q[idx] = ((unsigned long long)(state >> 2) << 63) | ((unsigned long long)i << 31) | (unsigned long long)j;
        state = 1;
      } else if (ag[0] <= l16) {
        state = 2;
      }
      if (PACK) {
        reinterpret_cast<uint4 *>(a.tcagg)[at] = make_uint4(w[0], w[1], w[2], w[3] | state << 16);
      } else if (a.tc16) {
        reinterpret_cast<uint4 *>(a.tcagg)[at] =
            make_uint4((uint32_t)ag[0] | (uint32_t)ag[1] << 16, (uint32_t)ag[2] | (uint32_t)ag[3] << 16,
                       (uint32_t)ag[4] | (uint32_t)ag[5] << 16, (uint32_t)ag[6] | state << 16);
      } else {
        uint4 *d = reinterpret_cast<uint4 *>(a.tcagg) + 2 * at;
        d[0] = make_uint4((uint32_t)ag[0], (uint32_t)ag[1], (uint32_t)ag[2], (uint32_t)ag[3]);
        d[1] = make_uint4((uint32_t)ag[4], (uint32_t)ag[5], (uint32_t)ag[6], state);
      }
    }
  }
}

template <bool WPLANE, bool PACK>
__global__ void __launch_bounds__(kEvThreads, 2) event_kernel(PairArgs a)
{
  event_tile<WPLANE, PACK>(a, blockIdx.x, blockIdx.y);
}

// A batch of alignments: each block's (descriptor, bx, by, z). A descriptor's copy in shared memory, for all threads.
__device__ __forceinline__ const PairArgs &batch_args(const PairArgs *descs, int k)
{
  __shared__ __align__(16) unsigned char raw[sizeof(PairArgs)];
  for (int q = threadIdx.x; q < (int)(sizeof(PairArgs) / 4); q += blockDim.x)
    reinterpret_cast<int32_t *>(raw)[q] = reinterpret_cast<const int32_t *>(&descs[k])[q];
  __syncthreads();
  return *reinterpret_cast<const PairArgs *>(raw);
}

template <bool WPLANE, bool PACK>
__global__ void __launch_bounds__(kEvThreads, 2) event_batch_kernel(const PairArgs *descs, const int4 *blocks)
{
  const int4 b = blocks[blockIdx.x];
  event_tile<WPLANE, PACK>(batch_args(descs, b.x), b.y, b.z);
}

// Whether pair (i, j) has a contribution that is not a multiple of 1/16 in a run whose records hold everything else: the
// three-fold events of either sequence against the other's codes. Out of line: few sequences have one.
__device__ __noinline__ bool three_pair(const uint8_t *flag, const uint8_t *three, const uint32_t *ev_off,
                                        const uint32_t *ev, const uint8_t *ccT, uint32_t Np, int i, int j)
{
  uint32_t f = 0;
  if (three[i]) f |= three_flags(flag, ev, ccT + j, Np, ev_off[i], ev_off[i + 1]);
  if (three[j]) f |= three_flags(flag, ev, ccT + i, Np, ev_off[j], ev_off[j + 1]);
  return f >> 30 & 1u;
}

// The formula for the records that event_kernel finished (state 0; 1: queued for the site-order walk, 2: skipped by -l).
// A warp takes a segment of segw columns of rpw rows; the launch's columns are [jlo, jhi), jhi at most cend. The record's x16 integers go into the formula as they are: every
// quantity scales by a power of two, so each quotient is the same double. A logarithm that the C library may round the
// other way (17% of the pairs have one, so nearly every warp step would run the certificate for a few lanes) puts the
// pair's range in a per-warp queue, and the certificate runs for 32 queued pairs at a time.
// LIN (average, gapmm, skip): the records come straight from the count kernel, in sixteenths with the ambiguity codes'
// weights in them. What is left is the constant columns, under gapmm the sites where both have a gap (counted as N
// against N by the weights, nothing to tn93; from the gap words of the row), the -l test and the pairs with three-fold
// codes. Against the event kernel of those modes: 6,700 x 1,500 pair stage 1.95 -> 1.48 ms under average, 2.77 -> 1.61 ms
// under gapmm.
constexpr int kFmQueue = 64;
template <bool REC16, bool LIN>
__device__ __forceinline__ void formula_rows(const PairArgs &a, long jlo, long jhi, int segw, int rpw, int bx, int by)
{
  __shared__ double qlo[kWarps][kFmQueue], qhi[kWarps][kFmQueue];
  __shared__ int qi[kWarps][kFmQueue], qj[kWarps][kFmQueue];
  const RunConsts &rc = a.rc;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long tn = a.tcncols ? a.tcncols : a.ncols, tb = a.tcncols ? a.tccolbase : a.colbase;
  const int l16 = overlap16(rc);
  int namb = 0, nund = 0, qn = 0, wunit = -1;
  AmbLane al;  // lanes' totals of the warp's unit wunit
  al.unit = -1;
  auto drain = [&](int n) {  // the certificate of the n <= 32 oldest queued pairs, one per lane
    int unit = -1;
    double lo = 0., hi = 0., w = 0.;
    if (lane < n) {
      Dist D;
      D.lo = qlo[warp][lane];
      D.hi = qhi[warp][lane];
      const long i = qi[warp][lane], j = qj[warp][lane];
      if (rc.resolve_all || !certified(D, rc)) {
        nund++;
        if (a.ex.und_list) {
          const unsigned idx = atomicAdd(a.ex.und_n, 1u);
          if (idx < a.ex.und_cap) {
            a.ex.und_list[2 * (size_t)idx] = (unsigned long long)a.ex.und_k;
            a.ex.und_list[2 * (size_t)idx + 1] = ((unsigned long long)i << 32) | (unsigned long long)j;
          }
        }
      }
      if (a.ex.amb) {
        unit = a.ex.colunit ? a.ex.colunit[j - a.colbase] : fst_bin(rc, i, j);
        w = (double)(a.ex.counts[i] * a.ex.counts[j]);
        lo = D.lo <= 0. ? 0. : D.lo;
        hi = D.hi <= 0. ? 0. : D.hi;
      }
    }
    if (!a.ex.amb) return;
    // lanes of the warp's own unit keep their totals; the pairs of any other unit are added up and sent at once
    if (wunit < 0) wunit = __shfl_sync(0xffffffffu, unit, 0);
    AmbLane other;
    other.unit = -1;
    if (unit == wunit)
      amb_add(a.ex.amb, al, unit, lo, hi, w);
    else if (unit >= 0)
      amb_add(a.ex.amb, other, unit, lo, hi, w);
    amb_warp_flush(a.ex.amb, other);
  };
  const long ra = a.r0 + (bx * (long)kWarps + warp) * rpw, rb = min(a.r1, ra + rpw);
  for (long i = ra; i < rb; i++) {
    const long lb = rc.cross ? rc.n1 : i + 1;
    const long s0 = (rc.cross ? jlo : max(lb, jlo)) + (long)by * segw;
    const long c0 = max(lb, s0), c1 = min(jhi, s0 + segw);
    const size_t rec0 = (size_t)(i - a.r0) * tn - tb;
    double *const drow = a.dist + (size_t)(i - a.r0) * a.ncols - a.colbase;
    uint32_t q0 = 0, q1 = 0;
    uint64_t gw = 0;
    bool ti = false;
    if (LIN) {
      if (rc.gapmm) {
        if (a.wl_off) {
          q0 = a.wl_off[i];
          q1 = a.wl_off[i + 1];
        } else {
          // no word lists (a batch): the row's nonzero gap words among the first 64 as a mask, the words past them all (24
          // alignments of 900-3,000 columns: 0.33 ms of formula with every word read, 0.24 so)
          const uint64_t *G = a.planes + 4 * rc.Npad + i;
          const bool g0 = lane < rc.W && __ldg(G + (size_t)lane * rc.NP * rc.Npad);
          const bool g1 = lane + 32 < rc.W && __ldg(G + (size_t)(lane + 32) * rc.NP * rc.Npad);
          gw = (uint64_t)__ballot_sync(0xffffffffu, g0) | (uint64_t)__ballot_sync(0xffffffffu, g1) << 32;
          q0 = 64;
          q1 = (uint32_t)max(64l, rc.W);
        }
      }
      ti = a.three && a.three[i];
    }
    for (long j0 = c0; j0 < c1; j0 += 32) {
      const long j = j0 + lane;
      uint32_t state = 1;
      int ag[7];
      if (j < c1) {
        if (REC16) {
          const uint4 g = __ldcs(reinterpret_cast<const uint4 *>(a.tcagg) + rec0 + j);
          ag[0] = (int)(g.x & 0xFFFFu);
          ag[1] = (int)(g.x >> 16);
          ag[2] = (int)(g.y & 0xFFFFu);
          ag[3] = (int)(g.y >> 16);
          ag[4] = (int)(g.z & 0xFFFFu);
          ag[5] = (int)(g.z >> 16);
          ag[6] = (int)(g.w & 0xFFFFu);
          state = g.w >> 16;
        } else {
          const uint4 *g = reinterpret_cast<const uint4 *>(a.tcagg) + 2 * (rec0 + j);
          const uint4 g0 = __ldcs(g), g1 = __ldcs(g + 1);
          ag[0] = (int)g0.x;
          ag[1] = (int)g0.y;
          ag[2] = (int)g0.z;
          ag[3] = (int)g0.w;
          ag[4] = (int)g1.x;
          ag[5] = (int)g1.y;
          ag[6] = (int)g1.z;
          state = g1.w;
        }
        if (LIN) {
          state = 0;
          ag[0] += 16 * (int)rc.constT;
          ag[1] += 16 * (int)rc.constT;
          ag[4] += 16 * (int)rc.constNf[0];
          ag[5] += 16 * (int)rc.constNf[1];
          ag[6] += 16 * (int)rc.constNf[2];
          if (rc.gapmm) {
            int n = 0;
            auto gaps = [&](uint32_t w) {
              const uint64_t *G = a.planes + ((size_t)w * rc.NP + 4) * rc.Npad;
              n += popc(__ldg(G + i) & __ldg(G + j));
            };
            for (uint64_t m = gw; m; m &= m - 1) gaps((uint32_t)__ffsll((long long)m) - 1);
            for (uint32_t q = q0; q < q1; q++) gaps(a.wl_off ? __ldg(a.wl + q) : q);
            ag[0] -= 16 * n;
            ag[1] -= 4 * n;
            ag[2] -= 2 * n;
            ag[3] -= 2 * n;
            ag[4] -= 8 * n;
            ag[5] -= 8 * n;
            ag[6] -= 8 * n;
          }
          if (a.three && (ti || a.three[j]) &&
              three_pair(a.tab->events.flag, a.three, a.ev_off, a.ev, a.ccT, (uint32_t)rc.Npad, (int)i, (int)j)) {
            const unsigned idx = atomicAdd(a.replay_n, 1u);
            if (idx < a.replay_cap) a.replay_q[idx] = ((unsigned long long)i << 31) | (unsigned long long)j;
            state = 1;
          } else if (ag[0] <= l16) {
            state = 2;
          }
        }
        if (state == 2) drow[j] = __longlong_as_double((long long)kSkipBits);
      }
      bool amb = false;
      double lo = 0., hi = 0.;
      if (state == 0) {
        const double nf[4] = {(double)ag[4], (double)ag[5], (double)ag[6], (double)(2 * ag[0] - ag[4] - ag[5] - ag[6])};
        const Dist D = tn93_distance(*a.logt, nf, (double)ag[1], (double)ag[2], (double)ag[3], rc.log_band, rc.log_spread);
        drow[j] = D.d;
        amb = D.amb != 0;
        lo = D.lo;
        hi = D.hi;
      }
      const unsigned m = __ballot_sync(0xffffffffu, amb);
      if (m) {
        if (amb) {
          const int at = qn + __popc(m & lanemask_lt());
          qlo[warp][at] = lo;
          qhi[warp][at] = hi;
          qi[warp][at] = (int)i;
          qj[warp][at] = (int)j;
          namb++;
        }
        qn += __popc(m);
        __syncwarp();
        if (qn >= 32) {
          drain(32);
          qn -= 32;
          const double l2 = qlo[warp][32 + lane], h2 = qhi[warp][32 + lane];
          const int i2 = qi[warp][32 + lane], j2 = qj[warp][32 + lane];
          __syncwarp();
          if (lane < qn) {
            qlo[warp][lane] = l2;
            qhi[warp][lane] = h2;
            qi[warp][lane] = i2;
            qj[warp][lane] = j2;
          }
          __syncwarp();
        }
      }
    }
  }
  if (qn) drain(qn);
  count_flags(a.counters, namb, nund);
  if (a.ex.amb) amb_warp_flush(a.ex.amb, al);
}

template <bool REC16, bool LIN>
__global__ void __launch_bounds__(256, 3) formula_kernel(PairArgs a, long jlo, long jhi, int segw, int rpw)
{
  formula_rows<REC16, LIN>(a, jlo, jhi, segw, rpw, blockIdx.x, blockIdx.y);
}

// a batch of alignments: each block's (descriptor, bx, by, rows per warp * 2048 + columns of a segment)
template <bool REC16, bool LIN>
__global__ void __launch_bounds__(256, 3) formula_batch_kernel(const PairArgs *descs, const int4 *blocks)
{
  const int4 b = blocks[blockIdx.x];
  const PairArgs &a = batch_args(descs, b.x);
  formula_rows<REC16, LIN>(a, 0, a.cend, b.w & 2047, b.w >> 11, b.y, b.z);
}
