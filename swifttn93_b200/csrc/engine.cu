// engine.cu -- sm_100a kernels of the all-pairs TN93 engine and the C ABI of include/tn93g.h.
//
// One run (tn93g_run) is a pipeline over bands of rows:
//   pack      colscan_kernel, pack_kernel, events_kernel, transpose_kernel: constant-column fold, bit planes,
//             compressed codes and sparse event lists (replaces Engine::prepare, swifttn93.cpp:570-1044)
//   pair      pair_kernel: per pair the clean-site counts by AND/XOR + POPC over 64-column plane words, the
//             N-plane cross counts, the sparse ambiguity events through the x16 tables, tn93's -l / -g
//             decisions, the TN93 formula in FP64 and the log certificate; writes the raw distance
//             (replaces kernel8/kernel16/kernelW/sparse_*/phaseA/tail8, swifttn93.cpp:1241-2170)
//   replay    replay_kernel: pairs with a contribution that is not a multiple of 1/16 are recomputed by a
//             site-order walk with tn93's float sums (replaces replay/ordered, swifttn93.cpp:1050-1232)
//   rows      stats_kernel (per row segment: histogram, links, skipped pairs, maxima, text length) and
//             sum_kernel (per row, the FP64 sums in tn93's column order) (phase C, swifttn93.cpp:2479-2604)
//   write     write_kernel: the distance-file text of the band at scanned segment offsets (the ordered writer,
//             swifttn93.cpp:2811-2858, and fastfmt)
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <math.h>

#include <algorithm>
#include <chrono>
#include <atomic>
#include <mutex>
#include <string>
#include <system_error>
#include <thread>
#include <vector>

#include "kernels.cuh"
#include "chain_sum.cuh"
#include "tc_count.cuh"
#include "tn93g.h"

namespace tn93 {
void build_log_table(LogTable *T);
}

using namespace tn93;

namespace {

constexpr int kWarps = 8;  // warps per block of the pair / row kernels

__device__ __forceinline__ int popc(uint64_t x) { return __popcll(x); }
__device__ __forceinline__ unsigned lanemask_lt() { return (1u << (threadIdx.x & 31)) - 1u; }

__device__ __forceinline__ bool sparse_code(int c, bool wplane) { return c >= 4 && c < 17 && !(wplane && c == 15); }

//------------------------------------------------------------------------------------------------ pack
// Each packing kernel's body takes its block coordinates as arguments, so that a batch of alignments can run one
// launch for all of them (the *_batch_kernel forms below map each block to its alignment and local block).

// per column: the set of codes seen (bit c), per launch the number of N codes; block (bx, by) covers 256 columns
// of 64 sequences
__device__ __forceinline__ void colscan_body(const uint8_t *__restrict__ codes, long N, long L, uint32_t *seen,
                                             unsigned long long *nN, long bx, long by)
{
  const long p = bx * 256l + threadIdx.x;
  const long i0 = by * 64l, i1 = min(N, i0 + 64);
  uint32_t m = 0;
  unsigned cn = 0;
  if (p < L)
    for (long i = i0; i < i1; i++) {
      const unsigned c = codes[i * L + p];
      m |= 1u << c;
      cn += c == 15;
    }
  if (p < L && m) atomicOr(&seen[p], m);
  for (int o = 16; o; o >>= 1) cn += __shfl_xor_sync(0xffffffffu, cn, o);
  if ((threadIdx.x & 31) == 0 && cn) atomicAdd(nN, (unsigned long long)cn);
}

__global__ void colscan_kernel(const uint8_t *__restrict__ codes, long N, long L, uint32_t *seen,
                               unsigned long long *nN)
{
  colscan_body(codes, N, L, seen, nN, blockIdx.x, blockIdx.y);
}

// one warp per (sequence, 64-column word): bit planes, compressed codes, sparse event counts; block bx covers 8
// sequences, and the words w0, w0 + wstep, ...
__device__ __forceinline__ void pack_body(const PackArgs &a, long bx, long w0, long wstep)
{
  const int lane = threadIdx.x & 31;
  const long i = bx * (long)kWarps + (threadIdx.x >> 5);
  if (i >= a.N) return;
  for (long w = w0; w < a.W; w += wstep) {
  const long k0 = w * 64 + lane, k1 = k0 + 32;
  const int c0 = k0 < a.Lc ? a.codes[i * a.L + a.varcol[k0]] : 17;
  const int c1 = k1 < a.Lc ? a.codes[i * a.L + a.varcol[k1]] : 17;
  if (k0 < a.Lc) a.cc[i * a.Lc + k0] = (uint8_t)c0;
  if (k1 < a.Lc) a.cc[i * a.Lc + k1] = (uint8_t)c1;
  auto both = [&](bool p0, bool p1) -> uint64_t {
    return (uint64_t)__ballot_sync(0xffffffffu, p0) | ((uint64_t)__ballot_sync(0xffffffffu, p1) << 32);
  };
  const uint64_t clean = both(c0 < 4, c1 < 4);
  const uint64_t hi = both(c0 < 4 && (c0 & 1), c1 < 4 && (c1 & 1));
  const uint64_t lo = both(c0 < 4 && (c0 & 2), c1 < 4 && (c1 & 2));
  const bool g0 = k0 < a.Lc && c0 == 17, g1 = k1 < a.Lc && c1 == 17;
  const uint64_t wn = a.wplane ? both(c0 == 15 || (a.gapmm && g0), c1 == 15 || (a.gapmm && g1)) : 0;
  const uint64_t gp = a.gapmm ? both(g0, g1) : 0;
  const uint64_t sp = both(sparse_code(c0, a.wplane), sparse_code(c1, a.wplane));
  if (lane == 0) {
    uint64_t *P = a.planes + (size_t)w * a.NP * a.Npad + i;
    P[0] = hi;
    P[a.Npad] = lo;
    P[2 * a.Npad] = clean;
    P[3 * a.Npad] = wn;
    if (a.NP > 4) P[4 * a.Npad] = gp;
    if (sp) atomicAdd(&a.evcount[i], (unsigned)popc(sp));
  }
  }
}

__global__ void pack_kernel(PackArgs a) { pack_body(a, blockIdx.x, blockIdx.y, gridDim.y); }

// The nonzero N-plane words (plane 3 of each word) of 32 sequences by a block of 16 warps: lanes over the sequences, so
// that loads coalesce, warps over 16 stretches of the words (one thread a sequence walked 468 words alone: 2,000 x 29,900
// 91 us to count and 226 us to list, 8 and 21 us so).
constexpr int kWlWarps = 16;

__device__ __forceinline__ bool w_word(const uint64_t *planes, long w, int NP, long Npad, long i)
{
  return planes[((size_t)w * NP + 3) * Npad + i] != 0;
}

// wcount[i]: how many of sequence i's words are nonzero
__global__ void __launch_bounds__(32 * kWlWarps) wcount_kernel(const uint64_t *planes, long N, long W, int NP, long Npad,
                                                               uint32_t *wcount)
{
  __shared__ uint32_t part[kWlWarps][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long i = blockIdx.x * 32l + lane;  // below Npad, a multiple of 32
  uint32_t n = 0;
#pragma unroll 4
  for (long w = W * warp / kWlWarps; w < W * (warp + 1) / kWlWarps; w++) n += w_word(planes, w, NP, Npad, i);
  part[warp][lane] = n;
  __syncthreads();
  if (warp == 0 && i < N) {
    for (int k = 1; k < kWlWarps; k++) n += part[k][lane];
    wcount[i] = n;
  }
}

// wl: the indices of sequence i's nonzero words, in order, from wl_off[i]
__global__ void __launch_bounds__(32 * kWlWarps) wlist_kernel(const uint64_t *planes, long N, long W, int NP, long Npad,
                                                              const uint32_t *wl_off, uint32_t *wl)
{
  __shared__ uint32_t part[kWlWarps][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long i = blockIdx.x * 32l + lane;
  const long w0 = W * warp / kWlWarps, w1 = W * (warp + 1) / kWlWarps;
  uint32_t n = 0;
#pragma unroll 4
  for (long w = w0; w < w1; w++) n += w_word(planes, w, NP, Npad, i);
  part[warp][lane] = n;
  __syncthreads();
  if (i >= N || n == 0) return;
  uint32_t o = wl_off[i];
  for (int k = 0; k < warp; k++) o += part[k][lane];
#pragma unroll 4
  for (long w = w0; w < w1; w++)
    if (w_word(planes, w, NP, Npad, i)) wl[o++] = (uint32_t)w;
}

__device__ __forceinline__ void put_event(const PackArgs &a, uint32_t at, uint32_t k, int c)
{
  a.ev[at] = k << 5 | (uint32_t)c;
  if (a.ev2) a.ev2[at] = make_uint2(k * a.ev2_Npad, (uint32_t)(c - kSparse0) * (kCodes * 8));
}

// one warp per sequence: its sparse events in site order (block bx: 8 sequences)
__device__ __forceinline__ void events_body(const PackArgs &a, long bx)
{
  const int lane = threadIdx.x & 31;
  const long i = bx * (long)kWarps + (threadIdx.x >> 5);
  if (i >= a.N) return;
  uint32_t off = a.ev_off[i];
  const uint8_t *row = a.cc + i * a.Lc;
  bool three = false;
  // 256 columns a step, their codes loaded before any is looked at (2,000 x 29,900: 188 us with 64 a step, 90 us so)
  for (long k0 = lane; k0 - lane < a.Lc; k0 += 256) {
    int c[8];
#pragma unroll
    for (int q = 0; q < 8; q++) c[q] = k0 + 32 * q < a.Lc ? row[k0 + 32 * q] : 17;
#pragma unroll
    for (int q = 0; q < 8; q++) {
      const bool s = sparse_code(c[q], a.wplane);
      const unsigned b = __ballot_sync(0xffffffffu, s);
      if (s) put_event(a, off + __popc(b & lanemask_lt()), (uint32_t)(k0 + 32 * q), c[q]);
      off += __popc(b);
      three |= c[q] >= 11 && c[q] <= 14;
    }
  }
  // null events (no site, the tables' zero row) up to the list's padded end
  if (lane < (int)(a.ev_off[i + 1] - off)) put_event(a, off + lane, 0, kGap);
  if (a.three) {
    three = __any_sync(0xffffffffu, three);
    if (lane == 0) a.three[i] = three;
  }
}

__global__ void events_kernel(PackArgs a) { events_body(a, blockIdx.x); }

// ccT[k][i] = cc[i][k] (padding sequences read as gaps); block (bx, by) of 32 x 8 threads: 128 columns x 32 sequences,
// stored four sequences to a word where the matrix starts on one (2,000 x 29,900: 124 us with 32 x 32 bytes a block,
// 47 us so)
constexpr int kTransK = 128;
__device__ __forceinline__ void transpose_body(const uint8_t *__restrict__ cc, uint8_t *ccT, long N, long Lc, long Npad,
                                               long bx, long by)
{
  __shared__ uint8_t tile[32][kTransK + 4];
  const long k0 = bx * kTransK, i0 = by * 32l;
  const int tx = threadIdx.x, ty = threadIdx.y;
  for (int r = ty; r < 32; r += 8) {
    const long i = i0 + r;
#pragma unroll
    for (int q = 0; q < kTransK; q += 32) {
      const long k = k0 + q + tx;
      tile[r][q + tx] = (i < N && k < Lc) ? cc[i * Lc + k] : (uint8_t)17;
    }
  }
  __syncthreads();
  const int g = 4 * (tx & 7);
  const bool words = ((reinterpret_cast<uintptr_t>(ccT) | (uintptr_t)Npad) & 3) == 0;
#pragma unroll
  for (int q = 0; q < kTransK; q += 32) {
    const int kk = q + ty * 4 + (tx >> 3);
    if (k0 + kk >= Lc) continue;
    uint8_t *const o = ccT + (k0 + kk) * Npad + i0 + g;
    if (words && i0 + g < Npad) {
      *reinterpret_cast<uint32_t *>(o) = (uint32_t)tile[g][kk] | (uint32_t)tile[g + 1][kk] << 8 | (uint32_t)tile[g + 2][kk] << 16 |
                                         (uint32_t)tile[g + 3][kk] << 24;
    } else {
      for (int b = 0; b < 4; b++)
        if (i0 + g + b < Npad) o[b] = tile[g + b][kk];
    }
  }
}

__global__ void transpose_kernel(const uint8_t *__restrict__ cc, uint8_t *ccT, long N, long Lc, long Npad)
{
  transpose_body(cc, ccT, N, Lc, Npad, blockIdx.x, blockIdx.y);
}

//------------------------------------------------------------------------------------------------ pair
// powers of ten for the certificate's fast test
__device__ __constant__ double kP10[12] = {1e-5, 1e-4, 1e-3, 1e-2, 1e-1, 1e0, 1e1, 1e2, 1e3, 1e4, 1e5, 1e6};
__device__ __constant__ double kScale[11] = {1e10, 1e9, 1e8, 1e7, 1e6, 1e5, 1e4, 1e3, 1e2, 1e1, 1e0};

// Do lo <= hi print the same six significant digits? Fast test: scale both into [1e5, 1e6) and require the same
// integer part with both fractions clear of 1/2 by 1e-4 (the scaled doubles are within 1e-9 of the exact scaled
// values). Returns -1 when the test cannot decide (then the caller compares the printed strings).
__device__ __forceinline__ int same_g_fast(double lo, double hi)
{
  if (!(lo >= 1e-5 && hi < 1e5)) return -1;
  int X = 0;
#pragma unroll
  for (int k = 1; k < 10; k++) X += lo >= kP10[k];
  const double s = kScale[X];
  const double ta = __dmul_rn(lo, s), tb = __dmul_rn(hi, s);
  if (!(ta >= 1e5 && tb < 1e6)) return -1;
  const double fa = floor(ta), fb = floor(tb);
  if (fa != fb) return -1;
  const double ra = ta - fa, rb = tb - fb;
  if (rb < 0.4999 || ra > 0.5001) return 1;
  return -1;
}

// Do lo and hi print the same text? The certificate's exact test when the fast one cannot decide; out of line, so
// that the big-number scratch of the decimal conversion lives in its own stack frame, not in its callers'.
__device__ __noinline__ bool same_g_text(double lo, double hi)
{
  char x[24], y[24];
  const int nx = fmt_g(lo, x), ny = fmt_g(hi, y);
  if (nx != ny) return false;
  for (int k = 0; k < nx; k++)
    if (x[k] != y[k]) return false;
  return true;
}

// decision-stability certificate: do the histogram bin, the link decision and the printed text agree for
// every distance the C library's log may lead to?
__device__ bool certified(const Dist &D, const RunConsts &rc)
{
  if (hist_bin(D.lo) != hist_bin(D.hi)) return false;
  const double tlo = D.lo <= 0. ? 0. : D.lo, thi = D.hi <= 0. ? 0. : D.hi;
  const bool llo = tlo >= rc.min_distance && tlo <= rc.threshold;
  const bool lhi = thi >= rc.min_distance && thi <= rc.threshold;
  if (llo != lhi) return false;
  if (!llo && tlo < rc.min_distance && thi > rc.threshold) return false;
  if (llo && rc.emit && tlo != thi) {
    const int f = same_g_fast(tlo, thi);
    if (f >= 0) return f == 1;
    return same_g_text(tlo, thi);
  }
  return true;
}

// Per-lane running totals of the ambiguous pairs' effect on one summary unit (ExactSink::amb): flushed with
// atomics when the unit changes, and warp by warp at the end of a tile.
struct AmbLane {
  int unit;  // -1: empty
  int n;     // ambiguous pairs
  double lo, hi, spread;
};

__device__ __forceinline__ void amb_flush(unsigned long long *acc, int unit, int n, double lo, double hi,
                                          double spread)
{
  unsigned long long *w = acc + 4 * unit;
  atomicMax(&w[0], (unsigned long long)__double_as_longlong(lo));
  atomicMax(&w[1], (unsigned long long)__double_as_longlong(hi));
  atomicAdd(reinterpret_cast<double *>(&w[2]), spread);
  atomicAdd(&w[3], (unsigned long long)n);
}

__device__ __forceinline__ void amb_add(unsigned long long *acc, AmbLane &L, int unit, double lo, double hi, double w)
{
  if (L.unit != unit) {
    if (L.unit >= 0) amb_flush(acc, L.unit, L.n, L.lo, L.hi, L.spread);
    L.unit = unit;
    L.n = 0;
    L.lo = L.hi = L.spread = 0.;
  }
  L.n++;
  L.lo = fmax(L.lo, lo);
  L.hi = fmax(L.hi, hi);
  L.spread += (hi - lo) * w;
}

// all 32 lanes: each unit held by some lane is reduced over the warp and added once
__device__ __forceinline__ void amb_warp_flush(unsigned long long *acc, AmbLane &L)
{
  for (;;) {
    const unsigned act = __ballot_sync(0xffffffffu, L.unit >= 0);
    if (!act) break;
    const int u = __shfl_sync(0xffffffffu, L.unit, __ffs(act) - 1);
    const bool me = L.unit == u;
    double lo = me ? L.lo : 0., hi = me ? L.hi : 0., sp = me ? L.spread : 0.;
    int n = me ? L.n : 0;
    for (int o = 16; o; o >>= 1) {
      lo = fmax(lo, __shfl_xor_sync(0xffffffffu, lo, o));
      hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
      sp += __shfl_xor_sync(0xffffffffu, sp, o);
      n += __shfl_xor_sync(0xffffffffu, n, o);
    }
    if ((threadIdx.x & 31) == 0) amb_flush(acc, u, n, lo, hi, sp);
    if (me) L.unit = -1;
  }
}

// histogram bin of pair (i, j) under -m (0 within the first file, 1 within the second, 2 between them)
__device__ __forceinline__ int fst_bin(const RunConsts &rc, long i, long j)
{
  return rc.fst ? (i < rc.n1 ? (j >= rc.n1 ? 2 : 0) : 1) : 0;
}

// The formula and its certificate for exact inputs; returns the raw distance (from the correctly rounded
// logarithms). A pair whose printed bytes or decisions depend on the C library's rounding (or, in resolve-all
// mode, any pair with an ambiguous logarithm) is appended to the undecided list, to be finished with the C
// library's own logarithms; every pair with an ambiguous logarithm widens its summary unit's bounds.
__device__ __forceinline__ double finish_exact(const LogTable &T, const RunConsts &rc, const ExactSink &ex,
                                               const double nf[4], double diag, double ag, double ct, long i, long j,
                                               long colbase, int &namb, int &nund, AmbLane &al)
{
  const Dist D = tn93_distance(T, nf, diag, ag, ct, rc.log_band, rc.log_spread);
  if (D.amb) {
    namb++;
    if (rc.resolve_all || !certified(D, rc)) {
      nund++;
      if (ex.und_list) {
        const unsigned idx = atomicAdd(ex.und_n, 1u);
        if (idx < ex.und_cap) {
          ex.und_list[2 * (size_t)idx] = (unsigned long long)ex.und_k;
          ex.und_list[2 * (size_t)idx + 1] = ((unsigned long long)i << 32) | (unsigned long long)j;
        }
      }
    }
    if (ex.amb) {
      const int unit = ex.colunit ? ex.colunit[j - colbase] : fst_bin(rc, i, j);
      const double w = (double)(ex.counts[i] * ex.counts[j]);
      amb_add(ex.amb, al, unit, D.lo <= 0. ? 0. : D.lo, D.hi <= 0. ? 0. : D.hi, w);
    }
  }
  return D.d;
}

// warp-level total of the per-lane counts, one atomic per warp (all 32 lanes must call it)
__device__ __forceinline__ void count_flags(unsigned long long *counters, int namb, int nund)
{
  for (int o = 16; o; o >>= 1) {
    namb += __shfl_xor_sync(0xffffffffu, namb, o);
    nund += __shfl_xor_sync(0xffffffffu, nund, o);
  }
  if ((threadIdx.x & 31) == 0) {
    if (namb) atomicAdd(&counters[0], (unsigned long long)namb);
    if (nund) atomicAdd(&counters[1], (unsigned long long)nund);
  }
}

__device__ __forceinline__ void add_entry(int acc[9], const int32_t *t)
{
#pragma unroll
  for (int q = 0; q < 8; q++) acc[q] += t[q];
  acc[8] |= t[8];
}

// Block tile of the pair kernel: 32 rows x 32 columns, 8 warps. Column-side sparse events are summed with the
// lanes over the tile's rows (warp-uniform event lists, coalesced position-major partner codes) into shared
// memory; then each warp takes 4 of the tile's rows, one at a time, with the lanes over the columns: clean-site
// counts, row-side events (warp-uniform list) and the epilogue.
constexpr int kTile = 32;
constexpr int kRowsPerWarp = kTile / kWarps;
constexpr int kColAccStride = kTile * 9 + 1;  // ints per tile row (+1: conflict-free in both phases)
constexpr int kAggInts = (kSparseCodes * kCodes + 5) * kLanes;
// shared-memory tables of a pair block: the x16 table (unpacked runs), or the packed table and the N-plane entries
constexpr size_t kPackedSmem = sizeof(PackedTables) + 5 * sizeof(AggEntry);
constexpr size_t kTabSmem = ((size_t)kAggInts * 4 > kPackedSmem ? (size_t)kAggInts * 4 : kPackedSmem + 15) / 16 * 16;
constexpr size_t kPairSmem = kTabSmem + (size_t)kTile * kColAccStride * 4;

// copies the run's tables into the block's shared memory (all threads; the caller synchronises); the AVERAGE sums
// only when the run has a -g test that may need them
__device__ __forceinline__ void load_pair_tables(const PairTables *g, unsigned char *smem, bool packed, bool fallback)
{
  if (packed) {
    const int n0 = (int)((fallback ? sizeof(PackedTables) : offsetof(PackedTables, avg)) / 16);
    const int n1 = (int)(5 * sizeof(AggEntry) / 16), at1 = (int)(sizeof(PackedTables) / 16);
    const uint4 *src = reinterpret_cast<const uint4 *>(&g->packed);
    const uint4 *src2 = reinterpret_cast<const uint4 *>(&g->agg[kEvEntries]);
    uint4 *dst = reinterpret_cast<uint4 *>(smem);
    for (int t = threadIdx.x; t < n0 + n1; t += blockDim.x) {
      if (t < n0)
        dst[t] = src[t];
      else
        dst[at1 + t - n0] = src2[t - n0];
    }
  } else {
    const uint4 *src = reinterpret_cast<const uint4 *>(g->agg);
    uint4 *dst = reinterpret_cast<uint4 *>(smem);
    for (int t = threadIdx.x; t < kAggInts / 4; t += blockDim.x) dst[t] = src[t];
  }
}

// the N-plane entries (ew[4], eww) in the block's tables
__device__ __forceinline__ const AggEntry *ew_entries(const unsigned char *smem, bool packed)
{
  return packed ? reinterpret_cast<const AggEntry *>(smem + sizeof(PackedTables))
                : reinterpret_cast<const AggEntry *>(smem) + kEvEntries;
}

struct Counts {
  int T, MM, TS, CT, Y1, Y2, L1, L2, T1, T2;
  int nWc, nWh, nWl, nWt, nWW, nGG;
};

// What AVERAGE mode adds to the x16 event sums of one pair (PackedTables::avg words) that the -g test sends there: the
// events of sequence i against the codes of j, then those of j where i is not a sparse code itself (such a site is
// counted once, from i's side). Each calling lane walks its own pair's two lists, a dozen to a few hundred table reads,
// where the site-order walk of the replay kernel visits every word of the alignment with a whole warp. Out of line: few
// lanes of an ordinary run come here, and its registers stay out of the caller's (the run's arrays come as scalars,
// since a reference would put the kernel's parameters on every thread's stack).
__device__ __noinline__ uint4 avg_events(const uint32_t (*tab)[4], bool wplane, const uint32_t *ev_off,
                                         const uint32_t *ev, const uint8_t *ccT, long Np, int i, int j)
{
  uint4 s = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll 1
  for (int side = 0; side < 2; side++) {
    const int own = side ? j : i, other = side ? i : j;
    const uint32_t e1 = ev_off[own + 1];
    for (uint32_t e = ev_off[own]; e < e1; e++) {
      const uint32_t v = __ldg(ev + e);
      const int pc = __ldg(ccT + (size_t)(v >> 5) * Np + other);
      if (side && sparse_code(pc, wplane)) continue;
      const uint4 t = *reinterpret_cast<const uint4 *>(tab[((v & 31) - 4) * kCodes + pc]);
      s.x += t.x;
      s.y += t.y;
      s.z += t.z;
      s.w += t.w;
    }
  }
  return s;
}

// the same with the unpacked table (a sequence with more than kPackedMaxEvents events): lane q of 0..6
__device__ __noinline__ int avg_events_lane(const AggEntry *tab, bool wplane, const uint32_t *ev_off,
                                            const uint32_t *ev, const uint8_t *ccT, long Np, int i, int j, int q)
{
  int s = 0;
#pragma unroll 1
  for (int side = 0; side < 2; side++) {
    const int own = side ? j : i, other = side ? i : j;
    const uint32_t e1 = ev_off[own + 1];
    for (uint32_t e = ev_off[own]; e < e1; e++) {
      const uint32_t v = __ldg(ev + e);
      const int pc = __ldg(ccT + (size_t)(v >> 5) * Np + other);
      if (side && sparse_code(pc, wplane)) continue;
      const int32_t *t = tab[((v & 31) - 4) * kCodes + pc].v;
      s += t[9 + q] - t[q];
    }
  }
  return s;
}

// the signed low and high 16-bit lanes of a word of sums
__device__ __forceinline__ int lane_lo(uint32_t w) { return (int)(int16_t)(w & 0xFFFFu); }
__device__ __forceinline__ int lane_hi(uint32_t w) { return (int)(w - (uint32_t)lane_lo(w)) >> 16; }

// the per-pair epilogue: exact x16 aggregates, tn93's -l / -g / order decisions, formula, certificate (AVG: the -g test's
// AVERAGE pairs are finished here)
template <bool WPLANE, bool AVG>
// cl: the clean-site aggregates of the pair (jointly clean sites, matches, A<->G and C<->T transitions, A, C and G
// base counts over both sequences), from the popcount loop or the tensor-core count kernel; c: N-plane counts
__device__ __forceinline__ void pair_epilogue(const PairArgs &a, const unsigned char *smem, const AggEntry *EW,
                                              const Counts &c, const int cl[7], const int acc[9], long i, long j,
                                              int &namb, int &nund, AmbLane &al)
{
  const RunConsts &rc = a.rc;
  const int base[7] = {16 * (cl[0] + (int)rc.constT), 16 * (cl[1] + (int)rc.constT), 16 * cl[2], 16 * cl[3],
                       16 * (cl[4] + (int)rc.constNf[0]), 16 * (cl[5] + (int)rc.constNf[1]),
                       16 * (cl[6] + (int)rc.constNf[2])};
  int wb[4] = {0, 0, 0, 0}, nww = 0;
  if (WPLANE) {
    wb[3] = c.nWt;
    wb[1] = c.nWh - c.nWt;
    wb[2] = c.nWl - c.nWt;
    wb[0] = c.nWc - wb[1] - wb[2] - wb[3];
    nww = c.nWW - c.nGG;
  }
  int ag[7];
#pragma unroll
  for (int q = 0; q < 7; q++) {
    int v = base[q] + acc[q];
    if (WPLANE) v += wb[0] * EW[0].v[q] + wb[1] * EW[1].v[q] + wb[2] * EW[2].v[q] + wb[3] * EW[3].v[q] + nww * EW[4].v[q];
    ag[q] = v;
  }
  int amb = acc[7];
  if (WPLANE) amb += wb[0] * EW[0].v[7] + wb[1] * EW[1].v[7] + wb[2] * EW[2].v[7] + wb[3] * EW[3].v[7] + nww * EW[4].v[7];
  double *slot = a.dist + (size_t)(i - a.r0) * a.ncols + (j - a.colbase);
  unsigned long long qentry = 0;
  bool to_replay = false;
  if (acc[8] & 1) {
    to_replay = true;  // order-dependent float sums in the main mode
  } else {
    double tng = (double)ag[0] / 16.0;
    if (tng > (double)rc.min_overlap && rc.fallback_avg && tng * rc.resolve_fraction <= (double)amb) {
      // tn93 recomputes the pair with -a average (refkernel.cpp:742-750): with the AVERAGE sums, exact in any order
      // when they are multiples of 1/16, or else by the site-order path. Only with the N plane on: N runs are what
      // sends most pairs of a set here (2,000 x 29,900, 1.2 M of 2 M pairs past -g 0.05: 224 ms a run with the walk,
      // 9.7 ms so); without it few pairs come, and the code costs the kernel at 64 registers more than they do
      // (6,700 x 1,500: 5.30 ms a run with it, 5.15 ms without).
      if (!AVG || (acc[8] & 2)) {
        to_replay = true;
        qentry = 1ull << 63;
      } else {
        if (rc.packed) {
          const uint4 d = avg_events(reinterpret_cast<const PackedTables *>(smem)->avg, rc.wplane, a.ev_off, a.ev, a.ccT,
                                     rc.Npad, (int)i, (int)j);
          ag[0] += lane_lo(d.x);
          ag[1] += lane_hi(d.x);
          ag[2] += lane_lo(d.y);
          ag[3] += lane_hi(d.y);
          ag[4] += lane_lo(d.z);
          ag[5] += lane_hi(d.z);
          ag[6] += (int)d.w;
        } else {
          for (int q = 0; q < 7; q++)
            ag[q] += avg_events_lane(reinterpret_cast<const AggEntry *>(smem), rc.wplane, a.ev_off, a.ev, a.ccT, rc.Npad,
                                     (int)i, (int)j, q);
        }
        if (WPLANE) {
#pragma unroll
          for (int q = 0; q < 7; q++)
            ag[q] += wb[0] * (EW[0].v[9 + q] - EW[0].v[q]) + wb[1] * (EW[1].v[9 + q] - EW[1].v[q]) +
                     wb[2] * (EW[2].v[9 + q] - EW[2].v[q]) + wb[3] * (EW[3].v[9 + q] - EW[3].v[q]) +
                     nww * (EW[4].v[9 + q] - EW[4].v[q]);
        }
        tng = (double)ag[0] / 16.0;
      }
    }
    if (to_replay) {
    } else if (tng <= (double)rc.min_overlap) {
      *slot = __longlong_as_double((long long)kSkipBits);
    } else {
      const double nf[4] = {(double)ag[4] / 16.0, (double)ag[5] / 16.0, (double)ag[6] / 16.0,
                            (double)(2 * ag[0] - ag[4] - ag[5] - ag[6]) / 16.0};
      *slot = finish_exact(*a.logt, rc, a.ex, nf, (double)ag[1] / 16.0, (double)ag[2] / 16.0, (double)ag[3] / 16.0, i,
                           j, a.colbase, namb, nund, al);
    }
  }
  if (to_replay) {
    const unsigned idx = atomicAdd(a.replay_n, 1u);
    if (idx < a.replay_cap) a.replay_q[idx] = qentry | ((unsigned long long)i << 31) | (unsigned long long)j;
  }
}

// packed event sums (PackedTables) of one lane: four words of 16-bit lanes and the non-dyadic flag
struct PackedAcc {
  uint32_t w0, w1, w2, w3, f;
};

__device__ __forceinline__ void add_packed(PackedAcc &p, const uint32_t (*tab)[4], const uint32_t *flags, int k)
{
  const uint4 t = *reinterpret_cast<const uint4 *>(tab[k]);
  p.w0 += t.x;
  p.w1 += t.y;
  p.w2 += t.z;
  p.w3 += t.w;
  p.f |= flags[k];
}

// Drops from L2 the tensor-core records of one tile row once every lane of the warp has read its own (all 32 lanes
// call it): the 128-byte lines wholly inside the tile row's records [rec0, rec0 + nrec) (nrec <= 32: the tile's
// columns that lie in this row of the record array) are invalidated without being written back
// (discard.global.L2), so records that the count kernel left in L2 never travel to DRAM. A line that straddles
// either edge also holds records of another tile or row and is kept. Each record is read once, by this warp.
__device__ __forceinline__ void discard_records(const void *base, size_t rec0, long nrec, int rec_bytes, int lane)
{
  __syncwarp();
  const uintptr_t lo = (uintptr_t)base + rec0 * (uintptr_t)rec_bytes, hi = lo + (uintptr_t)nrec * rec_bytes;
  const uintptr_t line = ((lo + 127) & ~(uintptr_t)127) + (uintptr_t)lane * 128;
  if (line + 128 <= hi) asm volatile("discard.global.L2 [%0], 128;" ::"l"(line) : "memory");
}

// Adds the packed table entries of the events [e0, e1) of one sequence against the partner at column p of the
// position-major code matrix. Four events per step: their words and partner codes are loaded before any sum, so
// that four partner-code loads (mostly from L2) are in flight at once.
__device__ __forceinline__ void add_events(PackedAcc &p, const uint32_t (*tab)[4], const uint32_t *flags,
                                           const uint32_t *ev, const uint8_t *ccT, long Np, long partner,
                                           uint32_t e0, uint32_t e1)
{
  uint32_t e = e0;
  for (; e + 4 <= e1; e += 4) {
    uint32_t v[4];
    int pc[4];
#pragma unroll
    for (int q = 0; q < 4; q++) v[q] = __ldg(ev + e + q);
#pragma unroll
    for (int q = 0; q < 4; q++) pc[q] = __ldg(ccT + (size_t)(v[q] >> 5) * Np + partner);
#pragma unroll
    for (int q = 0; q < 4; q++) add_packed(p, tab, flags, ((v[q] & 31) - 4) * kCodes + pc[q]);
  }
  for (; e < e1; e++) {
    const uint32_t v = __ldg(ev + e);
    add_packed(p, tab, flags, ((v & 31) - 4) * kCodes + __ldg(ccT + (size_t)(v >> 5) * Np + partner));
  }
}

// One tile of pairs: rows [i0, i0 + 8 * rpw) (rpw = rows per warp, 1..4) x columns [j0, j0 + 32). The block's
// tables must be in smem (load_pair_tables). All threads of the block call it with the same arguments.
template <bool WPLANE, bool GAPMM>
__device__ __forceinline__ void pair_tile(const PairArgs &a, const unsigned char *smem, int *colacc, long i0, long j0,
                                          int rpw)
{
  const RunConsts &rc = a.rc;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int trows = kWarps * rpw;
  const bool packed = rc.packed;
  const AggEntry *sagg = reinterpret_cast<const AggEntry *>(smem);
  const PackedTables &PT = *reinterpret_cast<const PackedTables *>(smem);
  const AggEntry *EW = ew_entries(smem, packed);
  // block-uniform exits: no valid pair in the tile
  if (i0 >= a.r1 || j0 >= a.cend) return;
  if (!rc.cross && j0 + kTile - 1 <= i0) return;
  const long Np = rc.Npad;
  // N-plane cross terms from the sequences' nonzero N words (row side and column side), when the clean-site counts
  // come from the tensor cores and the events are packed (the column accumulator has room); else every word
  const bool sparse_w = WPLANE && packed && a.tcagg != nullptr && a.wl_off != nullptr;
  // ---- column-side sparse events: lane = tile row, warp-uniform column; skipped where the row is sparse too
  // (packed: the column-side table holds zeros there)
  if (lane < trows) {
    const long ib = min(i0 + lane, rc.N - 1);
    for (int cl = warp; cl < kTile; cl += kWarps) {
      const long j = j0 + cl;
      int *dst = colacc + lane * kColAccStride + cl * 9;
      if (packed) {
        PackedAcc p = {0u, 0u, 0u, 0u, 0u};
        if (j < rc.N) add_events(p, PT.col, PT.colf, a.ev, a.ccT, Np, ib, a.ev_off[j], a.ev_off[j + 1]);
        dst[0] = (int)p.w0;
        dst[1] = (int)p.w1;
        dst[2] = (int)p.w2;
        dst[3] = (int)p.w3;
        dst[4] = (int)p.f;
        if (sparse_w) {
          // the column's N sites against the row's clean bases (its share of the N-plane cross terms)
          int xc = 0, xh = 0, xl = 0, xt = 0;
          if (j < rc.N)
            for (uint32_t q = a.wl_off[j]; q < a.wl_off[j + 1]; q++) {
              const uint64_t *P = a.planes + (size_t)__ldg(a.wl + q) * rc.NP * Np;
              const uint64_t nj = __ldg(P + 3 * Np + j);
              const uint64_t hi = __ldg(P + ib), lo = __ldg(P + Np + ib), ci = __ldg(P + 2 * Np + ib);
              xc += popc(nj & ci);
              xh += popc(nj & hi);
              xl += popc(nj & lo);
              xt += popc(nj & hi & lo);
            }
          dst[5] = xc;
          dst[6] = xh;
          dst[7] = xl;
          dst[8] = xt;
        }
      } else {
        int acc[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
        if (j < rc.N) {
          const uint32_t f0 = a.ev_off[j], f1 = a.ev_off[j + 1];
          for (uint32_t e = f0; e < f1; e++) {
            const uint32_t v = __ldg(a.ev + e);
            const int pc = a.ccT[(size_t)(v >> 5) * Np + ib];
            if (sparse_code(pc, WPLANE)) continue;
            add_entry(acc, sagg[((v & 31) - 4) * kCodes + pc].v);
          }
        }
#pragma unroll
        for (int q = 0; q < 9; q++) dst[q] = acc[q];
      }
    }
  }
  __syncthreads();
  // ---- per row of this warp (4 rows, one at a time): clean-site counts against lane = column, the row-side
  // sparse events (warp-uniform list), then the epilogue
  const long j = j0 + lane;
  const long jj = j < rc.N ? j : rc.N - 1;
  int namb = 0, nund = 0;
  AmbLane al;
  al.unit = -1;
#pragma unroll 1
  for (int r = 0; r < rpw; r++) {
    const long i = i0 + warp + kWarps * r;
    if (i >= a.r1) break;
    const long lb = rc.cross ? rc.n1 : i + 1;
    const bool valid = j >= lb && j < a.cend;
    if (!__any_sync(0xffffffffu, valid)) continue;
    Counts c = Counts{0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
    const bool tc = a.tcagg != nullptr;  // clean-site counts from the tensor-core kernel
    const int *src = colacc + (int)(i - i0) * kColAccStride + lane * 9;
    if (sparse_w) {
      // the row's N sites against the column's clean bases and N sites (warp-uniform word list), then the column's
      // share from the column phase: each union term of the dense loop below splits into these disjoint parts
      for (uint32_t q = a.wl_off[i]; q < a.wl_off[i + 1]; q++) {
        const uint64_t *Pw = a.planes + (size_t)__ldg(a.wl + q) * rc.NP * Np;
        const uint64_t ni = __ldg(Pw + 3 * Np + i);
        const uint64_t hj = __ldg(Pw + jj), lj = __ldg(Pw + Np + jj), cj = __ldg(Pw + 2 * Np + jj);
        const uint64_t nj = __ldg(Pw + 3 * Np + jj);
        c.nWc += popc(ni & cj);
        c.nWh += popc(ni & hj);
        c.nWl += popc(ni & lj);
        c.nWt += popc(ni & hj & lj);
        c.nWW += popc(ni & nj);
        if (GAPMM) c.nGG += popc(__ldg(Pw + 4 * Np + i) & __ldg(Pw + 4 * Np + jj));
      }
      c.nWc += src[5];
      c.nWh += src[6];
      c.nWl += src[7];
      c.nWt += src[8];
    }
    const uint64_t *P = a.planes;
    for (long w = 0; w < ((tc && (!WPLANE || sparse_w)) ? 0 : rc.W); w++, P += (size_t)rc.NP * Np) {
      const uint64_t hj = __ldg(P + jj), lj = __ldg(P + Np + jj), cj = __ldg(P + 2 * Np + jj);
      const uint64_t hi = __ldg(P + i), lo = __ldg(P + Np + i), ci = __ldg(P + 2 * Np + i);
      if (!tc) {
        const uint64_t b = ci & cj, x = hi ^ hj, y = lo ^ lj;
        const uint64_t ts = b & ~x & y;
        c.T += popc(b);
        c.MM += popc(b & (x | y));
        c.TS += popc(ts);
        c.CT += popc(ts & hi);
        c.Y1 += popc(b & hi);
        c.Y2 += popc(b & hj);
        c.L1 += popc(b & lo);
        c.L2 += popc(b & lj);
        c.T1 += popc(b & hi & lo);
        c.T2 += popc(b & hj & lj);
      }
      if (WPLANE) {
        // The N plane and the clean plane of one sequence are disjoint, so each pair of cross terms (this row's N
        // sites against the column's clean bases, and the other way round) covers disjoint sites: one popcount
        // of their union counts both.
        const uint64_t ni = __ldg(P + 3 * Np + i), nj = __ldg(P + 3 * Np + jj);
        c.nWc += popc((ni & cj) | (nj & ci));
        c.nWh += popc((ni & hj) | (nj & hi));
        c.nWl += popc((ni & lj) | (nj & lo));
        c.nWt += popc((ni & hj & lj) | (nj & hi & lo));
        c.nWW += popc(ni & nj);
        if (GAPMM) c.nGG += popc(__ldg(P + 4 * Np + i) & __ldg(P + 4 * Np + jj));
      }
    }
    int acc[9];
    const uint32_t e0 = a.ev_off[i], e1 = a.ev_off[i + 1];
    if (packed) {
      PackedAcc p = {(uint32_t)src[0], (uint32_t)src[1], (uint32_t)src[2], (uint32_t)src[3], (uint32_t)src[4]};
      add_events(p, PT.row, PT.rowf, a.ev, a.ccT, Np, jj, e0, e1);
      acc[0] = (int)(p.w0 & 0xFFFFu);
      acc[1] = (int)(p.w0 >> 16);
      acc[2] = (int)(p.w1 & 0xFFFFu);
      acc[3] = (int)(p.w1 >> 16);
      acc[4] = (int)(p.w2 & 0xFFFFu);
      acc[5] = (int)(p.w2 >> 16);
      acc[6] = (int)(p.w3 & 0xFFFFu);
      acc[7] = (int)(p.w3 >> 16);
      acc[8] = (int)p.f;
    } else {
#pragma unroll
      for (int q = 0; q < 9; q++) acc[q] = src[q];
      for (uint32_t e = e0; e < e1; e++) {
        const uint32_t v = __ldg(a.ev + e);
        const int pc = a.ccT[(size_t)(v >> 5) * Np + jj];
        add_entry(acc, sagg[((v & 31) - 4) * kCodes + pc].v);
      }
    }
    int cl[7];
    if (tc) {
      // the pair's record from the tensor-core kernel (8 lanes, 7 used)
      const long tn = a.tcncols ? a.tcncols : a.ncols, tb = a.tcncols ? a.tccolbase : a.colbase;
      const size_t at = (size_t)(i - a.r0) * tn + (jj - tb);
      if (a.tc16) {
        const uint4 *gp = reinterpret_cast<const uint4 *>(a.tcagg) + at;
        const uint4 g = valid ? __ldg(gp) : make_uint4(0, 0, 0, 0);
        cl[0] = (int)(g.x & 0xFFFFu);
        cl[1] = (int)(g.x >> 16);
        cl[2] = (int)(g.y & 0xFFFFu);
        cl[3] = (int)(g.y >> 16);
        cl[4] = (int)(g.z & 0xFFFFu);
        cl[5] = (int)(g.z >> 16);
        cl[6] = (int)(g.w & 0xFFFFu);
      } else {
        const uint4 *g = reinterpret_cast<const uint4 *>(a.tcagg) + 2 * at;
        const uint4 g0 = valid ? __ldg(g) : make_uint4(0, 0, 0, 0);
        const uint4 g1 = valid ? __ldg(g + 1) : make_uint4(0, 0, 0, 0);
        cl[0] = (int)g0.x;
        cl[1] = (int)g0.y;
        cl[2] = (int)g0.z;
        cl[3] = (int)g0.w;
        cl[4] = (int)g1.x;
        cl[5] = (int)g1.y;
        cl[6] = (int)g1.z;
      }
      discard_records(a.tcagg, (size_t)(i - a.r0) * tn + (size_t)(j0 - tb), min((long)kTile, tb + tn - j0),
                      a.tc16 ? 16 : 32, lane);
    } else {
      const int nfT = c.T1 + c.T2, nfC = c.Y1 + c.Y2 - nfT, nfG = c.L1 + c.L2 - nfT;
      cl[0] = c.T;
      cl[1] = c.T - c.MM;
      cl[2] = c.TS - c.CT;
      cl[3] = c.CT;
      cl[4] = 2 * c.T - nfC - nfG - nfT;
      cl[5] = nfC;
      cl[6] = nfG;
    }
    if (valid) pair_epilogue<WPLANE, WPLANE && !GAPMM>(a, smem, EW, c, cl, acc, i, j, namb, nund, al);
  }
  count_flags(a.counters, namb, nund);
  if (a.ex.amb) amb_warp_flush(a.ex.amb, al);
}

template <bool WPLANE, bool GAPMM, int MINB>
__global__ void __launch_bounds__(256, MINB) pair_kernel(PairArgs a)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  int *colacc = reinterpret_cast<int *>(smem_raw + kTabSmem);
  const long i0 = a.r0 + blockIdx.y * (long)kTile;
  const long j0 = a.cstart + blockIdx.x * (long)kTile;
  if (i0 >= a.r1 || j0 >= a.cend || (!a.rc.cross && j0 + kTile - 1 <= i0)) return;
  load_pair_tables(a.tab, smem_raw, a.rc.packed, WPLANE && a.rc.fallback_avg);
  __syncthreads();
  pair_tile<WPLANE, GAPMM>(a, smem_raw, colacc, i0, j0, kRowsPerWarp);
}

// Columns per segment of the formula, stats and write kernels: a warp handles one (row, segment), so a band of a few
// long rows still fills the GPU.
constexpr int kSeg = 1024;

#include "split_pair.cuh"

static_assert(sizeof(PairArgs) % 4 == 0, "PairArgs is copied as 32-bit words");

// A tile of a batch: alignment k, first row i0, first column j0, rows per warp.
struct BatchTile {
  int k, rpw;
  int i0, j0;
};

// Batched pair kernel over many alignments: a persistent grid takes tiles from a queue (one atomic per tile),
// loads the tile's alignment descriptor and agg table into shared memory when the alignment changes, and runs
// pair_tile. Tiles are ordered longest alignments first, so the tail is short.
template <bool WPLANE, bool GAPMM, int MINB>
__global__ void __launch_bounds__(256, MINB)
    pair_batch_kernel(const PairArgs *descs, const BatchTile *tiles, int ntiles, unsigned *next)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  int *colacc = reinterpret_cast<int *>(smem_raw + kTabSmem);
  __shared__ __align__(16) unsigned char sd_raw[sizeof(PairArgs)];
  const PairArgs &sd = *reinterpret_cast<const PairArgs *>(sd_raw);
  __shared__ int s_t;
  int cur = -1;
  for (;;) {
    if (threadIdx.x == 0) s_t = (int)atomicAdd(next, 1u);
    __syncthreads();
    const int t = s_t;
    if (t >= ntiles) break;
    const BatchTile T = tiles[t];
    if (T.k != cur) {
      for (int q = threadIdx.x; q < (int)(sizeof(PairArgs) / 4); q += blockDim.x)
        reinterpret_cast<int32_t *>(sd_raw)[q] = reinterpret_cast<const int32_t *>(&descs[T.k])[q];
      __syncthreads();
      load_pair_tables(sd.tab, smem_raw, sd.rc.packed, WPLANE && sd.rc.fallback_avg);
      cur = T.k;
    }
    __syncthreads();
    pair_tile<WPLANE, GAPMM>(sd, smem_raw, colacc, T.i0, T.j0, T.rpw);
    __syncthreads();
  }
}

//------------------------------------------------------------------------------------------------ replay
// position of the n-th set bit (0-based) of x; x has more than n set bits
__device__ __forceinline__ int nth_bit32(unsigned x, int n)
{
  int pos = 0;
#pragma unroll
  for (int s = 16; s; s >>= 1) {
    const int c = __popc(x & ((1u << s) - 1u));
    if (n >= c) {
      n -= c;
      x >>= s;
      pos += s;
    }
  }
  return pos;
}

// tn93's own per-pair computation (refkernel.cpp:622-750) for one pair, by one warp:
//   * clean/clean cells: the 4x4 table from the bit planes (lanes over 64-column words);
//   * every other site in site order: lane q adds the site's contribution to float cell q, so each cell is summed in site
//     order as tn93 does; lanes 16..19 add the integer diagonal resolutions, lane 20 the ambiguity count. The sites are the
//     two sequences' events, merged (sites with a gap contribute nothing, so they are left out), where their lists are at
//     hand, hold everything else (no N plane, not gapmm) and have 32 events or fewer; else the lanes fetch the codes of
//     each word's non-clean sites;
//   * tn93's c1-major merge of float and integer cells and the -l / -g tests, leaving the formula's exact inputs. t = 1
//     starts in AVERAGE mode (a pair the -g test already sent there).
// All lanes call it; the result is the same in all of them.
struct WalkOut {
  bool skip;  // below the overlap (-l)
  double nf[4], diag, ag, ct;
};

__device__ WalkOut walk_pair(const ReplayArgs &a, long i, long j, int t, unsigned char *sc1, unsigned char *sc2)
{
  const int lane = threadIdx.x & 31;
  const RunConsts &rc = a.rc;
  const long Np = rc.Npad;
  const uint64_t last_valid = (rc.Lc & 63) ? ((1ull << (rc.Lc & 63)) - 1ull) : ~0ull;
  const uint8_t *s1 = a.cc + (size_t)i * rc.Lc, *s2 = a.cc + (size_t)j * rc.Lc;
  // clean/clean 4x4 counts (the same in every mode)
  int cnt[16];
#pragma unroll
  for (int q = 0; q < 16; q++) cnt[q] = 0;
  for (long w = lane; w < rc.W; w += 32) {
    const uint64_t *P = a.planes + (size_t)w * rc.NP * Np;
    const uint64_t hi = P[i], lo = P[Np + i], ci = P[2 * Np + i];
    const uint64_t hj = P[j], lj = P[Np + j], cj = P[2 * Np + j];
    const uint64_t xi[4] = {ci & ~hi & ~lo, ci & hi & ~lo, ci & ~hi & lo, ci & hi & lo};
    const uint64_t xj[4] = {cj & ~hj & ~lj, cj & hj & ~lj, cj & ~hj & lj, cj & hj & lj};
#pragma unroll
    for (int x = 0; x < 4; x++)
#pragma unroll
      for (int y = 0; y < 4; y++) cnt[x * 4 + y] += popc(xi[x] & xj[y]);
  }
  if (rc.Lc < 65536) {  // two cells to a word
#pragma unroll
    for (int q = 0; q < 8; q++) {
      const uint32_t x = __reduce_add_sync(0xffffffffu, (uint32_t)cnt[q] | (uint32_t)cnt[q + 8] << 16);
      cnt[q] = (int)(x & 0xFFFFu);
      cnt[q + 8] = (int)(x >> 16);
    }
  } else {
#pragma unroll
    for (int q = 0; q < 16; q++) cnt[q] = __reduce_add_sync(0xffffffffu, cnt[q]);
  }
  // the merged events: sc1, sc2 hold the codes of ns sites (-1: walked word by word)
  int ns = -1;
  if (a.ev && !rc.wplane && !rc.gapmm) {
    const uint32_t e0 = a.ev_off[i], f0 = a.ev_off[j];
    const int ni = (int)(a.ev_off[i + 1] - e0), nj = (int)(a.ev_off[j + 1] - f0);
    if (ni <= 32 && nj <= 32) {
      const uint32_t vi = lane < ni ? __ldg(a.ev + e0 + lane) : (uint32_t)kGap;  // null events have a gap's code
      const uint32_t vj = lane < nj ? __ldg(a.ev + f0 + lane) : (uint32_t)kGap;
      const int ci = (int)(vi & 31), cj = (int)(vj & 31);
      const uint32_t ki = vi >> 5, kj = vj >> 5;
      const int oj = ci != kGap ? s2[ki] : kGap, oi = cj != kGap ? s1[kj] : kGap;
      const bool ui = oj != kGap, uj = oi != kGap && !sparse_code(oi, false);  // an event of both comes from i's list
      const unsigned mi = __ballot_sync(0xffffffffu, ui), mj = __ballot_sync(0xffffffffu, uj);
      int ri = __popc(mi & lanemask_lt()), rj = __popc(mj & lanemask_lt());
      for (unsigned m = mj; m; m &= m - 1) ri += __shfl_sync(0xffffffffu, kj, __ffs(m) - 1) < ki;
      for (unsigned m = mi; m; m &= m - 1) rj += __shfl_sync(0xffffffffu, ki, __ffs(m) - 1) < kj;
      if (ui) {
        sc1[ri] = (unsigned char)ci;
        sc2[ri] = (unsigned char)oj;
      }
      if (uj) {
        sc1[rj] = (unsigned char)oi;
        sc2[rj] = (unsigned char)cj;
      }
      ns = __popc(mi) + __popc(mj);
      __syncwarp();
    }
  }
  WalkOut R;
  R.skip = false;
  R.diag = R.ag = R.ct = 0.;
  R.nf[0] = R.nf[1] = R.nf[2] = R.nf[3] = 0.;
  for (;;) {
    const SiteEntry *S = a.site + t * kCodes * kCodes;
    double acc = 0.;  // lane q < 16: float cell q
    long iacc = 0;    // lanes 16..19: diagonal resolutions, lane 20: ambiguity count
    auto add_sites = [&](int n) {
#pragma unroll 4
      for (int l = 0; l < n; l++) {
        const SiteEntry &E = S[sc1[l] * kCodes + sc2[l]];
        if (lane < 16)
          acc = __dadd_rn(acc, E.fc[lane]);  // adding 0.0 changes nothing: no cell is ever -0.0
        else if (lane < 21)
          iacc += reinterpret_cast<const int32_t *>(&E)[offsetof(SiteEntry, icd) / 4 + lane - 16];  // icd[4], then amb
      }
    };
    if (ns >= 0) add_sites(ns);
    for (long w = 0; ns < 0 && w < rc.W; w++) {
      const uint64_t *P = a.planes + (size_t)w * rc.NP * Np;
      uint64_t E = ~(P[2 * Np + i] & P[2 * Np + j]);
      if (w == rc.W - 1) E &= last_valid;
      if (!E) continue;
      const int ne = __popcll(E), nlo = __popc((unsigned)E);
      for (int rk = lane; rk < ne; rk += 32) {
        const int bit = rk < nlo ? nth_bit32((unsigned)E, rk) : 32 + nth_bit32((unsigned)(E >> 32), rk - nlo);
        const long k = w * 64 + bit;
        sc1[rk] = s1[k];
        sc2[rk] = s2[k];
      }
      __syncwarp();
      add_sites(ne);
      __syncwarp();
    }
    // the cells in every lane, then tn93's merge and decisions
    double fc[16];
    long icd[4];
#pragma unroll
    for (int q = 0; q < 16; q++) fc[q] = __shfl_sync(0xffffffffu, acc, q);
#pragma unroll
    for (int q = 0; q < 4; q++) icd[q] = __shfl_sync(0xffffffffu, iacc, 16 + q);
    const long amb = __shfl_sync(0xffffffffu, iacc, 20);
    bool next = false;  // recompute with -a average
    {
      long ic[16];
      for (int q = 0; q < 16; q++) ic[q] = cnt[q];
      for (int x = 0; x < 4; x++) ic[x * 5] += icd[x] + rc.constCnt[x];
      double tot = 0., nf[4] = {0., 0., 0., 0.};
      for (int c1 = 0; c1 < 4; c1++)
        for (int c2 = 0; c2 < 4; c2++) {
          const double pc = fc[c1 * 4 + c2] = __dadd_rn(fc[c1 * 4 + c2], (double)ic[c1 * 4 + c2]);
          tot = __dadd_rn(tot, pc);
          nf[c1] = __dadd_rn(nf[c1], pc);
          nf[c2] = __dadd_rn(nf[c2], pc);
        }
      if (tot <= (double)rc.min_overlap) {
        R.skip = true;
      } else if (t == 0 && rc.fallback_avg && __dmul_rn(tot, rc.resolve_fraction) <= (double)(unsigned long)amb) {
        next = true;
      } else {
        R.diag = __dadd_rn(__dadd_rn(__dadd_rn(fc[0], fc[5]), fc[10]), fc[15]);
        R.ag = __dadd_rn(fc[2], fc[8]);
        R.ct = __dadd_rn(fc[7], fc[13]);
        for (int q = 0; q < 4; q++) R.nf[q] = nf[q];
      }
    }
    if (!next) break;
    t = 1;
  }
  __syncwarp();  // the next pair's sites take the place of these
  return R;
}

// The order-dependent pairs (a contribution that is not a multiple of 1/16). A warp walks up to 32 pairs of the queue one
// after the other, keeps each pair's sums in a lane, and then evaluates the formula for all of them at once (a pair's
// formula takes as many instructions for one lane as for 32). Fewer where the queue is short, so that every warp has some.
// 3,001 x 1,065 with 3e-5 three-fold codes: 644 us with the formula in one lane and the sites word by word, 161 us so.
__device__ __forceinline__ void replay_run(const ReplayArgs &a)
{
  __shared__ unsigned char sc1[kWarps][64], sc2[kWarps][64];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned long long n = min((unsigned long long)*a.qn, a.qcap), warps = (unsigned long long)gridDim.x * kWarps;
  if (blockIdx.x == 0 && threadIdx.x == 0 && n) atomicAdd(&a.counters[2], n);
  const int group = (int)min(32ull, (n + warps - 1) / warps);
  int namb = 0, nund = 0;
  AmbLane al;
  al.unit = -1;
  for (unsigned long long base = ((unsigned long long)blockIdx.x * kWarps + warp) * group; base < n; base += warps * group) {
    const int m = (int)min((unsigned long long)group, n - base);
    const unsigned long long mine = lane < m ? a.q[base + lane] : 0ull;
    WalkOut W;
    W.skip = true;
    for (int r = 0; r < m; r++) {
      const unsigned long long e = __shfl_sync(0xffffffffu, mine, r);
      const WalkOut X = walk_pair(a, (long)((e >> 31) & 0xFFFFFFFFull), (long)(e & 0x7FFFFFFFull), (int)(e >> 63), sc1[warp],
                                  sc2[warp]);
      if (lane == r) W = X;
    }
    if (lane < m) {
      const long i = (long)((mine >> 31) & 0xFFFFFFFFull), j = (long)(mine & 0x7FFFFFFFull);
      a.dist[(size_t)(i - a.r0) * a.ncols + (j - a.colbase)] =
          W.skip ? __longlong_as_double((long long)kSkipBits)
                 : finish_exact(*a.logt, a.rc, a.ex, W.nf, W.diag, W.ag, W.ct, i, j, a.colbase, namb, nund, al);
    }
  }
  count_flags(a.counters, namb, nund);
  if (a.ex.amb) amb_warp_flush(a.ex.amb, al);
}

// Undecided pairs, step 1 (one warp per listed pair): the site-order walk gives the formula's exact inputs in any
// mode (for a pair the pair kernel finished, its x16 aggregates and the walk's float sums are the same numbers),
// then the arguments of its logarithms. descs[k] describes run k of the list's entries.
__global__ void __launch_bounds__(256) und_args_kernel(const ReplayArgs *descs, const unsigned long long *list,
                                                       unsigned n, UndEntry *out)
{
  __shared__ unsigned char sc1[kWarps][64], sc2[kWarps][64];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (unsigned idx = blockIdx.x * kWarps + warp; idx < n; idx += gridDim.x * kWarps) {
    const int k = (int)list[2 * (size_t)idx];
    const unsigned long long ij = list[2 * (size_t)idx + 1];
    const long i = (long)(ij >> 32), j = (long)(ij & 0xFFFFFFFFull);
    const ReplayArgs &a = descs[k];
    const WalkOut W = walk_pair(a, i, j, 0, sc1[warp], sc2[warp]);
    if (lane == 0) {
      UndEntry &E = out[idx];
      E.k = k;
      E.slot = (long)((i - a.r0) * a.ncols + (j - a.colbase));
      E.state = W.skip ? 1 : 0;
      E.nlog = 0;
      for (int q = 0; q < 4; q++) E.in[q] = W.nf[q];
      E.in[4] = W.diag;
      E.in[5] = W.ag;
      E.in[6] = W.ct;
      E.arg[0] = E.arg[1] = E.arg[2] = 1.0;
      if (!W.skip) {
        const Prep P = tn93_prep(W.nf, W.diag, W.ag, W.ct);
        E.nlog = P.nlog;
        for (int q = 0; q < 3; q++) E.arg[q] = P.arg[q];
      }
    }
  }
}

// Undecided pairs, step 2 (one thread per pair): the formula from the C library's logarithms (UndEntry::lg)
__global__ void und_finish_kernel(const ReplayArgs *descs, const UndEntry *e, unsigned n)
{
  const unsigned idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= n) return;
  const UndEntry &E = e[idx];
  if (E.state) return;
  const double nf[4] = {E.in[0], E.in[1], E.in[2], E.in[3]};
  const Prep P = tn93_prep(nf, E.in[4], E.in[5], E.in[6]);
  descs[E.k].dist[E.slot] = tn93_combine(P, E.lg[0], E.lg[1], E.lg[2]);
}

__global__ void __launch_bounds__(256) replay_kernel(ReplayArgs a) { replay_run(a); }

// the replay queues of a batch's alignments, one after the other (each is usually empty or short)
__global__ void __launch_bounds__(256) replay_batch_kernel(const ReplayArgs *descs, int K)
{
  for (int k = 0; k < K; k++)
    if (*descs[k].qn) replay_run(descs[k]);
}

// exclusive scan of a band's segment byte counts (one block), and the band total: 4,096 counts at a time, four to a
// thread, the next ones loaded while these are scanned. (46,900 counts: 58 us with a stretch of 46 to each thread, whose
// loads do not coalesce, 35 us so.)
__global__ void __launch_bounds__(1024) scan_kernel(const unsigned long long *in, unsigned long long *out, long n,
                                                   unsigned long long *total)
{
  __shared__ unsigned long long part[2][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned long long v[4], carry = 0;
  auto load = [&](long b) {
#pragma unroll
    for (int k = 0; k < 4; k++) v[k] = b + k < n ? in[b + k] : 0;
  };
  long b = threadIdx.x * 4l;
  load(b);
  for (long b0 = 0, t = 0; b0 < n; b0 += 4096, b += 4096, t++) {
    const unsigned long long x[4] = {v[0], v[1], v[2], v[3]}, own = x[0] + x[1] + x[2] + x[3];
    load(b + 4096);
    unsigned long long inc = own;
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long y = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += y;
    }
    if (lane == 31) part[t & 1][warp] = inc;
    __syncthreads();  // the other buffer is free: every warp has passed the barrier after it read that one
    unsigned long long w = part[t & 1][lane];
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    unsigned long long run = carry + inc - own;
    const unsigned long long before = __shfl_sync(0xffffffffu, w, (warp + 31) & 31);
    if (warp) run += before;
    carry += __shfl_sync(0xffffffffu, w, 31);
#pragma unroll
    for (int k = 0; k < 4; k++) {
      if (b + k < n) out[b + k] = run;
      run += x[k];
    }
  }
  if (threadIdx.x == 0) *total = carry;
}

// Large exclusive scans in three coalesced passes: tile sums, a scan of the tile sums (scan_kernel), then each
// tile's scan from its offset. A tile is 256 threads x 16 consecutive elements.
constexpr int kScanTile = 4096;

__global__ void __launch_bounds__(256) tile_sum_kernel(const unsigned long long *in, long n,
                                                       unsigned long long *tile_sum)
{
  __shared__ unsigned long long ws[8];
  const long b = blockIdx.x * (long)kScanTile;
  unsigned long long s = 0;
  for (int k = threadIdx.x; k < kScanTile; k += 256) {
    const long e = b + k;
    if (e < n) s += in[e];
  }
  for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long t = 0;
    for (int w = 0; w < 8; w++) t += ws[w];
    tile_sum[blockIdx.x] = t;
  }
}

__global__ void __launch_bounds__(256) tile_scan_kernel(const unsigned long long *in, unsigned long long *out, long n,
                                                        const unsigned long long *tile_off)
{
  __shared__ unsigned long long ws[8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long b = blockIdx.x * (long)kScanTile + threadIdx.x * 16l;
  unsigned long long v[16], s = 0;
#pragma unroll
  for (int k = 0; k < 16; k++) {
    v[k] = b + k < n ? in[b + k] : 0;
    s += v[k];
  }
  // exclusive scan of the per-thread sums over the block
  unsigned long long inc = s;
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  if (lane == 31) ws[warp] = inc;
  __syncthreads();
  unsigned long long base = tile_off[blockIdx.x];
  for (int w = 0; w < warp; w++) base += ws[w];
  unsigned long long run = base + inc - s;
#pragma unroll
  for (int k = 0; k < 16; k++) {
    if (b + k < n) out[b + k] = run;
    run += v[k];
  }
}

// exclusive scan of n counters into out, the sum into *total; tmp holds 2 * ceil(n / kScanTile) + 1 counters
cudaError_t launch_scan(const unsigned long long *in, unsigned long long *out, long n, unsigned long long *total,
                        unsigned long long *tmp, cudaStream_t st)
{
  if (n <= 65536) {
    scan_kernel<<<1, 1024, 0, st>>>(in, out, n, total);
    return cudaGetLastError();
  }
  const long nt = (n + kScanTile - 1) / kScanTile;
  tile_sum_kernel<<<(unsigned)nt, 256, 0, st>>>(in, n, tmp);
  scan_kernel<<<1, 1024, 0, st>>>(tmp, tmp + nt, nt, total);
  tile_scan_kernel<<<(unsigned)nt, 256, 0, st>>>(in, out, n, tmp + nt);
  return cudaGetLastError();
}

//------------------------------------------------------------------------------------------------ rows
__device__ __forceinline__ int digits_of(long v)  // of 0 <= v < 2^31 (a sequence's number)
{
  const uint32_t u = (uint32_t)v;
  return 1 + (u >= 10u) + (u >= 100u) + (u >= 1000u) + (u >= 10000u) + (u >= 100000u) + (u >= 1000000u) + (u >= 10000000u) +
         (u >= 100000000u) + (u >= 1000000000u);
}

struct PairView {
  bool valid, computed, linked, counted;  // counted: contributes to the sums (not a -l skip)
  int bin, hb;
  long w;
  double thisD;
};

__device__ __forceinline__ double raw_pair(const RowArgs &a, long i, long j)
{
  return a.dist[(size_t)(i - a.r0) * a.ncols + (j - a.colbase)];
}

// pair (i, j), whose raw distance the caller has read (for j < N)
__device__ __forceinline__ PairView view_pair(const RowArgs &a, long i, long j, long cnt_i, double raw)
{
  const RunConsts &rc = a.rc;
  PairView v;
  v.valid = j < rc.N;
  v.computed = v.linked = v.counted = false;
  v.bin = 0;
  v.hb = 0;
  v.w = 0;
  v.thisD = -1.0;
  if (!v.valid) return v;
  v.w = cnt_i * a.counts[j];
  if (rc.fst) v.bin = i < rc.n1 ? (j >= rc.n1 ? 2 : 0) : 1;
  if ((uint64_t)__double_as_longlong(raw) != kSkipBits) {
    v.computed = true;
    v.hb = hist_bin(raw);
    v.thisD = raw <= 0. ? 0. : raw;
  }
  v.linked = v.thisD >= rc.min_distance && v.thisD <= rc.threshold;
  v.counted = !(v.thisD <= -0.5);
  return v;
}

// A printed distance handed from the stats kernel to the writer, one 32-bit word per pair slot: 0 = not printed;
// kind 1 (bits 30-31) = the six digits q (bits 0-19) and the decimal exponent X + 16 (bits 20-25) of a value in
// [1e-5, 1e5); kind 2 = zero ("0"); kind 3 = any other value (the writer formats the double itself). len receives
// the length of the text. d is a reported distance: not negative, not NaN.
__device__ __forceinline__ uint32_t print_code(double d, int &len)
{
  if (d == 0.0) {
    len = 1;
    return 2u << 30;
  }
  if (d >= 1e-5 && d < 1e5) {
    const Dec D = decimal6(d);
    len = dec_len(D);
    return (1u << 30) | ((uint32_t)(D.X + 16) << 20) | D.q;
  }
  len = fmt_g_len(d);
  return 3u << 30;
}

// the text of a printed-distance code (d: the distance, read only for kind 3); returns the length
__device__ __forceinline__ int fmt_code(uint32_t code, double d, char *out)
{
  const uint32_t kind = code >> 30;
  if (kind == 1) {
    Dec D;
    D.q = code & 0xFFFFFu;
    D.X = (int)((code >> 20) & 63u) - 16;
    return fmt_dec(D, out);
  }
  if (kind == 2) {
    out[0] = '0';
    return 1;
  }
  return fmt_g(d, out);
}

// what the text writers need of a pair: whether it is reported, and its printed distance (tn93's "<= 0 -> 0")
__device__ __forceinline__ bool linked_pair(const RowArgs &a, long i, long j, double &thisD)
{
  const RunConsts &rc = a.rc;
  if (j >= rc.N) return false;
  const double raw = a.dist[(size_t)(i - a.r0) * a.ncols + (j - a.colbase)];
  if ((uint64_t)__double_as_longlong(raw) == kSkipBits) return false;
  thisD = raw <= 0. ? 0. : raw;
  return thisD >= rc.min_distance && thisD <= rc.threshold;
}

__device__ __forceinline__ int self_len(const RowArgs &a, long i)
{
  if (!a.rc.report_self || a.rc.cross) return 0;
  if (a.rc.format == 0) return 2 * a.name_len[i] + 4;
  if (a.rc.format == 1) return 2 * digits_of(i) + 4;
  return 0;
}

// one warp per (row, segment): histogram, links, skips, maxima and the byte count of the segment's text
__device__ __forceinline__ void stats_rows(const RowArgs &a, long bx, int sg)
{
  __shared__ unsigned long long sh[3 * kHistBins];
  for (int t = threadIdx.x; t < 3 * kHistBins; t += blockDim.x) sh[t] = 0;
  __syncthreads();
  const RunConsts &rc = a.rc;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long i = a.r0 + bx * kWarps + warp;
  if (i < a.r1) {
    const long r = i - a.r0;
    const long slot = r * a.maxseg + sg;
    const long lb = rc.cross ? rc.n1 : i + 1;
    const long c0 = lb + (long)sg * kSeg, c1 = min(rc.N, c0 + kSeg);
    const long cnt_i = a.counts[i];
    const int nli = a.name_len[i];
    const int dli = rc.format == 1 ? digits_of(i) : 0;
    double m0 = 0., m1 = 0., m2 = 0.;
    long long links = 0, skipped = 0;
    unsigned long long bytes = 0;
    if (sg == 0 && !rc.cross) {
      if (cnt_i > 1 && lane == 0) {
        const unsigned long long svs = (unsigned long long)(cnt_i * (cnt_i - 1l)) >> 1;
        atomicAdd(&sh[i < rc.n1 ? 0 : kHistBins], svs);
      }
      if (lane == 0 && rc.emit) bytes += self_len(a, i);
    }
    for (long j0 = c0; j0 < c1; j0 += 32) {
      const long j = j0 + lane;
      PairView v = view_pair(a, i, j, cnt_i, j < rc.N ? raw_pair(a, i, j) : 0.);
      if (j >= c1) v.valid = v.computed = v.linked = false;
      // histogram: lanes with the same bin add once (their weights summed when all are 1)
      const int key = v.computed ? v.bin * kHistBins + v.hb : -1;
      const unsigned peers = __match_any_sync(0xffffffffu, key);
      if (__all_sync(0xffffffffu, !v.computed || v.w == 1)) {
        if (v.computed && lane == __ffs(peers) - 1) atomicAdd(&sh[key], (unsigned long long)__popc(peers));
      } else if (v.computed) {
        atomicAdd(&sh[key], (unsigned long long)v.w);
      }
      uint32_t code = 0;
      if (v.valid && v.linked) {
        links += v.w;
        if (rc.emit) {
          if (rc.format != 2) {
            int gl;
            if (a.dcode)
              code = print_code(v.thisD, gl);
            else
              gl = fmt_g_len(v.thisD);
            bytes += rc.format == 0 ? nli + a.name_len[j] + gl + 3 : dli + digits_of(j) + gl + 3;
          } else {
            a.hy[(size_t)i * rc.N + j] = v.thisD;
            a.hy[(size_t)j * rc.N + i] = v.thisD;
          }
        }
      }
      if (a.dcode && v.valid) a.dcode[(size_t)(i - a.r0) * a.ncols + (j - a.colbase)] = code;
      if (v.valid && !v.counted) skipped++;
      if (v.valid && v.counted) {
        if (v.bin == 0) m0 = v.thisD > m0 ? v.thisD : m0;
        else if (v.bin == 1) m1 = v.thisD > m1 ? v.thisD : m1;
        else m2 = v.thisD > m2 ? v.thisD : m2;
      }
    }
    for (int o = 16; o; o >>= 1) {
      links += __shfl_xor_sync(0xffffffffu, links, o);
      skipped += __shfl_xor_sync(0xffffffffu, skipped, o);
      bytes += __shfl_xor_sync(0xffffffffu, bytes, o);
      m0 = fmax(m0, __shfl_xor_sync(0xffffffffu, m0, o));
      m1 = fmax(m1, __shfl_xor_sync(0xffffffffu, m1, o));
      m2 = fmax(m2, __shfl_xor_sync(0xffffffffu, m2, o));
    }
    if (lane == 0) {
      a.seg_bytes[slot] = bytes;
      a.seg_links[slot] = links;
      a.seg_skip[slot] = skipped;
      a.seg_max[slot * 3] = m0;
      a.seg_max[slot * 3 + 1] = m1;
      a.seg_max[slot * 3 + 2] = m2;
    }
  }
  __syncthreads();
  for (int t = threadIdx.x; t < 3 * kHistBins; t += blockDim.x)
    if (sh[t]) atomicAdd(&a.hist[t], sh[t]);
}

// Resident blocks per SM for the stats and write kernels 4 (64 registers): same box, per 22.4 M pairs, row stage (stats,
// sums, scan, totals) 0.50 ms with 4, 0.56 with 5, 0.54 with 6; write 0.60 ms with 4, 0.69 with 3, 0.91 with 6.
__global__ void __launch_bounds__(256, 4) stats_kernel(RowArgs a) { stats_rows(a, blockIdx.x, blockIdx.y); }


// Sums in order by a warp (chain_sum.cuh): s and the result are the same in every lane.
__device__ __forceinline__ double warp_total(double x)
{
  for (int o = 16; o; o >>= 1) x = __dadd_rn(x, __shfl_xor_sync(0xffffffffu, x, o));
  return x;
}

// s plus the 32 lanes' terms, lane 0's first
__device__ __forceinline__ double chain_add32(double s, double t)
{
  ChainBinade c;
  bool ok = chain_binade(s, c);
  const double s1 = __dadd_rn(s, warp_total(chain_round(c, t, ok)));
  if (__all_sync(0xffffffffu, (ok && s1 < c.end) || t == 0.)) return __any_sync(0xffffffffu, t != 0.) ? s1 : s;
#pragma unroll
  for (int l = 0; l < 32; l++) s = __dadd_rn(s, __shfl_sync(0xffffffffu, t, l));
  return s;
}

// s plus 128 terms: the lanes' t[0], then their t[1], ...
__device__ __forceinline__ double chain_add128(double s, const double (&t)[4])
{
  ChainBinade c;
  bool ok = chain_binade(s, c);
  double x = 0.;
#pragma unroll
  for (int q = 0; q < 4; q++) x = __dadd_rn(x, chain_round(c, t[q], ok));
  const double s1 = __dadd_rn(s, warp_total(x));
  if (__all_sync(0xffffffffu, ok && s1 < c.end)) return s1;
#pragma unroll 1
  for (int q = 0; q < 4; q++) s = chain_add32(s, q == 0 ? t[0] : q == 1 ? t[1] : q == 2 ? t[2] : t[3]);
  return s;
}

// s plus x[0], x[1], ... x[n - 1] (shared memory), in groups that grow to 1,024 while they succeed
__device__ __forceinline__ double chain_shared(const double *x, int n, double s)
{
  const int lane = threadIdx.x & 31;
  int len = 32;
  for (int at = 0; at < n;) {
    const int m = min(len, n - at);
    ChainBinade c;
    bool ok = chain_binade(s, c);
    double y = 0.;
    for (int k = lane; k < m; k += 32) y = __dadd_rn(y, chain_round(c, x[at + k], ok));
    const double s1 = __dadd_rn(s, warp_total(y));
    if (__all_sync(0xffffffffu, ok && s1 < c.end)) {
      s = s1;
      at += m;
      len = min(2 * len, 1024);
    } else if (m <= 32) {
#pragma unroll 8
      for (int k = 0; k < m; k++) s = __dadd_rn(s, x[at + k]);
      at += m;
    } else {
      len = max(32, len / 4);
    }
  }
  return s;
}

// tn93's sum over a unit's rows in row order (swifttn93.cpp:2838-2848), *s0 = rs[0] + rs[STRIDE] + ... of n rows, by one block.
// The block stages 2,048 rows in shared memory, loading the next ones meanwhile; each warp adds its share of them for the
// binade that the sum stands in, and warp 0 puts the shares together: a share with a half-way term or past the binade is
// added in smaller groups, and past the binade the shares that follow are formed anew. 30,000 rows: 291 us with one thread
// adding them one by one, 105 us with one warp in groups, 80 us so.
constexpr int kReduceChunk = 2048;
template <int THREADS, int STRIDE>
__device__ __forceinline__ void chain_rows(const double *rs, long n, double *s0)
{
  constexpr int kPer = kReduceChunk / THREADS, kW = THREADS / 32, kShare = kReduceChunk / kW;
  __shared__ double ss[kReduceChunk], part[kW], s_sh;
  __shared__ int state[kW], from_sh;  // state of a share: 0 not addable, 1 addable, 2 all zero
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double a[kPer], s = 0.;
  auto load = [&](long r0) {
#pragma unroll
    for (int k = 0; k < kPer; k++) {
      const long r = r0 + k * THREADS + threadIdx.x;
      a[k] = r < n ? rs[r * STRIDE] : 0.;
    }
  };
  load(0);
  for (long r0 = 0; r0 < n; r0 += kReduceChunk) {
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kPer; k++) ss[k * THREADS + threadIdx.x] = a[k];
    __syncthreads();
    load(r0 + kReduceChunk);
    const int m = (int)min((long)kReduceChunk, n - r0);  // past m: zeros
    for (int from = 0; from < kW && from * kShare < m;) {
      ChainBinade c;
      const bool valid = chain_binade(s, c);
      if (warp >= from) {
        bool ok = valid, zero = true;
        double y = 0.;
#pragma unroll
        for (int k = 0; k < kPer; k++) {
          const double t = ss[warp * kShare + 32 * k + lane];
          y = __dadd_rn(y, chain_round(c, t, ok));
          zero &= t == 0.;
        }
        y = warp_total(y);
        ok = __all_sync(0xffffffffu, ok);
        zero = __all_sync(0xffffffffu, zero);
        if (lane == 0) {
          part[warp] = y;
          state[warp] = zero ? 2 : ok ? 1 : 0;
        }
      }
      __syncthreads();
      if (warp == 0) {
        int w = from;
        while (w < kW && w * kShare < m) {
          const int st = state[w];
          const double s1 = __dadd_rn(s, part[w]);
          if (st == 2 || (st == 1 && s1 < c.end)) {
            if (st == 1) s = s1;
            w++;
            continue;
          }
          s = chain_shared(ss + w * kShare, min(kShare, m - w * kShare), s);
          w++;
          if (!valid || !(s < c.end)) break;
        }
        if (lane == 0) {
          s_sh = s;
          from_sh = w;
        }
      }
      __syncthreads();
      s = s_sh;
      from = from_sh;
    }
  }
  if (threadIdx.x == 0) *s0 = s;
}

// the sum of weights, whole numbers: exact in any order while below 2^53 (chain_weights adds them one by one past that).
// Every thread brings its part and whether all its terms were whole; the result is valid in thread 0.
template <int THREADS, int STRIDE>
__device__ __forceinline__ void chain_weights(const double *rw, long n, double part, bool whole, double *w0)
{
  __shared__ double ws[THREADS / 32];
  part = warp_total(part);
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = part;
  whole = __syncthreads_and(whole);
  if (threadIdx.x == 0) {
    double w = 0.;
    for (int k = 0; k < THREADS / 32; k++) w = __dadd_rn(w, ws[k]);
    if (!whole || !(w < 0x1p53)) {
      w = 0.;
      for (long r = 0; r < n; r++) w = __dadd_rn(w, rw[r * STRIDE]);
    }
    *w0 = w;
  }
}

// one warp per row: tn93's row sums in column order (swifttn93.cpp:2594-2602). The self-pair weights come first, as tn93
// adds them when the row starts (swifttn93.cpp:2405-2415). Without -m the terms are added 128 at a time with the bits of
// one after the other (chain_sum.cuh): 22.4 M pairs 231 us
// with one shuffle and add a term, 81 us so.
__device__ __forceinline__ void sum_rows(const RowArgs &a, long bx)
{
  __shared__ double sterm[kWarps][32], sw[kWarps][32];
  __shared__ unsigned char sbin[kWarps][32];
  const RunConsts &rc = a.rc;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long i = a.r0 + bx * kWarps + warp;
  if (i >= a.r1) return;
  const long cnt_i = a.counts[i];
  double s0 = 0., s1 = 0., s2 = 0., w0 = 0., w1 = 0., w2 = 0.;
  const long lb = rc.cross ? rc.n1 : i + 1, cend = rc.N, out_row = i - a.r0;
  if (!rc.cross && cnt_i > 1) {
    const unsigned long long svs = (unsigned long long)(cnt_i * (cnt_i - 1l)) >> 1;
    if (i < rc.n1)
      w0 += (double)svs;
    else
      w1 += (double)svs;
  }
  const double *drow = a.dist + (size_t)(i - a.r0) * a.ncols - a.colbase;
  if (!rc.fst) {
    // Single bin: 128 columns at a time; skipped pairs and columns past the end add +0.0, which leaves a non-negative sum
    // unchanged. The weights are integers: their double sum is exact, in any order, while the total stays below
    // 2^53, so they are added as integers (and re-added one by one in the rare case the total is larger).
    // The next columns' distances and counts are loaded before these are added, so the loads overlap the chain.
    unsigned long long wsum = 0;
    double raw[4];
    long cj[4];
    auto load = [&](long j0) {
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const long j = j0 + 32 * q + lane;
        raw[q] = j < cend ? drow[j] : __longlong_as_double((long long)kSkipBits);
        cj[q] = j < cend ? a.counts[j] : 0;
      }
    };
    load(lb);
    for (long j0 = lb; j0 < cend; j0 += 128) {
      double t[4];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        t[q] = 0.;
        if ((uint64_t)__double_as_longlong(raw[q]) != kSkipBits) {
          const long w = cnt_i * cj[q];
          t[q] = __dmul_rn(raw[q] <= 0. ? 0. : raw[q], (double)w);
          wsum += (unsigned long long)w;
        }
      }
      load(j0 + 128);
      s0 = chain_add128(s0, t);
    }
    for (int o = 16; o; o >>= 1) wsum += __shfl_xor_sync(0xffffffffu, wsum, o);
    const unsigned long long svs = (!rc.cross && cnt_i > 1) ? (unsigned long long)(cnt_i * (cnt_i - 1l)) >> 1 : 0;
    if (wsum + svs < (1ull << 53)) {
      w0 = (double)(wsum + svs);
    } else {
      w0 = (double)svs;
      for (long j0 = lb; j0 < cend; j0 += 32) {
        const long j = j0 + lane;
        double wl = 0.;
        if (j < cend && (uint64_t)__double_as_longlong(drow[j]) != kSkipBits) wl = (double)(cnt_i * a.counts[j]);
#pragma unroll
        for (int l = 0; l < 32; l++) w0 = __dadd_rn(w0, __shfl_sync(0xffffffffu, wl, l));
      }
    }
    if (lane == 0) {
      const long r = out_row;
      a.row_sum[r * 3] = s0;
      a.row_sum[r * 3 + 1] = 0.;
      a.row_sum[r * 3 + 2] = 0.;
      a.row_w[r * 3] = w0;
      a.row_w[r * 3 + 1] = 0.;
      a.row_w[r * 3 + 2] = 0.;
    }
    return;
  }
  for (long j0 = lb; j0 < cend; j0 += 32) {
    const long j = j0 + lane;
    bool inc = false;
    double term = 0., wl = 0.;
    int bin = 0;
    if (j < cend) {
      const double raw = drow[j];
      if ((uint64_t)__double_as_longlong(raw) != kSkipBits) {
        const double t = raw <= 0. ? 0. : raw;
        const long w = cnt_i * a.counts[j];
        if (rc.fst) bin = i < rc.n1 ? (j >= rc.n1 ? 2 : 0) : 1;
        inc = true;
        term = __dmul_rn(t, (double)w);
        wl = (double)w;
      }
    }
    sterm[warp][lane] = term;
    sw[warp][lane] = wl;
    sbin[warp][lane] = inc ? (unsigned char)bin : (unsigned char)255;
    __syncwarp();
    if (lane == 0) {
      const int n = (int)min(32l, cend - j0);
      if (!rc.fst) {
        for (int l = 0; l < n; l++)
          if (sbin[warp][l] == 0) {
            s0 = __dadd_rn(s0, sterm[warp][l]);
            w0 = __dadd_rn(w0, sw[warp][l]);
          }
      } else {
        for (int l = 0; l < n; l++) {
          const int bl = sbin[warp][l];
          if (bl == 0) {
            s0 = __dadd_rn(s0, sterm[warp][l]);
            w0 = __dadd_rn(w0, sw[warp][l]);
          } else if (bl == 1) {
            s1 = __dadd_rn(s1, sterm[warp][l]);
            w1 = __dadd_rn(w1, sw[warp][l]);
          } else if (bl == 2) {
            s2 = __dadd_rn(s2, sterm[warp][l]);
            w2 = __dadd_rn(w2, sw[warp][l]);
          }
        }
      }
    }
    __syncwarp();
  }
  if (lane == 0) {
    const long r = out_row;
    a.row_sum[r * 3] = s0;
    a.row_sum[r * 3 + 1] = s1;
    a.row_sum[r * 3 + 2] = s2;
    a.row_w[r * 3] = w0;
    a.row_w[r * 3 + 1] = w1;
    a.row_w[r * 3 + 2] = w2;
  }
}

__global__ void __launch_bounds__(256) sum_kernel(RowArgs a) { sum_rows(a, blockIdx.x); }

__device__ __forceinline__ char *put_bytes(char *o, const char *s, int n)
{
  for (int k = 0; k < n; k++) o[k] = s[k];
  return o + n;
}

// the text of one reported pair at o (generic pointer: shared staging or global); csvn prints column j as j - jshift
__device__ __forceinline__ void put_line(char *o, const RowArgs &a, long i, long j, long jshift, const char *ni,
                                         int nli, const char *g, int gl)
{
  const RunConsts &rc = a.rc;
  if (rc.format == 0) {
    o = put_bytes(o, ni, nli);
    *o++ = rc.delim;
    o = put_bytes(o, a.names + a.name_off[j], a.name_len[j]);
    *o++ = rc.delim;
  } else {
    char t[24];
    int n = fmt_long(i, t);
    o = put_bytes(o, t, n);
    *o++ = rc.delim;
    n = fmt_long(j - jshift, t);
    o = put_bytes(o, t, n);
    *o++ = rc.delim;
  }
  o = put_bytes(o, g, gl);
  *o = '\n';
}

// Output staging: each warp assembles its lines in shared memory at the same offset modulo 16 as their
// destination, then stores whole 16-byte blocks (edges byte by byte), so global writes are coalesced. Nothing is
// written at or past the end of the counted range.
constexpr int kStage = 4096;

struct Stager {
  char *buf;       // this warp's staging buffer (16-byte aligned)
  uintptr_t gpos;  // global address of the first staged byte
  uintptr_t gend;  // end of the counted range
  int head, fill;  // buf[head .. head + fill) holds global [gpos, gpos + fill)
  bool over;       // the text ran past its counted length (reported as an internal error)
  __device__ void flush(int lane)
  {
    const uintptr_t g0 = gpos - (uintptr_t)head;
    if (gpos + fill > gend) over = true;
    const int end = (int)min((uintptr_t)(head + fill), gend > g0 ? gend - g0 : 0), nblk = (end + 15) >> 4;
    for (int b = lane; b < nblk; b += 32) {
      const int lo = b << 4, hi = lo + 16;
      if (lo >= head && hi <= end)
        *reinterpret_cast<uint4 *>(g0 + lo) = *reinterpret_cast<const uint4 *>(buf + lo);
      else
        for (int k = max(lo, head); k < min(hi, end); k++) *reinterpret_cast<char *>(g0 + k) = buf[k];
    }
    __syncwarp();
    gpos += fill;
    head = (int)(gpos & 15);
    fill = 0;
  }
};

// Lines in 8-byte words. A byte at a time (load a byte, store a byte) a line of 36 bytes took about 500 instructions of a
// warp for 32 of them and 22.4 M of them 611-649 us; by words of 8 shifted into place 602 us (630 since the exact
// digits of rare values are a call), column numbers (-f csvn) 449 -> 325 us per 1.6 M. What bounds it is latency: loading the next columns' codes and names early (more registers, 3 blocks
// instead of 4 on an SM) took 687 us.
constexpr int kLineName = 64;  // longest name (and start of a line) written by words

// the end of a line as little-endian words: delimiter, distance, newline (16 bytes at most); bytes past n are zero
struct LineEnd {
  uint64_t lo, hi;
  int n;
};

// any distance, by fmt_code (out of line: its scratch and the big-number conversion stay out of the writer's registers)
__device__ __noinline__ LineEnd line_end_any(uint32_t code, double d, char delim)
{
  LineEnd e;
  char g[24];
  const int n = fmt_code(code, d, g);
  e.lo = (unsigned char)delim;
  e.hi = 0;
  for (int k = 0; k <= n; k++) {
    const uint64_t c = k < n ? (unsigned char)g[k] : 10u;
    if (k < 7)
      e.lo |= c << 8 * (k + 1);
    else
      e.hi |= c << 8 * (k - 7);
  }
  e.n = n + 2;
  return e;
}

__device__ __forceinline__ LineEnd line_end(uint32_t code, double d, char delim)
{
  const int X = (int)((code >> 20) & 63u) - 16;
  LineEnd e;
  if (code >> 30 == 1 && X < 0 && X >= -4) {
    // "0." , -X - 1 zeros, the digits without their trailing zeros. The six digits as bytes: q = 1000 a + b, both in
    // 16-bit lanes, hundreds by 41 / 4096 and tens by 103 / 1024 (exact below 1,000 and below 100).
    const uint32_t q = code & 0xFFFFFu, hi3 = q / 1000u, v = hi3 | (q - 1000u * hi3) << 16;
    const uint32_t h = (v * 41u >> 12) & 0x000F000Fu, r = v - 100u * h, t = (r * 103u >> 10) & 0x000F000Fu, u = r - 10u * t;
    const uint64_t D = (uint64_t)((h & 0xFFFFu) | (t & 0xFFFFu) << 8 | (u & 0xFFFFu) << 16) |
                       (uint64_t)((h >> 16) | (t >> 16) << 8 | (u >> 16) << 16) << 24;
    const int nd = (71 - __clzll((long long)D)) >> 3, z = -X - 1;
    const uint64_t body = ((D | 0x303030303030ull) & ((1ull << 8 * nd) - 1)) | 10ull << 8 * nd;
    const uint64_t pre = (uint64_t)(unsigned char)delim | 0x2E3000ull | (0x303030000000ull & ((1ull << 8 * (3 + z)) - 1));
    const int s = 8 * (3 + z);
    e.lo = pre | body << s;
    e.hi = body >> (64 - s);
    e.n = 3 + z + nd + 1;
    return e;
  }
  return line_end_any(code, d, delim);
}

// a line byte by byte (out of line, as few lines come here)
__device__ __noinline__ void put_line_bytes(char *o, const RowArgs &a, long i, long j, const LineEnd &e)
{
  char g[16];
  for (int k = 0; k < e.n - 2; k++) g[k] = (char)((k < 7 ? e.lo >> 8 * (k + 1) : e.hi >> 8 * (k - 7)));
  put_line(o, a, i, j, 0, a.names + a.name_off[i], a.name_len[i], g, e.n - 2);
}

// the decimal digits of v < 10^8, first digit in the low byte: four 2-digit lanes (100 by 5243 / 2^19, exact below 43,699;
// 10 by 103 / 1024), leading zeros shifted out
__device__ __forceinline__ uint64_t number_word(uint32_t v)
{
  const uint32_t a = v / 10000u, b = v - 10000u * a;
  const uint32_t a1 = a * 5243u >> 19, b1 = b * 5243u >> 19;
  const uint64_t t = (uint64_t)(a1 | (a - 100u * a1) << 16) | (uint64_t)(b1 | (b - 100u * b1) << 16) << 32;
  const uint64_t u = (t * 103u >> 10) & 0x000F000F000F000Full;
  const uint64_t d = u | (t - 10u * u) << 8;
  const int z = v ? (__ffsll((long long)d) - 1) & ~7 : 56;
  return (d | 0x3030303030303030ull) >> z;
}

// a stream of bytes on its way to aligned words: acc holds the s / 8 bytes of the word at p that came so far
struct LineWords {
  uint64_t *p, acc;
  int s;
  __device__ __forceinline__ void put8(uint64_t x)
  {
    *p++ = acc | x << s;
    acc = x >> 1 >> (63 - s);
  }
  __device__ __forceinline__ void put(uint64_t x, int n)  // the n low bytes of x (1 to 8); the others are zero
  {
    acc |= x << s;
    const int t = s + 8 * n;
    if (t >= 64) {
      *p++ = acc;
      acc = x >> 1 >> (63 - s);
    }
    s = t & 63;
  }
  // n bytes (0 or more) from the unaligned address src, by the aligned words that hold them
  __device__ __forceinline__ void put_name(const char *src, int n)
  {
    const uint64_t *q = reinterpret_cast<const uint64_t *>(reinterpret_cast<uintptr_t>(src) & ~(uintptr_t)7);
    const int o = (int)(reinterpret_cast<uintptr_t>(src) & 7), words = (o + n + 7) >> 3, f = 8 * o;
    uint64_t cur = words ? __ldg(q) : 0;
    for (int left = n, k = 1; left > 0; left -= 8, k++) {
      const uint64_t nxt = k < words ? __ldg(q + k) : 0;
      const uint64_t x = cur >> f | nxt << 1 << (63 - f);
      cur = nxt;
      if (left >= 8)
        put8(x);
      else
        put(x & ((1ull << 8 * left) - 1), left);
    }
  }
};

// one warp per (row, segment): the segment's text at its scanned offset (the row's self line in segment 0)
template <bool DCODE>
__device__ __forceinline__ void write_rows(const RowArgs &a, long bx, int sg)
{
  __shared__ __align__(16) char stage[kWarps][kStage];
  __shared__ uint64_t prefix[kWarps][kLineName / 8 + 1];
  const RunConsts &rc = a.rc;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long i = a.r0 + bx * kWarps + warp;
  if (i >= a.r1) return;
  const long slot = (i - a.r0) * a.maxseg + sg;
  const long lb = rc.cross ? rc.n1 : i + 1;
  const long c0 = lb + (long)sg * kSeg, c1 = min(rc.N, c0 + kSeg);
  if (a.seg_bytes[slot] == 0) return;
  const int nli = a.name_len[i];
  const char *ni = a.names + a.name_off[i];
  Stager S;
  S.buf = stage[warp];
  S.gpos = (uintptr_t)(a.out + a.seg_off[slot]);
  S.gend = S.gpos + a.seg_bytes[slot];
  S.head = (int)(S.gpos & 15);
  S.fill = 0;
  S.over = false;
  const int sl = sg == 0 ? self_len(a, i) : 0;
  if (sl) {
    const bool direct = S.head + sl > kStage;
    if (direct && S.gpos + sl > S.gend) {
      if (lane == 0) atomicAdd(a.err, 1ull);
      return;
    }
    if (lane == 0) {
      char *o = direct ? (char *)S.gpos : S.buf + S.head;
      if (rc.format == 0) {
        o = put_bytes(o, ni, nli);
        *o++ = rc.delim;
        o = put_bytes(o, ni, nli);
        *o++ = rc.delim;
      } else {
        char t[24];
        const int n = fmt_long(i, t);
        o = put_bytes(o, t, n);
        *o++ = rc.delim;
        o = put_bytes(o, t, n);
        *o++ = rc.delim;
      }
      *o++ = '0';
      *o = '\n';
    }
    __syncwarp();
    if (direct) {
      S.gpos += sl;
      S.head = (int)(S.gpos & 15);
    } else
      S.fill = sl;
  }
  // the lines' common start in words: name i (or its number) and a delimiter
  const int n1 = (rc.format == 0 ? nli : digits_of(i)) + 1;
  uint64_t *const pw = prefix[warp];
  if (n1 <= kLineName) {
    if (lane <= kLineName / 8) pw[lane] = 0;
    __syncwarp();
    char *const pc = reinterpret_cast<char *>(pw);
    if (rc.format == 0) {
      for (int k = lane; k < nli; k += 32) pc[k] = ni[k];
    } else if (lane == 0) {
      fmt_long(i, pc);
    }
    if (lane == 0) pc[n1 - 1] = rc.delim;
    __syncwarp();
  }
  for (long j0 = c0; j0 < c1; j0 += 32) {
    const long j = j0 + lane;
    double thisD = 0.;
    bool put;
    uint32_t code = 0;
    if (DCODE) {
      // the stats kernel's code of this pair: printed or not, and its digits
      code = j < c1 ? a.dcode[(size_t)(i - a.r0) * a.ncols + (j - a.colbase)] : 0u;
      put = code != 0;
      if (put && (code >> 30) == 3u) linked_pair(a, i, j, thisD);
    } else {
      put = j < c1 && linked_pair(a, i, j, thisD);
      int gl;
      if (put) code = print_code(thisD, gl);
    }
    LineEnd e = {0, 0, 0};
    int n2 = 0, len = 0;
    if (put) {
      e = line_end(code, thisD, rc.delim);
      n2 = rc.format == 0 ? a.name_len[j] : digits_of(j);
      len = n1 + n2 + e.n;
    }
    int pre = len;
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, pre, o);
      if (lane >= o) pre += t;
    }
    const int total = __shfl_sync(0xffffffffu, pre, 31);
    if (total == 0) continue;
    if (S.head + S.fill + total > kStage) S.flush(lane);
    const bool whole = S.head + total > kStage;  // larger than the staging buffer (very long names): written in place
    if (whole && S.gpos + total > S.gend) {
      S.over = true;
      break;
    }
    const unsigned puts = __ballot_sync(0xffffffffu, put);
    if (whole || n1 > kLineName || __any_sync(0xffffffffu, put && (n2 > (rc.format == 0 ? kLineName : 8) || len < 8))) {
      if (put) {
        put_line_bytes(whole ? (char *)(S.gpos + pre - len) : S.buf + S.head + S.fill + (pre - len), a, i, j, e);
      }
    } else {
      // Lines meet inside 8-byte words: a lane leaves the bytes before its line zero in its first word (the first lane
      // keeps what stands there), and adds its own last bytes to the next lane's first word once that is stored. Lines of
      // 8 bytes or more: a word holds bytes of two lines at most.
      LineWords w;
      if (put) {
        const int at = S.head + S.fill + (pre - len);
        w.p = reinterpret_cast<uint64_t *>(S.buf + (at & ~7));
        w.s = 8 * (at & 7);
        w.acc = (puts & lanemask_lt()) ? 0 : *w.p & ((1ull << w.s) - 1);
        for (int k = 0; k < n1 >> 3; k++) w.put8(pw[k]);
        if (n1 & 7) w.put(pw[n1 >> 3], n1 & 7);
        if (rc.format == 0)
          w.put_name(a.names + a.name_off[j], n2);
        else
          w.put(number_word((uint32_t)j), n2);
        w.put(e.lo, min(e.n, 8));
        if (e.n > 8) w.put(e.hi, e.n - 8);
      }
      __syncwarp();
      const bool last = lane == 31 - __clz(puts);
      if (put && w.s) *w.p = last ? w.acc : *w.p | w.acc;
    }
    __syncwarp();
    if (whole) {
      S.gpos += total;
      S.head = (int)(S.gpos & 15);
    } else {
      S.fill += total;
    }
  }
  S.flush(lane);
  if (S.over && lane == 0) atomicAdd(a.err, 1ull);
}

__global__ void __launch_bounds__(256, 4) write_kernel(const __grid_constant__ RowArgs a) { write_rows<true>(a, blockIdx.x, blockIdx.y); }

// Batched row stage: block b of the batch is row block blocks[b].y of alignment blocks[b].x; blockIdx.y is the
// segment (blocks past an alignment's segment count exit).
__global__ void __launch_bounds__(256) stats_batch_kernel(const RowArgs *descs, const int2 *blocks)
{
  const int2 B = blocks[blockIdx.x];
  const RowArgs &a = descs[B.x];
  if ((long)blockIdx.y >= a.maxseg) return;
  stats_rows(a, B.y, blockIdx.y);
}

__global__ void __launch_bounds__(256) sum_batch_kernel(const RowArgs *descs, const int2 *blocks)
{
  const int2 B = blocks[blockIdx.x];
  sum_rows(descs[B.x], B.y);
}

__global__ void __launch_bounds__(256, 3) write_batch_kernel(const RowArgs *descs, const int2 *blocks)
{
  const int2 B = blocks[blockIdx.x];
  const RowArgs &a = descs[B.x];
  if ((long)blockIdx.y >= a.maxseg) return;
  write_rows<false>(a, B.y, blockIdx.y);
}

// Per alignment of a batch (single-file runs, bin 0 only): links, skips and maximum over its (row, segment)
// slots, and tn93's mean numerator and weight: the rows' sums added in row order from 0 (swifttn93.cpp:2838-2848).
// One block per alignment.
__global__ void __launch_bounds__(256) aln_reduce_kernel(const RowArgs *descs, double *out /* [K][3] */,
                                                         long long *cnt /* [K][2] */)
{
  __shared__ long long rl[8], rs[8];
  __shared__ double rm[8];
  const RowArgs &a = descs[blockIdx.x];
  const long nr = a.r1 - a.r0, ms = a.maxseg;
  long long links = 0, skipped = 0;
  double m = 0.;
  for (long g = threadIdx.x; g < nr * ms; g += 256) {
    links += a.seg_links[g];
    skipped += a.seg_skip[g];
    m = fmax(m, a.seg_max[g * 3]);
  }
  double w = 0.;
  bool whole = true;
  for (long r = threadIdx.x; r < nr; r += 256) {
    const double x = a.row_w[r * 3];
    whole &= x >= 0. && x == floor(x);
    w = __dadd_rn(w, x);
  }
  chain_weights<256, 3>(a.row_w, nr, w, whole, out + blockIdx.x * 3 + 2);
  chain_rows<256, 3>(a.row_sum, nr, out + blockIdx.x * 3 + 1);
  for (int o = 16; o; o >>= 1) {
    links += __shfl_xor_sync(0xffffffffu, links, o);
    skipped += __shfl_xor_sync(0xffffffffu, skipped, o);
    m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  }
  if ((threadIdx.x & 31) == 0) {
    rl[threadIdx.x >> 5] = links;
    rs[threadIdx.x >> 5] = skipped;
    rm[threadIdx.x >> 5] = m;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; w++) {
      links += rl[w];
      skipped += rs[w];
      m = fmax(m, rm[w]);
    }
    out[blockIdx.x * 3] = m;
    cnt[blockIdx.x * 2] = links;
    cnt[blockIdx.x * 2 + 1] = skipped;
  }
}

// -f hyphy: per matrix row the byte count, then the text: "\n{" d(r,0) "," ... "}" with 0 on the diagonal, the
// reported distance where the pair was reported and 100 elsewhere (swifttn93.cpp:2869-2897)
__device__ __forceinline__ int hy_entry(const double *hy, long N, long r, long c, char *buf)
{
  if (c == r) {
    buf[0] = '0';
    return 1;
  }
  const double d = hy[(size_t)r * N + c];
  if (d != d) {
    buf[0] = '1';
    buf[1] = '0';
    buf[2] = '0';
    return 3;
  }
  return fmt_g(d, buf);
}

__global__ void hy_len_kernel(const double *hy, long N, unsigned long long *row_bytes)
{
  const int lane = threadIdx.x & 31;
  const long r = blockIdx.x * (long)kWarps + (threadIdx.x >> 5);
  if (r >= N) return;
  unsigned long long b = 0;
  for (long c = lane; c < N; c += 32) {
    char t[24];
    b += hy_entry(hy, N, r, c, t) + (c ? 1 : 0);
  }
  for (int o = 16; o; o >>= 1) b += __shfl_xor_sync(0xffffffffu, b, o);
  if (lane == 0) row_bytes[r] = b + 3;  // "\n{" and "}"
}

__global__ void hy_write_kernel(const double *hy, long N, const unsigned long long *row_off, char *out)
{
  const int lane = threadIdx.x & 31;
  const long r = blockIdx.x * (long)kWarps + (threadIdx.x >> 5);
  if (r >= N) return;
  char *o = out + row_off[r];
  if (lane == 0) {
    o[0] = '\n';
    o[1] = '{';
  }
  o += 2;
  for (long c0 = 0; c0 < N; c0 += 32) {
    const long c = c0 + lane;
    char t[24];
    int len = 0;
    if (c < N) len = hy_entry(hy, N, r, c, t) + (c ? 1 : 0);
    int pre = len;
    for (int s = 1; s < 32; s <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, pre, s);
      if (lane >= s) pre += v;
    }
    const int total = __shfl_sync(0xffffffffu, pre, 31);
    if (c < N) {
      char *p = o + (pre - len);
      if (c) *p++ = ',';
      put_bytes(p, t, len - (c ? 1 : 0));
    }
    o += total;
  }
  if (lane == 0) *o = '}';
}

__global__ void fill_nan_kernel(double *p, size_t n)
{
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x)
    p[k] = __longlong_as_double(0x7FF8000000000000ll);
}

// Kernel attributes (the opt-in to more than 48 KB of dynamic shared memory) belong to each device's context, so
// they are set once per device. PerDevice::once runs set() for the current device unless it already succeeded
// there; callers on other threads wait for it (the lock is held while set() runs), and a failed set() is retried
// by the next call, so no launch can see the flag before the attribute is in place.
struct PerDevice {
  std::mutex mu;
  std::atomic<unsigned long long> done{0};
  template <class F>
  cudaError_t once(F set)
  {
    int d = 0;
    cudaError_t e = cudaGetDevice(&d);
    if (e != cudaSuccess) return e;
    const unsigned long long bit = 1ull << (d & 63);
    if (done.load(std::memory_order_acquire) & bit) return cudaSuccess;
    std::lock_guard<std::mutex> g(mu);
    if (done.load(std::memory_order_relaxed) & bit) return cudaSuccess;
    e = set();
    if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_release);
    return e;
  }
};

// pair kernel launch (dynamic shared memory above the 48 KB default needs the opt-in attribute once per device).
// Register budgets: 2 blocks per SM (128 registers, no spills), 3 (80 registers, some spills) or 4 (64).
template <int MINB>
cudaError_t launch_pair_t(const PairArgs &A, dim3 g, cudaStream_t st)
{
  static PerDevice attr;
  cudaError_t e = attr.once([] {
    cudaError_t r;
    if ((r = cudaFuncSetAttribute(pair_kernel<false, false, MINB>,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPairSmem)) != cudaSuccess)
      return r;
    if ((r = cudaFuncSetAttribute(pair_kernel<true, false, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)kPairSmem)) != cudaSuccess)
      return r;
    return cudaFuncSetAttribute(pair_kernel<true, true, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)kPairSmem);
  });
  if (e != cudaSuccess) return e;
  if (A.rc.wplane) {
    if (A.rc.gapmm)
      pair_kernel<true, true, MINB><<<g, 256, kPairSmem, st>>>(A);
    else
      pair_kernel<true, false, MINB><<<g, 256, kPairSmem, st>>>(A);
  } else
    pair_kernel<false, false, MINB><<<g, 256, kPairSmem, st>>>(A);
  return cudaGetLastError();
}

template <bool WPLANE, bool PACK>
cudaError_t launch_event_t(const PairArgs &A, dim3 g, cudaStream_t st)
{
  static PerDevice attr;
  const cudaError_t e = attr.once([] {
    return cudaFuncSetAttribute(event_kernel<WPLANE, PACK>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)EvTile<WPLANE>::smem);
  });
  if (e != cudaSuccess) return e;
  event_kernel<WPLANE, PACK><<<g, kEvThreads, EvTile<WPLANE>::smem, st>>>(A);
  return cudaGetLastError();
}

// Whether a pair launch takes the split form (event_kernel, then formula_kernel): with the tensor-core records, whose
// slots hold the final aggregates, packed event sums (16-bit lanes), a code matrix that 32-bit offsets reach and, under
// the N plane, the sequences' N words. (gapmm has weighted records, or takes the fused kernel: event_kernel does not know
// sites where both have a gap.)
bool pair_split(const PairArgs &A)
{
  if (A.lin) return true;
  return A.tcagg && A.ev2 && !A.rc.gapmm && A.rc.packed && A.rc.Lc * A.rc.Npad < (1l << 32) && (!A.rc.wplane || A.wl_off);
}

// Columns of a segment and rows of a warp in the formula kernel, for nrows x ncols pairs: a warp takes one segment of a few
// rows, or, where each column has a summary unit of its own (a server batch), a strip of 32 columns down many rows, so that
// a warp's pairs belong to one or two units. Long segments and several rows keep the atomics of a warp's totals rare (22.4 M
// pairs: 0.85 ms with 1,024 columns, 0.90 with 512); small launches take shorter segments, down to 128 columns, so that the
// SMs have two waves of warps (1,801 x 1,203 in bands of 0.2-0.4 M pairs: 0.10 -> 0.05 ms a band), and rows are added up
// only past four waves, strips past one (a strip's row has few pairs, and its warp four atomics on its query's words: 32
// columns x 30,000 rows 109 us with a row to a warp, 59 us with 8).
void formula_shape(long nrows, long ncols, bool units, int sms, int &segw, int &rpw)
{
  segw = units ? 32 : kSeg;
  while (segw > 128 && nrows * ((ncols + segw - 1) / segw) < sms * 48l) segw /= 2;
  const long nseg = (ncols + segw - 1) / segw;
  rpw = (int)std::max<long>(1, std::min<long>(1024 / std::min<long>(segw, ncols), nrows * nseg / (sms * (units ? 24l : 128l))));
}

// The pair stage of rows [A.r0, A.r1) and the columns from A.cstart (32 ncolblocks of them). Fused kernel: 4 resident
// blocks per SM (64 registers a thread) with the tensor-core counts and no N plane, 3 (80) with it, 2 with the popcount
// loop, which needs the registers. TN93G_PAIR_BLOCKS=2|3|4 overrides.
cudaError_t launch_pair(const PairArgs &A, long ncolblocks, long nrows, int sms, cudaStream_t st)
{
  static const int forced = [] {
    const char *e = getenv("TN93G_PAIR_BLOCKS");
    return e ? (atoi(e) == 4 ? 4 : atoi(e) == 3 ? 3 : 2) : 0;
  }();
  dim3 g((unsigned)ncolblocks, (unsigned)((nrows + kTile - 1) / kTile));
  if (pair_split(A)) {
    const long jend = std::min<long>(A.cend, A.cstart + ncolblocks * kTile), jbeg = A.cstart & ~1l, ibeg = A.r0 & ~1l;
    const long rows = A.rc.wplane ? EvTile<true>::rows : EvTile<false>::rows;
    const dim3 ge((unsigned)((jend - jbeg + kEvCols - 1) / kEvCols), (unsigned)((A.r1 - ibeg + rows - 1) / rows));
    const cudaError_t e = A.lin         ? cudaSuccess
                          : A.rc.wplane ? launch_event_t<true, false>(A, ge, st)
                          : A.tc16      ? launch_event_t<false, true>(A, ge, st)
                                        : launch_event_t<false, false>(A, ge, st);
    if (e != cudaSuccess) return e;
    const long jlo = std::max(A.cstart, A.tcncols ? A.tccolbase : A.colbase);
    int segw, rpw;
    formula_shape(nrows, jend - jlo, A.ex.colunit != nullptr, sms, segw, rpw);
    const long nseg = (jend - jlo + segw - 1) / segw;
    const dim3 gf((unsigned)((nrows + kWarps * rpw - 1) / (kWarps * rpw)), (unsigned)nseg);
    if (A.lin) {
      if (A.tc16)
        formula_kernel<true, true><<<gf, 256, 0, st>>>(A, jlo, jend, segw, rpw);
      else
        formula_kernel<false, true><<<gf, 256, 0, st>>>(A, jlo, jend, segw, rpw);
    } else if (A.tc16)
      formula_kernel<true, false><<<gf, 256, 0, st>>>(A, jlo, jend, segw, rpw);
    else
      formula_kernel<false, false><<<gf, 256, 0, st>>>(A, jlo, jend, segw, rpw);
    return cudaGetLastError();
  }
  const int minb = forced ? forced : (A.tcagg ? (A.rc.wplane ? 3 : 4) : 2);
  if (minb == 4) return launch_pair_t<4>(A, g, st);
  return minb == 3 ? launch_pair_t<3>(A, g, st) : launch_pair_t<2>(A, g, st);
}

// the tensor-core count kernels' opt-in to their dynamic shared memory, once per device
cudaError_t tc_attr_once()
{
  static PerDevice attr;
  return attr.once([] {
    cudaError_t e = cudaFuncSetAttribute(count_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTcSmem);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(count_tc_batch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTcSmem);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(count_tc_persist_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPSmem);
  });
}

// TN93G_TC_KERNEL=tile selects the one-tile-per-CTA count kernel instead of the persistent one (same records)
bool tc_tile_kernel()
{
  static const bool tile = [] {
    const char *e = getenv("TN93G_TC_KERNEL");
    return e && strcmp(e, "tile") == 0;
  }();
  return tile;
}

// Tensor-core counts over the count_tc_kernel grid (gx column tiles x gy row tiles) of T: the persistent kernel on
// min(tiles, SMs) CTAs, or one CTA per tile.
cudaError_t launch_count_grid(const TcArgs &T, long gx, long gy, int sms, cudaStream_t st)
{
  cudaError_t e = tc_attr_once();
  if (e != cudaSuccess) return e;
  if (tc_tile_kernel()) {
    count_tc_kernel<<<dim3((unsigned)gx, (unsigned)gy), 128, kTcSmem, st>>>(T);
  } else {
    const long nt = gx * gy;
    count_tc_persist_kernel<<<(unsigned)std::min<long>(nt, sms), kPThreads, kPSmem, st>>>(T, nullptr, nullptr, 0);
  }
  return cudaGetLastError();
}

// the same over a list of (descriptor, first row, first column) tiles; G carries the wait limit, the error word
// and the test hook for the persistent kernel
cudaError_t launch_count_list(const TcArgs &G, const TcArgs *descs, const int4 *tiles, int ntiles, int sms,
                              cudaStream_t st)
{
  cudaError_t e = tc_attr_once();
  if (e != cudaSuccess) return e;
  if (tc_tile_kernel())
    count_tc_batch_kernel<<<(unsigned)ntiles, 128, kTcSmem, st>>>(descs, tiles);
  else
    count_tc_persist_kernel<<<(unsigned)std::min(ntiles, sms), kPThreads, kPSmem, st>>>(G, descs, tiles, ntiles);
  return cudaGetLastError();
}

}  // namespace

//================================================================================================== host side

struct DevBuf {
  void *p = nullptr;
  size_t n = 0;
};

// the buffers of tn93g_batch_run
enum BatchBuf {
  BB_CODES, BB_SEEN, BB_NN, BB_VARCOL, BB_PLANES, BB_CC, BB_CCT, BB_EVCOUNT, BB_EVOFF, BB_EV, BB_AGG, BB_SITE,
  BB_NAMES, BB_NAMEOFF, BB_NAMELEN, BB_COUNTS, BB_DIST, BB_RQ, BB_RQN, BB_COUNTERS, BB_PDESC, BB_RDESC, BB_ROWDESC,
  BB_TILES, BB_NEXT, BB_BLOCKS, BB_SBYTES, BB_SOFF, BB_SLINKS, BB_SSKIP, BB_SMAX, BB_RSUM, BB_RW, BB_HIST, BB_TOTAL,
  BB_SCANTMP, BB_RED, BB_REDC, BB_FIRST, BB_FIRSTIDX, BB_OUT, BB_OH, BB_TCAGG, BB_TCDESC, BB_TCTILES, BB_TCERR,
  BB_UND, BB_UNDN, BB_AMB, BB_SCANDESC, BB_PACKDESC, BB_TRDESC, BB_OHDESC, BB_BOFF, BB_EV2, BB_THREE, BB_SPLIT, BB_COUNT
};
constexpr int kMaxTcChunks = 48;         // row chunks of a band on the tensor-core count path
// Pairs per chunk of the tensor-core path (count kernel, then pair kernel): 16 M pairs, 256 MB of 16-byte records.
// Larger chunks amortise the persistent count kernel's pipeline fill and drain and the pair kernel's last wave
// (6,700 x 1,500 benchmark set, resolve pair stage per 22.4 M pairs: 3.17 ms with 2 M-pair chunks, 2.94 with 4 M,
// 2.77 with 8 M, 2.71 with 16 M, 2.67 with one chunk); the records then travel through HBM, which the pair stage
// leaves almost idle. TN93G_TC_CHUNK_PAIRS overrides.
constexpr long kTcChunkPairs = 16l << 20;

struct tn93g_set {
  long N = 0, L = 0;
  size_t cap[5] = {0, 0, 0, 0, 0};  // bytes of d_codes, d_counts, d_names, d_name_off, d_name_len
  uint8_t *d_codes = nullptr;
  long *d_counts = nullptr;
  char *d_names = nullptr;
  uint64_t *d_name_off = nullptr;
  int32_t *d_name_len = nullptr;
  std::vector<long> counts, name_len;
};

constexpr int kUploadThreads = 4;  // upload_host's

struct tn93g_ctx {
  int device = 0;
  size_t budget = 0, used = 0;
  cudaStream_t stream = nullptr;
  std::string err;
  LogTable *d_logt = nullptr;
  Tables *h_tab = nullptr;
  PairTables *h_ptab = nullptr;  // host staging of the pair stage's tables
  DevBuf seen, nN, varcol, planes, cc, ccT, evcount, evoff, ev, ev2, three, agg, site, dist, dcode, wcount, wloff, wl, rq, rqn, counters,
      rbytes, rsum, rw, fraw, fspan, flen, fcode,
      rmax, rlinks, rskip, hist, roff, out, hy;
  void *pinned = nullptr;
  size_t pinned_n = 0;
  cudaEvent_t evs[16];
  cudaStream_t copy_stream = nullptr;   // device->host copies of finished bands
  cudaStream_t write_stream = nullptr;  // text writers of finished bands (beside the next bands' kernels)
  cudaEvent_t evw0[2], evw1[2], evc0[2], evc1[2];
  cudaEvent_t evrow[2];  // per band parity: its text is written
  cudaEvent_t evk[2][5];  // per band parity: start, after pair, after replay, after stats+sums+scan, stats on host
  cudaEvent_t evcnt[2][2 * kMaxTcChunks];  // per band parity: around each chunk's tensor-core count kernel
  DevBuf out2[2], total;
  void *pin2[2] = {nullptr, nullptr};
  size_t pin2_n[2] = {0, 0};
  void *pstats = nullptr;
  size_t pstats_n = 0;
  std::vector<std::pair<int, std::string>> batch_keys, batch_site_keys;  // what BB_AGG and BB_SITE hold
  std::string tab_key;   // what agg and site hold (run_impl; empty: nothing)
  void *hrun = nullptr;  // pinned block of a run's small transfers
  size_t hrun_n = 0;
  void *upload_pin = nullptr;  // upload_host's pieces (two a thread), and the events of their copies, made with the context
  cudaEvent_t upload_ev[2 * kUploadThreads] = {nullptr};
  // device buffers of freed sets, kept for the next upload (repeated upload/free skips the allocator)
  std::vector<std::pair<void *, size_t>> set_pool;
  double timings[8] = {0};
  long launches = 0;
  size_t dev_out_n = 0;
  DevBuf bb[BB_COUNT];  // buffers of tn93g_batch_run (indexed by BatchBuf)
  int count_path = 1;  // clean-site counts: 0 popcounts on the CUDA cores, 1 tensor cores (tcgen05)
  int sms = 148;       // streaming multiprocessors of the device (persistent and grid-stride launches)
  DevBuf ohimg, tcagg;
  uint64_t wait_ns = kTcWaitNs;  // limit of each bounded device wait
  bool exact_sums = false;       // tn93g_set_exact_sums
  int fault = TN93G_FAULT_NONE;  // test hook for the next run (tn93g_inject_fault)
  // exactness: undecided lists and counts per band parity, the summary units' bounds, the resolver's entries and
  // run descriptors, and the logarithm's band and candidate spread (tn93g_set_log_band)
  DevBuf und[2], undn, undwork, rdesc;
  double log_band = kLogBand, log_spread = kLogSpread;
  std::vector<tn93g_server *> servers;  // on this context
  bool bands_busy = false;    // a run is using its band buffers
  bool records_busy = false;  // a batch's pair stage has yet to read bb[BB_EV2] and bb[BB_TCAGG]
};

namespace {

#define CU(call)                                                                      \
  do {                                                                                \
    cudaError_t e_ = (call);                                                          \
    if (e_ != cudaSuccess) {                                                          \
      ctx->err = std::string(#call) + ": " + cudaGetErrorString(e_);                  \
      return e_ == cudaErrorMemoryAllocation ? TN93G_ENOMEM : TN93G_ECUDA;            \
    }                                                                                 \
  } while (0)

// length of an event list with its null events
uint32_t pad_events(uint32_t n) { return (n + kEvPad - 1) / kEvPad * kEvPad; }

// gives b back; the stream's work on it ends first (cudaFree waits for the device)
void release(tn93g_ctx *ctx, DevBuf &b)
{
  if (!b.p) return;
  cudaFree(b.p);
  ctx->used -= b.n;
  b.p = nullptr;
  b.n = 0;
}

void server_reclaim(tn93g_server *srv);

// Gives back the memory that only saves time, for a call that has no room without it: a run's and the servers' event offsets
// (the pair stage takes the fused kernel from then on, with the same results), the servers' larger chunks, the records that
// the last batch left, and the band and text buffers that the last run left. Kernels get such a buffer's address from the context or the server at each launch, never from an
// earlier one. False when there was nothing to give.
bool reclaim(tn93g_ctx *ctx)
{
  const size_t before = ctx->used;
  for (cudaStream_t s : {ctx->stream, ctx->write_stream, ctx->copy_stream}) cudaStreamSynchronize(s);
  release(ctx, ctx->ev2);
  if (!ctx->records_busy) {
    release(ctx, ctx->bb[BB_EV2]);
    release(ctx, ctx->bb[BB_TCAGG]);
  }
  if (!ctx->bands_busy)
    for (DevBuf *b : {&ctx->dist, &ctx->dcode, &ctx->tcagg, &ctx->rq, &ctx->und[0], &ctx->und[1], &ctx->out2[0], &ctx->out2[1]})
      release(ctx, *b);
  for (tn93g_server *s : ctx->servers) server_reclaim(s);
  return ctx->used < before;
}

// bytes of device memory within the budget; TN93G_ENOMEM where they do not fit
int take_device(tn93g_ctx *ctx, void **p, size_t bytes)
{
  if (ctx->budget && ctx->used + bytes > ctx->budget) {
    ctx->err = "over the context's HBM budget";
    return TN93G_ENOMEM;
  }
  const cudaError_t e = cudaMalloc(p, bytes);
  if (e != cudaSuccess) {
    cudaGetLastError();  // the caller may do without
    ctx->err = std::string("cudaMalloc: ") + cudaGetErrorString(e);
    return e == cudaErrorMemoryAllocation ? TN93G_ENOMEM : TN93G_ECUDA;
  }
  ctx->used += bytes;
  return TN93G_OK;
}

// b of at least `bytes`, its contents lost when it grows. spare: memory that the caller can do without (nothing is given back
// for it, and no message is left)
int ensure(tn93g_ctx *ctx, DevBuf &b, size_t bytes, bool spare = false)
{
  if (bytes <= b.n && b.p) return TN93G_OK;
  release(ctx, b);
  bytes = std::max<size_t>(bytes, 256);
  int r = take_device(ctx, &b.p, bytes);
  while (r == TN93G_ENOMEM && !spare && reclaim(ctx)) r = take_device(ctx, &b.p, bytes);
  if (r == TN93G_OK)
    b.n = bytes;
  else if (r == TN93G_ENOMEM && spare)
    ctx->err.clear();
  return r;
}

int ensure_pinned(tn93g_ctx *ctx, size_t bytes)
{
  if (bytes <= ctx->pinned_n) return TN93G_OK;
  if (ctx->pinned) cudaFreeHost(ctx->pinned);
  ctx->pinned = nullptr;
  ctx->pinned_n = 0;
  bytes = std::max<size_t>(bytes + bytes / 4, 1 << 20);
  CU(cudaHostAlloc(&ctx->pinned, bytes, cudaHostAllocDefault));
  ctx->pinned_n = bytes;
  return TN93G_OK;
}

int ensure_pinned_at(tn93g_ctx *ctx, void *&p, size_t &n, size_t bytes, unsigned flags = cudaHostAllocDefault)
{
  if (bytes <= n && p) return TN93G_OK;
  if (p) cudaFreeHost(p);
  p = nullptr;
  n = 0;
  bytes = std::max<size_t>(bytes + bytes / 4, 1 << 20);
  CU(cudaHostAlloc(&p, bytes, flags));
  n = bytes;
  return TN93G_OK;
}

// grows b to `bytes`, keeping its first `keep` bytes (stream-ordered copy)
int ensure_keep(tn93g_ctx *ctx, DevBuf &b, size_t bytes, size_t keep)
{
  if (bytes <= b.n && b.p) return TN93G_OK;
  bytes = std::max<size_t>(bytes + bytes / 2, 1 << 20);
  void *p = nullptr;
  int r = take_device(ctx, &p, bytes);
  while (r == TN93G_ENOMEM && reclaim(ctx)) r = take_device(ctx, &p, bytes);
  if (r != TN93G_OK) return r;
  if (keep && b.p) CU(cudaMemcpyAsync(p, b.p, keep, cudaMemcpyDeviceToDevice, ctx->stream));
  if (b.p) {
    CU(cudaStreamSynchronize(ctx->stream));
    cudaFree(b.p);
    ctx->used -= b.n;
  }
  b.p = p;
  b.n = bytes;
  return TN93G_OK;
}

#define TRY(x)                   \
  do {                           \
    int r_ = (x);                \
    if (r_ != TN93G_OK) return r_; \
  } while (0)

// Host memory on its way to the device: n bytes from src to dst, behind the work of the context's stream.
struct HostSpan {
  void *dst;
  const void *src;
  size_t n;
};

// Queues the copies of the spans on the context's stream; pageable memory has been read when it returns. A copy from
// pageable memory goes through the driver's staging buffer, filled by the calling thread alone (16-18 GB/s here, a third of
// the link). From kUploadMin bytes on, up to kUploadThreads threads fill pinned buffers of the context instead, piece by
// piece, and queue each piece's copy: 60 MB 3.4 -> 1.4 ms. The threads end with the call; where one cannot be started, or
// the buffers cannot be allocated, the rest do its work.
constexpr size_t kUploadPiece = 1 << 20;
constexpr size_t kUploadMin = 4 << 20;

int upload_host(tn93g_ctx *ctx, const std::vector<HostSpan> &spans)
{
  struct Piece {
    char *dst;
    const char *src;
    size_t n;
  };
  std::vector<Piece> pieces;
  std::vector<const HostSpan *> pageable;
  for (const HostSpan &h : spans) {
    cudaPointerAttributes pa;
    bool direct = h.n < kUploadMin / 16;  // many small copies cost more than the staging saves
    if (!direct) {
      const cudaError_t e = cudaPointerGetAttributes(&pa, h.src);
      if (e != cudaSuccess) cudaGetLastError();
      direct = e == cudaSuccess && pa.type != cudaMemoryTypeUnregistered;  // pinned already
    }
    if (direct) {
      if (h.n) CU(cudaMemcpyAsync(h.dst, h.src, h.n, cudaMemcpyHostToDevice, ctx->stream));
      continue;
    }
    pageable.push_back(&h);
    for (size_t at = 0; at < h.n; at += kUploadPiece)
      pieces.push_back({(char *)h.dst + at, (const char *)h.src + at, std::min(kUploadPiece, h.n - at)});
  }
  size_t bytes = 0;
  for (const Piece &p : pieces) bytes += p.n;
  bool staged = bytes >= kUploadMin;
  if (staged && !ctx->upload_pin) {
    if (cudaHostAlloc(&ctx->upload_pin, 2 * kUploadThreads * kUploadPiece, cudaHostAllocDefault) != cudaSuccess) {
      cudaGetLastError();
      ctx->upload_pin = nullptr;
      staged = false;
    }
  }
  if (!staged) {
    for (const HostSpan *h : pageable) CU(cudaMemcpyAsync(h->dst, h->src, h->n, cudaMemcpyHostToDevice, ctx->stream));
    return TN93G_OK;
  }
  std::atomic<size_t> next{0};
  std::atomic<int> failed{0};
  auto work = [&](int t) {
    cudaSetDevice(ctx->device);
    for (int turn = 0;; turn++) {
      const size_t k = next++;
      if (k >= pieces.size() || failed) break;
      const int b = 2 * t + (turn & 1);
      char *pin = (char *)ctx->upload_pin + b * kUploadPiece;
      cudaError_t e = cudaEventSynchronize(ctx->upload_ev[b]);  // the buffer's previous copy (an earlier call's too)
      if (e == cudaSuccess) {
        memcpy(pin, pieces[k].src, pieces[k].n);
        e = cudaMemcpyAsync(pieces[k].dst, pin, pieces[k].n, cudaMemcpyHostToDevice, ctx->stream);
      }
      if (e == cudaSuccess) e = cudaEventRecord(ctx->upload_ev[b], ctx->stream);
      if (e != cudaSuccess) failed = (int)e;
    }
  };
  std::thread helpers[kUploadThreads - 1];
  const int most = std::min<int>(kUploadThreads, std::max(1u, std::thread::hardware_concurrency()));
  for (int t = 1; t < most; t++) {
    try {
      helpers[t - 1] = std::thread(work, t);
    } catch (const std::system_error &) {
      break;
    }
  }
  work(0);
  for (std::thread &h : helpers)
    if (h.joinable()) h.join();
  CU((cudaError_t)(int)failed);
  return TN93G_OK;
}

// The host's C library log of every listed argument: the decision oracle for pairs whose printed bytes or
// decisions depend on how that log rounds (the reference calls the same function, swifttn93.cpp:1954-2001).
// Large lists (resolve-all passes) are split over the host's threads.
void host_logs(std::vector<UndEntry> &E)
{
  auto work = [&E](size_t b, size_t e) {
    for (size_t k = b; k < e; k++)
      for (int q = 0; q < 3; q++) E[k].lg[q] = q < E[k].nlog ? log(E[k].arg[q]) : 0.;
  };
  const size_t n = E.size();
  const unsigned nt = std::max(1u, std::min(std::thread::hardware_concurrency(), (unsigned)(n / 65536 + 1)));
  if (nt == 1) {
    work(0, n);
    return;
  }
  std::vector<std::thread> th;
  for (unsigned t = 0; t < nt; t++) th.emplace_back(work, n * t / nt, n * (t + 1) / nt);
  for (auto &t : th) t.join();
}

// Finishes the n listed pairs (entries (k, i << 32 | j), run k described by d_descs[k] in device memory) with the
// C library's logarithms: the site-order walk gives each pair's formula arguments on the device, the host takes
// their logs, and the device evaluates the formula with them into the pair's raw-distance slot.
int resolve_listed(tn93g_ctx *ctx, const ReplayArgs *d_descs, const unsigned long long *d_list, unsigned n,
                   cudaStream_t st)
{
  if (!n) return TN93G_OK;
  unsigned piece = n;  // pairs at a time: all, or as many as there is room for
  int r;
  while ((r = ensure(ctx, ctx->undwork, (size_t)piece * sizeof(UndEntry))) == TN93G_ENOMEM && piece > 4096) piece = (piece + 1) / 2;
  TRY(r);
  UndEntry *dw = (UndEntry *)ctx->undwork.p;
  std::vector<UndEntry> h;
  for (size_t at = 0; at < n; at += piece) {
    const unsigned m = (unsigned)std::min<size_t>(piece, n - at);
    und_args_kernel<<<(unsigned)std::min<unsigned long>((m + kWarps - 1) / kWarps, 8ul * ctx->sms), 256, 0, st>>>(
        d_descs, d_list + 2 * at, m, dw);
    CU(cudaGetLastError());
    h.resize(m);
    CU(cudaMemcpyAsync(h.data(), dw, (size_t)m * sizeof(UndEntry), cudaMemcpyDeviceToHost, st));
    CU(cudaStreamSynchronize(st));
    host_logs(h);
    CU(cudaMemcpyAsync(dw, h.data(), (size_t)m * sizeof(UndEntry), cudaMemcpyHostToDevice, st));
    und_finish_kernel<<<(m + 255) / 256, 256, 0, st>>>(d_descs, dw, m);
    CU(cudaGetLastError());
    ctx->launches += 2;
  }
  return TN93G_OK;
}

// a tn93g_sink that appends to the std::string at user
int append_sink(void *user, const char *bytes, size_t n)
{
  static_cast<std::string *>(user)->append(bytes, n);
  return 0;
}

// the pair stage's tables for a run: the x16 event table (with the N-plane entries) and its packed form
void fill_pair_tables(const Tables &T, bool wplane, PairTables *out)
{
  memcpy(out->agg, T.ev, sizeof out->agg);
  pack_tables(T, wplane, &out->packed);
  event_tables(T, wplane, &out->events);
}

// Whether a run's records hold whole pairs (TcClasses weights): the modes without resolution, on the tensor cores
bool weighted_mode(int mode) { return mode == TN93G_AVERAGE || mode == TN93G_GAPMM || mode == TN93G_SKIP; }

TcClasses tc_classes(int mode, bool weighted)
{
  TcClasses C;
  class_weights(mode, weighted, C.w);
  return C;
}

// the summary units' bounds (ExactSink::amb words) as doubles: {largest low, largest high, spread, count}
void amb_bounds(const unsigned long long *w, double out[4])
{
  memcpy(&out[0], &w[0], 8);
  memcpy(&out[1], &w[1], 8);
  memcpy(&out[2], &w[2], 8);
  out[3] = (double)w[3];
}

}  // namespace

namespace tn93 {
bool summary_certified(const tn93g_summary *s, const double bounds[3][4], long chain, int fst);
}

extern "C" {

const char *tn93g_strerror(int code)
{
  switch (code) {
    case TN93G_OK: return "ok";
    case TN93G_EINVAL: return "invalid argument";
    case TN93G_ECUDA: return "CUDA runtime error";
    case TN93G_ENOMEM: return "out of device or pinned memory";
    case TN93G_ESINK: return "output callback aborted the run";
    case TN93G_ENODEV: return "no usable CUDA device";
    case TN93G_ETIMEOUT: return "device wait timed out";
    case TN93G_ETOOBIG: return "alignment too long (L >= 2^25)";
    case TN93G_ESCRATCH: return "alignment exceeds the allocation-free entry point's limits (N <= 512, L <= 4096)";
    case TN93G_EFASTA: return "the FASTA reader refused the input";
    case TN93G_EUNDECIDED: return "a distance could not be decided exactly";
    default: return "unknown error";
  }
}

const char *tn93g_last_cuda_error(tn93g_ctx *ctx) { return ctx ? ctx->err.c_str() : ""; }

int tn93g_set_count_path(tn93g_ctx *ctx, int path)
{
  if (!ctx || path < 0 || path > 1) return TN93G_EINVAL;
  ctx->count_path = path;
  return TN93G_OK;
}

int tn93g_set_log_band(tn93g_ctx *ctx, double band_ulps, double spread_ulps)
{
  if (!ctx || !(band_ulps >= kLogBand && band_ulps <= 0.5) || !(spread_ulps >= 1.0 && spread_ulps <= 0x1p40))
    return TN93G_EINVAL;
  ctx->log_band = band_ulps;
  ctx->log_spread = floor(spread_ulps);
  return TN93G_OK;
}

int tn93g_set_exact_sums(tn93g_ctx *ctx, int on)
{
  if (!ctx) return TN93G_EINVAL;
  ctx->exact_sums = on != 0;
  return TN93G_OK;
}

int tn93g_set_wait_limit(tn93g_ctx *ctx, double seconds)
{
  if (!ctx || !(seconds > 0. && seconds <= 60.)) return TN93G_EINVAL;
  ctx->wait_ns = (uint64_t)(seconds * 1e9);
  return TN93G_OK;
}

int tn93g_inject_fault(tn93g_ctx *ctx, int fault)
{
  if (!ctx || fault < TN93G_FAULT_NONE || fault > TN93G_FAULT_SKIP_FILL) return TN93G_EINVAL;
  ctx->fault = fault;
  return TN93G_OK;
}

// A band's links, skips and maxima over its n (row, segment) slots into tot[5] (zeroed before): links, skips, and the three
// maxima as bit patterns (not negative). The host took them from a copy of every slot: 2.2 MB over the link for 6,700 rows
// of 7 segments (51 us of gather_kernel, and the host's loop over them), 0.1 MB so: 0.14 ms less a run of 22.4 M pairs.
__global__ void __launch_bounds__(256) band_totals_kernel(const long long *links, const long long *skip, const double *mx,
                                                          long n, unsigned long long *tot)
{
  long long l = 0, k = 0;
  double m[3] = {0., 0., 0.};
  for (long t = blockIdx.x * 256l + threadIdx.x; t < n; t += gridDim.x * 256l) {
    l += links[t];
    k += skip[t];
    for (int q = 0; q < 3; q++) m[q] = fmax(m[q], mx[t * 3 + q]);
  }
  for (int o = 16; o; o >>= 1) {
    l += __shfl_xor_sync(0xffffffffu, l, o);
    k += __shfl_xor_sync(0xffffffffu, k, o);
    for (int q = 0; q < 3; q++) m[q] = fmax(m[q], __shfl_xor_sync(0xffffffffu, m[q], o));
  }
  if ((threadIdx.x & 31) == 0) {
    if (l) atomicAdd(&tot[0], (unsigned long long)l);
    if (k) atomicAdd(&tot[1], (unsigned long long)k);
    for (int q = 0; q < 3; q++)
      if (m[q] > 0.) atomicMax(&tot[2 + q], (unsigned long long)__double_as_longlong(m[q]));
  }
}

// Copies up to nine ranges of 8-byte words into pinned host memory that the device maps (a band's statistics), so
// that they reach the host without a copy-engine transfer, which would queue behind the band texts in flight.
struct Gather {
  const unsigned long long *src[9];
  unsigned long long *dst[9];
  long n[9];
  int stride[9];  // words from one source word to the next
  int k;
};

__global__ void __launch_bounds__(256) gather_kernel(Gather g)
{
  const long stride = (long)gridDim.x * blockDim.x;
  for (int r = 0; r < g.k; r++)
    for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < g.n[r]; t += stride) g.dst[r][t] = g.src[r][t * g.stride[r]];
}

//------------------------------------------------------------------------------------------------ self-test
// one thread per input: the formula up to its logarithms (in: nf[4], diag, ag, ct; out: nlog, k2p, K1..K3, arg[3]),
// and the quotient xb[0] / xb[1] by div_by against the device's division (bad: differing bits)
__global__ void selftest_division_kernel(const double *in, double *out, const double *xb, long n,
                                         unsigned long long *bad)
{
  const long t = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (t >= n) return;
  const double *p = in + 7 * t;
  const double nf[4] = {p[0], p[1], p[2], p[3]};
  const Prep P = tn93_prep(nf, p[4], p[5], p[6]);
  double *o = out + 8 * t;
  o[0] = P.nlog;
  o[1] = P.k2p;
  o[2] = P.K1;
  o[3] = P.K2;
  o[4] = P.K3;
  o[5] = P.arg[0];
  o[6] = P.arg[1];
  o[7] = P.arg[2];
  const double x = xb[2 * t], b = xb[2 * t + 1];
  const double q = div_by(x, b, __ddiv_rn(1.0, b)), r = __ddiv_rn(x, b);
  if (__double_as_longlong(q) != __double_as_longlong(r)) atomicAdd(bad, 1ull);
}

int tn93g_selftest_division(tn93g_ctx *ctx, long n, unsigned long long seed, long mismatches[2])
{
  if (!ctx || n <= 0 || !mismatches) return TN93G_EINVAL;
  cudaSetDevice(ctx->device);
  uint64_t st = seed * 2654435761ull + 0x9E3779B97F4A7C15ull;
  auto rnd = [&]() {
    st ^= st << 13;
    st ^= st >> 7;
    st ^= st << 17;
    return st;
  };
  std::vector<double> in(7 * (size_t)n), out(8 * (size_t)n), xb(2 * (size_t)n);
  for (long t = 0; t < n; t++) {
    // counts as the pair kernel forms them: T clean-equivalent sites (sixteenths), base totals over both sequences
    // summing to 2T, matches, and A<->G / C<->T transitions among the mismatches; some inputs have a base absent
    // (K2P) or more mismatches than the formula takes (no logarithms)
    const long L = 50 + (long)(rnd() % 30000);
    const long T16 = 16 * (L / 2) + (long)(rnd() % (16 * (L / 2)));
    long rest = 2 * T16, nf16[4];
    for (int k = 0; k < 3; k++) {
      nf16[k] = (rnd() % 8 == 0) ? 0 : (long)(rnd() % (uint64_t)(rest / 2 + 1));
      rest -= nf16[k];
    }
    nf16[3] = rest;
    const long mis16 = (long)(rnd() % (uint64_t)(T16 / (rnd() % 4 == 0 ? 1 : 8) + 1));
    const long ag16 = (long)(rnd() % (uint64_t)(mis16 + 1)), ct16 = (long)(rnd() % (uint64_t)(mis16 - ag16 + 1));
    double *p = &in[7 * (size_t)t];
    for (int k = 0; k < 4; k++) p[k] = (double)nf16[k] / 16.0;
    p[4] = (double)(T16 - mis16) / 16.0;
    p[5] = (double)ag16 / 16.0;
    p[6] = (double)ct16 / 16.0;
    // quotients over 80 binades of divisor, either sign of dividend
    const double m = 1.0 + (double)(rnd() >> 12) * 0x1p-52, mb = 1.0 + (double)(rnd() >> 12) * 0x1p-52;
    const int ex = (int)(rnd() % 81) - 40, eb = (int)(rnd() % 81) - 40;
    xb[2 * (size_t)t] = ldexp(rnd() & 1 ? -m : m, ex);
    xb[2 * (size_t)t + 1] = ldexp(mb, eb);
  }
  DevBuf din, dout, dxb, dbad;
  const cudaStream_t st2 = ctx->stream;
  int rc = TN93G_OK;
  do {
    if ((rc = ensure(ctx, din, in.size() * 8)) != TN93G_OK || (rc = ensure(ctx, dout, out.size() * 8)) != TN93G_OK ||
        (rc = ensure(ctx, dxb, xb.size() * 8)) != TN93G_OK || (rc = ensure(ctx, dbad, 8)) != TN93G_OK)
      break;
    unsigned long long bad = 0;
    if (cudaMemcpyAsync(din.p, in.data(), in.size() * 8, cudaMemcpyHostToDevice, st2) != cudaSuccess ||
        cudaMemcpyAsync(dxb.p, xb.data(), xb.size() * 8, cudaMemcpyHostToDevice, st2) != cudaSuccess ||
        cudaMemsetAsync(dbad.p, 0, 8, st2) != cudaSuccess) {
      rc = TN93G_ECUDA;
      break;
    }
    selftest_division_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st2>>>(
        (const double *)din.p, (double *)dout.p, (const double *)dxb.p, n, (unsigned long long *)dbad.p);
    if (cudaGetLastError() != cudaSuccess ||
        cudaMemcpyAsync(out.data(), dout.p, out.size() * 8, cudaMemcpyDeviceToHost, st2) != cudaSuccess ||
        cudaMemcpyAsync(&bad, dbad.p, 8, cudaMemcpyDeviceToHost, st2) != cudaSuccess ||
        cudaStreamSynchronize(st2) != cudaSuccess) {
      rc = TN93G_ECUDA;
      break;
    }
    long diff = 0;
    for (long t = 0; t < n; t++) {
      const double *p = &in[7 * (size_t)t];
      const double nf[4] = {p[0], p[1], p[2], p[3]};
      const Prep P = tn93_prep(nf, p[4], p[5], p[6]);
      const double want[8] = {(double)P.nlog, (double)P.k2p, P.K1, P.K2, P.K3, P.arg[0], P.arg[1], P.arg[2]};
      if (memcmp(want, &out[8 * (size_t)t], sizeof want) != 0) diff++;
    }
    mismatches[0] = diff;
    mismatches[1] = (long)bad;
  } while (0);
  for (DevBuf *b : {&din, &dout, &dxb, &dbad})
    if (b->p) {
      cudaFree(b->p);
      ctx->used -= b->n;
    }
  return rc;
}

int tn93g_create(tn93g_ctx **out, int device, size_t hbm_budget)
{
  if (!out) return TN93G_EINVAL;
  *out = nullptr;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev <= device || device < 0) return TN93G_ENODEV;
  tn93g_ctx *ctx = new tn93g_ctx();
  ctx->device = device;
  ctx->budget = hbm_budget;
  int rc = TN93G_OK;
  do {
    if (cudaSetDevice(device) != cudaSuccess) {
      rc = TN93G_ENODEV;
      break;
    }
    if (cudaStreamCreateWithFlags(&ctx->stream, cudaStreamNonBlocking) != cudaSuccess) {
      rc = TN93G_ECUDA;
      break;
    }
    for (auto &e : ctx->evs)
      if (cudaEventCreate(&e) != cudaSuccess) rc = TN93G_ECUDA;
    for (int q = 0; q < 2; q++) {
      if (cudaEventCreate(&ctx->evw0[q]) != cudaSuccess || cudaEventCreate(&ctx->evw1[q]) != cudaSuccess ||
          cudaEventCreate(&ctx->evc0[q]) != cudaSuccess || cudaEventCreate(&ctx->evc1[q]) != cudaSuccess ||
          cudaEventCreateWithFlags(&ctx->evrow[q], cudaEventDisableTiming) != cudaSuccess)
        rc = TN93G_ECUDA;
      for (auto &e : ctx->evk[q])
        if (cudaEventCreate(&e) != cudaSuccess) rc = TN93G_ECUDA;
      for (auto &e : ctx->evcnt[q])
        if (cudaEventCreate(&e) != cudaSuccess) rc = TN93G_ECUDA;
    }
    for (auto &e : ctx->upload_ev)
      if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) rc = TN93G_ECUDA;
    if (cudaStreamCreateWithFlags(&ctx->copy_stream, cudaStreamNonBlocking) != cudaSuccess) rc = TN93G_ECUDA;
    if (cudaStreamCreateWithFlags(&ctx->write_stream, cudaStreamNonBlocking) != cudaSuccess) rc = TN93G_ECUDA;
    if (const char *e = getenv("TN93G_COUNT")) ctx->count_path = strcmp(e, "popc") == 0 ? 0 : 1;
    {
      const char *b = getenv("TN93G_LOG_BAND"), *p = getenv("TN93G_LOG_SPREAD");
      if (b || p) tn93g_set_log_band(ctx, b ? atof(b) : kLogBand, p ? atof(p) : kLogSpread);
    }
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) == cudaSuccess && sms > 0)
      ctx->sms = sms;
    LogTable h;
    build_log_table(&h);
    if (cudaMalloc(&ctx->d_logt, sizeof(LogTable)) != cudaSuccess ||
        cudaMemcpy(ctx->d_logt, &h, sizeof h, cudaMemcpyHostToDevice) != cudaSuccess)
      rc = TN93G_ECUDA;
    ctx->h_tab = new Tables();
    ctx->h_ptab = new PairTables();
  } while (0);
  if (rc != TN93G_OK) {
    tn93g_destroy(ctx);
    return rc;
  }
  *out = ctx;
  return TN93G_OK;
}

void tn93g_destroy(tn93g_ctx *ctx)
{
  if (!ctx) return;
  cudaSetDevice(ctx->device);
  DevBuf *bufs[] = {&ctx->seen, &ctx->nN, &ctx->varcol, &ctx->planes, &ctx->cc, &ctx->ccT, &ctx->evcount,
                    &ctx->evoff, &ctx->ev, &ctx->ev2, &ctx->three, &ctx->agg, &ctx->site, &ctx->dist, &ctx->dcode, &ctx->wcount, &ctx->wloff, &ctx->wl, &ctx->fraw, &ctx->fspan, &ctx->flen, &ctx->fcode, &ctx->rq, &ctx->rqn, &ctx->counters,
                    &ctx->rbytes, &ctx->rsum, &ctx->rw, &ctx->rmax, &ctx->rlinks, &ctx->rskip, &ctx->hist,
                    &ctx->roff, &ctx->out, &ctx->hy};
  for (DevBuf *b : bufs)
    if (b->p) cudaFree(b->p);
  for (DevBuf &b : ctx->bb)
    if (b.p) cudaFree(b.p);
  for (DevBuf *b : {&ctx->ohimg, &ctx->tcagg, &ctx->und[0], &ctx->und[1], &ctx->undn,
                    &ctx->undwork, &ctx->rdesc})
    if (b->p) cudaFree(b->p);
  if (ctx->d_logt) cudaFree(ctx->d_logt);
  if (ctx->pinned) cudaFreeHost(ctx->pinned);
  for (int q = 0; q < 2; q++) {
    if (ctx->out2[q].p) cudaFree(ctx->out2[q].p);
    if (ctx->pin2[q]) cudaFreeHost(ctx->pin2[q]);
    for (cudaEvent_t e : {ctx->evw0[q], ctx->evw1[q], ctx->evc0[q], ctx->evc1[q], ctx->evrow[q]})
      if (e) cudaEventDestroy(e);
    for (cudaEvent_t e : ctx->evk[q])
      if (e) cudaEventDestroy(e);
    for (cudaEvent_t e : ctx->evcnt[q])
      if (e) cudaEventDestroy(e);
  }
  if (ctx->total.p) cudaFree(ctx->total.p);
  if (ctx->hrun) cudaFreeHost(ctx->hrun);
  if (ctx->upload_pin) cudaFreeHost(ctx->upload_pin);
  for (cudaEvent_t e : ctx->upload_ev)
    if (e) cudaEventDestroy(e);
  for (auto &b : ctx->set_pool) cudaFree(b.first);
  if (ctx->pstats) cudaFreeHost(ctx->pstats);
  if (ctx->copy_stream) cudaStreamDestroy(ctx->copy_stream);
  if (ctx->write_stream) cudaStreamDestroy(ctx->write_stream);
  for (auto &e : ctx->evs)
    if (e) cudaEventDestroy(e);
  if (ctx->stream) cudaStreamDestroy(ctx->stream);
  delete ctx->h_tab;
  delete ctx->h_ptab;
  delete ctx;
}

// A new set from codes (host memory, or device memory when codes_kind says so), copy numbers and names (host).
static int upload_set(tn93g_ctx *ctx, tn93g_set **out, const uint8_t *codes, cudaMemcpyKind codes_kind, long N, long L,
                      const long *copy_counts, const char *names, const size_t *name_off, const long *name_len);

int tn93g_upload(tn93g_ctx *ctx, tn93g_set **out, const uint8_t *codes, long N, long L, const long *copy_counts,
                 const char *names, const size_t *name_off, const long *name_len)
{
  return upload_set(ctx, out, codes, cudaMemcpyHostToDevice, N, L, copy_counts, names, name_off, name_len);
}

static int upload_set(tn93g_ctx *ctx, tn93g_set **out, const uint8_t *codes, cudaMemcpyKind codes_kind, long N, long L,
                      const long *copy_counts, const char *names, const size_t *name_off, const long *name_len)
{
  if (!ctx || !out || !codes || N <= 0 || L <= 0 || !copy_counts || !names || !name_off || !name_len)
    return TN93G_EINVAL;
  if (L >= (1l << 25)) return TN93G_ETOOBIG;
  cudaSetDevice(ctx->device);
  tn93g_set *s = new tn93g_set();
  s->N = N;
  s->L = L;
  s->counts.assign(copy_counts, copy_counts + N);
  s->name_len.assign(name_len, name_len + N);
  size_t nbytes = 0;
  for (long i = 0; i < N; i++) nbytes = std::max(nbytes, name_off[i] + (size_t)name_len[i]);
  std::vector<uint64_t> off(name_off, name_off + N);
  std::vector<int32_t> nl(N);
  for (long i = 0; i < N; i++) nl[i] = (int32_t)name_len[i];
  auto fail = [&](cudaError_t e) {
    cudaGetLastError();
    ctx->err = cudaGetErrorString(e);
    tn93g_free_set(ctx, s);
    return e == cudaErrorMemoryAllocation ? TN93G_ENOMEM : TN93G_ECUDA;
  };
  cudaError_t e;
  // smallest pooled buffer that fits, else a new allocation
  auto take = [&](void **p, size_t bytes, int k) -> cudaError_t {
    bytes = std::max<size_t>(bytes, 256);
    long best = -1;
    for (size_t q = 0; q < ctx->set_pool.size(); q++)
      if (ctx->set_pool[q].second >= bytes && (best < 0 || ctx->set_pool[q].second < ctx->set_pool[best].second))
        best = (long)q;
    if (best >= 0) {
      *p = ctx->set_pool[best].first;
      s->cap[k] = ctx->set_pool[best].second;
      ctx->set_pool.erase(ctx->set_pool.begin() + best);
      return cudaSuccess;
    }
    s->cap[k] = bytes;
    cudaError_t m = cudaMalloc(p, bytes);
    while (m == cudaErrorMemoryAllocation && reclaim(ctx)) {
      cudaGetLastError();
      m = cudaMalloc(p, bytes);
    }
    return m;
  };
  if ((e = take((void **)&s->d_codes, (size_t)N * L, 0)) != cudaSuccess) return fail(e);
  if ((e = take((void **)&s->d_counts, N * sizeof(long), 1)) != cudaSuccess) return fail(e);
  if ((e = take((void **)&s->d_names, nbytes + 8, 2)) != cudaSuccess) return fail(e);
  if ((e = take((void **)&s->d_name_off, N * sizeof(uint64_t), 3)) != cudaSuccess) return fail(e);
  if ((e = take((void **)&s->d_name_len, N * sizeof(int32_t), 4)) != cudaSuccess) return fail(e);
  if (codes_kind == cudaMemcpyHostToDevice) {
    const int rc = upload_host(ctx, {{s->d_codes, codes, (size_t)N * L}});
    if (rc != TN93G_OK) {
      tn93g_free_set(ctx, s);
      return rc;
    }
  } else if ((e = cudaMemcpyAsync(s->d_codes, codes, (size_t)N * L, codes_kind, ctx->stream)) != cudaSuccess) {
    return fail(e);
  }
  if ((e = cudaMemcpyAsync(s->d_counts, copy_counts, N * sizeof(long), cudaMemcpyHostToDevice, ctx->stream)) !=
      cudaSuccess)
    return fail(e);
  if (nbytes && (e = cudaMemcpyAsync(s->d_names, names, nbytes, cudaMemcpyHostToDevice, ctx->stream)) != cudaSuccess)
    return fail(e);
  if ((e = cudaMemcpyAsync(s->d_name_off, off.data(), N * sizeof(uint64_t), cudaMemcpyHostToDevice, ctx->stream)) !=
      cudaSuccess)
    return fail(e);
  if ((e = cudaMemcpyAsync(s->d_name_len, nl.data(), N * sizeof(int32_t), cudaMemcpyHostToDevice, ctx->stream)) !=
      cudaSuccess)
    return fail(e);
  if ((e = cudaStreamSynchronize(ctx->stream)) != cudaSuccess) return fail(e);
  *out = s;
  return TN93G_OK;
}

//------------------------------------------------------------------------------------------------ FASTA on device
// The byte map of tn93's reader: the index of a byte in "ACGTURYSWKMBDHVN?-" (either case), -1 for any other byte
struct ByteMap {
  signed char v[256];
};

static ByteMap make_byte_map()
{
  ByteMap m;
  static const char kValid[] = "ACGTURYSWKMBDHVN?-";
  for (int c = 0; c < 256; c++) {
    m.v[c] = -1;
    const int u = (c >= 'a' && c <= 'z') ? c - 32 : c;
    if (!u) continue;
    const char *f = strchr(kValid, u);
    if (f) m.v[c] = (signed char)(f - kValid);
  }
  return m;
}

// one warp per record: how many of the bytes in its sequence range [span.x, span.y) of raw are letters of the map
__global__ void __launch_bounds__(256) fasta_count_kernel(const unsigned char *raw, const ulonglong2 *spans, long m,
                                                          ByteMap map, long *len)
{
  __shared__ signed char sm[256];
  for (int t = threadIdx.x; t < 256; t += blockDim.x) sm[t] = map.v[t];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const long k = blockIdx.x * (long)kWarps + (threadIdx.x >> 5);
  if (k >= m) return;
  const unsigned long long b = spans[k].x, e = spans[k].y;
  long n = 0;
  for (unsigned long long p = b + lane; p < e; p += 32) n += sm[raw[p]] >= 0;
  for (int o = 16; o; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
  if (lane == 0) len[k] = n;
}

// one warp per record: its sequence letters mapped to codes and compressed, in file order, to codes[k * L ...] (every
// record has L letters, checked on the host before the launch)
__global__ void __launch_bounds__(256) fasta_compress_kernel(const unsigned char *raw, const ulonglong2 *spans, long m,
                                                             ByteMap map, long L, uint8_t *codes)
{
  __shared__ signed char sm[256];
  for (int t = threadIdx.x; t < 256; t += blockDim.x) sm[t] = map.v[t];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const long k = blockIdx.x * (long)kWarps + (threadIdx.x >> 5);
  if (k >= m) return;
  const unsigned long long b = spans[k].x, e = spans[k].y;
  uint8_t *row = codes + (size_t)k * L;
  long base = 0;
  for (unsigned long long p0 = b; p0 < e; p0 += 32) {
    const unsigned long long p = p0 + lane;
    const int v = p < e ? sm[raw[p]] : -1;
    const unsigned mask = __ballot_sync(0xffffffffu, v >= 0);
    if (v >= 0) row[base + __popc(mask & ((1u << lane) - 1u))] = (uint8_t)v;
    base += __popc(mask);
  }
}

// The records of a FASTA file as tn93's reader finds them (swifttn93.cpp:259-406): '>' or '#' opens a record whose
// name runs to the end of the line, and its sequence is every byte up to the next '>' or '#'. memchr (vectorised in
// the C library) finds those bytes, so the host does not touch the sequence letters.
struct FastaRecords {
  std::vector<char> names;
  std::vector<size_t> name_off;
  std::vector<long> name_len, counts;
  std::vector<ulonglong2> spans;
  int eof_state = 2;     // the reader's state at the end of the file (2: inside a sequence, the normal end)
  std::string name_err;  // the record after the last span has an empty name (reported after the spans' lengths)
};

static void fasta_records(const char *bytes, size_t n, char counts_sep, FastaRecords &R)
{
  // the next '>' and '#' at or after the last search start (n: none); still the next ones for any later start that
  // does not pass them
  size_t ngt = 0, nhs = 0;
  bool have = false;
  auto next_open = [&](size_t i) -> size_t {
    if (!have || ngt < i) {
      const void *g = i < n ? memchr(bytes + i, '>', n - i) : nullptr;
      ngt = g ? (size_t)((const char *)g - bytes) : n;
    }
    if (!have || nhs < i) {
      const void *h = i < n ? memchr(bytes + i, '#', n - i) : nullptr;
      nhs = h ? (size_t)((const char *)h - bytes) : n;
    }
    have = true;
    return std::min(ngt, nhs);
  };
  size_t o = next_open(0);
  if (o == n) {
    R.eof_state = 0;
    return;
  }
  size_t i = o + 1;
  for (;;) {
    size_t q = i;
    while (q < n && bytes[q] != '\n' && bytes[q] != '\r') q++;
    if (q == n) {
      R.eof_state = 1;
      return;
    }
    const long len = (long)(q - i);
    if (len <= 0) {
      R.name_err = "Sequence names must be non-empty.\n";
      return;
    }
    const size_t begin = R.names.size();
    R.names.insert(R.names.end(), bytes + i, bytes + q);
    R.names.push_back('\0');
    unsigned long count = 1;
    if (len >= 3) {
      const char *nm = R.names.data() + begin;
      long k = len - 2;
      while (k >= 1 && nm[k] != counts_sep) k--;
      if (k >= 1) count = (unsigned long)(long)(int)strtol(nm + k + 1, nullptr, 10);
      if (count < 1) count = 1;
    }
    R.counts.push_back((long)count);
    R.name_off.push_back(begin);
    R.name_len.push_back(len);
    i = q + 1;
    o = next_open(i);
    R.spans.push_back(make_ulonglong2(i, o));
    if (o == n) {
      R.eof_state = 2;
      return;
    }
    i = o + 1;
  }
}

// The reader's checks in its order, given each record's letter count: each length when its sequence closes, then
// what stopped the scan. Returns the message (empty when the file is accepted) and the length in *first_len.
static std::string fasta_check(const FastaRecords &R, const std::vector<long> &lens, long expect_len, long *first_len)
{
  std::string err;
  const long m = (long)R.spans.size();
  const bool have_len = expect_len > 0;
  long L = have_len ? expect_len : 0;
  for (long k = 0; k < m && err.empty(); k++) {
    if (k == 0 && !have_len) {
      L = lens[0];
      if (L <= 0) err = "First sequence length must be positive.\n";
    } else if (lens[k] != L) {
      err = "All sequences must have the same length (" + std::to_string(L) + "), but sequence '" +
            std::string(R.names.data() + R.name_off[k]) + "' had length " + std::to_string(lens[k]);
    }
  }
  if (err.empty() && !R.name_err.empty()) err = R.name_err;
  if (err.empty() && R.eof_state != 2) err = "Unexpected end of file: state " + std::to_string(R.eof_state) + "\n";
  *first_len = L;
  return err;
}

static void copy_msg(const std::string &err, char *msg, size_t msg_cap)
{
  if (!msg || !msg_cap) return;
  const size_t k = err.size() < msg_cap ? err.size() : msg_cap - 1;
  memcpy(msg, err.data(), k);
  msg[k] = 0;
}

// The device ingest's host half with the letters counted on the host: its record scan and checks, for tests on
// machines without a GPU. Returns TN93G_OK (with the size in n_out, L_out) or TN93G_EFASTA (message in msg).
int tn93g_fasta_check(const char *bytes, size_t nbytes, long expect_len, char counts_sep, long *n_out, long *L_out,
                      char *msg, size_t msg_cap)
{
  if (!bytes && nbytes) return TN93G_EINVAL;
  FastaRecords R;
  fasta_records(bytes, nbytes, counts_sep, R);
  const ByteMap map = make_byte_map();
  std::vector<long> lens(R.spans.size());
  for (size_t k = 0; k < R.spans.size(); k++) {
    long c = 0;
    for (unsigned long long p = R.spans[k].x; p < R.spans[k].y; p++) c += map.v[(unsigned char)bytes[p]] >= 0;
    lens[k] = c;
  }
  long L = 0;
  const std::string err = fasta_check(R, lens, expect_len, &L);
  copy_msg(err, msg, msg_cap);
  if (!err.empty()) return TN93G_EFASTA;
  if (n_out) *n_out = (long)R.spans.size();
  if (L_out) *L_out = L;
  return TN93G_OK;
}

int tn93g_upload_fasta(tn93g_ctx *ctx, tn93g_set **out, const char *bytes, size_t nbytes, long expect_len,
                       char counts_sep, long *n_out, long *L_out, char *msg, size_t msg_cap)
{
  if (!ctx || !out || (!bytes && nbytes)) return TN93G_EINVAL;
  *out = nullptr;
  cudaSetDevice(ctx->device);
  const cudaStream_t st = ctx->stream;
  FastaRecords R;
  fasta_records(bytes, nbytes, counts_sep, R);
  const long m = (long)R.spans.size();
  std::vector<long> lens(m);
  const ByteMap map = make_byte_map();
  if (m) {
    TRY(ensure(ctx, ctx->fraw, nbytes));
    TRY(ensure(ctx, ctx->fspan, m * sizeof(ulonglong2)));
    TRY(ensure(ctx, ctx->flen, m * sizeof(long)));
    CU(cudaMemcpyAsync(ctx->fraw.p, bytes, nbytes, cudaMemcpyHostToDevice, st));
    CU(cudaMemcpyAsync(ctx->fspan.p, R.spans.data(), m * sizeof(ulonglong2), cudaMemcpyHostToDevice, st));
    fasta_count_kernel<<<(unsigned)((m + kWarps - 1) / kWarps), 256, 0, st>>>(
        (const unsigned char *)ctx->fraw.p, (const ulonglong2 *)ctx->fspan.p, m, map, (long *)ctx->flen.p);
    CU(cudaGetLastError());
    CU(cudaMemcpyAsync(lens.data(), ctx->flen.p, m * sizeof(long), cudaMemcpyDeviceToHost, st));
    CU(cudaStreamSynchronize(st));
  }
  long first_len = 0;
  const std::string err = fasta_check(R, lens, expect_len, &first_len);
  copy_msg(err, msg, msg_cap);
  if (!err.empty()) return TN93G_EFASTA;
  if (first_len >= (1l << 25)) return TN93G_ETOOBIG;
  TRY(ensure(ctx, ctx->fcode, (size_t)m * first_len));
  fasta_compress_kernel<<<(unsigned)((m + kWarps - 1) / kWarps), 256, 0, st>>>(
      (const unsigned char *)ctx->fraw.p, (const ulonglong2 *)ctx->fspan.p, m, map, first_len, (uint8_t *)ctx->fcode.p);
  CU(cudaGetLastError());
  const int rc = upload_set(ctx, out, (const uint8_t *)ctx->fcode.p, cudaMemcpyDeviceToDevice, m, first_len,
                            R.counts.data(), R.names.data(), R.name_off.data(), R.name_len.data());
  if (rc != TN93G_OK) return rc;
  if (n_out) *n_out = m;
  if (L_out) *L_out = first_len;
  return TN93G_OK;
}

void tn93g_free_set(tn93g_ctx *ctx, tn93g_set *s)
{
  if (!s) return;
  void *bufs[5] = {s->d_codes, s->d_counts, s->d_names, s->d_name_off, s->d_name_len};
  if (ctx) {
    // the buffers go back to the context's pool (the context's stream has no work left on them: every run and
    // upload synchronises it before returning)
    for (int k = 0; k < 5; k++)
      if (bufs[k]) ctx->set_pool.push_back({bufs[k], s->cap[k]});
  } else {
    for (int k = 0; k < 5; k++)
      if (bufs[k]) cudaFree(bufs[k]);
  }
  delete s;
}

int tn93g_last_timings(tn93g_ctx *ctx, double *ms, int n)
{
  if (!ctx || !ms) return 0;
  const int k = std::min(n, 8);
  for (int q = 0; q < k; q++) ms[q] = ctx->timings[q];
  return k;
}

void *tn93g_stream(tn93g_ctx *ctx) { return ctx ? (void *)ctx->stream : nullptr; }

long tn93g_last_launches(tn93g_ctx *ctx) { return ctx ? ctx->launches : 0; }

// flags of run_impl: a second, exact pass for the JSON numbers (every ambiguous logarithm taken from the C library)
constexpr int kRunResolveAll = 1;
static int run_impl(tn93g_ctx *ctx, const tn93g_set *set, long n1, const tn93g_opts *opts, tn93g_sink sink, void *user,
                    tn93g_summary *sum, bool to_device, long row_begin = 0, long row_end = -1,
                    double *row_sums = nullptr, int flags = 0);

int tn93g_run(tn93g_ctx *ctx, const tn93g_set *set, long n1, const tn93g_opts *opts, tn93g_sink sink, void *user,
              tn93g_summary *sum)
{
  return run_impl(ctx, set, n1, opts, sink, user, sum, false);
}

int tn93g_run_rows(tn93g_ctx *ctx, const tn93g_set *set, long n1, const tn93g_opts *opts, long row_begin,
                   long row_end, tn93g_sink sink, void *user, double *row_sums, tn93g_summary *sum)
{
  if (!opts || opts->format == TN93G_HYPHY || row_begin < 0 || row_end < row_begin) return TN93G_EINVAL;
  return run_impl(ctx, set, n1, opts, sink, user, sum, false, row_begin, row_end, row_sums);
}

int tn93g_run_to_device(tn93g_ctx *ctx, const tn93g_set *set, long n1, const tn93g_opts *opts, void **dev_out,
                        size_t *nbytes, tn93g_summary *sum)
{
  if (!dev_out || !nbytes) return TN93G_EINVAL;
  const int rc = run_impl(ctx, set, n1, opts, nullptr, nullptr, sum, true);
  *dev_out = rc == TN93G_OK ? ctx->out.p : nullptr;
  *nbytes = rc == TN93G_OK ? ctx->dev_out_n : 0;
  return rc;
}

constexpr long kBandWords = 3 * kHistBins + 5;  // a band's histograms and totals (band_totals_kernel)
constexpr size_t kRunScalars = 17;       // words of a run's scalars (run_impl)
constexpr size_t kRunPinned = 4 << 20;  // pinned bytes kept for a run's small transfers

static int run_impl(tn93g_ctx *ctx, const tn93g_set *set, long n1, const tn93g_opts *opts, tn93g_sink sink, void *user,
                    tn93g_summary *sum, bool to_device, long row_begin, long row_end, double *row_sums, int flags)
{
  if (!ctx || !set || !opts || !sum || n1 <= 0 || n1 > set->N) return TN93G_EINVAL;
  if (opts->mode < 0 || opts->mode > 4 || opts->format < 0 || opts->format > 2) return TN93G_EINVAL;
  cudaSetDevice(ctx->device);
  cudaStream_t st = ctx->stream;
  const long N = set->N, L = set->L;
  memset(sum, 0, sizeof *sum);
  for (double &t : ctx->timings) t = 0;
  ctx->launches = 0;
  ctx->dev_out_n = 0;
  size_t dev_off = 0;  // to_device: bytes of the distance file already in ctx->out
  RunConsts rc;
  memset(&rc, 0, sizeof rc);
  rc.N = N;
  rc.n1 = n1;
  rc.mode = opts->mode;
  rc.gapmm = opts->mode == TN93G_GAPMM;
  rc.fst = n1 < N && opts->do_fst;
  rc.cross = n1 < N && !opts->do_fst;
  rc.fallback_avg = (opts->mode == TN93G_RESOLVE || opts->mode == TN93G_SUBSET) && opts->resolve_fraction < 1.;
  rc.emit = !opts->count_only;
  rc.format = opts->format;
  rc.delim = opts->delimiter;
  rc.report_self = opts->report_self && !rc.cross && n1 == N && rc.emit;
  rc.threshold = opts->threshold;
  rc.min_distance = opts->min_distance;
  rc.resolve_fraction = opts->resolve_fraction;
  rc.min_overlap = opts->min_overlap;
  rc.log_band = ctx->log_band;
  rc.log_spread = ctx->log_spread;
  rc.resolve_all = (flags & kRunResolveAll) != 0 || ctx->exact_sums;
  struct Busy {  // (an exact-sums pass is a run inside a run)
    bool &flag, was;
    ~Busy() { flag = was; }
  } busy = {ctx->bands_busy, ctx->bands_busy};
  ctx->bands_busy = true;
  bool fault_pending = ctx->fault == TN93G_FAULT_SKIP_FILL;  // injected into the first count launch only
  ctx->fault = TN93G_FAULT_NONE;
  const bool hyphy = rc.emit && opts->format == TN93G_HYPHY;
  cudaEvent_t *E = ctx->evs;
  CU(cudaEventRecord(E[0], st));

  //------------------------------------------------------------------ pack
  // The host's side of the small transfers: one pinned block (a copy to or from pageable memory costs about 10 us more), or
  // pageable memory for very long or many sequences. The device's scalars and column masks are each one buffer, cleared
  // and copied in one piece.
  const size_t seen_n = ((size_t)L * sizeof(uint32_t) + 7) / 8 * 8 + sizeof(unsigned long long);  // masks, then the N count
  const size_t host_part[6] = {seen_n, (size_t)L * sizeof(int32_t), N * sizeof(uint32_t), (N + 1) * sizeof(uint32_t),
                               N * sizeof(uint32_t), (N + 1) * sizeof(uint32_t)};
  size_t host_at[7] = {kRunScalars * sizeof(unsigned long long)};
  for (int q = 0; q < 6; q++) host_at[q + 1] = (host_at[q] + host_part[q] + 7) / 8 * 8;
  std::vector<char> host_big;
  char *host = nullptr;
  if (host_at[6] <= kRunPinned) {
    TRY(ensure_pinned_at(ctx, ctx->hrun, ctx->hrun_n, kRunPinned));
    host = (char *)ctx->hrun;
  } else {
    host_big.resize(host_at[6]);
    host = host_big.data();
  }
  unsigned long long *const h_scalars = (unsigned long long *)host;
  const uint32_t *const seen = (const uint32_t *)(host + host_at[0]);
  int32_t *const h_varcol = (int32_t *)(host + host_at[1]);
  uint32_t *const evc = (uint32_t *)(host + host_at[2]), *const evoff = (uint32_t *)(host + host_at[3]);
  uint32_t *const wcnt = (uint32_t *)(host + host_at[4]), *const woff = (uint32_t *)(host + host_at[5]);
  TRY(ensure(ctx, ctx->seen, seen_n));
  CU(cudaMemsetAsync(ctx->seen.p, 0, seen_n, st));
  {
    dim3 g((unsigned)((L + 255) / 256), (unsigned)((N + 63) / 64));
    colscan_kernel<<<g, 256, 0, st>>>(set->d_codes, N, L, (uint32_t *)ctx->seen.p,
                                      (unsigned long long *)((char *)ctx->seen.p + seen_n) - 1);
    CU(cudaGetLastError());
    ctx->launches++;
  }
  CU(cudaMemcpyAsync(host + host_at[0], ctx->seen.p, seen_n, cudaMemcpyDeviceToHost, st));
  CU(cudaStreamSynchronize(st));
  const unsigned long long nN = *((const unsigned long long *)(host + host_at[0] + seen_n) - 1);
  // a column is constant when every sequence has the same clean base there: each pair gets (b, b)
  long Lc = 0;
  bool three = false;
  for (long p = 0; p < L; p++) {
    const uint32_t m = seen[p];
    three |= (m & 0x7800u) != 0;
    if (m && !(m & (m - 1)) && m < 16) {
      const int b = __builtin_ctz(m);
      rc.constT++;
      rc.constNf[b] += 2;
      rc.constCnt[b]++;
    } else
      h_varcol[Lc++] = (int32_t)p;
  }
  const long W = (Lc + 63) / 64;
  const long Npad = (N + 31) / 32 * 32;
  rc.Lc = Lc;
  rc.W = W;
  rc.Npad = Npad;
  // N gets its own bit plane when frequent (more than 16 per sequence); gapmm always (gaps join it)
  rc.wplane = rc.gapmm || nN > 16ull * (unsigned long long)N;
  rc.NP = rc.gapmm ? 5 : 4;
  TRY(ensure(ctx, ctx->varcol, std::max<long>(Lc, 1) * sizeof(int32_t)));
  TRY(ensure(ctx, ctx->planes, (size_t)std::max<long>(W, 1) * rc.NP * Npad * sizeof(uint64_t)));
  TRY(ensure(ctx, ctx->cc, (size_t)N * std::max<long>(Lc, 1) + 8));  // read by the aligned words that hold its codes
  TRY(ensure(ctx, ctx->ccT, (size_t)std::max<long>(Lc, 1) * Npad));
  TRY(ensure(ctx, ctx->evcount, N * sizeof(uint32_t)));
  TRY(ensure(ctx, ctx->evoff, (N + 1) * sizeof(uint32_t)));
  TRY(ensure(ctx, ctx->three, N));
  if (Lc) CU(cudaMemcpyAsync(ctx->varcol.p, h_varcol, Lc * sizeof(int32_t), cudaMemcpyHostToDevice, st));
  CU(cudaMemsetAsync(ctx->planes.p, 0, (size_t)std::max<long>(W, 1) * rc.NP * Npad * sizeof(uint64_t), st));
  CU(cudaMemsetAsync(ctx->evcount.p, 0, N * sizeof(uint32_t), st));
  PackArgs pa;
  pa.codes = set->d_codes;
  pa.N = N;
  pa.L = L;
  pa.Lc = Lc;
  pa.W = W;
  pa.Npad = Npad;
  pa.varcol = (const int32_t *)ctx->varcol.p;
  pa.NP = rc.NP;
  pa.wplane = rc.wplane;
  pa.gapmm = rc.gapmm;
  pa.planes = (uint64_t *)ctx->planes.p;
  pa.cc = (uint8_t *)ctx->cc.p;
  pa.evcount = (uint32_t *)ctx->evcount.p;
  pa.ev_off = (const uint32_t *)ctx->evoff.p;
  // three-fold codes anywhere: the events kernel then marks their sequences
  pa.three = three && opts->mode != TN93G_SKIP ? (uint8_t *)ctx->three.p : nullptr;
  if (W) {
    pack_kernel<<<dim3((unsigned)((N + kWarps - 1) / kWarps), (unsigned)std::min<long>(W, 65535)), 256, 0, st>>>(pa);
    CU(cudaGetLastError());
    ctx->launches++;
    transpose_kernel<<<dim3((unsigned)((Lc + kTransK - 1) / kTransK), (unsigned)(Npad / 32)), dim3(32, 8), 0, st>>>(
        (const uint8_t *)ctx->cc.p, (uint8_t *)ctx->ccT.p, N, Lc, Npad);
    CU(cudaGetLastError());
    ctx->launches++;
  }
  const bool use_tc = ctx->count_path == 1 && Lc > 0;
  const bool lin = use_tc && weighted_mode(opts->mode);  // the records will hold the ambiguity codes
  const bool use_ev = !lin || (three && opts->mode != TN93G_SKIP);  // events are needed: all, or for three-fold codes
  // per sequence, its nonzero N-plane words (the pair kernel's sparse N-plane pass); counted here, listed below
  bool sparse_w = rc.wplane && W > 0 && (!lin || rc.gapmm);
  if (sparse_w) {
    TRY(ensure(ctx, ctx->wcount, N * sizeof(uint32_t)));
    wcount_kernel<<<(unsigned)((N + 31) / 32), 32 * kWlWarps, 0, st>>>((const uint64_t *)ctx->planes.p, N, W, rc.NP, Npad,
                                                                (uint32_t *)ctx->wcount.p);
    CU(cudaGetLastError());
    ctx->launches++;
    CU(cudaMemcpyAsync(wcnt, ctx->wcount.p, N * sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
  }
  if (use_ev) CU(cudaMemcpyAsync(evc, ctx->evcount.p, N * sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
  if (use_ev || sparse_w) CU(cudaStreamSynchronize(st));
  if (sparse_w) {
    unsigned long long t = 0;
    for (long i = 0; i < N; i++) {
      woff[i] = (uint32_t)t;
      t += wcnt[i];
    }
    sparse_w = t < 0xFFFFFFFFull;  // 32-bit offsets; beyond them every word is visited
    if (sparse_w) {
      woff[N] = (uint32_t)t;
      TRY(ensure(ctx, ctx->wloff, (N + 1) * sizeof(uint32_t)));
      TRY(ensure(ctx, ctx->wl, std::max<size_t>(t, 1) * sizeof(uint32_t)));
      CU(cudaMemcpyAsync(ctx->wloff.p, woff, (N + 1) * sizeof(uint32_t), cudaMemcpyHostToDevice, st));
      wlist_kernel<<<(unsigned)((N + 31) / 32), 32 * kWlWarps, 0, st>>>((const uint64_t *)ctx->planes.p, N, W, rc.NP, Npad,
                                                                 (const uint32_t *)ctx->wloff.p, (uint32_t *)ctx->wl.p);
      CU(cudaGetLastError());
      ctx->launches++;
    }
  }
  uint32_t max_ev = 0;  // null events add nothing to the packed sums
  unsigned long long nev = 0;
  for (long i = 0; i < N; i++) {
    evoff[i] = (uint32_t)nev;
    if (!use_ev) continue;
    nev += pad_events(evc[i]);
    max_ev = std::max(max_ev, evc[i]);
  }
  if (nev >= (1ull << 32)) return TN93G_ETOOBIG;  // 32-bit offsets
  evoff[N] = (uint32_t)nev;
  rc.packed = max_ev <= (uint32_t)kPackedMaxEvents;
  TRY(ensure(ctx, ctx->ev, std::max<size_t>(evoff[N], 1) * sizeof(uint32_t)));
  // The events again as event_kernel reads them, where the pair stage takes it (pair_split) and there is room: 8 bytes an
  // event beside the 4 of the list. Without them the fused kernel runs.
  bool use_ev2 = use_tc && !lin && rc.packed && Lc * Npad < (1l << 32) && (!rc.wplane || sparse_w);
  if (use_ev2) {
    const int r = ensure(ctx, ctx->ev2, std::max<size_t>(evoff[N], 1) * sizeof(uint2), true);
    if (r != TN93G_ENOMEM) TRY(r);
    use_ev2 = r == TN93G_OK;
  }
  CU(cudaMemcpyAsync(ctx->evoff.p, evoff, (N + 1) * sizeof(uint32_t), cudaMemcpyHostToDevice, st));
  pa.ev = (uint32_t *)ctx->ev.p;
  pa.ev2 = use_ev2 ? (uint2 *)ctx->ev2.p : nullptr;
  pa.ev2_Npad = (uint32_t)Npad;
  if (W && evoff[N]) {  // no list: nothing reads one
    events_kernel<<<(unsigned)((N + kWarps - 1) / kWarps), 256, 0, st>>>(pa);
    CU(cudaGetLastError());
    ctx->launches++;
  }
  // tables of this mode: they depend on the mode, the subset of codes and the N plane alone, so the last run's stay on the
  // device until a run needs others (with the small transfers above, building and copying them took 0.15 of the 0.49 ms of a 50 x 900 run)
  std::string tab_key(1, (char)(2 * opts->mode + (rc.wplane ? 1 : 0)));
  if (opts->mode == TN93G_SUBSET) tab_key.append((const char *)opts->subset, sizeof opts->subset);
  if (tab_key != ctx->tab_key) {
    ctx->tab_key.clear();
    build_tables(ctx->h_tab, opts->mode, opts->subset);
    fill_pair_tables(*ctx->h_tab, rc.wplane, ctx->h_ptab);
    TRY(ensure(ctx, ctx->agg, sizeof(PairTables)));
    TRY(ensure(ctx, ctx->site, sizeof(ctx->h_tab->site)));
    CU(cudaMemcpyAsync(ctx->agg.p, ctx->h_ptab, sizeof(PairTables), cudaMemcpyHostToDevice, st));
    CU(cudaMemcpyAsync(ctx->site.p, ctx->h_tab->site, sizeof(ctx->h_tab->site), cudaMemcpyHostToDevice, st));
    ctx->tab_key = tab_key;
  }
  // tensor-core count path: the one-hot operand image of every sequence (an extra 32-sequence block at the end,
  // which the last 64-column tile reads)
  const long tc_NB = (N + 31) / 32 + 1, tc_KS = (Lc + kTcStageK - 1) / kTcStageK;
  if (use_tc) {
    TRY(ensure(ctx, ctx->ohimg, (size_t)tc_KS * tc_NB * kTcBlockBytes));
    const long nthr = tc_NB * 32 * tc_KS * (kTcStageK / 16);
    onehot_kernel<<<(unsigned)((nthr + 255) / 256), 256, 0, st>>>((const uint8_t *)ctx->cc.p, N, Lc, tc_NB, tc_KS,
                                                                  (uint8_t *)ctx->ohimg.p, 0, tc_NB * 32,
                                                                  tc_classes(opts->mode, lin));
    CU(cudaGetLastError());
    ctx->launches++;
    CU(tc_attr_once());
  }
  CU(cudaEventRecord(E[1], st));

  //------------------------------------------------------------------ bands
  // rows of the pair triangle (or of the first file under -s): all of them, or the caller's range
  const long all_rows = rc.cross ? n1 : N;
  if (row_end < 0) row_end = all_rows;
  if (row_begin > all_rows || row_end > all_rows) return TN93G_EINVAL;
  const long upper = row_end;
  const long colbase = rc.cross ? n1 : 0;
  const long ncols = N - colbase;
  if (rc.cross)
    sum->pairwise = (unsigned long)(N - n1) * (unsigned long)(row_end - row_begin);
  else  // pairs (i, j > i) of rows [row_begin, row_end)
    sum->pairwise = (unsigned long)((row_end - row_begin) * (2 * N - row_begin - row_end - 1) / 2);
  // Band schedule. When the text goes to the host, a band holds about 3 M pairs (at most 16 M pair slots), so
  // that the copy of one band overlaps the kernels of the next; otherwise up to 64 M slots.
  const bool stream_text = !(to_device || hyphy || !rc.emit);
  static const long forced_band = [] {
    const char *e = getenv("TN93G_BAND_PAIRS");  // tuning knob: pairs per band when streaming text
    return e ? std::max(atol(e), 0l) : 0l;
  }();
  const long band_pairs = forced_band ? forced_band : (3l << 20);
  // When the text streams to the host, the bands ramp up from 1/16 of the target, 1.4 times larger each (a band's
  // kernels take about 0.7 of its copy's time, so each band's kernels end before the previous band's copy does and
  // the copies run back to back), and taper at the end (half of what is left, down to 1/8), so that the first copy
  // starts early and the last one, which nothing overlaps, is short. When the first band shows that little is
  // reported, there is nothing to overlap and the rest runs as large bands (below).
  using Bands = std::vector<std::pair<long, long>>;
  auto row_pairs = [&](long r) { return rc.cross ? ncols : N - r - 1; };
  auto count_pairs = [&](long b, long e) {
    long p = 0;
    for (long r = b; r < e; r++) p += row_pairs(r);
    return p;
  };
  // the rows from `from` on in bands of target pairs and at most cap pair slots; step: place in the ramp of the first one
  auto plan_bands = [&](long from, long target, long cap, bool ramps, int step) {
    Bands out;
    long left = count_pairs(from, upper);
    for (long r0 = from; r0 < upper; step++) {
      long tgt = target;
      if (ramps) {
        const double ramp = std::pow(1.4, (double)step) / 16.0;
        if (ramp < 1.0) tgt = std::max<long>(1, (long)((double)target * ramp));
        if (left < 2 * target) tgt = std::min(tgt, std::max(target / 8, left / 2));
      }
      long r = r0, pairs = 0;
      while (r < upper && (r == r0 || ((r - r0 + 1) * ncols <= cap && pairs < tgt && r - r0 < 65535l * kTile))) {
        pairs += row_pairs(r);
        r++;
      }
      out.push_back({r0, r});
      left -= pairs;
      r0 = r;
    }
    return out;
  };
  constexpr long kBigSlots = 64l << 20;    // pair slots of a band that need not overlap a copy (512 MB of distances)
  constexpr long kSmallSlots = 16l << 20;  // of the other bands
  Bands bands = (stream_text || rc.resolve_all) ? plan_bands(row_begin, band_pairs, kSmallSlots, stream_text, 0)
                                                : plan_bands(row_begin, 1l << 62, kBigSlots, false, 0);
  const long maxseg = std::max<long>(1, (ncols + kSeg - 1) / kSeg);
  if (hyphy) {
    TRY(ensure(ctx, ctx->hy, (size_t)N * N * sizeof(double)));
    fill_nan_kernel<<<1024, 256, 0, st>>>((double *)ctx->hy.p, (size_t)N * N);
    CU(cudaGetLastError());
    ctx->launches++;
  }
  const int tc16 = 32 * L < 65536;  // the final x16 aggregates fit 16-bit lanes
  long band = 1, nseg = 1;
  size_t dslots = 1, stat_stride = 0;
  std::vector<Bands> band_chunks;  // the tensor-core path's row chunks per band
  int nchunks[2] = {0, 0};
  unsigned und_cap_par[2] = {0, 0};  // grown per parity when a band lists more
  char *d_pstats = nullptr;          // the device's address of the statistics' staging
  // the row chunks of the bands from `first` on, boundaries on the count kernel's 32-row tiles; returns the pair slots of the
  // largest one
  auto plan_chunks = [&](size_t first) {
    band_chunks.resize(bands.size());
    size_t slots = 1;
    for (size_t b = first; b < bands.size(); b++) {
      band_chunks[b].clear();
      if (!use_tc) continue;
      const long r0 = bands[b].first, r1 = bands[b].second;
      static const long chunk_pairs = [] {
        const char *e = getenv("TN93G_TC_CHUNK_PAIRS");  // tuning knob: pairs per count/pair chunk
        return e && atol(e) > 0 ? atol(e) : kTcChunkPairs;
      }();
      const long target = std::max(chunk_pairs, (count_pairs(r0, r1) + kMaxTcChunks - 2) / (kMaxTcChunks - 1));
      for (long c0 = r0; c0 < r1;) {
        long c1 = c0, pairs = 0;
        while (c1 < r1 && (c1 == c0 || pairs < target)) {
          pairs += row_pairs(c1);
          c1++;
        }
        c1 = std::min(r1, (c1 + kTcRows - 1) / kTcRows * kTcRows);
        if ((int)band_chunks[b].size() == kMaxTcChunks - 1) c1 = r1;  // never more chunks than events
        band_chunks[b].push_back({c0, c1});
        slots = std::max(slots, (size_t)(c1 - c0) * ncols);
        c0 = c1;
      }
    }
    return slots;
  };
  auto max_rows = [](const Bands &v, size_t first) {
    long n = 1;
    for (size_t b = first; b < v.size(); b++) n = std::max(n, v[b].second - v[b].first);
    return n;
  };
  auto und_entries = [&](size_t slots) {
    return (unsigned)std::min<size_t>(rc.resolve_all ? slots : std::max<size_t>(4096, slots / 64), 0xFFFFFFF0u);
  };
  // per band parity (double-buffered): distances, segment statistics, row sums; the replay queue is per band
  auto band_buffers = [&](long rows, size_t chunk_slots) {
    const size_t slots = (size_t)rows * ncols, segs = (size_t)rows * maxseg, w = sizeof(unsigned long long);
    const size_t und = (size_t)und_entries(slots) * 2 * w;
    std::vector<std::pair<DevBuf *, size_t>> v = {{&ctx->dist, 2 * slots * w},       {&ctx->rq, slots * w},
                                                  {&ctx->rbytes, 2 * segs * w},      {&ctx->roff, 2 * segs * w},
                                                  {&ctx->rsum, 2 * (size_t)rows * 3 * w}, {&ctx->rw, 2 * (size_t)rows * 3 * w},
                                                  {&ctx->rmax, 2 * segs * 3 * w},    {&ctx->rlinks, 2 * segs * w},
                                                  {&ctx->rskip, 2 * segs * w},       {&ctx->und[0], und},
                                                  {&ctx->und[1], und}};
    if (rc.emit && !hyphy) v.push_back({&ctx->dcode, 2 * slots * sizeof(uint32_t)});
    if (use_tc) v.push_back({&ctx->tcagg, chunk_slots * (tc16 ? 16 : 32)});
    return v;
  };
  // Sizes them for the largest of the bands from the first one on; called again, with nothing in flight, when the schedule
  // changes. spare: the caller can go on without.
  auto size_buffers = [&](size_t first, bool spare) -> int {
    const size_t chunk_slots = plan_chunks(first);
    band = max_rows(bands, first);
    nseg = band * maxseg;
    dslots = (size_t)band * ncols;
    for (const auto &b : band_buffers(band, chunk_slots)) TRY(ensure(ctx, *b.first, b.second, spare));
    for (unsigned &cap : und_cap_par) cap = und_entries(dslots);
    // pinned staging of a band's statistics: row sums and weights (3 each at most), total bytes, the band's histogram and
    // totals, its undecided count and the count kernel's error word
    stat_stride = (size_t)band * 6 * sizeof(double) + (3 + kBandWords) * sizeof(unsigned long long);
    TRY(ensure_pinned_at(ctx, ctx->pstats, ctx->pstats_n, 2 * stat_stride, cudaHostAllocMapped));
    CU(cudaHostGetDevicePointer((void **)&d_pstats, ctx->pstats, 0));
    return TN93G_OK;
  };
  TRY(size_buffers(0, false));
  TRY(ensure(ctx, ctx->rqn, sizeof(unsigned)));
  // the run's scalars: 4 counters, the 3 summary units' bounds (4 words each), the count kernel's error word
  TRY(ensure(ctx, ctx->counters, kRunScalars * sizeof(unsigned long long)));
  CU(cudaMemsetAsync(ctx->counters.p, 0, kRunScalars * sizeof(unsigned long long), st));
  unsigned long long *const d_amb = (unsigned long long *)ctx->counters.p + 4, *const d_tcerr = d_amb + 12;
  // per band parity: its histogram (added on the host, so a band's row stage can run again), its undecided list
  TRY(ensure(ctx, ctx->hist, 2 * kBandWords * sizeof(unsigned long long)));
  TRY(ensure(ctx, ctx->total, 2 * sizeof(unsigned long long)));
  TRY(ensure(ctx, ctx->undn, 2 * sizeof(unsigned long long)));
  TRY(ensure(ctx, ctx->rdesc, 2 * sizeof(ReplayArgs)));
  double max_[3] = {0, 0, 0}, mean[3] = {0, 0, 0}, wc[3] = {0, 0, 0};
  unsigned long long hist_total[3 * kHistBins];
  memset(hist_total, 0, sizeof hist_total);
  long links = 0, skipped = 0, resolved = 0;
  float ms = 0;
  const int bins = rc.fst ? 3 : 1;  // sums of a row that can be other than zero
  struct HostStats {
    double *sum, *w;  // [row][bins]
    unsigned long long *total, *hist, *und, *tcerr;
  };
  auto host_stats = [&](int par) {
    char *base = (char *)ctx->pstats + par * stat_stride;
    HostStats h;
    h.sum = (double *)base;
    h.w = h.sum + band * 3;
    h.total = (unsigned long long *)(h.w + band * 3);
    h.hist = h.total + 1;
    h.und = h.hist + kBandWords;
    h.tcerr = h.und + 1;
    return h;
  };
  ReplayArgs rdesc_h[2];
  auto row_args = [&](int bi) {
    const int par = bi & 1;
    RowArgs RA;
    RA.rc = rc;
    RA.dist = (const double *)ctx->dist.p + par * dslots;
    RA.r0 = bands[bi].first;
    RA.r1 = bands[bi].second;
    RA.ncols = ncols;
    RA.colbase = colbase;
    RA.counts = set->d_counts;
    RA.name_len = set->d_name_len;
    RA.name_off = set->d_name_off;
    RA.names = set->d_names;
    RA.maxseg = maxseg;
    RA.seg_bytes = (unsigned long long *)ctx->rbytes.p + par * nseg;
    RA.seg_links = (long long *)ctx->rlinks.p + par * nseg;
    RA.seg_skip = (long long *)ctx->rskip.p + par * nseg;
    RA.seg_max = (double *)ctx->rmax.p + par * nseg * 3;
    RA.row_sum = (double *)ctx->rsum.p + par * band * 3;
    RA.row_w = (double *)ctx->rw.p + par * band * 3;
    RA.hist = (unsigned long long *)ctx->hist.p + par * kBandWords;
    RA.seg_off = (const unsigned long long *)ctx->roff.p + par * nseg;
    RA.seg_cols = nullptr;
    RA.nrows = RA.r1 - RA.r0;
    RA.out = nullptr;
    RA.hy = (double *)ctx->hy.p;
    RA.err = (unsigned long long *)ctx->counters.p + 3;
    RA.dcode = (rc.emit && !hyphy) ? (uint32_t *)ctx->dcode.p + par * dslots : nullptr;
    return RA;
  };
  // stats -> sums -> scan of band bi, then its statistics to the host (on the compute stream)
  auto enqueue_rows = [&](int bi) -> int {
    const int par = bi & 1;
    const long nr = bands[bi].second - bands[bi].first;
    cudaEvent_t *K = ctx->evk[par];
    RowArgs RA = row_args(bi);
    CU(cudaMemsetAsync(RA.hist, 0, kBandWords * sizeof(unsigned long long), st));
    stats_kernel<<<dim3((unsigned)((nr + kWarps - 1) / kWarps), (unsigned)maxseg), 256, 0, st>>>(RA);
    CU(cudaGetLastError());
    ctx->launches++;
    sum_kernel<<<(unsigned)((nr + kWarps - 1) / kWarps), 256, 0, st>>>(RA);
    CU(cudaGetLastError());
    ctx->launches++;
    unsigned long long *dtot = (unsigned long long *)ctx->total.p + par;
    scan_kernel<<<1, 1024, 0, st>>>(RA.seg_bytes, (unsigned long long *)RA.seg_off, nr * maxseg, dtot);
    CU(cudaGetLastError());
    ctx->launches++;
    band_totals_kernel<<<(unsigned)std::min<long>(64, (nr * maxseg + 255) / 256), 256, 0, st>>>(
        RA.seg_links, RA.seg_skip, RA.seg_max, nr * maxseg, RA.hist + 3 * kHistBins);
    CU(cudaGetLastError());
    ctx->launches++;
    CU(cudaEventRecord(K[3], st));
    // the band's statistics into the mapped staging (device addresses at the same offsets as host_stats')
    const HostStats h = host_stats(par);
    auto dev = [&](const void *hp) {
      return (unsigned long long *)(d_pstats + ((const char *)hp - (const char *)ctx->pstats));
    };
    Gather g;
    g.k = 0;
    auto add = [&](const void *src, const void *hdst, long nwords, int stride = 1) {
      g.src[g.k] = (const unsigned long long *)src;
      g.dst[g.k] = dev(hdst);
      g.stride[g.k] = stride;
      g.n[g.k++] = nwords;
    };
    add(RA.row_sum, h.sum, nr * bins, 3 / bins);
    add(RA.row_w, h.w, nr * bins, 3 / bins);
    add(dtot, h.total, 1);
    add(RA.hist, h.hist, kBandWords);
    add((unsigned long long *)ctx->undn.p + par, h.und, 1);
    if (use_tc)
      add(d_tcerr, h.tcerr, 1);
    else
      *h.tcerr = 0;
    gather_kernel<<<32, 256, 0, st>>>(g);
    CU(cudaGetLastError());
    ctx->launches++;
    CU(cudaEventRecord(K[4], st));
    return TN93G_OK;
  };
  // pair -> replay of band bi, then its row stage
  auto enqueue_compute = [&](int bi) -> int {
    const int par = bi & 1;
    const long r0 = bands[bi].first, r1 = bands[bi].second, nr = r1 - r0;
    cudaEvent_t *K = ctx->evk[par];
    // this parity's distances, codes and row arrays are read by band bi - 2's text writer on the write stream
    if (bi >= 2 && stream_text) CU(cudaStreamWaitEvent(st, ctx->evrow[par], 0));
    CU(cudaEventRecord(K[0], st));
    CU(cudaMemsetAsync(ctx->rqn.p, 0, sizeof(unsigned), st));
    CU(cudaMemsetAsync((unsigned long long *)ctx->undn.p + par, 0, sizeof(unsigned long long), st));
    ExactSink ex;
    ex.und_list = (unsigned long long *)ctx->und[par].p;
    ex.und_n = (unsigned *)((unsigned long long *)ctx->undn.p + par);
    ex.und_cap = und_cap_par[par];
    ex.und_k = 0;
    ex.amb = d_amb;
    ex.counts = set->d_counts;
    ex.colunit = nullptr;
    PairArgs A;
    A.rc = rc;
    A.planes = (const uint64_t *)ctx->planes.p;
    A.cc = (const uint8_t *)ctx->cc.p;
    A.ccT = (const uint8_t *)ctx->ccT.p;
    A.ev_off = (const uint32_t *)ctx->evoff.p;
    A.ev = (const uint32_t *)ctx->ev.p;
    A.ev2 = use_ev2 ? (const uint2 *)ctx->ev2.p : nullptr;
    A.three = pa.three;
    A.lin = lin;
    A.tab = (const PairTables *)ctx->agg.p;
    A.r0 = r0;
    A.r1 = r1;
    A.ncols = ncols;
    A.colbase = colbase;
    A.cend = N;
    A.dist = (double *)ctx->dist.p + par * dslots;
    A.replay_q = (unsigned long long *)ctx->rq.p;
    A.replay_n = (unsigned *)ctx->rqn.p;
    A.replay_cap = (unsigned long long)dslots;
    A.counters = (unsigned long long *)ctx->counters.p;
    A.logt = ctx->d_logt;
    A.ex = ex;
    A.wl_off = sparse_w ? (const uint32_t *)ctx->wloff.p : nullptr;
    A.wl = sparse_w ? (const uint32_t *)ctx->wl.p : nullptr;
    // columns: the smallest lower bound of the band's rows onwards
    const long cstart = rc.cross ? n1 : r0 + 1;
    const long cblk0 = (cstart - colbase) / 32;
    const long cblks = (ncols + 31) / 32 - cblk0;
    if (use_tc && cblks > 0) {
      // Clean-site aggregates on the tensor cores, then the pair kernel, chunk by chunk of rows (about kTcChunkPairs
      // pairs each); the pair kernel reads each record once and drops its cache line.
      const std::vector<std::pair<long, long>> &chunks = band_chunks[bi];
      for (size_t q = 0; q < chunks.size(); q++) {
        const long c0 = chunks[q].first, c1 = chunks[q].second;
        const long ccs = rc.cross ? n1 : c0 + 1;
        TcArgs T;
        T.onehot = (const uint8_t *)ctx->ohimg.p;
        T.NB = tc_NB;
        T.KS = tc_KS;
        T.N = N;
        T.n1 = n1;
        T.cross = rc.cross;
        T.r0 = c0;
        T.r1 = c1;
        T.ncols = ncols;
        T.colbase = colbase;
        T.cstart = ccs / kTcCols * kTcCols;
        T.cend = N;
        T.agg = ctx->tcagg.p;
        T.agg16 = tc16;
        T.err = d_tcerr;
        T.wait_ns = ctx->wait_ns;
        T.skip_fill_block = fault_pending ? 0 : -1;
        fault_pending = false;
        const long rt0 = c0 / kTcRows * kTcRows;
        const dim3 g((unsigned)((N - T.cstart + kTcCols - 1) / kTcCols), (unsigned)((c1 - rt0 + kTcRows - 1) / kTcRows));
        CU(cudaEventRecord(ctx->evcnt[par][2 * q], st));
        CU(launch_count_grid(T, g.x, g.y, ctx->sms, st));
        CU(cudaEventRecord(ctx->evcnt[par][2 * q + 1], st));
        ctx->launches++;
        PairArgs AC = A;
        AC.r0 = c0;
        AC.r1 = c1;
        AC.dist = A.dist + (size_t)(c0 - r0) * ncols;
        AC.tcagg = ctx->tcagg.p;
        AC.tc16 = tc16;
        const long cb0 = (ccs - colbase) / 32, cbs = (ncols + 31) / 32 - cb0;
        if (cbs > 0) {
          AC.cstart = colbase + cb0 * 32;
          CU(launch_pair(AC, cbs, c1 - c0, ctx->sms, st));
          ctx->launches += pair_split(AC) && !AC.lin ? 2 : 1;
        }
      }
      nchunks[par] = (int)chunks.size();
    } else if (cblks > 0) {
      A.cstart = colbase + cblk0 * 32;
      CU(launch_pair(A, cblks, nr, ctx->sms, st));
      ctx->launches++;
      nchunks[par] = 0;
    } else {
      nchunks[par] = 0;
    }
    CU(cudaEventRecord(K[1], st));
    ReplayArgs R;
    R.rc = rc;
    R.cc = (const uint8_t *)ctx->cc.p;
    R.planes = (const uint64_t *)ctx->planes.p;
    R.site = (const SiteEntry *)ctx->site.p;
    R.ev_off = A.ev_off;
    R.ev = use_ev ? A.ev : nullptr;
    R.q = (const unsigned long long *)ctx->rq.p;
    R.qn = (const unsigned *)ctx->rqn.p;
    R.qcap = (unsigned long long)dslots;
    R.r0 = r0;
    R.ncols = ncols;
    R.colbase = colbase;
    R.dist = A.dist;
    R.counters = (unsigned long long *)ctx->counters.p;
    R.logt = ctx->d_logt;
    R.ex = ex;
    rdesc_h[par] = R;
    replay_kernel<<<2 * ctx->sms, 256, 0, st>>>(R);
    CU(cudaGetLastError());
    ctx->launches++;
    CU(cudaEventRecord(K[2], st));
    return enqueue_rows(bi);
  };
  // texts on their way to the host: their buffers (out2, pin2), oldest first
  int pend_buf[2] = {0, 0}, pend_n = 0, next_buf = 0;
  size_t pend_bytes[2] = {0, 0};
  bool buf_used[2] = {false, false};
  // TN93G_TRACE=1: one stderr line per delivered text (device milliseconds from the run's first event: write
  // start and end, copy start and end; host milliseconds when the copy was seen complete), for pipeline tuning
  static const bool trace = getenv("TN93G_TRACE") != nullptr;
  const auto host0 = std::chrono::steady_clock::now();
  int delivered = 0;
  auto deliver_oldest = [&]() -> int {
    const int q = pend_buf[0];
    CU(cudaEventSynchronize(ctx->evc1[q]));
    CU(cudaEventElapsedTime(&ms, ctx->evw0[q], ctx->evw1[q]));
    ctx->timings[4] += ms;
    CU(cudaEventElapsedTime(&ms, ctx->evc0[q], ctx->evc1[q]));
    ctx->timings[5] += ms;
    if (trace) {
      float w0, w1, c0, c1;
      CU(cudaEventElapsedTime(&w0, E[0], ctx->evw0[q]));
      CU(cudaEventElapsedTime(&w1, E[0], ctx->evw1[q]));
      CU(cudaEventElapsedTime(&c0, E[0], ctx->evc0[q]));
      CU(cudaEventElapsedTime(&c1, E[0], ctx->evc1[q]));
      const double h = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - host0).count();
      fprintf(stderr, "tn93g trace: text %d bytes %zu write %.3f-%.3f copy %.3f-%.3f host %.3f\n", delivered++,
              pend_bytes[q], w0, w1, c0, c1, h);
    }
    pend_buf[0] = pend_buf[1];
    pend_n--;
    if (sink && sink(user, (const char *)ctx->pin2[q], pend_bytes[q])) return TN93G_ESINK;
    return TN93G_OK;
  };
  // Text of band bi: its rows [ra, rb), the n bytes from byte `at` of the band's text on. It is written on the write stream,
  // beside the next band's kernels, once the band's statistics are final (K[4]), then copied on the copy stream. The text
  // that holds the same buffer pair goes to the sink first: its copy has then left the device buffer, the sink has taken the
  // pinned buffer, and its events are free to record this one's. Meanwhile the copy engine works on the text in between.
  auto send_text = [&](int bi, long ra, long rb, size_t at, size_t n) -> int {
    const int q = next_buf;
    for (;;) {
      bool held = false;
      for (int k = 0; k < pend_n; k++) held |= pend_buf[k] == q;
      if (!held) break;
      TRY(deliver_oldest());
    }
    TRY(ensure(ctx, ctx->out2[q], n));
    TRY(ensure_pinned_at(ctx, ctx->pin2[q], ctx->pin2_n[q], n));
    RowArgs RA = row_args(bi);
    RA.r1 = RA.r0 + rb;
    RA.r0 += ra;
    RA.nrows = rb - ra;
    RA.dist += (size_t)ra * ncols;
    RA.dcode += (size_t)ra * ncols;
    RA.seg_bytes += ra * maxseg;
    RA.seg_off += ra * maxseg;
    RA.out = (char *)((uintptr_t)ctx->out2[q].p - at);  // seg_off counts from the band's first byte
    const cudaStream_t ws = ctx->write_stream;
    CU(cudaStreamWaitEvent(ws, ctx->evk[bi & 1][4], 0));
    if (buf_used[q]) CU(cudaStreamWaitEvent(ws, ctx->evc1[q], 0));
    CU(cudaEventRecord(ctx->evw0[q], ws));
    write_kernel<<<dim3((unsigned)((rb - ra + kWarps - 1) / kWarps), (unsigned)maxseg), 256, 0, ws>>>(RA);
    CU(cudaGetLastError());
    ctx->launches++;
    CU(cudaEventRecord(ctx->evw1[q], ws));
    CU(cudaStreamWaitEvent(ctx->copy_stream, ctx->evw1[q], 0));
    CU(cudaEventRecord(ctx->evc0[q], ctx->copy_stream));
    CU(cudaMemcpyAsync(ctx->pin2[q], ctx->out2[q].p, n, cudaMemcpyDeviceToHost, ctx->copy_stream));
    CU(cudaEventRecord(ctx->evc1[q], ctx->copy_stream));
    buf_used[q] = true;
    pend_bytes[q] = n;
    pend_buf[pend_n++] = q;
    next_buf ^= 1;
    return TN93G_OK;
  };
  // The whole text of band bi, tot bytes: in pieces of whole rows where a band larger than the streaming ones reports much (a
  // band of 64 M slots may have gigabytes, of which a piece is copied while the next is written), and where the buffers for
  // more do not fit.
  constexpr size_t kTextPiece = 64 << 20;
  auto send_band = [&](int bi, size_t tot) -> int {
    const long nr = bands[bi].second - bands[bi].first;
    const bool large = count_pairs(bands[bi].first, bands[bi].second) > band_pairs + ncols;
    size_t limit = large ? std::min(tot, kTextPiece) : tot;
    std::vector<unsigned long long> off;  // where each row's text starts, when it is taken in pieces
    for (long ra = 0; ra < nr;) {
      long rb = nr;
      size_t at = 0, n = tot;
      if (limit < tot) {
        if (off.empty()) {
          off.resize(nr + 1);
          CU(cudaMemcpy2DAsync(off.data(), sizeof off[0], row_args(bi).seg_off, maxseg * sizeof off[0], sizeof off[0], nr,
                               cudaMemcpyDeviceToHost, ctx->write_stream));
          CU(cudaStreamSynchronize(ctx->write_stream));
          off[nr] = tot;
        }
        at = off[ra];
        rb = std::max(ra + 1, (long)(std::upper_bound(off.begin() + ra, off.end(), at + limit) - off.begin()) - 1);
        n = off[rb] - at;
      }
      if (n) {
        const int r = send_text(bi, ra, rb, at, n);
        if (r == TN93G_ENOMEM && rb - ra > 1) {
          ctx->err.clear();
          limit = n / 2;
          continue;
        }
        TRY(r);
      }
      ra = rb;
    }
    CU(cudaEventRecord(ctx->evrow[bi & 1], ctx->write_stream));
    return TN93G_OK;
  };
  size_t band_text = 0;  // bytes that the last finished band reported
  // statistics of band bi in row order, then its text: written on the compute stream (behind the next band's
  // kernels) and copied to the host on the copy stream
  auto finish = [&](int bi) -> int {
    const int par = bi & 1;
    const long nr = bands[bi].second - bands[bi].first;
    cudaEvent_t *K = ctx->evk[par];
    CU(cudaEventSynchronize(K[4]));
    CU(cudaEventElapsedTime(&ms, K[0], K[1]));
    ctx->timings[1] += ms;
    for (int q = 0; q < nchunks[par]; q++) {
      CU(cudaEventElapsedTime(&ms, ctx->evcnt[par][2 * q], ctx->evcnt[par][2 * q + 1]));
      ctx->timings[7] += ms;
    }
    CU(cudaEventElapsedTime(&ms, K[1], K[2]));
    ctx->timings[2] += ms;
    CU(cudaEventElapsedTime(&ms, K[2], K[3]));
    ctx->timings[3] += ms;
    const HostStats h = host_stats(par);
    if (*h.tcerr) {
      // the next band's kernels may still be queued: let them drain so the context is idle for the next run
      cudaStreamSynchronize(st);
      ctx->err = "the tensor-core count kernel timed out waiting for its pipeline";
      return TN93G_ETIMEOUT;
    }
    if (*h.und) {
      // pairs whose bytes or decisions depend on the C library's rounding of a logarithm: finish them with its
      // logarithms, then run the band's row stage again
      if (*h.und > und_cap_par[par]) {
        // more than the list holds: grow this parity's list and run the band's pair stage again (the same pairs
        // are listed; the summary bounds only widen, which keeps them valid)
        const unsigned long long lim = std::min<unsigned long long>(dslots, 0xFFFFFFF0ull);
        const unsigned need = (unsigned)std::min<unsigned long long>(
            std::max<unsigned long long>(*h.und + *h.und / 4 + 1024, 2ull * und_cap_par[par]), lim);
        CU(cudaStreamSynchronize(st));
        TRY(ensure(ctx, ctx->und[par], (size_t)need * 2 * sizeof(unsigned long long)));
        und_cap_par[par] = need;
        TRY(enqueue_compute(bi));
        CU(cudaEventSynchronize(K[4]));
        if (*h.und > und_cap_par[par]) {
          ctx->err = "more undecided pairs in a band than its list holds";
          return TN93G_EUNDECIDED;
        }
      }
      ReplayArgs *dd = (ReplayArgs *)ctx->rdesc.p + par;
      CU(cudaMemcpyAsync(dd, &rdesc_h[par], sizeof(ReplayArgs), cudaMemcpyHostToDevice, st));
      TRY(resolve_listed(ctx, dd, (const unsigned long long *)ctx->und[par].p, (unsigned)*h.und, st));
      resolved += (long)*h.und;
      TRY(enqueue_rows(bi));
      CU(cudaEventSynchronize(K[4]));
    }
    for (int q = 0; q < 3 * kHistBins; q++) hist_total[q] += h.hist[q];
    const unsigned long long *const bt = h.hist + 3 * kHistBins;
    links += (long)bt[0];
    skipped += (long)bt[1];
    for (int q = 0; q < 3; q++) {
      double m;
      memcpy(&m, &bt[2 + q], sizeof m);
      max_[q] = std::max(max_[q], m);
    }
    // rows in order (swifttn93.cpp:2838-2848)
    for (long r = 0; r < nr; r++)
      for (int q = 0; q < bins; q++) {
        mean[q] += h.sum[r * bins + q];
        wc[q] += h.w[r * bins + q];
      }
    if (row_sums)
      for (long r = 0; r < nr; r++) {
        double *o = row_sums + (size_t)(bands[bi].first - row_begin + r) * 6;
        for (int q = 0; q < 3; q++) {
          o[q] = q < bins ? h.sum[r * bins + q] : 0.;
          o[3 + q] = q < bins ? h.w[r * bins + q] : 0.;
        }
      }
    const unsigned long long tot = *h.total;
    band_text = rc.emit && !hyphy ? tot : 0;
    if (!band_text) return TN93G_OK;
    sum->output_bytes += tot;
    if (to_device) {
      RowArgs RA = row_args(bi);
      const dim3 wgrid((unsigned)((nr + kWarps - 1) / kWarps), (unsigned)maxseg);
      TRY(ensure_keep(ctx, ctx->out, dev_off + tot, dev_off));
      RA.out = (char *)ctx->out.p + dev_off;
      CU(cudaEventRecord(ctx->evw0[0], st));
      write_kernel<<<wgrid, 256, 0, st>>>(RA);
      CU(cudaGetLastError());
      ctx->launches++;
      CU(cudaEventRecord(ctx->evw1[0], st));
      CU(cudaEventSynchronize(ctx->evw1[0]));
      CU(cudaEventElapsedTime(&ms, ctx->evw0[0], ctx->evw1[0]));
      ctx->timings[4] += ms;
      dev_off += tot;
      return TN93G_OK;
    }
    return send_band(bi, tot);
  };
  // Band bi + 1's kernels are queued before band bi is finished, so the device computes while the host takes band
  // bi's statistics; texts reach the sink when their pinned buffer is needed again, or at the end (at most one band
  // per parity waits).
  // A streamed run whose first band reports few pairs (less than 2 bytes of text a pair, so copying a band takes less than a
  // sixth of computing it) has nothing to overlap: what is left after the second runs as large bands, whose kernels fill the GPU (each
  // kernel's last wave, the row sums' chains and the replays cost a band about as much whatever its size: 6,700 x 1,500 at
  // -t 0.015 took 17 bands and 7.2 ms of device time, 4.9 ms so). The first rows may not be like the rest: the first large
  // band takes a quarter of what is left, so that, where it reports much, the next one's kernels run under its copies, and
  // what is not queued by then goes on in small bands (6,700 x 1,500, 100 unrelated rows and the rest linked: 8.5 ms, 9.6
  // with the rest in one band, 9.7 in small bands; nothing linked: 3.88, 3.91 and 7.05). Less than four small bands' worth
  // is one band: another would cost more than it could overlap (3,001 x 1,065: 1.36 and 1.49 ms, 4,000 x 1,500: 1.91 and
  // 1.96). If the larger buffers do not fit, the small bands go on.
  const bool may_grow = stream_text && !rc.resolve_all && !forced_band;
  auto few = [&](int bi) { return band_text < 2 * (size_t)count_pairs(bands[bi].first, bands[bi].second); };
  // the rows from band 2 on in large bands, with buffers for them; where those do not fit the schedule stays as it was
  bool large = false;
  auto grow_bands = [&]() -> int {
    const Bands small = bands;
    const long from = small[2].first;
    bool tried = false;
    int r = TN93G_ENOMEM;
    for (long cap = kBigSlots; cap > kSmallSlots && r == TN93G_ENOMEM; cap /= 2) {
      bands.resize(2);
      const long left = count_pairs(from, upper);
      bands.push_back(plan_bands(from, left < 4 * band_pairs ? left + 1 : std::max(band_pairs, left / 4), cap, false, 0)[0]);
      for (const auto &b : plan_bands(bands[2].second, left + 1, cap, false, 0)) bands.push_back(b);
      const long rows = max_rows(bands, 2);
      if (ctx->budget) {
        // Room for the larger buffers, for texts, and for what a run may need later and needed with the small bands too:
        // undecided lists of every pair, of these bands or of an exact-sums pass
        size_t need = ctx->used + 2 * kTextPiece;
        for (const auto &b : band_buffers(rows, plan_chunks(2))) need += b.second > b.first->n ? b.second - b.first->n : 0;
        const long exact = max_rows(plan_bands(row_begin, band_pairs, kSmallSlots, false, 0), 0);
        need += 4 * (size_t)std::max(rows, exact) * ncols * sizeof(unsigned long long);
        if (need > ctx->budget) continue;
      }
      tried = true;
      r = size_buffers(2, true);
    }
    large = r == TN93G_OK;
    if (r == TN93G_ENOMEM) {
      if (tried)  // what has grown makes room for the small bands' buffers again
        for (const auto &b : band_buffers(1, 1)) release(ctx, *b.first);
      bands = small;
      r = size_buffers(2, false);
    }
    return r;
  };
  int nb = (int)bands.size();
  for (int bi = 0; bi <= nb; bi++) {
    if (bi < nb) TRY(enqueue_compute(bi));
    if (bi >= 1) TRY(finish(bi - 1));
    if (bi == 1 && may_grow && nb > 3 && few(0)) {
      TRY(finish(1));
      while (pend_n) TRY(deliver_oldest());
      TRY(grow_bands());
      nb = (int)bands.size();
      bi = 2;
      TRY(enqueue_compute(2));
    } else if (large && bi >= 3 && bi + 1 < nb && !few(bi - 1)) {
      large = false;
      const Bands was = bands;
      bands.resize(bi + 1);
      for (const auto &b : plan_bands(was[bi].second, band_pairs, kSmallSlots, true, 99)) bands.push_back(b);
      const size_t records = plan_chunks(bi + 1) * (tc16 ? 16 : 32);
      if (max_rows(bands, bi + 1) > band || (use_tc && records > ctx->tcagg.n)) {  // (they fit the larger bands' buffers)
        bands = was;
        plan_chunks(bi + 1);
      }
      nb = (int)bands.size();
    }
  }
  while (pend_n) TRY(deliver_oldest());
  if (hyphy) {
    TRY(ensure(ctx, ctx->rbytes, N * sizeof(unsigned long long)));
    TRY(ensure(ctx, ctx->roff, N * sizeof(unsigned long long)));
    const unsigned blocks = (unsigned)((N + kWarps - 1) / kWarps);
    CU(cudaEventRecord(E[6], st));
    hy_len_kernel<<<blocks, 256, 0, st>>>((const double *)ctx->hy.p, N, (unsigned long long *)ctx->rbytes.p);
    CU(cudaGetLastError());
    ctx->launches++;
    std::vector<unsigned long long> hb(N), ho(N);
    CU(cudaMemcpyAsync(hb.data(), ctx->rbytes.p, N * sizeof(unsigned long long), cudaMemcpyDeviceToHost, st));
    CU(cudaStreamSynchronize(st));
    unsigned long long tot = 1;  // leading "{"
    for (long r = 0; r < N; r++) {
      ho[r] = tot;
      tot += hb[r];
    }
    tot += 2;  // "\n}"
    TRY(ensure(ctx, ctx->out, tot));
    if (!to_device) TRY(ensure_pinned(ctx, tot));
    CU(cudaMemcpyAsync(ctx->roff.p, ho.data(), N * sizeof(unsigned long long), cudaMemcpyHostToDevice, st));
    CU(cudaMemcpyAsync(ctx->out.p, "{", 1, cudaMemcpyHostToDevice, st));
    hy_write_kernel<<<blocks, 256, 0, st>>>((const double *)ctx->hy.p, N, (const unsigned long long *)ctx->roff.p,
                                            (char *)ctx->out.p);
    CU(cudaGetLastError());
    ctx->launches++;
    CU(cudaMemcpyAsync((char *)ctx->out.p + tot - 2, "\n}", 2, cudaMemcpyHostToDevice, st));
    CU(cudaEventRecord(E[7], st));
    if (!to_device) CU(cudaMemcpyAsync(ctx->pinned, ctx->out.p, tot, cudaMemcpyDeviceToHost, st));
    CU(cudaEventRecord(E[8], st));
    CU(cudaStreamSynchronize(st));
    CU(cudaEventElapsedTime(&ms, E[6], E[7]));
    ctx->timings[4] += ms;
    CU(cudaEventElapsedTime(&ms, E[7], E[8]));
    ctx->timings[5] += ms;
    sum->output_bytes += tot;
    dev_off = tot;
    if (!to_device && sink && sink(user, (const char *)ctx->pinned, tot)) return TN93G_ESINK;
  }
  CU(cudaMemcpyAsync(h_scalars, ctx->counters.p, kRunScalars * sizeof(unsigned long long), cudaMemcpyDeviceToHost, st));
  CU(cudaEventRecord(E[9], st));
  CU(cudaStreamSynchronize(st));
  unsigned long long counters[4], ambw[12];
  memcpy(counters, h_scalars, sizeof counters);
  memcpy(ambw, h_scalars + 4, sizeof ambw);
  const unsigned long long tcerr = h_scalars[16];
  if (trace) {
    float d9;
    CU(cudaEventElapsedTime(&d9, E[0], E[9]));
    fprintf(stderr, "tn93g trace: end device %.3f host %.3f bands %d\n", d9,
            std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - host0).count(), nb);
  }
  CU(cudaEventElapsedTime(&ms, E[0], E[1]));
  ctx->timings[0] = ms;
  CU(cudaEventElapsedTime(&ms, E[0], E[9]));
  ctx->timings[6] = ms;
  for (int q = 0; q < 3; q++) {
    sum->max[q] = max_[q];
    sum->mean[q] = mean[q];
    sum->weighted[q] = wc[q];
    for (int k = 0; k < kHistBins; k++) sum->hist[q][k] = hist_total[q * kHistBins + k];
  }
  sum->links = links;
  sum->skipped = skipped;
  sum->logs_ambiguous = (long)counters[0];
  sum->logs_resolved = resolved;
  sum->undecided = 0;  // every listed pair was finished with the C library's logarithms
  sum->pairs_replayed = (long)counters[2];
  ctx->dev_out_n = dev_off;
  if (tcerr) {
    ctx->err = "the tensor-core count kernel timed out waiting for its pipeline";
    return TN93G_ETIMEOUT;
  }
  if (counters[3]) {
    ctx->err = "internal error: a row's text did not match its counted length";
    return TN93G_ECUDA;
  }
  // The JSON numbers (maximum, means): certain for every rounding of the C library's log, or taken from a second
  // pass that finishes every pair with an ambiguous logarithm with the C library's own (rows in the same order).
  // (A proper range of rows is a part of a larger run: its caller certifies the merged summary.)
  for (int u = 0; u < 3; u++) amb_bounds(ambw + 4 * u, sum->amb_bounds[u]);
  if (rc.resolve_all) memset(sum->amb_bounds, 0, sizeof sum->amb_bounds);  // every ambiguous pair was finished exactly
  const long chain = (rc.cross ? N - n1 : N) + (row_end - row_begin) + 2;
  const bool whole = row_begin == 0 && row_end == all_rows;
  if (!rc.resolve_all && whole && !summary_certified(sum, sum->amb_bounds, chain, rc.fst)) {
    tn93g_opts o2 = *opts;
    o2.count_only = 1;
    tn93g_summary s2;
    std::vector<double> rs2(row_sums ? (size_t)(row_end - row_begin) * 6 : 0);
    const double t6 = ctx->timings[6];
    TRY(run_impl(ctx, set, n1, &o2, nullptr, nullptr, &s2, false, row_begin, row_end,
                 row_sums ? rs2.data() : nullptr, kRunResolveAll));
    for (int q = 0; q < 3; q++) {
      sum->max[q] = s2.max[q];
      sum->mean[q] = s2.mean[q];
    }
    if (row_sums) memcpy(row_sums, rs2.data(), rs2.size() * sizeof(double));
    sum->logs_resolved += s2.logs_resolved;
    sum->sums_repass = 1;
    memset(sum->amb_bounds, 0, sizeof sum->amb_bounds);
    ctx->timings[6] += t6;
    ctx->dev_out_n = dev_off;
  }
  return TN93G_OK;
}

}  // extern "C"

//================================================================================================== allocation-free entry point
// tn93g_pair_distances_noalloc: the pack -> pair -> site-order replay pipeline of tn93g_run for one alignment,
// with every intermediate buffer carved out of one fixed file-scope device array instead of cudaMalloc, for
// callers that must not allocate device memory. Inputs and outputs are the caller's device buffers.
namespace {

constexpr long kNaMaxN = 512;   // sequences
constexpr long kNaMaxL = 4096;  // columns
constexpr long kNaW = (kNaMaxL + 63) / 64;
constexpr size_t na_al(size_t x) { return (x + 255) / 256 * 256; }
constexpr size_t kNaLog = 0;
constexpr size_t kNaAgg = kNaLog + na_al(sizeof(LogTable));
constexpr size_t kNaSite = kNaAgg + na_al(sizeof(PairTables));
constexpr size_t kNaSeen = kNaSite + na_al(2 * kCodes * kCodes * sizeof(SiteEntry));
constexpr size_t kNaNN = kNaSeen + na_al(kNaMaxL * sizeof(uint32_t));
constexpr size_t kNaVarcol = kNaNN + na_al(sizeof(unsigned long long));
constexpr size_t kNaPlanes = kNaVarcol + na_al(kNaMaxL * sizeof(int32_t));
constexpr size_t kNaCC = kNaPlanes + na_al((size_t)kNaW * 5 * kNaMaxN * sizeof(uint64_t));
constexpr size_t kNaCCT = kNaCC + na_al((size_t)kNaMaxN * kNaMaxL);
constexpr size_t kNaEvcount = kNaCCT + na_al((size_t)kNaMaxL * kNaMaxN);
constexpr size_t kNaEvoff = kNaEvcount + na_al(kNaMaxN * sizeof(uint32_t));
constexpr size_t kNaEv = kNaEvoff + na_al((kNaMaxN + 1) * sizeof(uint32_t));
constexpr size_t kNaRq = kNaEv + na_al((size_t)kNaMaxN * kNaMaxL * sizeof(uint32_t));
constexpr size_t kNaRqn = kNaRq + na_al((size_t)kNaMaxN * kNaMaxN * sizeof(unsigned long long));
constexpr size_t kNaCounters = kNaRqn + na_al(sizeof(unsigned));
constexpr size_t kNaBytes = kNaCounters + na_al(4 * sizeof(unsigned long long));  // about 15.6 MB

// The scratch. Every GPU that loads this library holds it until the process exits.
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNaBytes];

// Per device: the scratch's device address (cudaGetSymbolAddress, taken with that device current) and whether
// the log table has been written into it. Host code must never pass the symbol itself to a kernel.
constexpr int kNaMaxDevices = 64;
std::mutex g_na_mu;
unsigned char *g_na_base[kNaMaxDevices];

// message of the last failure of a call made by this thread
thread_local char g_na_err[256];

void na_error(const char *what, cudaError_t e)
{
  snprintf(g_na_err, sizeof g_na_err, "%s: %s", what, cudaGetErrorString(e));
}

// caller holds g_na_mu
int noalloc_setup(int dev, unsigned char **base)
{
  if (dev < 0 || dev >= kNaMaxDevices) return TN93G_ENODEV;
  if (g_na_base[dev]) {
    *base = g_na_base[dev];
    return TN93G_OK;
  }
  unsigned char *p = nullptr;
  cudaError_t e = cudaGetSymbolAddress((void **)&p, g_noalloc_scratch);
  if (e != cudaSuccess || !p) {
    na_error("cudaGetSymbolAddress", e);
    return TN93G_ECUDA;
  }
  LogTable h;
  build_log_table(&h);
  e = cudaMemcpy(p + kNaLog, &h, sizeof h, cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    na_error("cudaMemcpy", e);
    return TN93G_ECUDA;
  }
  g_na_base[dev] = p;
  *base = p;
  return TN93G_OK;
}

Tables g_na_tables;     // host staging of the contribution tables (static storage; used with g_na_mu held)
PairTables g_na_ptab;  // and of the pair stage's form of them

// caller holds g_na_mu
int noalloc_run(const uint8_t *d_codes, long N, long L, const tn93g_opts *opts, double *d_dist, cudaStream_t st)
{
#define NA(call)                  \
  do {                            \
    cudaError_t e_ = (call);      \
    if (e_ != cudaSuccess) {      \
      na_error(#call, e_);        \
      return TN93G_ECUDA;         \
    }                             \
  } while (0)
  int dev = 0;
  NA(cudaGetDevice(&dev));
  unsigned char *S = nullptr;
  const int src = noalloc_setup(dev, &S);
  if (src != TN93G_OK) return src;
  RunConsts rc;
  memset(&rc, 0, sizeof rc);
  rc.N = N;
  rc.n1 = N;
  rc.mode = opts->mode;
  rc.gapmm = opts->mode == TN93G_GAPMM;
  rc.fallback_avg = (opts->mode == TN93G_RESOLVE || opts->mode == TN93G_SUBSET) && opts->resolve_fraction < 1.;
  rc.emit = !opts->count_only;
  rc.format = opts->format;
  rc.delim = opts->delimiter;
  rc.threshold = opts->threshold;
  rc.min_distance = opts->min_distance;
  rc.resolve_fraction = opts->resolve_fraction;
  rc.min_overlap = opts->min_overlap;
  rc.log_band = kLogBand;
  rc.log_spread = kLogSpread;
  rc.resolve_all = false;
  uint32_t *seen = (uint32_t *)(S + kNaSeen);
  unsigned long long *nN = (unsigned long long *)(S + kNaNN);
  NA(cudaMemsetAsync(seen, 0, L * sizeof(uint32_t), st));
  NA(cudaMemsetAsync(nN, 0, sizeof(unsigned long long), st));
  colscan_kernel<<<dim3((unsigned)((L + 255) / 256), (unsigned)((N + 63) / 64)), 256, 0, st>>>(d_codes, N, L, seen, nN);
  NA(cudaGetLastError());
  uint32_t h_seen[kNaMaxL];
  int32_t h_varcol[kNaMaxL];
  unsigned long long h_nN = 0;
  NA(cudaMemcpyAsync(h_seen, seen, L * sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
  NA(cudaMemcpyAsync(&h_nN, nN, sizeof h_nN, cudaMemcpyDeviceToHost, st));
  NA(cudaStreamSynchronize(st));
  long Lc = 0;
  for (long p = 0; p < L; p++) {
    const uint32_t m = h_seen[p];
    if (m && !(m & (m - 1)) && m < 16) {
      const int b = __builtin_ctz(m);
      rc.constT++;
      rc.constNf[b] += 2;
      rc.constCnt[b]++;
    } else
      h_varcol[Lc++] = (int32_t)p;
  }
  const long W = (Lc + 63) / 64, Npad = (N + 31) / 32 * 32;
  rc.Lc = Lc;
  rc.W = W;
  rc.Npad = Npad;
  rc.wplane = rc.gapmm || h_nN > 16ull * (unsigned long long)N;
  rc.NP = rc.gapmm ? 5 : 4;
  PackArgs pa;
  pa.codes = d_codes;
  pa.N = N;
  pa.L = L;
  pa.Lc = Lc;
  pa.W = W;
  pa.Npad = Npad;
  pa.varcol = (const int32_t *)(S + kNaVarcol);
  pa.NP = rc.NP;
  pa.wplane = rc.wplane;
  pa.gapmm = rc.gapmm;
  pa.planes = (uint64_t *)(S + kNaPlanes);
  pa.cc = S + kNaCC;
  pa.evcount = (uint32_t *)(S + kNaEvcount);
  pa.ev_off = (const uint32_t *)(S + kNaEvoff);
  pa.ev = (uint32_t *)(S + kNaEv);
  if (Lc) NA(cudaMemcpyAsync(S + kNaVarcol, h_varcol, Lc * sizeof(int32_t), cudaMemcpyHostToDevice, st));
  NA(cudaMemsetAsync(pa.planes, 0, (size_t)std::max<long>(W, 1) * rc.NP * Npad * sizeof(uint64_t), st));
  NA(cudaMemsetAsync(pa.evcount, 0, N * sizeof(uint32_t), st));
  if (W) {
    pack_kernel<<<dim3((unsigned)((N + kWarps - 1) / kWarps), (unsigned)W), 256, 0, st>>>(pa);
    NA(cudaGetLastError());
    transpose_kernel<<<dim3((unsigned)((Lc + kTransK - 1) / kTransK), (unsigned)(Npad / 32)), dim3(32, 8), 0, st>>>(
        pa.cc, S + kNaCCT, N, Lc, Npad);
    NA(cudaGetLastError());
  }
  uint32_t h_evc[kNaMaxN], h_evoff[kNaMaxN + 1];
  NA(cudaMemcpyAsync(h_evc, pa.evcount, N * sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
  NA(cudaStreamSynchronize(st));
  h_evoff[0] = 0;
  uint32_t max_ev = 0;
  for (long i = 0; i < N; i++) {
    h_evoff[i + 1] = h_evoff[i] + h_evc[i];
    max_ev = std::max(max_ev, h_evc[i]);
  }
  rc.packed = max_ev <= (uint32_t)kPackedMaxEvents;
  NA(cudaMemcpyAsync(S + kNaEvoff, h_evoff, (N + 1) * sizeof(uint32_t), cudaMemcpyHostToDevice, st));
  if (W && h_evoff[N]) {
    events_kernel<<<(unsigned)((N + kWarps - 1) / kWarps), 256, 0, st>>>(pa);
    NA(cudaGetLastError());
  }
  build_tables(&g_na_tables, opts->mode, opts->subset);
  fill_pair_tables(g_na_tables, rc.wplane, &g_na_ptab);
  NA(cudaMemcpyAsync(S + kNaAgg, &g_na_ptab, sizeof(PairTables), cudaMemcpyHostToDevice, st));
  NA(cudaMemcpyAsync(S + kNaSite, g_na_tables.site, sizeof(g_na_tables.site), cudaMemcpyHostToDevice, st));
  unsigned *rqn = (unsigned *)(S + kNaRqn);
  unsigned long long *counters = (unsigned long long *)(S + kNaCounters);
  NA(cudaMemsetAsync(rqn, 0, sizeof(unsigned), st));
  NA(cudaMemsetAsync(counters, 0, 4 * sizeof(unsigned long long), st));
  PairArgs A;
  A.rc = rc;
  A.planes = pa.planes;
  A.cc = pa.cc;
  A.ccT = S + kNaCCT;
  A.ev_off = pa.ev_off;
  A.ev = pa.ev;
  A.tab = (const PairTables *)(S + kNaAgg);
  A.r0 = 0;
  A.r1 = N;
  A.ncols = N;
  A.colbase = 0;
  A.cstart = 0;
  A.cend = N;
  A.dist = d_dist;
  A.replay_q = (unsigned long long *)(S + kNaRq);
  A.replay_n = rqn;
  A.replay_cap = (unsigned long long)kNaMaxN * kNaMaxN;
  A.counters = counters;
  A.logt = (const LogTable *)(S + kNaLog);
  memset(&A.ex, 0, sizeof A.ex);  // raw distances only: no undecided list, no summary bounds
  NA(launch_pair(A, (N + 31) / 32, N, 0 /* the fused kernel's grid does not use it */, st));
  unsigned nq = 0;
  NA(cudaMemcpyAsync(&nq, rqn, sizeof nq, cudaMemcpyDeviceToHost, st));
  NA(cudaStreamSynchronize(st));
  if (nq) {
    ReplayArgs R;
    R.rc = rc;
    R.cc = pa.cc;
    R.planes = pa.planes;
    R.site = (const SiteEntry *)(S + kNaSite);
    R.q = A.replay_q;
    R.qn = rqn;
    R.qcap = A.replay_cap;
    R.r0 = 0;
    R.ncols = N;
    R.colbase = 0;
    R.dist = d_dist;
    R.counters = counters;
    R.logt = A.logt;
    R.ex = A.ex;
    replay_kernel<<<(unsigned)std::min<unsigned>(296, (nq + kWarps - 1) / kWarps), 256, 0, st>>>(R);
    NA(cudaGetLastError());
  }
  NA(cudaStreamSynchronize(st));
  return TN93G_OK;
#undef NA
}

}  // namespace

extern "C" {

int tn93g_pair_distances_noalloc(const uint8_t *d_codes, long N, long L, const tn93g_opts *opts, double *d_dist,
                                 void *stream)
{
  if (!d_codes || !opts || !d_dist || N <= 0 || L <= 0) {
    snprintf(g_na_err, sizeof g_na_err, "invalid argument: a null pointer or a size <= 0 (N = %ld, L = %ld)", N, L);
    return TN93G_EINVAL;
  }
  if (opts->mode < 0 || opts->mode > 4) {
    snprintf(g_na_err, sizeof g_na_err, "invalid argument: ambiguity mode %d", opts->mode);
    return TN93G_EINVAL;
  }
  g_na_err[0] = 0;
  std::lock_guard<std::mutex> g(g_na_mu);
  if (N > kNaMaxN || L > kNaMaxL) {
    snprintf(g_na_err, sizeof g_na_err,
             "alignment of %ld x %ld exceeds the fixed scratch of the allocation-free entry point (N <= %ld, L <= %ld)",
             N, L, kNaMaxN, kNaMaxL);
    return TN93G_ESCRATCH;
  }
  return noalloc_run(d_codes, N, L, opts, d_dist, (cudaStream_t)stream);
}

const char *tn93g_noalloc_last_error(void) { return g_na_err; }

}  // extern "C"

//================================================================================================== resident-reference server
// The -s mode as a service: a reference alignment stays packed on the device (bit planes, codes, sparse events,
// with room after it for query sequences) and batches of query alignments are run against it. One batch is one
// cross run (rows = reference, columns = the batch's queries, as tn93 -s QUERY REF orders them,
// swifttn93.cpp:2321-2322, 2392) whose stats, sums and text are segmented by query, so every query gets the
// distance file and summary of its own tn93 run. Columns are not folded (a fold must hold for every query that
// will ever come), which changes no result.
namespace {

// Server rows: one thread per (reference row, query). The 256 threads of a block are 256 consecutive rows of one
// query, so a warp walks the query's columns together (warp-uniform loop) while each thread adds its row's terms
// in column order, the order tn93 adds a row's pairs in (swifttn93.cpp:2594-2602). Statistics and row sums are
// fused; the histogram is aggregated per warp (lanes with the same bin add once) and per block in shared memory.
__global__ void __launch_bounds__(256) qstats_kernel(RowArgs a)
{
  __shared__ unsigned long long sh[kHistBins];
  for (int t = threadIdx.x; t < kHistBins; t += blockDim.x) sh[t] = 0;
  __syncthreads();
  const RunConsts &rc = a.rc;
  const int q = blockIdx.y;
  const long i = a.r0 + blockIdx.x * 256l + threadIdx.x;
  const bool row = i < a.r1;
  const long c0 = a.seg_cols[q], c1 = a.seg_cols[q + 1], jshift = c0 - rc.n1;
  const long ii = row ? i : a.r0;
  const long cnt_i = a.counts[ii];
  const int nli = a.name_len[ii];
  const int dli = rc.format == 1 ? digits_of(ii) : 0;
  double mx = 0., s0 = 0., w0 = 0.;
  long long links = 0, skipped = 0;
  unsigned long long bytes = 0;
  // A thread's distances lie next to each other, its neighbours' a row apart: four are loaded together (a 32-byte sector),
  // before any is used (40 queries x 30,000 rows: 510 us one at a time, 446 us so).
  double raw[4];
  for (long j = c0; j < c1; j++) {
    const int at = (int)(j - c0) & 3;
    if (at == 0)
#pragma unroll
      for (int k = 0; k < 4; k++) raw[k] = j + k < c1 ? raw_pair(a, ii, j + k) : 0.;
    PairView v = view_pair(a, ii, j, cnt_i, at == 0 ? raw[0] : at == 1 ? raw[1] : at == 2 ? raw[2] : raw[3]);
    if (!row) v.valid = v.computed = v.linked = false;
    const int key = v.computed ? v.hb : -1;
    const unsigned peers = __match_any_sync(0xffffffffu, key);
    if (__all_sync(0xffffffffu, !v.computed || v.w == 1)) {
      if (v.computed && (threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&sh[key], (unsigned long long)__popc(peers));
    } else if (v.computed) {
      atomicAdd(&sh[key], (unsigned long long)v.w);
    }
    if (!v.valid) continue;
    if (v.linked) {
      links += v.w;
      if (rc.emit) {
        const int gl = fmt_g_len(v.thisD);
        bytes += rc.format == 0 ? nli + a.name_len[j] + gl + 3 : dli + digits_of(j - jshift) + gl + 3;
      }
    }
    if (!v.counted) {
      skipped++;
    } else {
      mx = v.thisD > mx ? v.thisD : mx;
      s0 = __dadd_rn(s0, __dmul_rn(v.thisD, (double)v.w));
      w0 = __dadd_rn(w0, (double)v.w);
    }
  }
  if (row) {
    const size_t slot = (size_t)q * a.nrows + (i - a.r0);
    a.seg_bytes[slot] = bytes;
    a.seg_links[slot] = links;
    a.seg_skip[slot] = skipped;
    a.seg_max[slot] = mx;  // one word a slot here: a batch has one histogram bin
    a.row_sum[slot] = s0;
    a.row_w[slot] = w0;
  }
  __syncthreads();
  unsigned long long *hist = a.hist + (size_t)q * 3 * kHistBins;
  for (int t = threadIdx.x; t < kHistBins; t += blockDim.x)
    if (sh[t]) atomicAdd(&hist[t], sh[t]);
}

// Server text: one thread per (reference row, query) writes that row's lines for the query's columns at its
// scanned offset (the text is sparse at serving thresholds, so direct byte stores suffice).
__global__ void __launch_bounds__(256) qwrite_kernel(RowArgs a)
{
  const RunConsts &rc = a.rc;
  const int q = blockIdx.y;
  const long i = a.r0 + blockIdx.x * 256l + threadIdx.x;
  if (i >= a.r1) return;
  const size_t slot = (size_t)q * a.nrows + (i - a.r0);
  const unsigned long long nb = a.seg_bytes[slot];
  if (nb == 0) return;
  const long c0 = a.seg_cols[q], c1 = a.seg_cols[q + 1], jshift = c0 - rc.n1;
  const int nli = a.name_len[i];
  const char *ni = a.names + a.name_off[i];
  const int dli = rc.format == 1 ? digits_of(i) : 0;
  char *o = a.out + a.seg_off[slot], *const end = o + nb;
  for (long j = c0; j < c1; j++) {
    double thisD = 0.;
    if (!linked_pair(a, i, j, thisD)) continue;
    char g[24];
    const int gl = fmt_g(thisD, g);
    const int len = rc.format == 0 ? nli + a.name_len[j] + gl + 3 : dli + digits_of(j - jshift) + gl + 3;
    if (o + len > end) {
      atomicAdd(a.err, 1ull);
      return;
    }
    put_line(o, a, i, j, jshift, ni, nli, g, gl);
    o += len;
  }
  if (o != end) atomicAdd(a.err, 1ull);
}

// Per query: links, skips and maxima over the reference rows, and tn93's mean numerator and weight: the rows' sums
// added in row order, as tn93's writer adds them (swifttn93.cpp:2838-2848). One block per query. Only bin 0 is used in a
// server batch (no -m).
__global__ void __launch_bounds__(512) query_reduce_kernel(RowArgs a, int nq, double *qout /* [nq][9] */,
                                                           long long *qlinks /* [nq][3]: links, skips, text offset */)
{
  __shared__ long long rl[16], rs[16];
  __shared__ double rm[16];
  const int q = blockIdx.x;
  const long nr = a.nrows;
  const size_t base = (size_t)q * nr;
  double *o = qout + (size_t)q * 9;
  long long links = 0, skipped = 0;
  double m = 0., w = 0.;
  bool whole = true;
#pragma unroll 4
  for (long r = threadIdx.x; r < nr; r += 512) {
    links += a.seg_links[base + r];
    skipped += a.seg_skip[base + r];
    m = fmax(m, a.seg_max[base + r]);
    const double x = a.row_w[base + r];
    whole &= x >= 0. && x == floor(x);
    w = __dadd_rn(w, x);
  }
  chain_weights<512, 1>(a.row_w + base, nr, w, whole, o + 6);
  chain_rows<512, 1>(a.row_sum + base, nr, o + 3);
  for (int o = 16; o; o >>= 1) {
    links += __shfl_xor_sync(0xffffffffu, links, o);
    skipped += __shfl_xor_sync(0xffffffffu, skipped, o);
    m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  }
  if ((threadIdx.x & 31) == 0) {
    rl[threadIdx.x >> 5] = links;
    rs[threadIdx.x >> 5] = skipped;
    rm[threadIdx.x >> 5] = m;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 16; w++) {
      links += rl[w];
      skipped += rs[w];
      m = fmax(m, rm[w]);
    }
    o[0] = m;
    o[1] = o[2] = 0.;
    o[4] = o[5] = 0.;
    o[7] = o[8] = 0.;
    qlinks[q * 3] = links;
    qlinks[q * 3 + 1] = skipped;
    qlinks[q * 3 + 2] = (long long)a.seg_off[base];
  }
}

}  // namespace

struct tn93g_server {
  tn93g_ctx *ctx = nullptr;
  RunConsts base;
  long Nref = 0, L = 0, W = 0, Npad = 0, cap_q = 0;
  int cap_nq = 0;
  size_t ev_ref = 0, ev_cap = 0, names_ref = 0;
  DevBuf planes, cc, ccT, evcount, evoff, ev, ev2, three, agg, site, varcol, qcodes, counts, names, name_off, name_len, dist, rq,
      rqn, counters, segcols, sbytes, soff, slinks, sskip, smax, rsum, rw, hist, total, out, qout, qlinks, scantmp;
  void *pin = nullptr;
  size_t pin_n = 0;
  // tensor-core counts: the one-hot image of the reference and the batch's queries, and the aggregates of one
  // chunk of query columns at a time
  bool tc = false;
  bool lin = false;  // the records hold the ambiguity codes (average, gapmm, skip)
  int tc16 = 0;
  long tc_NB = 0, tc_KS = 0, tc_chunk = 0;
  DevBuf ohimg, tcagg, tcerr;
  void *hstat = nullptr;  // a batch's statistics in host memory that the device maps
  size_t hstat_n = 0;
  // exactness: the undecided list (capacity und_cap entries; grown for an exact-sums pass), its count, the
  // per-query bounds, the query of each column, the replay descriptor the resolver reads
  DevBuf und, undn, amb, colunit, rdesc;
  unsigned und_cap = 0;
  uint32_t ref_max_ev = 0;  // most sparse events of a reference sequence (the packed sums need <= kPackedMaxEvents)
};

namespace {
// Query columns per chunk of the tensor-core records (counts, events, formula), a multiple of 64; chunks end on the count
// kernel's 64-column tiles, so the first one is up to 63 columns narrower, and the pair stage stops where the counts do
// (PairArgs::cend). 40 queries (1,280 columns) against 30,000 sequences, pair stage: 5.03 ms with chunks of 128 from the
// reference's last row (three 64-column tiles each), 3.91 so.
constexpr long kServerTcChunk = 512, kServerTcChunkMin = 128;

// bytes of the records of a chunk of cols query columns
size_t server_records(const tn93g_server *srv, long cols) { return (size_t)srv->Nref * cols * (srv->tc16 ? 16 : 32); }

// The events' offsets and the larger chunk of records go back to the context. Should the smallest chunk, taken out of what
// the larger one gave back, fail all the same, the server counts with POPC from then on (same results).
void server_reclaim(tn93g_server *srv)
{
  tn93g_ctx *ctx = srv->ctx;
  release(ctx, srv->ev2);
  if (!srv->tc || srv->tc_chunk <= kServerTcChunkMin) return;
  release(ctx, srv->tcagg);
  srv->tc_chunk = kServerTcChunkMin;
  srv->tc = ensure(ctx, srv->tcagg, server_records(srv, kServerTcChunkMin), true) == TN93G_OK;
}

// words of the statistics of a batch of nq queries: total, undecided, counters, error word, and per query 9 sums, 3 counts,
// 4 bounds and the histogram
size_t server_stats(size_t nq) { return 7 + nq * (9 + 3 + 4 + 3 * kHistBins); }

// opt-in to the count kernel's dynamic shared memory on the current device
int tc_attr(tn93g_ctx *ctx)
{
  CU(tc_attr_once());
  return TN93G_OK;
}
}  // namespace

extern "C" {

void tn93g_server_destroy(tn93g_server *srv)
{
  if (!srv) return;
  tn93g_ctx *ctx = srv->ctx;
  if (ctx) cudaSetDevice(ctx->device);
  DevBuf *bufs[] = {&srv->planes, &srv->cc, &srv->ccT, &srv->evcount, &srv->evoff, &srv->ev, &srv->ev2, &srv->three, &srv->agg, &srv->site,
                    &srv->varcol, &srv->qcodes, &srv->counts, &srv->names, &srv->name_off, &srv->name_len,
                    &srv->dist, &srv->rq, &srv->rqn, &srv->counters, &srv->segcols, &srv->sbytes, &srv->soff,
                    &srv->slinks, &srv->sskip, &srv->smax, &srv->rsum, &srv->rw, &srv->hist, &srv->total,
                    &srv->out, &srv->qout, &srv->qlinks, &srv->scantmp, &srv->ohimg, &srv->tcagg, &srv->tcerr,
                    &srv->und, &srv->undn, &srv->amb, &srv->colunit, &srv->rdesc};
  for (DevBuf *b : bufs)
    if (b->p) {
      cudaFree(b->p);
      if (ctx) ctx->used -= b->n;
    }
  if (srv->pin) cudaFreeHost(srv->pin);
  if (srv->hstat) cudaFreeHost(srv->hstat);
  if (ctx) ctx->servers.erase(std::remove(ctx->servers.begin(), ctx->servers.end(), srv), ctx->servers.end());
  delete srv;
}

int tn93g_server_create(tn93g_ctx *ctx, tn93g_server **out, const uint8_t *codes, long N, long L,
                        const long *copy_counts, const char *names, const size_t *name_off, const long *name_len,
                        const tn93g_opts *opts, long max_batch_sequences, int max_batch_queries)
{
  if (!ctx || !out || !codes || N <= 0 || L <= 0 || !copy_counts || !names || !name_off || !name_len || !opts ||
      max_batch_sequences <= 0 || max_batch_queries <= 0 || max_batch_queries > 65535)
    return TN93G_EINVAL;
  if (opts->mode < 0 || opts->mode > 4 || opts->format < 0 || opts->format > 1) return TN93G_EINVAL;
  if (L >= (1l << 25) || N > 65535l * 32 || (unsigned long)(N + max_batch_sequences) * (unsigned long)L >= (1ul << 32))
    return TN93G_ETOOBIG;
  *out = nullptr;
  cudaSetDevice(ctx->device);
  cudaStream_t st = ctx->stream;
  tn93g_server *srv = new tn93g_server();
  srv->ctx = ctx;
  int rc_ = TN93G_OK;
#define SV(x)                   \
  do {                          \
    rc_ = (x);                  \
    if (rc_ != TN93G_OK) {      \
      tn93g_server_destroy(srv); \
      return rc_;               \
    }                           \
  } while (0)
#define SVC(call)                                                     \
  do {                                                                \
    cudaError_t e_ = (call);                                          \
    if (e_ != cudaSuccess) {                                          \
      ctx->err = std::string(#call) + ": " + cudaGetErrorString(e_);  \
      tn93g_server_destroy(srv);                                      \
      return TN93G_ECUDA;                                             \
    }                                                                 \
  } while (0)
  RunConsts &rc = srv->base;
  memset(&rc, 0, sizeof rc);
  rc.mode = opts->mode;
  rc.gapmm = opts->mode == TN93G_GAPMM;
  rc.cross = true;
  rc.fallback_avg = (opts->mode == TN93G_RESOLVE || opts->mode == TN93G_SUBSET) && opts->resolve_fraction < 1.;
  rc.emit = !opts->count_only;
  rc.format = opts->format;
  rc.delim = opts->delimiter;
  rc.threshold = opts->threshold;
  rc.min_distance = opts->min_distance;
  rc.resolve_fraction = opts->resolve_fraction;
  rc.min_overlap = opts->min_overlap;
  rc.log_band = ctx->log_band;
  rc.log_spread = ctx->log_spread;
  rc.resolve_all = ctx->exact_sums;
  srv->Nref = N;
  srv->L = L;
  srv->W = (L + 63) / 64;
  srv->cap_q = max_batch_sequences;
  srv->cap_nq = max_batch_queries;
  srv->Npad = (N + max_batch_sequences + 63) / 32 * 32;
  const long cap_n = N + max_batch_sequences, Np = srv->Npad, W = srv->W;
  rc.Lc = L;
  rc.W = W;
  rc.Npad = Np;
  rc.NP = rc.gapmm ? 5 : 4;
  // the reference's codes, its N count (the N plane is used when N is frequent, as in tn93g_run)
  SV(ensure(ctx, srv->qcodes, std::max<size_t>((size_t)N, (size_t)max_batch_sequences) * L));
  SVC(cudaMemcpyAsync(srv->qcodes.p, codes, (size_t)N * L, cudaMemcpyHostToDevice, st));
  SV(ensure(ctx, ctx->seen, L * sizeof(uint32_t)));
  SV(ensure(ctx, ctx->nN, sizeof(unsigned long long)));
  SVC(cudaMemsetAsync(ctx->seen.p, 0, L * sizeof(uint32_t), st));
  SVC(cudaMemsetAsync(ctx->nN.p, 0, sizeof(unsigned long long), st));
  colscan_kernel<<<dim3((unsigned)((L + 255) / 256), (unsigned)((N + 63) / 64)), 256, 0, st>>>(
      (const uint8_t *)srv->qcodes.p, N, L, (uint32_t *)ctx->seen.p, (unsigned long long *)ctx->nN.p);
  SVC(cudaGetLastError());
  unsigned long long nN = 0;
  SVC(cudaMemcpyAsync(&nN, ctx->nN.p, sizeof nN, cudaMemcpyDeviceToHost, st));
  SVC(cudaStreamSynchronize(st));
  rc.wplane = rc.gapmm || nN > 16ull * (unsigned long long)N;
  // resident arrays with room for max_batch_sequences query sequences after the reference
  SV(ensure(ctx, srv->planes, (size_t)W * rc.NP * Np * sizeof(uint64_t)));
  SV(ensure(ctx, srv->cc, (size_t)cap_n * L + 8));
  SV(ensure(ctx, srv->ccT, (size_t)L * Np));
  SV(ensure(ctx, srv->evcount, cap_n * sizeof(uint32_t)));
  SV(ensure(ctx, srv->evoff, (cap_n + 1) * sizeof(uint32_t)));
  SV(ensure(ctx, srv->three, cap_n));
  SV(ensure(ctx, srv->varcol, L * sizeof(int32_t)));
  SVC(cudaMemsetAsync(srv->planes.p, 0, (size_t)W * rc.NP * Np * sizeof(uint64_t), st));
  SVC(cudaMemsetAsync(srv->evcount.p, 0, cap_n * sizeof(uint32_t), st));
  SVC(cudaMemsetAsync(srv->three.p, 0, cap_n, st));
  SVC(cudaMemsetAsync(srv->ccT.p, kGap, (size_t)L * Np, st));  // slots past the batch read as gaps
  {
    std::vector<int32_t> id(L);
    for (long p = 0; p < L; p++) id[p] = (int32_t)p;
    SVC(cudaMemcpy(srv->varcol.p, id.data(), L * sizeof(int32_t), cudaMemcpyHostToDevice));
  }
  PackArgs pa;
  pa.codes = (const uint8_t *)srv->qcodes.p;
  pa.N = N;
  pa.L = L;
  pa.Lc = L;
  pa.W = W;
  pa.Npad = Np;
  pa.varcol = (const int32_t *)srv->varcol.p;
  pa.NP = rc.NP;
  pa.wplane = rc.wplane;
  pa.gapmm = rc.gapmm;
  pa.planes = (uint64_t *)srv->planes.p;
  pa.cc = (uint8_t *)srv->cc.p;
  pa.evcount = (uint32_t *)srv->evcount.p;
  pack_kernel<<<dim3((unsigned)((N + kWarps - 1) / kWarps), (unsigned)std::min<long>(W, 65535)), 256, 0, st>>>(pa);
  SVC(cudaGetLastError());
  transpose_kernel<<<dim3((unsigned)((L + kTransK - 1) / kTransK), (unsigned)((N + 31) / 32)), dim3(32, 8), 0, st>>>(
      (const uint8_t *)srv->cc.p, (uint8_t *)srv->ccT.p, N, L, Np);
  SVC(cudaGetLastError());
  std::vector<uint32_t> evc(N), evo(N + 1);
  SVC(cudaMemcpyAsync(evc.data(), srv->evcount.p, N * sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
  SVC(cudaStreamSynchronize(st));
  for (long i = 0; i < N; i++) {
    evo[i] = (uint32_t)srv->ev_ref;
    srv->ev_ref += pad_events(evc[i]);
    srv->ref_max_ev = std::max(srv->ref_max_ev, evc[i]);
  }
  srv->ev_cap = srv->ev_ref + (size_t)max_batch_sequences * ((L + kEvPad - 1) / kEvPad * kEvPad);
  if (srv->ev_cap >= (1ull << 32)) SV(TN93G_ETOOBIG);  // 32-bit offsets
  evo[N] = (uint32_t)srv->ev_ref;
  SV(ensure(ctx, srv->ev, std::max<size_t>(srv->ev_cap, 1) * sizeof(uint32_t)));
  SVC(cudaMemcpyAsync(srv->evoff.p, evo.data(), (N + 1) * sizeof(uint32_t), cudaMemcpyHostToDevice, st));
  // tables of the server's mode
  build_tables(ctx->h_tab, opts->mode, opts->subset);
  fill_pair_tables(*ctx->h_tab, rc.wplane, ctx->h_ptab);
  SV(ensure(ctx, srv->agg, sizeof(PairTables)));
  SV(ensure(ctx, srv->site, sizeof(ctx->h_tab->site)));
  SVC(cudaMemcpyAsync(srv->agg.p, ctx->h_ptab, sizeof(PairTables), cudaMemcpyHostToDevice, st));
  SVC(cudaMemcpyAsync(srv->site.p, ctx->h_tab->site, sizeof(ctx->h_tab->site), cudaMemcpyHostToDevice, st));
  // names, name offsets and lengths, copy numbers of every sequence (the reference's now, the queries' per batch)
  size_t nbytes = 0;
  for (long i = 0; i < N; i++) nbytes = std::max(nbytes, name_off[i] + (size_t)name_len[i]);
  srv->names_ref = nbytes;
  SV(ensure(ctx, srv->names, nbytes + 1 + (size_t)max_batch_sequences * 64));
  SV(ensure(ctx, srv->name_off, cap_n * sizeof(uint64_t)));
  SV(ensure(ctx, srv->name_len, cap_n * sizeof(int32_t)));
  SV(ensure(ctx, srv->counts, cap_n * sizeof(long)));
  std::vector<uint64_t> off(name_off, name_off + N);
  std::vector<int32_t> nl(N);
  for (long i = 0; i < N; i++) nl[i] = (int32_t)name_len[i];
  if (nbytes) SVC(cudaMemcpyAsync(srv->names.p, names, nbytes, cudaMemcpyHostToDevice, st));
  SVC(cudaMemcpyAsync(srv->name_off.p, off.data(), N * sizeof(uint64_t), cudaMemcpyHostToDevice, st));
  SVC(cudaMemcpyAsync(srv->name_len.p, nl.data(), N * sizeof(int32_t), cudaMemcpyHostToDevice, st));
  SVC(cudaMemcpyAsync(srv->counts.p, copy_counts, N * sizeof(long), cudaMemcpyHostToDevice, st));
  // per-batch buffers at capacity (a batch never reallocates them): distances and the replay queue of every
  // pair, per (query, row) statistics, per-query histograms and results
  {
    const size_t dslots = (size_t)N * max_batch_sequences, nslot = (size_t)max_batch_queries * N;
    const int nq = max_batch_queries;
    SV(ensure(ctx, srv->dist, dslots * sizeof(double)));
    SV(ensure(ctx, srv->rq, dslots * sizeof(unsigned long long)));
    SV(ensure(ctx, srv->rqn, sizeof(unsigned)));
    SV(ensure(ctx, srv->counters, 4 * sizeof(unsigned long long)));
    SV(ensure(ctx, srv->sbytes, nslot * sizeof(unsigned long long)));
    SV(ensure(ctx, srv->soff, nslot * sizeof(unsigned long long)));
    SV(ensure(ctx, srv->slinks, nslot * sizeof(long long)));
    SV(ensure(ctx, srv->sskip, nslot * sizeof(long long)));
    SV(ensure(ctx, srv->smax, nslot * sizeof(double)));
    SV(ensure(ctx, srv->rsum, nslot * sizeof(double)));
    SV(ensure(ctx, srv->rw, nslot * sizeof(double)));
    SV(ensure(ctx, srv->hist, (size_t)nq * 3 * kHistBins * sizeof(unsigned long long)));
    SV(ensure(ctx, srv->total, sizeof(unsigned long long)));
    SV(ensure(ctx, srv->segcols, (nq + 1) * sizeof(long)));
    SV(ensure(ctx, srv->qout, (size_t)nq * 9 * sizeof(double)));
    SV(ensure(ctx, srv->qlinks, (size_t)nq * 3 * sizeof(long long)));
    SV(ensure_pinned_at(ctx, srv->hstat, srv->hstat_n, server_stats(nq) * sizeof(unsigned long long), cudaHostAllocMapped));
    SV(ensure(ctx, srv->scantmp, (2 * (nslot / kScanTile + 1) + 1) * sizeof(unsigned long long)));
    srv->und_cap = (unsigned)std::min<size_t>(std::max<size_t>(4096, dslots / 64), 0xFFFFFFF0u);
    SV(ensure(ctx, srv->und, (size_t)srv->und_cap * 2 * sizeof(unsigned long long)));
    SV(ensure(ctx, srv->undn, sizeof(unsigned long long)));
    SV(ensure(ctx, srv->amb, (size_t)nq * 4 * sizeof(unsigned long long)));
    SV(ensure(ctx, srv->colunit, (size_t)max_batch_sequences * sizeof(int)));
    SV(ensure(ctx, srv->rdesc, sizeof(ReplayArgs)));
    // a first text buffer (device and pinned host), so that early batches do not stall on growth
    const size_t text0 = 32u << 20;
    SV(ensure(ctx, srv->out, text0));
    SVC(cudaHostAlloc(&srv->pin, text0, cudaHostAllocDefault));
    srv->pin_n = text0;
  }
  // tensor-core counts (the context's count path): the reference's blocks of the one-hot image now, the blocks
  // holding queries per batch; when the budget cannot hold the image and one chunk of aggregates, the server
  // counts with POPC instead (same results)
  if (ctx->count_path == 1) {
    srv->tc_NB = (N + max_batch_sequences + 31) / 32 + 1;
    srv->tc_KS = (L + kTcStageK - 1) / kTcStageK;
    srv->tc16 = 32 * L < 65536;
    const size_t img = (size_t)srv->tc_KS * srv->tc_NB * kTcBlockBytes;
    // a chunk that holds the largest batch from any first column, or the smallest one where that does not fit
    srv->tc_chunk = std::min<long>(kServerTcChunk, std::max(kServerTcChunkMin, (max_batch_sequences + 127) / 64 * 64));
    const bool room = ensure(ctx, srv->ohimg, img) == TN93G_OK && ensure(ctx, srv->tcerr, sizeof(unsigned long long)) == TN93G_OK;
    if (room && ensure(ctx, srv->tcagg, server_records(srv, srv->tc_chunk), true) != TN93G_OK) srv->tc_chunk = kServerTcChunkMin;
    if (room && ensure(ctx, srv->tcagg, server_records(srv, srv->tc_chunk)) == TN93G_OK) {
      srv->tc = true;
      srv->lin = weighted_mode(opts->mode);
      SV(tc_attr(ctx));
      const long nfull = N / 32 * 32;  // whole reference blocks (the block shared with queries is built per batch)
      if (nfull) {
        const long nthr = nfull * srv->tc_KS * (kTcStageK / 16);
        onehot_kernel<<<(unsigned)((nthr + 255) / 256), 256, 0, st>>>((const uint8_t *)srv->cc.p, N, L, srv->tc_NB,
                                                                      srv->tc_KS, (uint8_t *)srv->ohimg.p, 0, nfull,
                                                                      tc_classes(opts->mode, srv->lin));
        SVC(cudaGetLastError());
      }
    } else {
      for (DevBuf *b : {&srv->ohimg, &srv->tcagg, &srv->tcerr}) release(ctx, *b);
      ctx->err.clear();
    }
  }
  // the events again as event_kernel reads them, where the pair stage takes it (pair_split) and there is room
  if (srv->tc && !srv->lin && !rc.wplane && srv->ref_max_ev <= (uint32_t)kPackedMaxEvents && L * Np < (1l << 32)) {
    const int r = ensure(ctx, srv->ev2, std::max<size_t>(srv->ev_cap, 1) * sizeof(uint2), true);
    if (r != TN93G_ENOMEM) SV(r);
  }
  pa.ev_off = (const uint32_t *)srv->evoff.p;
  pa.ev = (uint32_t *)srv->ev.p;
  pa.ev2 = (uint2 *)srv->ev2.p;
  pa.ev2_Npad = (uint32_t)Np;
  pa.three = (uint8_t *)srv->three.p;
  if (srv->ev_ref) {
    events_kernel<<<(unsigned)((N + kWarps - 1) / kWarps), 256, 0, st>>>(pa);
    SVC(cudaGetLastError());
  }
  SVC(cudaStreamSynchronize(st));
  ctx->servers.push_back(srv);
#undef SV
#undef SVC
  *out = srv;
  return TN93G_OK;
}

int tn93g_server_batch(tn93g_server *srv, int nq, const tn93g_alignment *queries, tn93g_query_sink sink, void *user,
                       tn93g_summary *sums)
{
  if (!srv || nq <= 0 || !queries || !sums) return TN93G_EINVAL;
  tn93g_ctx *ctx = srv->ctx;
  cudaSetDevice(ctx->device);
  cudaStream_t st = ctx->stream;
  ctx->launches = 0;
  for (double &t : ctx->timings) t = 0;
  cudaEvent_t *E = ctx->evs;  // stage boundaries: start, packed, pair, replay, rows, written, copied
  const long Nref = srv->Nref, L = srv->L, Np = srv->Npad, W = srv->W;
  if (nq > srv->cap_nq) {
    ctx->err = "more queries than the server's batch capacity";
    return TN93G_EINVAL;
  }
  std::vector<long> qstart(nq + 1);
  qstart[0] = 0;
  for (int q = 0; q < nq; q++) {
    if (queries[q].n <= 0 || queries[q].L != srv->L || !queries[q].codes || !queries[q].copy_counts ||
        !queries[q].names || !queries[q].name_off || !queries[q].name_len)
      return TN93G_EINVAL;
    qstart[q + 1] = qstart[q] + queries[q].n;
  }
  const long Q = qstart[nq];
  if (Q > srv->cap_q) {
    ctx->err = "batch larger than the server's query capacity";
    return TN93G_EINVAL;
  }
  // query codes, names, offsets, lengths and copy numbers into the slots after the reference
  std::vector<uint64_t> off(Q);
  std::vector<int32_t> nl(Q);
  std::vector<long> cnt(Q);
  size_t nb = srv->names_ref;
  std::string qnames;  // the queries' names, one after the other
  for (int q = 0; q < nq; q++) {
    size_t qn = 0;
    for (long k = 0; k < queries[q].n; k++) qn = std::max(qn, queries[q].name_off[k] + (size_t)queries[q].name_len[k]);
    qnames.append(queries[q].names, qn);
    for (long k = 0; k < queries[q].n; k++) {
      off[qstart[q] + k] = nb + queries[q].name_off[k];
      nl[qstart[q] + k] = (int32_t)queries[q].name_len[k];
      cnt[qstart[q] + k] = queries[q].copy_counts[k];
    }
    nb += qn;
  }
  TRY(ensure_keep(ctx, srv->names, nb + 1, srv->names_ref));
  CU(cudaEventRecord(E[0], st));
  for (int q = 0; q < nq; q++) {
    CU(cudaMemcpyAsync((uint8_t *)srv->qcodes.p + (size_t)qstart[q] * L, queries[q].codes, (size_t)queries[q].n * L,
                       cudaMemcpyHostToDevice, st));
  }
  if (!qnames.empty())
    CU(cudaMemcpyAsync((char *)srv->names.p + srv->names_ref, qnames.data(), qnames.size(), cudaMemcpyHostToDevice, st));
  CU(cudaMemcpyAsync((uint64_t *)srv->name_off.p + Nref, off.data(), Q * sizeof(uint64_t), cudaMemcpyHostToDevice, st));
  CU(cudaMemcpyAsync((int32_t *)srv->name_len.p + Nref, nl.data(), Q * sizeof(int32_t), cudaMemcpyHostToDevice, st));
  CU(cudaMemcpyAsync((long *)srv->counts.p + Nref, cnt.data(), Q * sizeof(long), cudaMemcpyHostToDevice, st));
  // pack the queries into their slots
  RunConsts rc = srv->base;
  rc.N = Nref + Q;
  rc.n1 = Nref;
  PackArgs pa;
  pa.codes = (const uint8_t *)srv->qcodes.p;
  pa.N = Q;
  pa.L = L;
  pa.Lc = L;
  pa.W = W;
  pa.Npad = Np;
  pa.varcol = (const int32_t *)srv->varcol.p;
  pa.NP = rc.NP;
  pa.wplane = rc.wplane;
  pa.gapmm = rc.gapmm;
  pa.planes = (uint64_t *)srv->planes.p + Nref;
  pa.cc = (uint8_t *)srv->cc.p + (size_t)Nref * L;
  pa.evcount = (uint32_t *)srv->evcount.p + Nref;
  CU(cudaMemsetAsync(pa.evcount, 0, Q * sizeof(uint32_t), st));
  pack_kernel<<<dim3((unsigned)((Q + kWarps - 1) / kWarps), (unsigned)std::min<long>(W, 65535)), 256, 0, st>>>(pa);
  CU(cudaGetLastError());
  ctx->launches++;
  transpose_kernel<<<dim3((unsigned)((L + kTransK - 1) / kTransK), (unsigned)((Q + 31) / 32)), dim3(32, 8), 0, st>>>(
      pa.cc, (uint8_t *)srv->ccT.p + Nref, Q, L, Np);
  CU(cudaGetLastError());
  ctx->launches++;
  std::vector<uint32_t> evc(Q), evo(Q + 1);
  CU(cudaMemcpyAsync(evc.data(), pa.evcount, Q * sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
  CU(cudaStreamSynchronize(st));
  evo[0] = (uint32_t)srv->ev_ref;
  uint32_t max_ev = srv->ref_max_ev;
  for (long k = 0; k < Q; k++) {
    evo[k + 1] = evo[k] + pad_events(evc[k]);
    max_ev = std::max(max_ev, evc[k]);
  }
  rc.packed = max_ev <= (uint32_t)kPackedMaxEvents;
  CU(cudaMemcpyAsync((uint32_t *)srv->evoff.p + Nref, evo.data(), (Q + 1) * sizeof(uint32_t), cudaMemcpyHostToDevice,
                     st));
  pa.ev_off = (const uint32_t *)srv->evoff.p + Nref;
  pa.ev = (uint32_t *)srv->ev.p;
  pa.ev2 = (uint2 *)srv->ev2.p;
  pa.ev2_Npad = (uint32_t)Np;
  pa.three = (uint8_t *)srv->three.p + Nref;
  if (evo[Q] > evo[0]) {
    events_kernel<<<(unsigned)((Q + kWarps - 1) / kWarps), 256, 0, st>>>(pa);
    CU(cudaGetLastError());
    ctx->launches++;
  }
  CU(cudaEventRecord(E[1], st));
  // the cross run: rows = reference, columns = the batch's queries
  const size_t dslots = (size_t)Nref * Q;
  const size_t nslot = (size_t)nq * Nref;
  CU(cudaMemsetAsync(srv->counters.p, 0, 4 * sizeof(unsigned long long), st));
  CU(cudaMemsetAsync(srv->amb.p, 0, (size_t)nq * 4 * sizeof(unsigned long long), st));
  std::vector<long> segc(nq + 1);
  for (int q = 0; q <= nq; q++) segc[q] = Nref + qstart[q];
  CU(cudaMemcpyAsync(srv->segcols.p, segc.data(), (nq + 1) * sizeof(long), cudaMemcpyHostToDevice, st));
  {
    std::vector<int> cu(Q);
    for (int q = 0; q < nq; q++)
      for (long k = qstart[q]; k < qstart[q + 1]; k++) cu[k] = q;
    CU(cudaMemcpyAsync(srv->colunit.p, cu.data(), Q * sizeof(int), cudaMemcpyHostToDevice, st));
  }
  if (srv->tc) {
    // the image blocks from the one shared by the reference's last rows and the first queries, through one zero
    // block past the last query
    const long b0 = Nref / 32, b1 = (Nref + Q + 31) / 32 + 1;
    const long nthr = (b1 - b0) * 32 * srv->tc_KS * (kTcStageK / 16);
    CU(cudaMemsetAsync(srv->tcerr.p, 0, sizeof(unsigned long long), st));
    onehot_kernel<<<(unsigned)((nthr + 255) / 256), 256, 0, st>>>((const uint8_t *)srv->cc.p, Nref + Q, L, srv->tc_NB,
                                                                  srv->tc_KS, (uint8_t *)srv->ohimg.p, b0 * 32,
                                                                  (b1 - b0) * 32, tc_classes(rc.mode, srv->lin));
    CU(cudaGetLastError());
    ctx->launches++;
  }
  ReplayArgs R;
  // pair stage (and the site-order replay) of the whole batch; resolve_all: an exact-sums pass
  auto enqueue_pairs = [&](bool resolve_all) -> int {
    RunConsts rcp = rc;
    rcp.resolve_all = rc.resolve_all || resolve_all;
    CU(cudaMemsetAsync(srv->rqn.p, 0, sizeof(unsigned), st));
    CU(cudaMemsetAsync(srv->undn.p, 0, sizeof(unsigned long long), st));
    ExactSink ex;
    ex.und_list = (unsigned long long *)srv->und.p;
    ex.und_n = (unsigned *)srv->undn.p;
    ex.und_cap = srv->und_cap;
    ex.und_k = 0;
    ex.amb = resolve_all ? nullptr : (unsigned long long *)srv->amb.p;
    ex.counts = (const long *)srv->counts.p;
    ex.colunit = (const int *)srv->colunit.p;
    PairArgs A;
    A.rc = rcp;
    A.planes = (const uint64_t *)srv->planes.p;
    A.cc = (const uint8_t *)srv->cc.p;
    A.ccT = (const uint8_t *)srv->ccT.p;
    A.ev_off = (const uint32_t *)srv->evoff.p;
    A.ev = (const uint32_t *)srv->ev.p;
    A.ev2 = (const uint2 *)srv->ev2.p;
    A.three = rc.mode != TN93G_SKIP ? (const uint8_t *)srv->three.p : nullptr;
    A.lin = srv->tc && srv->lin;
    A.tab = (const PairTables *)srv->agg.p;
    A.r0 = 0;
    A.r1 = Nref;
    A.ncols = Q;
    A.colbase = Nref;
    A.cstart = Nref;
    A.cend = Nref + Q;
    A.dist = (double *)srv->dist.p;
    A.replay_q = (unsigned long long *)srv->rq.p;
    A.replay_n = (unsigned *)srv->rqn.p;
    A.replay_cap = dslots;
    A.counters = (unsigned long long *)srv->counters.p;
    A.logt = ctx->d_logt;
    A.ex = ex;
    if (srv->tc) {
      // per chunk of query columns: counts on the tensor cores, then the pair kernel
      for (long c0 = Nref, c1; c0 < Nref + Q; c0 = c1) {
        c1 = std::min(Nref + Q, c0 / kTcCols * kTcCols + srv->tc_chunk);
        TcArgs T;
        T.onehot = (const uint8_t *)srv->ohimg.p;
        T.NB = srv->tc_NB;
        T.KS = srv->tc_KS;
        T.N = Nref + Q;
        T.n1 = Nref;
        T.cross = true;
        T.r0 = 0;
        T.r1 = Nref;
        T.ncols = srv->tc_chunk;
        T.colbase = c0;
        T.cstart = c0 / kTcCols * kTcCols;
        T.cend = c1;
        T.agg = srv->tcagg.p;
        T.agg16 = srv->tc16;
        T.err = (unsigned long long *)srv->tcerr.p;
        T.wait_ns = ctx->wait_ns;
        T.skip_fill_block = -1;
        const dim3 g((unsigned)((c1 - T.cstart + kTcCols - 1) / kTcCols), (unsigned)((Nref + kTcRows - 1) / kTcRows));
        CU(launch_count_grid(T, g.x, g.y, ctx->sms, st));
        PairArgs AC = A;
        AC.tcagg = srv->tcagg.p;
        AC.tc16 = srv->tc16;
        AC.tcncols = srv->tc_chunk;
        AC.tccolbase = c0;
        AC.cstart = c0;
        AC.cend = c1;  // the records past it are the next chunk's, not counted yet
        CU(launch_pair(AC, (c1 - c0 + 31) / 32, Nref, ctx->sms, st));
        ctx->launches += pair_split(AC) && !AC.lin ? 3 : 2;
      }
    } else {
      CU(launch_pair(A, (Q + 31) / 32, Nref, ctx->sms, st));
      ctx->launches++;
    }
    CU(cudaEventRecord(E[2], st));
    R.rc = rcp;
    R.cc = A.cc;
    R.planes = A.planes;
    R.site = (const SiteEntry *)srv->site.p;
    R.ev_off = A.ev_off;
    R.ev = A.ev;
    R.q = A.replay_q;
    R.qn = A.replay_n;
    R.qcap = dslots;
    R.r0 = 0;
    R.ncols = Q;
    R.colbase = Nref;
    R.dist = A.dist;
    R.counters = A.counters;
    R.logt = ctx->d_logt;
    R.ex = ex;
    replay_kernel<<<2 * ctx->sms, 256, 0, st>>>(R);
    CU(cudaGetLastError());
    ctx->launches++;
    CU(cudaEventRecord(E[3], st));
    return TN93G_OK;
  };
  RowArgs RA;
  RA.rc = rc;
  RA.dist = (const double *)srv->dist.p;
  RA.r0 = 0;
  RA.r1 = Nref;
  RA.ncols = Q;
  RA.colbase = Nref;
  RA.counts = (const long *)srv->counts.p;
  RA.name_len = (const int32_t *)srv->name_len.p;
  RA.name_off = (const uint64_t *)srv->name_off.p;
  RA.names = (const char *)srv->names.p;
  RA.maxseg = nq;
  RA.seg_cols = (const long *)srv->segcols.p;
  RA.nrows = Nref;
  RA.seg_bytes = (unsigned long long *)srv->sbytes.p;
  RA.seg_links = (long long *)srv->slinks.p;
  RA.seg_skip = (long long *)srv->sskip.p;
  RA.seg_max = (double *)srv->smax.p;
  RA.row_sum = (double *)srv->rsum.p;
  RA.row_w = (double *)srv->rw.p;
  RA.hist = (unsigned long long *)srv->hist.p;
  RA.seg_off = (const unsigned long long *)srv->soff.p;
  RA.hy = nullptr;
  RA.err = (unsigned long long *)srv->counters.p + 3;
  RA.out = nullptr;
  const dim3 g2((unsigned)((Nref + 255) / 256), (unsigned)nq);
  unsigned long long total = 0, und = 0;
  std::vector<double> qo((size_t)nq * 9);
  std::vector<long long> ql((size_t)nq * 3);
  std::vector<unsigned long long> qoff(nq + 1), hist((size_t)nq * 3 * kHistBins), ambw((size_t)nq * 4);
  unsigned long long counters[4], tcerr = 0;
  // row stage (per-query statistics and row sums, scan, per-query reduction) and its results on the host
  auto rows_and_read = [&]() -> int {
    CU(cudaMemsetAsync(srv->hist.p, 0, (size_t)nq * 3 * kHistBins * sizeof(unsigned long long), st));
    qstats_kernel<<<g2, 256, 0, st>>>(RA);
    CU(cudaGetLastError());
    ctx->launches++;
    CU(launch_scan(RA.seg_bytes, (unsigned long long *)RA.seg_off, (long)nslot, (unsigned long long *)srv->total.p,
                   (unsigned long long *)srv->scantmp.p, st));
    ctx->launches++;
    query_reduce_kernel<<<(unsigned)nq, 512, 0, st>>>(RA, nq, (double *)srv->qout.p, (long long *)srv->qlinks.p);
    CU(cudaGetLastError());
    ctx->launches++;
    CU(cudaEventRecord(E[4], st));
    // the statistics to the host in one kernel (a copy of a few words to pageable memory takes about 10 us; there were
    // six of them and one a query: 0.5 ms for 40 queries)
    unsigned long long *dst = nullptr;
    CU(cudaHostGetDevicePointer((void **)&dst, srv->hstat, 0));
    Gather g;
    g.k = 0;
    auto add = [&](const void *src, size_t nwords) {
      g.src[g.k] = (const unsigned long long *)src;
      g.dst[g.k] = dst;
      g.stride[g.k] = 1;
      g.n[g.k++] = (long)nwords;
      dst += nwords;
    };
    add(srv->total.p, 1);
    add(srv->undn.p, 1);
    add(srv->counters.p, 4);
    if (srv->tc) add(srv->tcerr.p, 1);
    add(srv->qout.p, qo.size());
    add(srv->qlinks.p, ql.size());
    add(srv->amb.p, ambw.size());
    add(srv->hist.p, hist.size());
    gather_kernel<<<16, 256, 0, st>>>(g);
    CU(cudaGetLastError());
    ctx->launches++;
    CU(cudaStreamSynchronize(st));
    const unsigned long long *h = (const unsigned long long *)srv->hstat;
    auto take = [&](void *to, size_t nwords) {
      memcpy(to, h, nwords * sizeof *h);
      h += nwords;
    };
    take(&total, 1);
    take(&und, 1);
    take(counters, 4);
    if (srv->tc) take(&tcerr, 1);
    take(qo.data(), qo.size());
    take(ql.data(), ql.size());
    take(ambw.data(), ambw.size());
    take(hist.data(), hist.size());
    for (int q = 0; q < nq; q++) qoff[q] = (unsigned long long)ql[q * 3 + 2];
    return TN93G_OK;
  };
  // finishes the listed undecided pairs with the C library's logarithms and runs the row stage again
  long resolved = 0;
  auto resolve_and_reread = [&]() -> int {
    if (und > srv->und_cap) {
      ctx->err = "more undecided pairs in a batch than its list holds";
      return TN93G_EUNDECIDED;
    }
    CU(cudaMemcpyAsync(srv->rdesc.p, &R, sizeof R, cudaMemcpyHostToDevice, st));
    TRY(resolve_listed(ctx, (const ReplayArgs *)srv->rdesc.p, (const unsigned long long *)srv->und.p, (unsigned)und,
                       st));
    resolved += (long)und;
    return rows_and_read();
  };
  TRY(enqueue_pairs(false));
  TRY(rows_and_read());
  if (tcerr) {
    ctx->err = "the tensor-core count kernel timed out waiting for its pipeline";
    return TN93G_ETIMEOUT;
  }
  const long ambiguous0 = (long)counters[0];
  // more undecided pairs than the list holds: grow it and run the batch's pair stage again (the same pairs are
  // listed; the per-query bounds only widen)
  auto grow_and_rerun = [&](bool resolve_all) -> int {
    const unsigned cap = (unsigned)std::min<unsigned long long>(
        std::max<unsigned long long>(und + und / 4 + 1024, 2ull * srv->und_cap), std::min<size_t>(dslots, 0xFFFFFFF0u));
    TRY(ensure(ctx, srv->und, (size_t)cap * 2 * sizeof(unsigned long long)));
    srv->und_cap = cap;
    TRY(enqueue_pairs(resolve_all));
    return rows_and_read();
  };
  if (und > srv->und_cap) TRY(grow_and_rerun(false));
  if (und) TRY(resolve_and_reread());
  // per query: the JSON numbers certain for every rounding of the C library's log, or an exact-sums pass
  std::vector<tn93g_summary> S(nq);
  auto fill_summaries = [&]() {
    for (int q = 0; q < nq; q++) {
      tn93g_summary &X = S[q];
      memset(&X, 0, sizeof X);
      X.pairwise = (unsigned long)Nref * (unsigned long)queries[q].n;
      X.links = (long)ql[q * 3];
      X.skipped = (long)ql[q * 3 + 1];
      for (int k = 0; k < 3; k++) {
        X.max[k] = qo[q * 9 + k];
        X.mean[k] = qo[q * 9 + 3 + k];
        X.weighted[k] = qo[q * 9 + 6 + k];
        for (int b = 0; b < kHistBins; b++) X.hist[k][b] = hist[((size_t)q * 3 + k) * kHistBins + b];
      }
    }
  };
  fill_summaries();
  bool repass = false;
  for (int q = 0; q < nq && !rc.resolve_all; q++) {
    amb_bounds(&ambw[(size_t)q * 4], S[q].amb_bounds[0]);
    if (!summary_certified(&S[q], S[q].amb_bounds, Nref + queries[q].n + 2, 0)) repass = true;
  }
  if (repass) {
    // every pair with an ambiguous logarithm finished with the C library's log (the list must hold all of them)
    const unsigned cap = (unsigned)std::min<size_t>(dslots, 0xFFFFFFF0u);
    if (cap > srv->und_cap) {
      TRY(ensure(ctx, srv->und, (size_t)cap * 2 * sizeof(unsigned long long)));
      srv->und_cap = cap;
    }
    TRY(enqueue_pairs(true));
    TRY(rows_and_read());
    if (und > srv->und_cap) TRY(grow_and_rerun(true));
    if (und) TRY(resolve_and_reread());
    fill_summaries();
  }
  qoff[nq] = total;
  if (rc.emit && total) {
    if (srv->out.n < total) TRY(ensure(ctx, srv->out, total + total / 2));
    if (srv->pin_n < total) {
      if (srv->pin) cudaFreeHost(srv->pin);
      srv->pin = nullptr;
      srv->pin_n = 0;
      CU(cudaHostAlloc(&srv->pin, total + total / 4, cudaHostAllocDefault));
      srv->pin_n = total + total / 4;
    }
    RA.out = (char *)srv->out.p;
    qwrite_kernel<<<g2, 256, 0, st>>>(RA);
    CU(cudaGetLastError());
    ctx->launches++;
    CU(cudaEventRecord(E[5], st));
    CU(cudaMemcpyAsync(srv->pin, srv->out.p, total, cudaMemcpyDeviceToHost, st));
    CU(cudaMemcpyAsync(srv->hstat, (unsigned long long *)srv->counters.p + 3, sizeof(unsigned long long),
                       cudaMemcpyDeviceToHost, st));
    CU(cudaEventRecord(E[6], st));
    CU(cudaStreamSynchronize(st));
    memcpy(&counters[3], srv->hstat, sizeof counters[3]);
    float ms = 0.f;
    CU(cudaEventElapsedTime(&ms, E[4], E[5]));
    ctx->timings[4] = ms;
    CU(cudaEventElapsedTime(&ms, E[5], E[6]));
    ctx->timings[5] = ms;
    CU(cudaEventElapsedTime(&ms, E[0], E[6]));
    ctx->timings[6] = ms;
  } else {
    float ms = 0.f;
    CU(cudaEventElapsedTime(&ms, E[0], E[4]));
    ctx->timings[6] = ms;
  }
  {
    float ms = 0.f;
    CU(cudaEventElapsedTime(&ms, E[0], E[1]));
    ctx->timings[0] = ms;
    CU(cudaEventElapsedTime(&ms, E[1], E[2]));
    ctx->timings[1] = ms;
    CU(cudaEventElapsedTime(&ms, E[2], E[3]));
    ctx->timings[2] = ms;
    CU(cudaEventElapsedTime(&ms, E[3], E[4]));
    ctx->timings[3] = ms;
  }
  if (counters[3]) {
    ctx->err = "internal error: a query's text did not match its counted length";
    return TN93G_ECUDA;
  }
  for (int q = 0; q < nq; q++) {
    tn93g_summary &X = sums[q];
    X = S[q];
    if (repass) memset(X.amb_bounds, 0, sizeof X.amb_bounds);
    X.output_bytes = qoff[q + 1] - qoff[q];
    if (q == 0) {
      X.pairs_replayed = (long)counters[2];
      X.logs_ambiguous = ambiguous0;
      X.logs_resolved = resolved;
      X.undecided = 0;  // every listed pair was finished with the C library's logarithms
      X.sums_repass = repass ? 1 : 0;
    }
    if (rc.emit && sink && sink(user, q, (const char *)srv->pin + qoff[q], (size_t)(qoff[q + 1] - qoff[q])))
      return TN93G_ESINK;
  }
  return TN93G_OK;
}

}  // extern "C"

//================================================================================================== batched runs
// Many independent alignments in one pass (each with its own options): every stage runs over all of them at once.
// Packing is per alignment on one stream; the pair stage is one persistent launch per kernel class over a queue of
// all alignments' tiles (longest alignments first); the replay, statistics, sums, scan, reduction and text are
// batched kernels over all alignments' rows. Each alignment's output equals its own tn93g_run byte for byte.
namespace {


// Packing of a batch, one launch per step over all alignments: block b belongs to the alignment k with
// off[k] <= b < off[k + 1] (off[] is the prefix sum of the alignments' block counts) and is its block b - off[k].
__device__ __forceinline__ int batch_owner(const int *off, int K, int b)
{
  int lo = 0, hi = K - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (off[mid] <= b)
      lo = mid;
    else
      hi = mid - 1;
  }
  return lo;
}

struct ScanDesc {
  const uint8_t *codes;
  long N, L;
  uint32_t *seen;
  unsigned long long *nN;
};
struct TransDesc {
  const uint8_t *cc;
  uint8_t *ccT;
  long N, Lc, Npad;
};
struct OneHotDesc {
  const uint8_t *cc;
  long N, Lc, NB, KS;
  uint8_t *img;
  TcClasses C;
};

__global__ void __launch_bounds__(256) colscan_batch_kernel(const ScanDesc *d, const int *off, int K)
{
  const int k = batch_owner(off, K, blockIdx.x);
  const long lb = (long)blockIdx.x - off[k];
  const ScanDesc &a = d[k];
  const long gx = (a.L + 255) / 256;
  colscan_body(a.codes, a.N, a.L, a.seen, a.nN, lb % gx, lb / gx);
}

// one block per (8 sequences, one 64-column word)
__global__ void __launch_bounds__(256) pack_batch_kernel(const PackArgs *d, const int *off, int K)
{
  const int k = batch_owner(off, K, blockIdx.x);
  const long lb = (long)blockIdx.x - off[k];
  const PackArgs &a = d[k];
  const long gx = (a.N + kWarps - 1) / kWarps;
  pack_body(a, lb % gx, lb / gx, a.W);
}

__global__ void __launch_bounds__(256) events_batch_kernel(const PackArgs *d, const int *off, int K)
{
  const int k = batch_owner(off, K, blockIdx.x);
  events_body(d[k], (long)blockIdx.x - off[k]);
}

__global__ void __launch_bounds__(256) transpose_batch_kernel(const TransDesc *d, const int *off, int K)
{
  const int k = batch_owner(off, K, blockIdx.x);
  const long lb = (long)blockIdx.x - off[k];
  const TransDesc &a = d[k];
  const long gx = (a.Lc + kTransK - 1) / kTransK;
  transpose_body(a.cc, a.ccT, a.N, a.Lc, a.Npad, lb % gx, lb / gx);
}

__global__ void __launch_bounds__(256) onehot_batch_kernel(const OneHotDesc *d, const int *off, int K)
{
  const int k = batch_owner(off, K, blockIdx.x);
  const OneHotDesc &a = d[k];
  onehot_body(a.cc, a.N, a.Lc, a.NB, a.KS, a.img, 0, a.NB * 32, (long)blockIdx.x - off[k], a.C);
}

// the prefix sum of per-alignment block counts, uploaded to slot q of the offsets buffer; returns the total
int upload_offsets(tn93g_ctx *ctx, DevBuf &buf, int q, int K, const std::vector<long> &blocks, cudaStream_t st,
                   int *total)
{
  std::vector<int> off(K + 1);
  long t = 0;
  for (int k = 0; k < K; k++) {
    off[k] = (int)t;
    t += blocks[k];
  }
  off[K] = (int)t;
  if (t >= (1l << 31)) return TN93G_ETOOBIG;
  CU(cudaMemcpyAsync((int *)buf.p + (size_t)q * (K + 1), off.data(), (K + 1) * sizeof(int), cudaMemcpyHostToDevice,
                     st));
  *total = (int)t;
  return TN93G_OK;
}

__global__ void gather_u64_kernel(const unsigned long long *src, const long *idx, unsigned long long *dst, int n)
{
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) dst[k] = src[idx[k]];
}

template <bool WPLANE, bool PACK>
cudaError_t launch_event_batch(const PairArgs *descs, const int4 *blocks, size_t n, cudaStream_t st)
{
  static PerDevice attr;
  const cudaError_t e = attr.once([] {
    return cudaFuncSetAttribute(event_batch_kernel<WPLANE, PACK>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)EvTile<WPLANE>::smem);
  });
  if (e != cudaSuccess) return e;
  event_batch_kernel<WPLANE, PACK><<<(unsigned)n, kEvThreads, EvTile<WPLANE>::smem, st>>>(descs, blocks);
  return cudaGetLastError();
}

template <int MINB>
cudaError_t launch_pair_batch_t(int sms, bool wplane, bool gapmm, const PairArgs *descs, const BatchTile *tiles,
                                int ntiles, unsigned *next, cudaStream_t st)
{
  static PerDevice attr;
  const cudaError_t e = attr.once([] {
    cudaError_t r;
    if ((r = cudaFuncSetAttribute(pair_batch_kernel<true, true, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)kPairSmem)) != cudaSuccess)
      return r;
    if ((r = cudaFuncSetAttribute(pair_batch_kernel<true, false, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)kPairSmem)) != cudaSuccess)
      return r;
    return cudaFuncSetAttribute(pair_batch_kernel<false, false, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)kPairSmem);
  });
  if (e != cudaSuccess) return e;
  const dim3 g((unsigned)(sms * MINB));
  if (gapmm)
    pair_batch_kernel<true, true, MINB><<<g, 256, kPairSmem, st>>>(descs, tiles, ntiles, next);
  else if (wplane)
    pair_batch_kernel<true, false, MINB><<<g, 256, kPairSmem, st>>>(descs, tiles, ntiles, next);
  else
    pair_batch_kernel<false, false, MINB><<<g, 256, kPairSmem, st>>>(descs, tiles, ntiles, next);
  return cudaGetLastError();
}

}  // namespace

// records: alignments may take the records path, whose event offsets and wider records are taken where there is room
static int batch_impl(tn93g_ctx *ctx, int K, const tn93g_alignment *alns, const tn93g_opts *opts, const int *rows_per_warp,
                      int pair_blocks, tn93g_query_sink sink, void *user, tn93g_summary *sums, bool records)
{
  if (!ctx || K <= 0 || !alns || !opts || !sums) return TN93G_EINVAL;
  for (int k = 0; k < K; k++) {
    const tn93g_alignment &A = alns[k];
    const tn93g_opts &o = opts[k];
    if (A.n <= 0 || A.L <= 0 || !A.codes || !A.copy_counts || !A.names || !A.name_off || !A.name_len)
      return TN93G_EINVAL;
    if (o.mode < 0 || o.mode > 4 || (o.format != TN93G_CSV && o.format != TN93G_CSVN) || o.do_fst) return TN93G_EINVAL;
    if (A.L >= (1l << 25) || A.n >= (1l << 31)) return TN93G_ETOOBIG;
    if (rows_per_warp && rows_per_warp[k] != 1 && rows_per_warp[k] != 2 && rows_per_warp[k] != 4) return TN93G_EINVAL;
  }
  if (pair_blocks == 0) pair_blocks = 2;
  if (pair_blocks != 2 && pair_blocks != 3) return TN93G_EINVAL;
  cudaSetDevice(ctx->device);
  cudaStream_t st = ctx->stream;
  for (double &t : ctx->timings) t = 0;
  ctx->launches = 0;
  DevBuf *bb = ctx->bb;
  cudaEvent_t *E = ctx->evs;
  float ms = 0.f;
  CU(cudaEventRecord(E[0], st));
  //------------------------------------------------------------------ inputs
  std::vector<size_t> code_off(K + 1), seen_off(K + 1), name_base(K + 1), row_base(K + 1);
  code_off[0] = seen_off[0] = name_base[0] = row_base[0] = 0;
  for (int k = 0; k < K; k++) {
    size_t nb = 0;
    for (long i = 0; i < alns[k].n; i++) nb = std::max(nb, alns[k].name_off[i] + (size_t)alns[k].name_len[i]);
    code_off[k + 1] = code_off[k] + (size_t)alns[k].n * alns[k].L;
    seen_off[k + 1] = seen_off[k] + alns[k].L;
    name_base[k + 1] = name_base[k] + nb;
    row_base[k + 1] = row_base[k] + alns[k].n;
  }
  const size_t NR = row_base[K];
  TRY(ensure(ctx, bb[BB_CODES], code_off[K]));
  TRY(ensure(ctx, bb[BB_NAMES], name_base[K] + 8));  // names are read by the aligned words that hold them
  TRY(ensure(ctx, bb[BB_NAMEOFF], NR * sizeof(uint64_t)));
  TRY(ensure(ctx, bb[BB_NAMELEN], NR * sizeof(int32_t)));
  TRY(ensure(ctx, bb[BB_COUNTS], NR * sizeof(long)));
  std::vector<uint64_t> noff(NR);
  std::vector<int32_t> nlen(NR);
  std::vector<long> cnts(NR);
  std::string names;  // the alignments' names, one after the other: one copy
  names.reserve(name_base[K]);
  std::vector<HostSpan> spans;
  for (int k = 0; k < K; k++)
    spans.push_back({(uint8_t *)bb[BB_CODES].p + code_off[k], alns[k].codes, code_off[k + 1] - code_off[k]});
  TRY(upload_host(ctx, spans));
  for (int k = 0; k < K; k++) {
    names.append(alns[k].names, name_base[k + 1] - name_base[k]);
    for (long i = 0; i < alns[k].n; i++) {
      noff[row_base[k] + i] = name_base[k] + alns[k].name_off[i];
      nlen[row_base[k] + i] = (int32_t)alns[k].name_len[i];
      cnts[row_base[k] + i] = alns[k].copy_counts[i];
    }
  }
  if (!names.empty()) CU(cudaMemcpyAsync(bb[BB_NAMES].p, names.data(), names.size(), cudaMemcpyHostToDevice, st));
  CU(cudaMemcpyAsync(bb[BB_NAMEOFF].p, noff.data(), NR * sizeof(uint64_t), cudaMemcpyHostToDevice, st));
  CU(cudaMemcpyAsync(bb[BB_NAMELEN].p, nlen.data(), NR * sizeof(int32_t), cudaMemcpyHostToDevice, st));
  CU(cudaMemcpyAsync(bb[BB_COUNTS].p, cnts.data(), NR * sizeof(long), cudaMemcpyHostToDevice, st));
  //------------------------------------------------------------------ column scan and folding
  TRY(ensure(ctx, bb[BB_SEEN], seen_off[K] * sizeof(uint32_t)));
  TRY(ensure(ctx, bb[BB_NN], K * sizeof(unsigned long long)));
  CU(cudaMemsetAsync(bb[BB_SEEN].p, 0, seen_off[K] * sizeof(uint32_t), st));
  CU(cudaMemsetAsync(bb[BB_NN].p, 0, K * sizeof(unsigned long long), st));
  TRY(ensure(ctx, bb[BB_BOFF], 5 * (size_t)(K + 1) * sizeof(int)));
  TRY(ensure(ctx, bb[BB_SCANDESC], K * sizeof(ScanDesc)));
  TRY(ensure(ctx, bb[BB_PACKDESC], K * sizeof(PackArgs)));
  TRY(ensure(ctx, bb[BB_TRDESC], K * sizeof(TransDesc)));
  TRY(ensure(ctx, bb[BB_OHDESC], K * sizeof(OneHotDesc)));
  const int *boff = (const int *)bb[BB_BOFF].p;
  {
    std::vector<ScanDesc> sd(K);
    std::vector<long> nb(K);
    for (int k = 0; k < K; k++) {
      const long N = alns[k].n, L = alns[k].L;
      sd[k] = ScanDesc{(const uint8_t *)bb[BB_CODES].p + code_off[k], N, L, (uint32_t *)bb[BB_SEEN].p + seen_off[k],
                       (unsigned long long *)bb[BB_NN].p + k};
      nb[k] = ((L + 255) / 256) * ((N + 63) / 64);
    }
    CU(cudaMemcpyAsync(bb[BB_SCANDESC].p, sd.data(), K * sizeof(ScanDesc), cudaMemcpyHostToDevice, st));
    int total = 0;
    TRY(upload_offsets(ctx, bb[BB_BOFF], 0, K, nb, st, &total));
    if (total) {
      colscan_batch_kernel<<<(unsigned)total, 256, 0, st>>>((const ScanDesc *)bb[BB_SCANDESC].p, boff, K);
      CU(cudaGetLastError());
      ctx->launches++;
    }
  }
  std::vector<uint32_t> seen(seen_off[K]);
  std::vector<unsigned long long> nN(K);
  CU(cudaMemcpyAsync(seen.data(), bb[BB_SEEN].p, seen_off[K] * sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
  CU(cudaMemcpyAsync(nN.data(), bb[BB_NN].p, K * sizeof(unsigned long long), cudaMemcpyDeviceToHost, st));
  CU(cudaStreamSynchronize(st));
  std::vector<RunConsts> RC(K);
  std::vector<int32_t> varcol;
  std::vector<char> three(K, 0);  // three-fold codes anywhere (not under skip): the events kernel marks their sequences
  std::vector<size_t> vc_off(K + 1), pl_off(K + 1), cc_off(K + 1), cct_off(K + 1), evo_off(K + 1);
  vc_off[0] = pl_off[0] = cc_off[0] = cct_off[0] = evo_off[0] = 0;
  for (int k = 0; k < K; k++) {
    const long N = alns[k].n, L = alns[k].L;
    const tn93g_opts *o = &opts[k];
    RunConsts &rc = RC[k];
    memset(&rc, 0, sizeof rc);
    rc.N = N;
    rc.n1 = N;
    rc.mode = o->mode;
    rc.gapmm = o->mode == TN93G_GAPMM;
    rc.fallback_avg = (o->mode == TN93G_RESOLVE || o->mode == TN93G_SUBSET) && o->resolve_fraction < 1.;
    rc.emit = !o->count_only;
    rc.format = o->format;
    rc.delim = o->delimiter;
    rc.report_self = o->report_self && rc.emit;
    rc.threshold = o->threshold;
    rc.min_distance = o->min_distance;
    rc.resolve_fraction = o->resolve_fraction;
    rc.min_overlap = o->min_overlap;
    rc.log_band = ctx->log_band;
    rc.log_spread = ctx->log_spread;
    rc.resolve_all = ctx->exact_sums;
    for (long p = 0; p < L; p++) {
      const uint32_t m = seen[seen_off[k] + p];
      three[k] |= (m & 0x7800u) != 0 && o->mode != TN93G_SKIP;
      if (m && !(m & (m - 1)) && m < 16) {
        const int b = __builtin_ctz(m);
        rc.constT++;
        rc.constNf[b] += 2;
        rc.constCnt[b]++;
      } else
        varcol.push_back((int32_t)p);
    }
    vc_off[k + 1] = varcol.size();
    rc.Lc = (long)(vc_off[k + 1] - vc_off[k]);
    rc.W = (rc.Lc + 63) / 64;
    rc.Npad = (N + 31) / 32 * 32;
    rc.wplane = rc.gapmm || nN[k] > 16ull * (unsigned long long)N;
    rc.NP = rc.gapmm ? 5 : 4;
    pl_off[k + 1] = pl_off[k] + (size_t)std::max<long>(rc.W, 1) * rc.NP * rc.Npad;
    cc_off[k + 1] = cc_off[k] + (size_t)N * std::max<long>(rc.Lc, 1);
    cct_off[k + 1] = cct_off[k] + (size_t)std::max<long>(rc.Lc, 1) * rc.Npad;
    evo_off[k + 1] = evo_off[k] + N + 1;
  }
  TRY(ensure(ctx, bb[BB_VARCOL], std::max<size_t>(varcol.size(), 1) * sizeof(int32_t)));
  TRY(ensure(ctx, bb[BB_PLANES], pl_off[K] * sizeof(uint64_t)));
  TRY(ensure(ctx, bb[BB_CC], cc_off[K] + 8));
  TRY(ensure(ctx, bb[BB_CCT], cct_off[K]));
  TRY(ensure(ctx, bb[BB_EVCOUNT], NR * sizeof(uint32_t)));
  TRY(ensure(ctx, bb[BB_EVOFF], evo_off[K] * sizeof(uint32_t)));
  if (!varcol.empty())
    CU(cudaMemcpyAsync(bb[BB_VARCOL].p, varcol.data(), varcol.size() * sizeof(int32_t), cudaMemcpyHostToDevice, st));
  CU(cudaMemsetAsync(bb[BB_PLANES].p, 0, pl_off[K] * sizeof(uint64_t), st));
  CU(cudaMemsetAsync(bb[BB_EVCOUNT].p, 0, NR * sizeof(uint32_t), st));
  std::vector<PackArgs> PA(K);
  for (int k = 0; k < K; k++) {
    const RunConsts &rc = RC[k];
    PackArgs &pa = PA[k];
    pa.codes = (const uint8_t *)bb[BB_CODES].p + code_off[k];
    pa.N = rc.N;
    pa.L = alns[k].L;
    pa.Lc = rc.Lc;
    pa.W = rc.W;
    pa.Npad = rc.Npad;
    pa.varcol = (const int32_t *)bb[BB_VARCOL].p + vc_off[k];
    pa.NP = rc.NP;
    pa.wplane = rc.wplane;
    pa.gapmm = rc.gapmm;
    pa.planes = (uint64_t *)bb[BB_PLANES].p + pl_off[k];
    pa.cc = (uint8_t *)bb[BB_CC].p + cc_off[k];
    pa.evcount = (uint32_t *)bb[BB_EVCOUNT].p + row_base[k];
    pa.ev_off = (const uint32_t *)bb[BB_EVOFF].p + evo_off[k];
    pa.ev = nullptr;
  }
  {
    // bit planes and codes (one block per 8 sequences and word), and the transposed codes, of every alignment
    std::vector<long> nbp(K), nbt(K);
    std::vector<TransDesc> td(K);
    for (int k = 0; k < K; k++) {
      const RunConsts &rc = RC[k];
      nbp[k] = rc.W ? ((rc.N + kWarps - 1) / kWarps) * rc.W : 0;
      nbt[k] = rc.W ? ((rc.Lc + kTransK - 1) / kTransK) * (rc.Npad / 32) : 0;
      td[k] = TransDesc{PA[k].cc, (uint8_t *)bb[BB_CCT].p + cct_off[k], rc.N, rc.Lc, rc.Npad};
    }
    CU(cudaMemcpyAsync(bb[BB_PACKDESC].p, PA.data(), K * sizeof(PackArgs), cudaMemcpyHostToDevice, st));
    CU(cudaMemcpyAsync(bb[BB_TRDESC].p, td.data(), K * sizeof(TransDesc), cudaMemcpyHostToDevice, st));
    int tp = 0, tt = 0;
    TRY(upload_offsets(ctx, bb[BB_BOFF], 1, K, nbp, st, &tp));
    TRY(upload_offsets(ctx, bb[BB_BOFF], 2, K, nbt, st, &tt));
    if (tp) {
      pack_batch_kernel<<<(unsigned)tp, 256, 0, st>>>((const PackArgs *)bb[BB_PACKDESC].p, boff + (K + 1), K);
      CU(cudaGetLastError());
      ctx->launches++;
    }
    if (tt) {
      transpose_batch_kernel<<<(unsigned)tt, dim3(32, 8), 0, st>>>((const TransDesc *)bb[BB_TRDESC].p,
                                                                  boff + 2 * (K + 1), K);
      CU(cudaGetLastError());
      ctx->launches++;
    }
  }
  std::vector<uint32_t> evc(NR), evo(evo_off[K]);
  CU(cudaMemcpyAsync(evc.data(), bb[BB_EVCOUNT].p, NR * sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
  CU(cudaStreamSynchronize(st));
  // Which alignments take the records path (event and formula kernels, as pair_split; average, gapmm and skip with the
  // weighted operand image): all with variable columns on the tensor-core path but those with more than kPackedMaxEvents
  // events in a sequence, with an N plane under resolve (the batch makes no N word lists) or with a code matrix past 32-bit
  // offsets. 24 alignments of 50-2,000 x 900-3,000 in three modes: pair stage and replay 2.12 -> 0.93 ms. When its
  // larger records do not fit, or leave no room for what comes after them (tn93g_batch_run), every alignment takes the fused
  // kernel.
  const bool use_tc = ctx->count_path == 1;
  std::vector<char> split(K, 0), lin(K, 0);
  std::vector<size_t> rec(K), ag_off(K + 1, 0);  // bytes of a pair's record; the alignments' records
  size_t nev = 0;
  auto plan_events = [&](bool may_split) -> int {
    nev = 0;
    for (int k = 0; k < K; k++) {
      const bool on = use_tc && RC[k].W > 0 && alns[k].n > 1;
      lin[k] = on && may_split && weighted_mode(opts[k].mode);
      const bool none = lin[k] && !three[k];  // no list: nothing reads one
      uint32_t max_ev = 0;
      for (long i = 0; i < alns[k].n; i++) {
        const uint32_t n = none ? 0 : evc[row_base[k] + i];
        evo[evo_off[k] + i] = (uint32_t)nev;
        nev += pad_events(n);
        max_ev = std::max(max_ev, n);
      }
      evo[evo_off[k] + alns[k].n] = (uint32_t)nev;
      RC[k].packed = max_ev <= (uint32_t)kPackedMaxEvents;
      split[k] = lin[k] || (on && may_split && RC[k].packed && !RC[k].wplane && RC[k].Lc * RC[k].Npad < (1l << 32));
      // the fused kernel reads whole counts; the others write a pair's final sixteenths back into its record
      rec[k] = (split[k] ? 32 * alns[k].L : 2 * RC[k].Lc) < 65536 ? 16 : 32;
      ag_off[k + 1] = ag_off[k] + (on ? (size_t)alns[k].n * alns[k].n * rec[k] : 0);
    }
    if (nev >= (1ull << 32)) return TN93G_ETOOBIG;
    TRY(ensure(ctx, bb[BB_EV], std::max<size_t>(nev, 1) * sizeof(uint32_t)));
    if (may_split) {
      TRY(ensure(ctx, bb[BB_EV2], std::max<size_t>(nev, 1) * sizeof(uint2), true));
      TRY(ensure(ctx, bb[BB_THREE], NR, true));
    }
    if (use_tc) TRY(ensure(ctx, bb[BB_TCAGG], std::max<size_t>(ag_off[K], 16), may_split));
    return TN93G_OK;
  };
  // the pair stage's other large buffers come first, so that only the records path itself can be what does not fit
  std::vector<size_t> d_off(K + 1), q_off(K + 1);
  d_off[0] = q_off[0] = 0;
  for (int k = 0; k < K; k++) {
    const size_t N = alns[k].n;
    d_off[k + 1] = d_off[k] + N * N;
    q_off[k + 1] = q_off[k] + std::max<size_t>(N * (N - 1) / 2, 1);
  }
  TRY(ensure(ctx, bb[BB_DIST], d_off[K] * sizeof(double)));
  TRY(ensure(ctx, bb[BB_RQ], q_off[K] * sizeof(unsigned long long)));
  ctx->records_busy = true;
  int planned = plan_events(use_tc && records);
  if (use_tc && records && planned == TN93G_ENOMEM) {
    release(ctx, bb[BB_EV2]);
    release(ctx, bb[BB_TCAGG]);
    planned = plan_events(false);
  }
  TRY(planned);
  CU(cudaMemcpyAsync(bb[BB_EVOFF].p, evo.data(), evo_off[K] * sizeof(uint32_t), cudaMemcpyHostToDevice, st));
  {
    // every alignment's sparse events (one block per 8 sequences)
    std::vector<long> nbe(K);
    for (int k = 0; k < K; k++) {
      PA[k].ev = (uint32_t *)bb[BB_EV].p;
      if (split[k]) {
        PA[k].ev2 = (uint2 *)bb[BB_EV2].p;
        PA[k].ev2_Npad = (uint32_t)RC[k].Npad;
        PA[k].three = three[k] ? (uint8_t *)bb[BB_THREE].p + row_base[k] : nullptr;
      }
      nbe[k] = (RC[k].W && evo[evo_off[k] + alns[k].n] > evo[evo_off[k]]) ? (RC[k].N + kWarps - 1) / kWarps : 0;
    }
    CU(cudaMemcpyAsync(bb[BB_PACKDESC].p, PA.data(), K * sizeof(PackArgs), cudaMemcpyHostToDevice, st));
    int te = 0;
    TRY(upload_offsets(ctx, bb[BB_BOFF], 3, K, nbe, st, &te));
    if (te) {
      events_batch_kernel<<<(unsigned)te, 256, 0, st>>>((const PackArgs *)bb[BB_PACKDESC].p, boff + 3 * (K + 1), K);
      CU(cudaGetLastError());
      ctx->launches++;
    }
  }
  // tables: one copy per distinct (mode, ambiguity subset, N plane); the site tables per (mode, subset)
  std::vector<int> tab_of(K), site_of(K);
  std::vector<std::pair<int, std::string>> keys, site_keys;
  std::vector<int> key_of, site_key_of;  // an alignment with that key
  for (int k = 0; k < K; k++) {
    const std::string sub((const char *)opts[k].subset, sizeof opts[k].subset);
    const std::string sk = opts[k].mode == TN93G_SUBSET ? sub : std::string();
    const std::pair<int, std::string> key(opts[k].mode * 2 + (RC[k].wplane ? 1 : 0), sk), skey(opts[k].mode, sk);
    int t = -1, u = -1;
    for (size_t q = 0; q < keys.size(); q++)
      if (keys[q] == key) t = (int)q;
    for (size_t q = 0; q < site_keys.size(); q++)
      if (site_keys[q] == skey) u = (int)q;
    if (t < 0) {
      t = (int)keys.size();
      keys.push_back(key);
      key_of.push_back(k);
    }
    if (u < 0) {
      u = (int)site_keys.size();
      site_keys.push_back(skey);
      site_key_of.push_back(k);
    }
    tab_of[k] = t;
    site_of[k] = u;
  }
  // the last batch's tables stay on the device until a batch needs others (they depend on these keys alone)
  const size_t site_n = sizeof(ctx->h_tab->site) / sizeof(SiteEntry);
  if (keys != ctx->batch_keys || site_keys != ctx->batch_site_keys) {
    ctx->batch_keys.clear();
    std::vector<PairTables> h_agg(keys.size());
    std::vector<SiteEntry> h_site;
    for (size_t q = 0; q < keys.size(); q++) {
      build_tables(ctx->h_tab, opts[key_of[q]].mode, opts[key_of[q]].subset);
      fill_pair_tables(*ctx->h_tab, RC[key_of[q]].wplane, &h_agg[q]);
    }
    for (int k : site_key_of) {
      build_tables(ctx->h_tab, opts[k].mode, opts[k].subset);
      const SiteEntry *se = &ctx->h_tab->site[0][0];
      h_site.insert(h_site.end(), se, se + site_n);
    }
    TRY(ensure(ctx, bb[BB_AGG], h_agg.size() * sizeof(PairTables)));
    TRY(ensure(ctx, bb[BB_SITE], h_site.size() * sizeof(SiteEntry)));
    CU(cudaMemcpyAsync(bb[BB_AGG].p, h_agg.data(), h_agg.size() * sizeof(PairTables), cudaMemcpyHostToDevice, st));
    CU(cudaMemcpyAsync(bb[BB_SITE].p, h_site.data(), h_site.size() * sizeof(SiteEntry), cudaMemcpyHostToDevice, st));
    CU(cudaStreamSynchronize(st));  // the host copies end here
    ctx->batch_keys = keys;
    ctx->batch_site_keys = site_keys;
  }
  CU(cudaEventRecord(E[1], st));
  //------------------------------------------------------------------ pair stage
  std::vector<size_t> seg_base(K + 1, 0);
  std::vector<long> maxseg(K);
  for (int k = 0; k < K; k++) {
    const size_t N = alns[k].n;
    maxseg[k] = std::max<long>(1, ((long)N + kSeg - 1) / kSeg);
    seg_base[k + 1] = seg_base[k] + N * maxseg[k];
  }
  TRY(ensure(ctx, bb[BB_RQN], K * sizeof(unsigned)));
  TRY(ensure(ctx, bb[BB_COUNTERS], (size_t)K * 4 * sizeof(unsigned long long)));
  CU(cudaMemsetAsync(bb[BB_RQN].p, 0, K * sizeof(unsigned), st));
  CU(cudaMemsetAsync(bb[BB_COUNTERS].p, 0, (size_t)K * 4 * sizeof(unsigned long long), st));
  // one undecided list for every alignment (entries carry the alignment), per-alignment summary bounds
  const unsigned und_cap = (unsigned)std::min<size_t>(std::max<size_t>(4096, q_off[K] / 64), 0xFFFFFFF0u);
  TRY(ensure(ctx, bb[BB_UND], (size_t)und_cap * 2 * sizeof(unsigned long long)));
  TRY(ensure(ctx, bb[BB_UNDN], sizeof(unsigned long long)));
  TRY(ensure(ctx, bb[BB_AMB], (size_t)K * 4 * sizeof(unsigned long long)));
  CU(cudaMemsetAsync(bb[BB_UNDN].p, 0, sizeof(unsigned long long), st));
  CU(cudaMemsetAsync(bb[BB_AMB].p, 0, (size_t)K * 4 * sizeof(unsigned long long), st));
  std::vector<PairArgs> PD(K);
  std::vector<ReplayArgs> RD(K);
  for (int k = 0; k < K; k++) {
    PairArgs &A = PD[k];
    memset(&A, 0, sizeof A);
    A.rc = RC[k];
    A.planes = (const uint64_t *)bb[BB_PLANES].p + pl_off[k];
    A.cc = (const uint8_t *)bb[BB_CC].p + cc_off[k];
    A.ccT = (const uint8_t *)bb[BB_CCT].p + cct_off[k];
    A.ev_off = (const uint32_t *)bb[BB_EVOFF].p + evo_off[k];
    A.ev = (const uint32_t *)bb[BB_EV].p;
    A.tab = (const PairTables *)bb[BB_AGG].p + tab_of[k];
    A.r0 = 0;
    A.r1 = alns[k].n;
    A.ncols = alns[k].n;
    A.colbase = 0;
    A.cstart = 0;
    A.cend = alns[k].n;
    A.dist = (double *)bb[BB_DIST].p + d_off[k];
    A.replay_q = (unsigned long long *)bb[BB_RQ].p + q_off[k];
    A.replay_n = (unsigned *)bb[BB_RQN].p + k;
    A.replay_cap = q_off[k + 1] - q_off[k];
    A.counters = (unsigned long long *)bb[BB_COUNTERS].p + 4 * k;
    A.logt = ctx->d_logt;
    A.ex.und_list = (unsigned long long *)bb[BB_UND].p;
    A.ex.und_n = (unsigned *)bb[BB_UNDN].p;
    A.ex.und_cap = und_cap;
    A.ex.und_k = k;
    A.ex.amb = (unsigned long long *)bb[BB_AMB].p + 4 * k;
    A.ex.counts = (const long *)bb[BB_COUNTS].p + row_base[k];
    A.ex.colunit = nullptr;
    ReplayArgs &R = RD[k];
    memset(&R, 0, sizeof R);
    R.rc = RC[k];
    R.cc = A.cc;
    R.planes = A.planes;
    R.site = (const SiteEntry *)bb[BB_SITE].p + (size_t)site_of[k] * site_n;
    R.ev_off = A.ev_off;
    R.ev = lin[k] && !three[k] ? nullptr : A.ev;  // such an alignment's lists are left empty
    R.q = A.replay_q;
    R.qn = A.replay_n;
    R.qcap = A.replay_cap;
    R.r0 = 0;
    R.ncols = A.ncols;
    R.colbase = 0;
    R.dist = A.dist;
    R.counters = A.counters;
    R.logt = ctx->d_logt;
    R.ex = A.ex;
  }
  std::vector<int> order(K);
  for (int k = 0; k < K; k++) order[k] = k;
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return RC[a].Lc > RC[b].Lc; });
  // tensor-core count path: per alignment an operand image and its pairs' records ([n][n]), computed by one launch over
  // every alignment's 32 x 64 tiles
  if (use_tc) {
    std::vector<size_t> oh_off(K + 1, 0);
    std::vector<TcArgs> TD(K);
    std::vector<int4> tct;
    for (int k = 0; k < K; k++) {
      const long N = alns[k].n;
      const bool on = RC[k].W > 0 && N > 1;
      const long NB = (N + 31) / 32 + 1, KS = (RC[k].Lc + kTcStageK - 1) / kTcStageK;
      oh_off[k + 1] = oh_off[k] + (on ? (size_t)KS * NB * kTcBlockBytes : 0);
      TcArgs &T = TD[k];
      memset(&T, 0, sizeof T);
      T.NB = NB;
      T.KS = KS;
      T.N = N;
      T.n1 = N;
      T.cross = false;
      T.r0 = 0;
      T.r1 = N;
      T.ncols = N;
      T.colbase = 0;
      T.cstart = 0;
      T.cend = N;
    }
    TRY(ensure(ctx, bb[BB_OH], std::max<size_t>(oh_off[K], 16)));
    TRY(ensure(ctx, bb[BB_TCERR], sizeof(unsigned long long)));
    CU(cudaMemsetAsync(bb[BB_TCERR].p, 0, sizeof(unsigned long long), st));
    std::vector<OneHotDesc> ohd(K);
    std::vector<long> nbo(K, 0);
    for (int k : order) {
      if (oh_off[k + 1] == oh_off[k]) continue;
      TcArgs &T = TD[k];
      T.onehot = (const uint8_t *)bb[BB_OH].p + oh_off[k];
      T.agg = (char *)bb[BB_TCAGG].p + ag_off[k];
      T.agg16 = rec[k] == 16;
      T.err = (unsigned long long *)bb[BB_TCERR].p;
      T.wait_ns = ctx->wait_ns;
      T.skip_fill_block = -1;
      ohd[k] = OneHotDesc{PA[k].cc, T.N, RC[k].Lc, T.NB, T.KS, (uint8_t *)bb[BB_OH].p + oh_off[k],
                          tc_classes(opts[k].mode, lin[k])};
      nbo[k] = (T.NB * 32 * T.KS * (kTcStageK / 16) + 255) / 256;
      for (long i0 = 0; i0 < T.N - 1; i0 += kTcRows)
        for (long j0 = (i0 + 1) / kTcCols * kTcCols; j0 < T.N; j0 += kTcCols) tct.push_back(make_int4(k, (int)i0, (int)j0, 0));
      PD[k].tcagg = T.agg;
      PD[k].tc16 = T.agg16;
      PD[k].lin = lin[k];
      PD[k].ev2 = PA[k].ev2;
      PD[k].three = PA[k].three;
    }
    {
      // every alignment's one-hot operand image in one launch
      int to = 0;
      TRY(upload_offsets(ctx, bb[BB_BOFF], 4, K, nbo, st, &to));
      CU(cudaMemcpyAsync(bb[BB_OHDESC].p, ohd.data(), K * sizeof(OneHotDesc), cudaMemcpyHostToDevice, st));
      if (to) {
        onehot_batch_kernel<<<(unsigned)to, 256, 0, st>>>((const OneHotDesc *)bb[BB_OHDESC].p, boff + 4 * (K + 1), K);
        CU(cudaGetLastError());
        ctx->launches++;
      }
    }
    if (!tct.empty()) {
      TRY(ensure(ctx, bb[BB_TCDESC], K * sizeof(TcArgs)));
      TRY(ensure(ctx, bb[BB_TCTILES], tct.size() * sizeof(int4)));
      CU(cudaMemcpyAsync(bb[BB_TCDESC].p, TD.data(), K * sizeof(TcArgs), cudaMemcpyHostToDevice, st));
      CU(cudaMemcpyAsync(bb[BB_TCTILES].p, tct.data(), tct.size() * sizeof(int4), cudaMemcpyHostToDevice, st));
      TcArgs G;
      memset(&G, 0, sizeof G);
      G.err = (unsigned long long *)bb[BB_TCERR].p;
      G.wait_ns = ctx->wait_ns;
      G.skip_fill_block = -1;
      CU(launch_count_list(G, (const TcArgs *)bb[BB_TCDESC].p, (const int4 *)bb[BB_TCTILES].p, (int)tct.size(),
                           ctx->sms, st));
      ctx->launches++;
    }
  }
  // the tile queue: per kernel class, longest alignments first
  std::vector<BatchTile> tiles;
  int cls_n[3] = {0, 0, 0};
  for (int cls = 0; cls < 3; cls++)
    for (int k : order) {
      const int kc = RC[k].gapmm ? 2 : RC[k].wplane ? 1 : 0;
      if (kc != cls || !RC[k].W || split[k]) continue;
      const int rpw = rows_per_warp ? rows_per_warp[k] : kRowsPerWarp, trows = kWarps * rpw;
      const long N = alns[k].n;
      for (long i0 = 0; i0 < N - 1; i0 += trows)
        for (long j0 = (i0 + 1) / kTile * kTile; j0 < N; j0 += kTile) {
          tiles.push_back(BatchTile{k, rpw, (int)i0, (int)j0});
          cls_n[cls]++;
        }
    }
  // alignments whose columns are all constant (Lc = 0) have no tiles: the epilogue runs on the constants alone
  // in tn93g_run; here they take the single-alignment kernel
  TRY(ensure(ctx, bb[BB_PDESC], K * sizeof(PairArgs)));
  TRY(ensure(ctx, bb[BB_RDESC], K * sizeof(ReplayArgs)));
  TRY(ensure(ctx, bb[BB_TILES], std::max<size_t>(tiles.size(), 1) * sizeof(BatchTile)));
  TRY(ensure(ctx, bb[BB_NEXT], 3 * sizeof(unsigned)));
  CU(cudaMemcpyAsync(bb[BB_PDESC].p, PD.data(), K * sizeof(PairArgs), cudaMemcpyHostToDevice, st));
  CU(cudaMemcpyAsync(bb[BB_RDESC].p, RD.data(), K * sizeof(ReplayArgs), cudaMemcpyHostToDevice, st));
  if (!tiles.empty())
    CU(cudaMemcpyAsync(bb[BB_TILES].p, tiles.data(), tiles.size() * sizeof(BatchTile), cudaMemcpyHostToDevice, st));
  CU(cudaMemsetAsync(bb[BB_NEXT].p, 0, 3 * sizeof(unsigned), st));
  int tbase = 0;
  for (int cls = 0; cls < 3; cls++) {
    if (!cls_n[cls]) continue;
    const BatchTile *tp = (const BatchTile *)bb[BB_TILES].p + tbase;
    unsigned *nx = (unsigned *)bb[BB_NEXT].p + cls;
    const PairArgs *dp = (const PairArgs *)bb[BB_PDESC].p;
    CU(pair_blocks == 3 ? launch_pair_batch_t<3>(ctx->sms, cls >= 1, cls == 2, dp, tp, cls_n[cls], nx, st)
                        : launch_pair_batch_t<2>(ctx->sms, cls >= 1, cls == 2, dp, tp, cls_n[cls], nx, st));
    ctx->launches++;
    tbase += cls_n[cls];
  }
  // the records path: event tiles (by record width), then formula blocks (by record width and weighted image)
  std::vector<int4> sb;
  size_t sb_at[7] = {0};
  for (int c = 0; c < 6; c++) {
    for (int k : order) {
      const long N = alns[k].n;
      const bool w16 = rec[k] == 16;
      if (!split[k]) continue;
      if (c < 2) {
        const int rows = EvTile<false>::rows;
        if (lin[k] || w16 != (c == 0)) continue;
        for (long i0 = 0; i0 < N - 1; i0 += rows)
          for (long j0 = i0 / kEvCols * kEvCols; j0 < N; j0 += kEvCols)
            sb.push_back(make_int4(k, (int)(j0 / kEvCols), (int)(i0 / rows), 0));
      } else if (w16 == (c % 2 == 0) && (bool)lin[k] == (c >= 4)) {
        int segw, rpw;
        formula_shape(N, N, false, ctx->sms, segw, rpw);
        for (long by = 0; by * segw < N - 1; by++)  // the segments of a row start at its first column
          for (long bx = 0; bx * kWarps * rpw < N - 1 - by * segw; bx++)
            sb.push_back(make_int4(k, (int)bx, (int)by, rpw << 11 | segw));
      }
    }
    sb_at[c + 1] = sb.size();
  }
  if (!sb.empty()) {
    TRY(ensure(ctx, bb[BB_SPLIT], sb.size() * sizeof(int4)));
    CU(cudaMemcpyAsync(bb[BB_SPLIT].p, sb.data(), sb.size() * sizeof(int4), cudaMemcpyHostToDevice, st));
    const PairArgs *dp = (const PairArgs *)bb[BB_PDESC].p;
    for (int c = 0; c < 6; c++) {
      const int4 *bl = (const int4 *)bb[BB_SPLIT].p + sb_at[c];
      const size_t n = sb_at[c + 1] - sb_at[c];
      if (!n) continue;
      if (c == 0) CU((launch_event_batch<false, true>(dp, bl, n, st)));
      if (c == 1) CU((launch_event_batch<false, false>(dp, bl, n, st)));
      if (c == 2) formula_batch_kernel<true, false><<<(unsigned)n, 256, 0, st>>>(dp, bl);
      if (c == 3) formula_batch_kernel<false, false><<<(unsigned)n, 256, 0, st>>>(dp, bl);
      if (c == 4) formula_batch_kernel<true, true><<<(unsigned)n, 256, 0, st>>>(dp, bl);
      if (c == 5) formula_batch_kernel<false, true><<<(unsigned)n, 256, 0, st>>>(dp, bl);
      CU(cudaGetLastError());
      ctx->launches++;
    }
  }
  for (int k = 0; k < K; k++)
    if (!RC[k].W && alns[k].n > 1) {
      CU(launch_pair(PD[k], (alns[k].n + kTile - 1) / kTile, alns[k].n, ctx->sms, st));
      ctx->launches++;
    }
  ctx->records_busy = false;  // what is launched from here on reads neither the records nor the offsets
  CU(cudaEventRecord(E[2], st));
  replay_batch_kernel<<<2 * ctx->sms, 256, 0, st>>>((const ReplayArgs *)bb[BB_RDESC].p, K);
  CU(cudaGetLastError());
  ctx->launches++;
  CU(cudaEventRecord(E[3], st));
  //------------------------------------------------------------------ rows
  const size_t NS = seg_base[K];
  TRY(ensure(ctx, bb[BB_SBYTES], NS * sizeof(unsigned long long)));
  TRY(ensure(ctx, bb[BB_SOFF], NS * sizeof(unsigned long long)));
  TRY(ensure(ctx, bb[BB_SLINKS], NS * sizeof(long long)));
  TRY(ensure(ctx, bb[BB_SSKIP], NS * sizeof(long long)));
  TRY(ensure(ctx, bb[BB_SMAX], NS * 3 * sizeof(double)));
  TRY(ensure(ctx, bb[BB_RSUM], NR * 3 * sizeof(double)));
  TRY(ensure(ctx, bb[BB_RW], NR * 3 * sizeof(double)));
  TRY(ensure(ctx, bb[BB_HIST], (size_t)K * 3 * kHistBins * sizeof(unsigned long long)));
  TRY(ensure(ctx, bb[BB_TOTAL], sizeof(unsigned long long)));
  TRY(ensure(ctx, bb[BB_SCANTMP], (2 * (NS / kScanTile + 1) + 1) * sizeof(unsigned long long)));
  TRY(ensure(ctx, bb[BB_RED], (size_t)K * 3 * sizeof(double)));
  TRY(ensure(ctx, bb[BB_REDC], (size_t)K * 2 * sizeof(long long)));
  TRY(ensure(ctx, bb[BB_FIRST], (size_t)K * sizeof(unsigned long long)));
  TRY(ensure(ctx, bb[BB_FIRSTIDX], (size_t)K * sizeof(long)));
  TRY(ensure(ctx, bb[BB_ROWDESC], K * sizeof(RowArgs)));
  CU(cudaMemsetAsync(bb[BB_HIST].p, 0, (size_t)K * 3 * kHistBins * sizeof(unsigned long long), st));
  std::vector<RowArgs> RA(K);
  std::vector<int2> blocks;
  long segmax = 1;
  std::vector<long> first_idx(K);
  for (int k = 0; k < K; k++) {
    RowArgs &a = RA[k];
    memset(&a, 0, sizeof a);
    a.rc = RC[k];
    a.dist = PD[k].dist;
    a.r0 = 0;
    a.r1 = alns[k].n;
    a.ncols = alns[k].n;
    a.colbase = 0;
    a.counts = (const long *)bb[BB_COUNTS].p + row_base[k];
    a.name_len = (const int32_t *)bb[BB_NAMELEN].p + row_base[k];
    a.name_off = (const uint64_t *)bb[BB_NAMEOFF].p + row_base[k];
    a.names = (const char *)bb[BB_NAMES].p;
    a.maxseg = maxseg[k];
    a.seg_cols = nullptr;
    a.nrows = alns[k].n;
    a.seg_bytes = (unsigned long long *)bb[BB_SBYTES].p + seg_base[k];
    a.seg_links = (long long *)bb[BB_SLINKS].p + seg_base[k];
    a.seg_skip = (long long *)bb[BB_SSKIP].p + seg_base[k];
    a.seg_max = (double *)bb[BB_SMAX].p + 3 * seg_base[k];
    a.row_sum = (double *)bb[BB_RSUM].p + 3 * row_base[k];
    a.row_w = (double *)bb[BB_RW].p + 3 * row_base[k];
    a.hist = (unsigned long long *)bb[BB_HIST].p + (size_t)k * 3 * kHistBins;
    a.seg_off = (const unsigned long long *)bb[BB_SOFF].p + seg_base[k];
    a.out = nullptr;
    a.hy = nullptr;
    a.err = (unsigned long long *)bb[BB_COUNTERS].p + 4 * k + 3;
    segmax = std::max(segmax, maxseg[k]);
    for (long bx = 0; bx < (alns[k].n + kWarps - 1) / kWarps; bx++) blocks.push_back(make_int2(k, (int)bx));
    first_idx[k] = (long)seg_base[k];
  }
  TRY(ensure(ctx, bb[BB_BLOCKS], blocks.size() * sizeof(int2)));
  CU(cudaMemcpyAsync(bb[BB_ROWDESC].p, RA.data(), K * sizeof(RowArgs), cudaMemcpyHostToDevice, st));
  CU(cudaMemcpyAsync(bb[BB_BLOCKS].p, blocks.data(), blocks.size() * sizeof(int2), cudaMemcpyHostToDevice, st));
  CU(cudaMemcpyAsync(bb[BB_FIRSTIDX].p, first_idx.data(), K * sizeof(long), cudaMemcpyHostToDevice, st));
  const RowArgs *rd = (const RowArgs *)bb[BB_ROWDESC].p;
  const int2 *bp = (const int2 *)bb[BB_BLOCKS].p;
  unsigned long long total = 0, und = 0;
  std::vector<double> red((size_t)K * 3);
  std::vector<long long> redc((size_t)K * 2);
  std::vector<unsigned long long> first(K + 1), hist((size_t)K * 3 * kHistBins), counters((size_t)K * 4);
  auto rows_and_read = [&]() -> int {
    CU(cudaMemsetAsync(bb[BB_HIST].p, 0, (size_t)K * 3 * kHistBins * sizeof(unsigned long long), st));
    stats_batch_kernel<<<dim3((unsigned)blocks.size(), (unsigned)segmax), 256, 0, st>>>(rd, bp);
    CU(cudaGetLastError());
    sum_batch_kernel<<<(unsigned)blocks.size(), 256, 0, st>>>(rd, bp);
    CU(cudaGetLastError());
    CU(launch_scan((const unsigned long long *)bb[BB_SBYTES].p, (unsigned long long *)bb[BB_SOFF].p, (long)NS,
                   (unsigned long long *)bb[BB_TOTAL].p, (unsigned long long *)bb[BB_SCANTMP].p, st));
    aln_reduce_kernel<<<K, 256, 0, st>>>(rd, (double *)bb[BB_RED].p, (long long *)bb[BB_REDC].p);
    CU(cudaGetLastError());
    gather_u64_kernel<<<(K + 255) / 256, 256, 0, st>>>((const unsigned long long *)bb[BB_SOFF].p,
                                                       (const long *)bb[BB_FIRSTIDX].p,
                                                       (unsigned long long *)bb[BB_FIRST].p, K);
    CU(cudaGetLastError());
    ctx->launches += 5;
    CU(cudaEventRecord(E[4], st));
    CU(cudaMemcpyAsync(&total, bb[BB_TOTAL].p, sizeof total, cudaMemcpyDeviceToHost, st));
    CU(cudaMemcpyAsync(red.data(), bb[BB_RED].p, red.size() * sizeof(double), cudaMemcpyDeviceToHost, st));
    CU(cudaMemcpyAsync(redc.data(), bb[BB_REDC].p, redc.size() * sizeof(long long), cudaMemcpyDeviceToHost, st));
    CU(cudaMemcpyAsync(first.data(), bb[BB_FIRST].p, K * sizeof(unsigned long long), cudaMemcpyDeviceToHost, st));
    CU(cudaMemcpyAsync(hist.data(), bb[BB_HIST].p, hist.size() * sizeof(unsigned long long), cudaMemcpyDeviceToHost,
                       st));
    CU(cudaMemcpyAsync(&und, bb[BB_UNDN].p, sizeof und, cudaMemcpyDeviceToHost, st));
    CU(cudaStreamSynchronize(st));
    return TN93G_OK;
  };
  TRY(rows_and_read());
  long resolved = 0;
  // more undecided pairs than the list holds: the alignments that listed any run again alone below
  const bool overflow = und > und_cap;
  if (und && !overflow) {
    // pairs whose bytes or decisions depend on the C library's rounding of a logarithm: finished with its
    // logarithms, then the row stage runs again
    TRY(resolve_listed(ctx, (const ReplayArgs *)bb[BB_RDESC].p, (const unsigned long long *)bb[BB_UND].p,
                       (unsigned)und, st));
    resolved = (long)und;
    TRY(rows_and_read());
  }
  first[K] = total;
  bool any_emit = false;
  for (int k = 0; k < K; k++) any_emit |= RC[k].emit;
  if (any_emit && total) {
    if (bb[BB_OUT].n < total) TRY(ensure(ctx, bb[BB_OUT], total + total / 4));
    TRY(ensure_pinned(ctx, total));
    for (int k = 0; k < K; k++) RA[k].out = (char *)bb[BB_OUT].p;
    CU(cudaMemcpyAsync(bb[BB_ROWDESC].p, RA.data(), K * sizeof(RowArgs), cudaMemcpyHostToDevice, st));
    write_batch_kernel<<<dim3((unsigned)blocks.size(), (unsigned)segmax), 256, 0, st>>>(rd, bp);
    CU(cudaGetLastError());
    ctx->launches++;
    CU(cudaEventRecord(E[5], st));
    CU(cudaMemcpyAsync(ctx->pinned, bb[BB_OUT].p, total, cudaMemcpyDeviceToHost, st));
  } else {
    CU(cudaEventRecord(E[5], st));
  }
  CU(cudaMemcpyAsync(counters.data(), bb[BB_COUNTERS].p, counters.size() * sizeof(unsigned long long),
                     cudaMemcpyDeviceToHost, st));
  CU(cudaEventRecord(E[6], st));
  CU(cudaStreamSynchronize(st));
  const int pairs_e[7][2] = {{0, 1}, {1, 2}, {2, 3}, {3, 4}, {4, 5}, {5, 6}, {0, 6}};
  for (int q = 0; q < 7; q++) {
    CU(cudaEventElapsedTime(&ms, E[pairs_e[q][0]], E[pairs_e[q][1]]));
    ctx->timings[q] = ms;
  }
  if (use_tc) {
    unsigned long long tcerr = 0;
    CU(cudaMemcpy(&tcerr, bb[BB_TCERR].p, sizeof tcerr, cudaMemcpyDeviceToHost));
    if (tcerr) {
      ctx->err = "the tensor-core count kernel timed out waiting for its pipeline";
      return TN93G_ETIMEOUT;
    }
  }
  for (int k = 0; k < K; k++) {
    if (counters[4 * k + 3]) {
      ctx->err = "internal error: a row's text did not match its counted length";
      return TN93G_ECUDA;
    }
    tn93g_summary &S = sums[k];
    memset(&S, 0, sizeof S);
    const unsigned long N = (unsigned long)alns[k].n;
    S.pairwise = N * (N - 1) / 2;
    S.links = (long)redc[2 * k];
    S.skipped = (long)redc[2 * k + 1];
    S.max[0] = red[3 * k];
    S.mean[0] = red[3 * k + 1];
    S.weighted[0] = red[3 * k + 2];
    for (int q = 0; q < 3; q++)
      for (int b = 0; b < kHistBins; b++) S.hist[q][b] = hist[((size_t)k * 3 + q) * kHistBins + b];
    S.logs_ambiguous = (long)counters[4 * k];
    S.logs_resolved = (long)counters[4 * k + 1];  // every listed pair was finished (resolved = the list's total)
    S.undecided = 0;
    S.pairs_replayed = (long)counters[4 * k + 2];
    S.output_bytes = RC[k].emit ? first[k + 1] - first[k] : 0;
  }
  (void)resolved;
  // After an overflow of the undecided list, every alignment that listed a pair runs again alone through
  // tn93g_run's path (which grows its list as needed): its text and summary replace the batch's.
  std::vector<std::string> redo_text(K);
  std::vector<char> redone(K, 0);
  if (overflow) {
    for (int k = 0; k < K; k++) {
      if (!counters[4 * k + 1]) continue;
      const tn93g_alignment &A = alns[k];
      tn93g_set *set = nullptr;
      TRY(tn93g_upload(ctx, &set, A.codes, A.n, A.L, A.copy_counts, A.names, A.name_off, A.name_len));
      tn93g_summary S2;
      const int r = run_impl(ctx, set, A.n, &opts[k], append_sink, &redo_text[k], &S2, false);
      tn93g_free_set(ctx, set);
      TRY(r);
      sums[k] = S2;
      redone[k] = 1;
    }
  }
  // Per alignment: the JSON numbers certain for every rounding of the C library's log, or the alignment runs
  // again alone through tn93g_run's path, whose exact-sums pass gives its maximum and mean (its text and counts
  // are certified pair by pair already).
  {
    std::vector<unsigned long long> ambw((size_t)K * 4);
    CU(cudaMemcpy(ambw.data(), bb[BB_AMB].p, ambw.size() * sizeof(unsigned long long), cudaMemcpyDeviceToHost));
    for (int k = 0; k < K; k++) {
      if (redone[k]) continue;
      tn93g_summary &S = sums[k];
      amb_bounds(&ambw[(size_t)k * 4], S.amb_bounds[0]);
      if (summary_certified(&S, S.amb_bounds, 2 * alns[k].n + 2, 0)) continue;
      const tn93g_alignment &A = alns[k];
      tn93g_set *set = nullptr;
      TRY(tn93g_upload(ctx, &set, A.codes, A.n, A.L, A.copy_counts, A.names, A.name_off, A.name_len));
      tn93g_opts o = opts[k];
      o.count_only = 1;
      tn93g_summary S2;
      const int r = run_impl(ctx, set, A.n, &o, nullptr, nullptr, &S2, false, 0, -1, nullptr, kRunResolveAll);
      tn93g_free_set(ctx, set);
      TRY(r);
      S.max[0] = S2.max[0];
      S.mean[0] = S2.mean[0];
      S.logs_resolved += S2.logs_resolved;
      S.sums_repass = 1;
      memset(S.amb_bounds, 0, sizeof S.amb_bounds);
    }
  }
  if (any_emit && sink)
    for (int k = 0; k < K; k++) {
      if (!RC[k].emit) continue;
      const int r = redone[k] ? sink(user, k, redo_text[k].data(), redo_text[k].size())
                              : sink(user, k, (const char *)ctx->pinned + first[k], (size_t)(first[k + 1] - first[k]));
      if (r) return TN93G_ESINK;
    }
  return TN93G_OK;
}

extern "C" int tn93g_batch_run(tn93g_ctx *ctx, int K, const tn93g_alignment *alns, const tn93g_opts *opts,
                               const int *rows_per_warp, int pair_blocks, tn93g_query_sink sink, void *user,
                               tn93g_summary *sums)
{
  if (!ctx) return TN93G_EINVAL;
  int r = batch_impl(ctx, K, alns, opts, rows_per_warp, pair_blocks, sink, user, sums, true);
  // no room for a later buffer beside the records path's (nothing has reached the sink by then): once more without it
  if (r == TN93G_ENOMEM && ctx->records_busy) {
    release(ctx, ctx->bb[BB_EV2]);
    release(ctx, ctx->bb[BB_TCAGG]);
    ctx->records_busy = false;
    ctx->err.clear();
    r = batch_impl(ctx, K, alns, opts, rows_per_warp, pair_blocks, sink, user, sums, false);
  }
  ctx->records_busy = false;
  return r;
}
