// xi_grid.cu — band-sweep kernel of the XiEstimator pair count (Cartesian
// and observing coordinates) for catalogues whose first-axis coordinate takes
// few distinct values: forests on a common log-wavelength grid, whose
// distances are one function of loglam (h5healxi.cc:196-203).
//
// With U the sorted distinct first-axis values of the catalogue and a
// sightline contiguous on U (its pixel p has value U[f + p]), the run
// boundaries of xi_sweep.cuh for a row x1 = U[g] along any column sightline j
// are the entries of one table row, in column order:
//   b_t(g) = B_t[g] - f_j clamped to [0, n_j],  t = 0 .. 2 n0 + 1,
// where B_t[g] is the first grid index whose value passes the boundary
// predicate of a threshold T[k] against U[g] (side 1 for t <= n0, side 0
// after it; k_grid_tables, engine.cu).  Band t of an item is the strip of
// columns [b_t(g), b_{t+1}(g)) over its rows g: one first-axis bin (band n0 is
// the |x1 - x2| < T[0] gap).  B_t[g] is non-decreasing in g and in t.
//
// The r_perp code (Cartesian) grows along a row, and up to the float rounding
// of d1*d1 along the rows, so an item has few code edges and each crosses a
// band within a few rows.  With F_g[c] the contribution of the columns [0, c)
// of row g (row factors times prefix sums of sightline j), the sum of band t
// below code edge m, whose first column in row g is e_m(g), is
//   U_t(m) = sum_g F_g[min(max(e_m, b_t), b_{t+1})] - F_g[b_t],
// and the bin (band t, code m - 1) is U_t(m) - U_t(m - 1).  With rho_t(m) the
// first row at which column b_t may have reached edge m (a bound with a
// margin over every rounding), rows below rho_{t+1}(m) lie under the edge in
// the whole band and rows from the first one that has passed it for sure lie
// above it, so
//   U_t(m) = V_{t+1}(rho_{t+1}(m)) - V_t(rho_t(m)) + X_t(m),
//   V_t(r) = sum over rows below r of F_g[b_t(g)],
// with X_t(m) over the few rows in between, where the edge's column is
// searched with the pixel-pair kernel's own binning decision.  So the inner
// loop (V) evaluates no bin at all: a lane owns boundary t and adds, row by
// row, six products of its row's (w*delta, w) and sightline j's prefix sums at
// one column.  The z sums and pair counts of a stretch of rows depend on the
// grid alone and come from prefix tables over the rows.  Where a sightline has
// gaps (GAPS) its missing pixels have zero weight, and pixel counts and loglam
// sums are two more products of row values and column prefix sums.
//
// What bounds it: shared-memory reads and the latency of the table reads
// around the inner loop (LSU data pipe 63 %, issue 41 %, most stalled cycles on
// L2 reads; ncu, 1,000 sightlines).  A step (one row of 32 boundaries) takes
// two 16-byte reads per lane at the least eight wavefronts; starting the lanes
// at row residues that keep both reads of eight lanes in different banks took
// the bank conflicts from 1.3e9 to 0.3e9 wavefronts of 2.5e9.
//
// Measured on a B200 against the version that evaluated the r_perp code at
// every boundary of every row and bisected each split run (one warp per item):
//                                            that  bands  + tables,  + arguments in
//                                                         pipeline   shared, turns
//   16,000 sightlines at 16/deg^2, 50 x 50   970   306    237        216 ms
//   2,000 sightlines on 100 deg^2            125   39.9   32.3       28.2
//   48 sightlines (one wave)                 1.58  0.17   0.18       0.17
//   observing, 500 sightlines                11.3  7.3    6.5        5.5
//   1,201 masked (pointer sweep: 133)                     21.0       19.4
// "Tables, pipeline": rows of code edges from a level table instead of a
// bisection (the bisection and its dependent reads took a fifth of the time),
// boundaries read from a skewed table (one sector for four lanes), two item
// buffers filled by bulk copies, the grid's values in shared memory.
#include <algorithm>
#include <type_traits>

#include "bulk_pipeline.cuh"
#include "xi_sweep.cuh"

namespace tos {
namespace {

// Warps per CTA; a CTA has two items in flight.  Sightlines with gaps take twice
// the shared memory an item, so twice the warps share a CTA's items there.
// Short items (kShortPixels) are bound by the chain of reads that prepares
// them, so each has one warp to itself, 16 CTAs an SM, and a claim takes up to
// 16 of them (neighbouring items add to the same bins: from one warp these adds
// do not meet).  Measured against four warps an item and the sweep before the
// band sweep, which had a warp an item (ms):
//                                               before   four   one
//   328,000 Cartesian items of 16 pixels          1.60   2.68   1.35
//   of 40                                         3.13   3.11   1.63
//   of 128                                       13.0    5.94   4.37
//   of 4 (the chain is longer than it was)        0.83   2.27   1.07
//   719,000 observing items of 16                 3.56   5.11   1.82
//   of 40                                         6.39   7.23   2.85
//   of 128                                       16.8   17.6    6.71
// With room for sightlines of 300 pixels fewer CTAs fit (16 pixels 2.3 ms, 128
// pixels 6.5): the limit is the longest for which 16 do.
enum Layout { kWhole, kShort, kGaps };
template <int L>
constexpr int kGridWarps = L == kGaps ? 8 : L == kShort ? 1 : 4;
constexpr int kShortClaim = 16;
constexpr int kBandsPerWarp = 31;  // 32 boundaries

// Sums of a stretch of rows: w d w d, w d, w d, w w, w, w (didj, di, dj, wgt,
// wi, wj), the centred z sum and the pair count.
template <bool GAPS>
struct BandSums {
  double s[6];
  double z;
  std::conditional_t<GAPS, double, uint32_t> n;
};

// One item as its warps see it.
struct BandItem {
  int fi, fj, ni, nj;  // first grid index and pixels of the two sightlines
  int tf, bands, per;  // first band with a pair, their number, bands per group (0 bands: the end)
  float ap;            // Cartesian: 2 (1 - c) inv1^2
  double c;
  const double2* P;    // prefix sums (w*delta, w) of sightline j, by column
  const double2* R;    // (w*delta, w) of sightline i, by row
  const double2* Ri;   // prefix sums of sightline i
  // sightlines with gaps (PairArgs::gap_*): column prefix sums of (pixels,
  // l'/2), row values (1 where there is a pixel, l'/2), and the prefix sums of
  // sightline i
  const double2 *C, *M, *Pi, *Ci;
  Dest d;
};

// The CTA's two items and the launch's arguments for the functions that are
// not inlined: through a reference to the kernel's parameters they would read
// them by generic loads.
__shared__ BandItem s_item[2];
__shared__ PairArgs s_args;
__shared__ Claim s_claim;  // of the warp that prepares an item

struct Sums6 {
  double a, b, c, d, e, f;
};

// ---- the item pipeline ----------------------------------------------------
// Two item buffers per CTA.  The warps take turns to prepare item k + 1 (claim
// it, find its bands, start the bulk copies of its prefix sums and row values)
// before their share of item k; each warp goes from item to item on its own, so
// a warp with fewer rows does not wait for the others unless it gets two items
// ahead.

// Row constants of the r_perp code of a row of distance d1.
__device__ __forceinline__ RowV code_row(const PairArgs& A, float ap, float d1) {
  RowV R;
  R.d1 = d1;
  const float p = __fmul_rn(R.d1, R.d1);
  const float err = __fmaf_rn(R.d1, R.d1, -p);  // d1*d1 = p + err exactly
  R.A1 = __fmul_rn(R.d1, ap);
  R.dl1 = __fmul_rn(-err, A.inv1sqf);
  return R;
}

// First column in [lo, hi) of row R with code >= m (hi when there is none).
// eb: the edge's bounds without the margin for the row's rounding term, which
// is part of u here.  Columns are compared in FP32 with the edge, and the few
// within its margin are binned as the pixel-pair kernel does.
template <bool MINPOS>
__device__ __forceinline__ int edge_column(const PairArgs& A, const RowV& R, const float* colx, double c,
                                           int lo, int hi, int m, float2 eb, unsigned& rech) {
  const int end = hi;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (fabsf(__fmaf_rn(R.A1, colx[mid], R.dl1)) >= eb.x) hi = mid; else lo = mid + 1;
  }
  while (lo < end && fabsf(__fmaf_rn(R.A1, colx[lo], R.dl1)) < eb.y &&
         perp_code<MINPOS>(A, R, colx[lo], c, rech) < m)
    ++lo;
  return lo;
}

// The six sums of band t in code c evaluated row by row from differences of
// prefix sums, for a bin whose telescoped sums cancel to rounding level: a
// bin all of whose weights are zero sums to exactly zero this way.
template <int COORD, bool MINPOS, bool GAPS>
__device__ __noinline__ Sums6 band_by_rows(const BandItem& it, const float* U, const uint16_t* tt, int g0, int g1,
                                           int code) {
  const PairArgs& A = s_args;
  double s[6] = {0, 0, 0, 0, 0, 0};
  unsigned rech = 0;
  const int fi = it.fi, fj = it.fj, nj = it.nj;
  for (int g = g0; g < g1; ++g) {
    int lo = min(max((int)tt[g] - fj, 0), nj), hi = min(max((int)tt[A.ngp + g] - fj, 0), nj);
    if (COORD == kCart) {
      const RowV V = code_row(A, it.ap, U[g]);
      const float4 e1 = A.edges[code + 1], e0 = A.edges[code];
      const int e = edge_column<MINPOS>(A, V, U + fj, it.c, lo, hi, code + 1, make_float2(e1.z, e1.w), rech);
      lo = edge_column<MINPOS>(A, V, U + fj, it.c, lo, e, code, make_float2(e0.z, e0.w), rech);
      hi = e;
    }
    if (hi <= lo) continue;
    const double2 a = it.P[lo], b = it.P[hi], r = it.R[g - fi];
    const double m = GAPS ? it.C[hi].x - it.C[lo].x : (double)(hi - lo), dwd = b.x - a.x, dw = b.y - a.y;
    const double one = GAPS ? it.M[g - fi].x : 1.0;
    s[0] += r.x * dwd;
    s[1] += r.x * m;
    s[2] += one * dwd;
    s[3] += r.y * dw;
    s[4] += r.y * m;
    s[5] += one * dw;
  }
  return Sums6{s[0], s[1], s[2], s[3], s[4], s[5]};
}

// Add the row values r (and m: with gaps) times the column sums p (and c).
__device__ __forceinline__ void add_gap_row(double (&a)[8], double2 r, double2 m, double2 p, double2 c) {
  a[0] = __fma_rn(r.x, p.x, a[0]);
  a[1] = __fma_rn(r.x, c.x, a[1]);
  a[2] = __fma_rn(m.x, p.x, a[2]);
  a[3] = __fma_rn(r.y, p.y, a[3]);
  a[4] = __fma_rn(r.y, c.x, a[4]);
  a[5] = __fma_rn(m.x, p.y, a[5]);
  a[6] = __fma_rn(m.y, c.x, __fma_rn(m.x, c.y, a[6]));
  a[7] = __fma_rn(m.x, c.x, a[7]);
}

// The same into X_t, of one row or of the sums of several.
__device__ __forceinline__ void add_gap_row(BandSums<true>& x, double2 r, double2 m, double2 p, double2 c) {
  double a[8] = {x.s[0], x.s[1], x.s[2], x.s[3], x.s[4], x.s[5], x.z, x.n};
  add_gap_row(a, r, m, p, c);
#pragma unroll
  for (int f = 0; f < 6; ++f) x.s[f] = a[f];
  x.z = a[6];
  x.n = a[7];
}

// Add grid row g's part of X_t (edge column q; from the row `rho` on less the
// columns below b0, which V_t no longer holds).
__device__ __forceinline__ void add_edge_row(const PairArgs& A, const BandItem& it, int g, int q, int b0, bool past,
                                             double lpj, BandSums<false>& x) {
  double2 p = it.P[q];
  const double2 r = it.R[g - it.fi];
  double bd = (double)q, l = A.glp[it.fj + q] - lpj;
  int bn = q;
  if (past) {
    const double2 p0 = it.P[b0];
    p.x -= p0.x;
    p.y -= p0.y;
    bn -= b0;
    bd = (double)bn;
    l -= A.glp[it.fj + b0] - lpj;
  }
  x.s[0] = __fma_rn(r.x, p.x, x.s[0]);
  x.s[1] = __fma_rn(r.x, bd, x.s[1]);
  x.s[2] += p.x;
  x.s[3] = __fma_rn(r.y, p.y, x.s[3]);
  x.s[4] = __fma_rn(r.y, bd, x.s[4]);
  x.s[5] += p.y;
  x.z = __fma_rn(0.5, __fma_rn((double)A.gl[g] - A.lmid, bd, l), x.z);
  x.n += (uint32_t)bn;
}

__device__ __forceinline__ void add_edge_row(const PairArgs&, const BandItem& it, int g, int q, int b0, bool past,
                                             double, BandSums<true>& x) {
  double2 p = it.P[q], c = it.C[q];
  if (past) {
    const double2 p0 = it.P[b0], c0 = it.C[b0];
    p.x -= p0.x;
    p.y -= p0.y;
    c.x -= c0.x;
    c.y -= c0.y;
  }
  add_gap_row(x, it.R[g - it.fi], it.M[g - it.fi], p, c);
}

// Bands t0 .. t0 + m - 1 of an item; lane = boundary t0 + lane (lane <= m).
// U: the grid's values (in shared memory where the kernel stages them).
template <int COORD, bool MINPOS, bool GAPS>
__device__ __forceinline__ void band_group(const PairArgs& A, const BandItem& it, const float* U, int t0, int m,
                                           int lane, int buf, unsigned long long* stats) {
  const int n0 = (int)A.g.n0, n1 = (int)A.g.n1;
  const int t = t0 + min(lane, m);
  const bool bound = lane <= m;           // this lane owns a boundary
  const bool owner = lane < m && t != n0; // and a band that is binned
  const int fi = it.fi, fj = it.fj, nj = it.nj, ge = it.fi + it.ni;
  const float ap = it.ap;
  const uint16_t* tt = A.gtab + (size_t)t * A.ngp;         // B_t by grid row
  const uint2* ts = A.gtabs + ((size_t)(t >> 5) * A.nblk + A.gskew[t]) * 32 + (t & 31);  // the same, skewed
  const size_t tr = (size_t)t * (A.ng + 1);
  const uint16_t* inv = A.ginv + tr;   // first row with B_t >= column
  const double* tz = A.gtz + tr;       // prefix sums over the rows
  const uint32_t* tb = A.gtb + tr;
  const double lpj = GAPS ? 0.0 : A.glp[fj], dfj = (double)fj;
  // rows with 0 < b_t < nj: [z, y)
  const int z = bound ? min(max((int)inv[fj + 1], fi), ge) : fi;
  const int y = bound ? min(max((int)inv[fj + nj], fi), ge) : fi;
  const int z1 = __shfl_down_sync(kFull, z, 1), y1 = __shfl_down_sync(kFull, y, 1);
  // codes the bands of the group can hold: edges m0 .. mtop, the last of them
  // (top) above every code unless it is n1
  int m0 = 1, mtop = 1;
  bool top = true;
  if (COORD == kCart) {
    float ulo = 1e30f, uhi = 0.f;
    if (owner && z1 < y) {  // rows of band t: from the first with b_{t+1} > 0 to the last with b_t < nj
      const int c0 = min(max((int)tt[z1] - fj, 0), nj - 1);
      const int c1 = min((int)tt[A.ngp + y - 1] - fj, nj) - 1;
      ulo = __fmul_rn(__fmul_rn(U[z1], ap), U[fj + c0]);
      uhi = __fmul_rn(__fmul_rn(U[y - 1], ap), U[fj + max(c1, 0)]);
    }
    ulo = __uint_as_float(__reduce_min_sync(kFull, __float_as_uint(ulo)));
    uhi = __uint_as_float(__reduce_max_sync(kFull, __float_as_uint(uhi)));
    if (ulo > uhi) return;  // no band of the group has a row
    const float tlo = sqrt_approx(ulo) + A.off1f, thi = sqrt_approx(uhi) + A.off1f;
    m0 = min(max((int)floorf(fminf(tlo, 1e9f)), 0), n1);
    while (m0 <= n1 && !(ulo < A.edges[m0].y)) ++m0;  // edges below every pair of the group
    while (m0 > 0 && ulo < A.edges[m0 - 1].y) --m0;
    mtop = min(max((int)floorf(fminf(thi, 1e9f)), m0), n1);
    while (mtop < n1 && !(uhi < A.edges[mtop + 1].x)) ++mtop;  // edges above every pair
    top = mtop < n1;           // the highest codes end with the band, not with an edge
    if (top) ++mtop;
    if (m0 > mtop) m0 = mtop;  // no edge crosses the group
  }
  if (!GAPS && owner && z1 < y) {  // pairs of the band, whatever their code
    const uint32_t nt = (tb[y] - tb[z]) - (uint32_t)fj * (uint32_t)(y - z);
    const uint32_t* tb1 = tb + (A.ng + 1);
    const uint32_t nt1 = (tb1[y1] - tb1[z1]) - (uint32_t)fj * (uint32_t)(y1 - z1) + (uint32_t)nj * (uint32_t)(y - y1);
    stats[0] += nt1 - nt;
  }
  // rho(e): a row of [z, y] below which u < edges[e].x at column b_t, from
  // the level table: u >= edges[e].x needs d1 d2 >= edges[e].x / ap
  const uint16_t* lev = A.glev + (size_t)t * (A.nlev + 1);
  const float rap = COORD == kCart ? __fdividef(A.lev_scale, ap) : 0.f;
  auto row_bound = [&](int e) {
    if (COORD == kObs || (top && e == mtop)) return y;
    const float l = __fmaf_rn(A.edges[e].x, rap, A.lev_off);
    return l >= 0.f ? min(max((int)lev[(int)fminf(l, (float)A.nlev)], z), y) : z;
  };
  unsigned rech = 0;
  int cur = z, rho = row_bound(m0);
  double tzc = 0.0, lpc = 0.0;
  uint32_t tbc = 0u;
  if (!GAPS) {
    tzc = tz[z];
    lpc = A.glp[z];
    tbc = tb[z];
  }
  BandSums<GAPS> xp;  // X_t of the edge before
#pragma unroll
  for (int f = 0; f < 6; ++f) xp.s[f] = 0.0;
  xp.z = 0.0;
  xp.n = 0;
  const double bias = 4503599627370496.0 + dfj;  // 2^52 + f_j
#pragma unroll 1
  for (int e = m0; e <= mtop; ++e) {
    const bool last = COORD == kObs || (top && e == mtop);
    // loads of this edge's row and the next edge's bound, used after the loop
    double tzr = 0.0, lpr = 0.0;
    uint32_t tbr = 0u;
    if (!GAPS) {
      tzr = tz[rho];
      lpr = A.glp[rho];
      tbr = tb[rho];
    }
    const int rho_next = e < mtop ? row_bound(e + 1) : y;
    // V: rows [cur, rho), four at a time.  A lane's row and column advance
    // together, so the banks that eight lanes read side by side (one 128-byte
    // wavefront when all differ) are set by where each starts: with lane l
    // starting in a row of residue m l mod 8 (m odd) its columns have the
    // residues m l + (column - row), and m = 1, 3, 5 or 7 is taken for the most
    // different ones.  A lane idles through the rows before cur.
    double a[GAPS ? 8 : 6];
#pragma unroll
    for (int f = 0; f < (GAPS ? 8 : 6); ++f) a[f] = 0.0;
    {
      const int l8 = lane & 7;
      const int lag = rho > cur ? (int)tt[cur] - cur : l8;
      unsigned used = (1u << ((l8 + lag) & 7)) | (0x100u << ((3 * l8 + lag) & 7)) | (0x10000u << ((5 * l8 + lag) & 7)) |
                      (0x1000000u << ((7 * l8 + lag) & 7));
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) used |= __shfl_xor_sync(kFull, used, o);
      int mul = 1, best = __popc(used & 0xFFu);
#pragma unroll
      for (int q = 1; q < 4; ++q) {
        const int n = __popc(used & (0xFFu << (8 * q)));
        if (n > best) {
          best = n;
          mul = 2 * q + 1;
        }
      }
      int g = cur - ((cur - mul * l8) & 7);
      const uint2* tp = ts + (g >> 2) * 32;
      const bool odd = g & 1, high = g & 2;  // the group's first row in its table entry
      const double2* rp = it.R + (g - fi);
      const double2* pj = it.P - fj;
      uint2 w = __ldg(tp), wn = __ldg(tp + 32);
      tp += 64;
#pragma unroll 1
      for (; g < rho; g += 4, rp += 4) {
        const uint2 wp = __ldg(tp);  // two groups ahead
        tp += 32;
        const uint32_t u0 = high ? w.y : w.x, u1 = high ? wn.x : w.y, u2 = high ? wn.y : wn.x;
        const uint32_t v0 = odd ? __funnelshift_r(u0, u1, 16) : u0, v1 = odd ? __funnelshift_r(u1, u2, 16) : u1;
        const uint32_t x[4] = {v0 & 0xFFFFu, v0 >> 16, v1 & 0xFFFFu, v1 >> 16};
        w = wn;
        wn = wp;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          if (g + q >= cur && g + q < rho) {
            const double2 p = pj[x[q]], r = rp[q];
            if constexpr (GAPS) {
              add_gap_row(a, r, it.M[g + q - fi], p, it.C[(int)x[q] - fj]);
              continue;
            }
            const double b = __hiloint2double(0x43300000, (int)x[q]) - bias;  // the column as a double
            a[0] = __fma_rn(r.x, p.x, a[0]);
            a[1] = __fma_rn(r.x, b, a[1]);
            a[2] += p.x;
            a[3] = __fma_rn(r.y, p.y, a[3]);
            a[4] = __fma_rn(r.y, b, a[4]);
            a[5] += p.y;
          }
        }
      }
    }
    // X: rows from rho1 in which the edge crosses the band
    const int rho1 = __shfl_down_sync(kFull, rho, 1);
    BandSums<GAPS> x;
#pragma unroll
    for (int f = 0; f < 6; ++f) x.s[f] = 0.0;
    x.z = 0.0;
    x.n = 0;
    if (owner) {
      if (last) {
        // the band's end: rows [y1, y) with every column from b_t on
        if constexpr (GAPS) {
          if (y > y1) {
            const double2 pa = it.Pi[y1 - fi], pb = it.Pi[y - fi], ca = it.Ci[y1 - fi], cb = it.Ci[y - fi];
            add_gap_row(x, make_double2(pb.x - pa.x, pb.y - pa.y), make_double2(cb.x - ca.x, cb.y - ca.y), it.P[nj],
                        it.C[nj]);
          }
        } else if (y > y1) {
          const double2 p = it.P[nj];
          const double2 ra = it.Ri[y1 - fi], rb = it.Ri[y - fi];
          const double dn = (double)nj, dr = (double)(y - y1);
          x.s[0] = (rb.x - ra.x) * p.x;
          x.s[1] = (rb.x - ra.x) * dn;
          x.s[2] = dr * p.x;
          x.s[3] = (rb.y - ra.y) * p.y;
          x.s[4] = (rb.y - ra.y) * dn;
          x.s[5] = dr * p.y;
          x.z = 0.5 * ((A.glp[y] - A.glp[y1]) * dn + (A.glp[fj + nj] - lpj) * dr);
          x.n = (uint32_t)nj * (uint32_t)(y - y1);
        }
      } else if (rho1 < y) {
        const float4 eb = A.edges[e];
        const float* colx = U + fj;
        const uint16_t* t1 = tt + A.ngp;
        int b0n = tt[rho1], b1n = t1[rho1];
        for (int g = rho1; g < y; ++g) {
          const int b0 = max(b0n - fj, 0), b1 = min(b1n - fj, nj);
          b0n = tt[g + 1];  // (a boundary's row of the table is longer than the grid)
          b1n = t1[g + 1];
          const RowV V = code_row(A, ap, U[g]);
          if (__fmul_rn(V.A1, colx[b0]) >= eb.y) break;  // this row and all after it lie above the edge
          const int q = edge_column<MINPOS>(A, V, colx, it.c, b0, b1, e, make_float2(eb.z, eb.w), rech);
          add_edge_row(A, it, g, q, b0, g >= rho, lpj, x);
        }
      }
    }
    // the bin of the codes between this edge and the one before: boundary
    // t + 1 less boundary t, and the edges' rows
    const int code = (COORD == kObs) ? 0 : e - 1;
    FAcc F;
    double zc;
    if constexpr (GAPS) {
      F.n = (uint32_t)(__shfl_down_sync(kFull, a[7], 1) - a[7] + x.n - xp.n);
      zc = __shfl_down_sync(kFull, a[6], 1) - a[6] + x.z - xp.z;
    } else {
      // z sum and pair count of the rows [cur, rho)
      const double vz = (tzr - tzc) - 0.5 * (dfj * (lpr - lpc) + lpj * (double)(rho - cur));
      const uint32_t vn = (tbr - tbc) - (uint32_t)fj * (uint32_t)(rho - cur);
      F.n = __shfl_down_sync(kFull, vn, 1) - vn + x.n - xp.n;
      zc = __shfl_down_sync(kFull, vz, 1) - vz + x.z - xp.z;
    }
    bool tiny = false;
#pragma unroll
    for (int f = 0; f < 6; ++f) {
      const double v = __shfl_down_sync(kFull, a[f], 1) - a[f];
      F.s[f] = v + x.s[f] - xp.s[f];
      // a sum that cancels to rounding level may be one whose every term is zero
      const double mag = fabs(a[f]) + fabs(v) + fabs(x.s[f]) + fabs(xp.s[f]);
      tiny = tiny || (F.s[f] != 0.0 && fabs(F.s[f]) < 0x1p-36 * mag);
    }
    if (owner && F.n != 0u && code >= 0) {
      if (tiny) {
        // (observing: by the caller's copy, which then lives in memory and leaves
        // the sweep its registers: 7.3 -> 6.4 ms for 500 sightlines)
        const Sums6 q =
            band_by_rows<COORD, MINPOS, GAPS>(COORD == kObs ? it : s_item[buf], U, tt, min(z1, y), y, code);
        F.s[0] = q.a, F.s[1] = q.b, F.s[2] = q.c, F.s[3] = q.d, F.s[4] = q.e, F.s[5] = q.f;
      }
      F.s[6] = __fma_rn(A.lmid, (double)F.n, zc);
      F.code = code;
      if (GAPS) stats[0] += F.n;
      add_bin<COORD>(A, it.d, (t < n0) ? n0 - 1 - t : t - n0 - 1, code, F);
    }
    xp = x;
    cur = rho;
    rho = rho_next;
    tzc = tzr;
    lpc = lpr;
    tbc = tbr;
  }
  stats[1] += rech;
}

// Prepare the next owned item into `h` (all lanes of one warp; SMEM: its data
// into buf, arriving on `full`).
template <int COORD, bool SMEM, int L>
__device__ __noinline__ int prepare_item(BandItem* h, int* next, double2* buf, unsigned long long* full, int lane) {
  constexpr bool GAPS = L == kGaps;
  const PairArgs& A = s_args;
  int taken = 0;
  const int nb = 2 * (int)A.g.n0 + 1;
  BandItem it;
  it.bands = 0;
  for (;;) {
    unsigned long long idx = 0;
    if (!claim_item(A, GAPS ? kOwnerGaps : L == kShort ? kOwnerShort : kOwnerGrid, s_claim, lane, idx,
                    L == kShort ? A.short_claim : 1)) break;
    ++taken;
    const uint32_t i = A.item_i[idx], j = A.item_j[idx];
    it.ni = (int)A.gspan[i];
    it.nj = (int)A.gspan[j];
    it.fi = (int)A.gfirst[i];
    it.fj = (int)A.gfirst[j];
    // bands that hold a pair: b_{t+1} > 0 in the last row, b_t < nj in the first
    int tf = nb, tl = -1;
    const int gl = it.fi + it.ni - 1;
    for (int b = 0; b < nb; b += 32) {
      const int t = b + lane;
      const bool in = t < nb && (int)A.gtab[(size_t)(t + 1) * A.ngp + gl] > it.fj &&
                      (int)A.gtab[(size_t)t * A.ngp + it.fi] < it.fj + it.nj;
      const unsigned q = __ballot_sync(kFull, in);
      if (q) {
        tf = min(tf, b + __ffs(q) - 1);
        tl = b + 31 - __clz(q);
      }
    }
    if (tl < tf) continue;
    it.c = A.item_c[idx];
    const double a = 2.0 * dsub(1.0, it.c);
    it.ap = (float)(a * A.g.inv1 * A.g.inv1);
    const int len = A.max_span + 1;
    const double2 *gP, *gR, *gC = nullptr, *gM = nullptr;
    if (GAPS) {
      const uint64_t oi = A.gap_off[i], oj = A.gap_off[j];
      gP = A.gap_pre + oj;
      gC = A.gap_cnt + oj;
      gR = A.gap_row + oi;
      gM = A.gap_one + oi;
      it.Pi = A.gap_pre + oi;
      it.Ci = A.gap_cnt + oi;
    } else {
      it.Ri = A.pre2 + A.off[i] + i;
      gP = A.pre2 + A.off[j] + j;
      gR = A.row2 + A.off[i];
    }
    it.P = SMEM ? buf : gP;
    it.R = SMEM ? buf + len : gR;
    it.C = SMEM ? buf + 2 * len : gC;
    it.M = SMEM ? buf + 3 * len : gM;
    const float4 ri = A.range[i], rj = A.range[j];
    it.d.zb = zbin_of_sum(__fadd_rn(ri.z, rj.z), A.g);
    it.d.cell = dest_row(A, i, j);
    it.d.sep = (COORD == kObs) ? A.item_sep[idx] : 0u;
    it.tf = tf;
    it.bands = tl - tf + 1;
    const int groups = (it.bands + kBandsPerWarp - 1) / kBandsPerWarp;
    it.per = (it.bands + groups - 1) / groups;
    if (lane == 0) {
      *h = it;
      *next = 0;
      if (SMEM) {
        const uint32_t bp = (uint32_t)(it.nj + 1) * 16u, br = (uint32_t)it.ni * 16u;
        bar_arrive_tx(full, GAPS ? 2 * (bp + br) : bp + br);
        bulk_load(buf, gP, bp, full);
        bulk_load(buf + len, gR, br, full);
        if (GAPS) {
          bulk_load(buf + 2 * len, gC, bp, full);
          bulk_load(buf + 3 * len, gM, br, full);
        }
      } else {
        bar_arrive(full);
      }
    }
    __syncwarp();
    return taken;
  }
  if (lane == 0) {  // no item left
    *h = it;
    bar_arrive(full);
  }
  __syncwarp();
  return taken;
}

// The arguments stay in the kernel's parameter space (__grid_constant__):
// the inlined sweep reads them as constant-bank operands.
template <int COORD, bool MINPOS, bool SMEM, int L>
__global__ void __launch_bounds__(kGridWarps<L> * 32, L == kGaps ? 2 : 16 / kGridWarps<L>) grid_kernel(const __grid_constant__ PairArgs A) {
  constexpr bool GAPS = L == kGaps;
  extern __shared__ double2 band_smem[];
  __shared__ int s_next[2];  // GAPS: next group of each item
  __shared__ unsigned long long s_full[2], s_empty[2];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int len = A.max_span + 1, buf_len = (GAPS ? 4 : 2) * len;
  const float* U = A.gU;
  if (SMEM && L != kShort) {
    float* u = reinterpret_cast<float*>(band_smem + 2 * (size_t)buf_len);
    for (int g = tid; g < A.ng; g += kGridWarps<L> * 32) u[g] = A.gU[g];
    U = u;
  }
  if (tid == 0) {
    s_args = A;
    s_claim.todo = 0u;
    for (int b = 0; b < 2; ++b) {
      bar_init(&s_full[b], 1);
      bar_init(&s_empty[b], kGridWarps<L>);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  unsigned long long stats[2] = {0ull, 0ull};  // pairs in bands, FP64 re-evaluations
  unsigned long long n_taken = 0;
  bool ok = true;
  if (warp == 0)
    n_taken += prepare_item<COORD, SMEM, L>(&s_item[0], &s_next[0], band_smem, &s_full[0], lane);
  for (uint32_t k = 0;; ++k) {
    const uint32_t b = k & 1u, parity = (k >> 1) & 1u;
    ok = bar_wait(&s_full[b], parity, A.wait_ms);
    if (!ok) {
      // the copies that this warp started must land before it ends
      if (k == 0 ? warp == 0 : ((warp - (int)(k - 1)) & (kGridWarps<L> - 1)) == kGridWarps<L> - 1)
        bar_wait(&s_full[b], parity, kWaitMs);
      break;
    }
    BandItem it = s_item[b];
    if (it.bands == 0) break;
    if (SMEM) {  // the same pointers, known to be in shared memory
      it.P = band_smem + (size_t)b * buf_len;
      it.R = it.P + len;
      it.C = it.P + 2 * len;
      it.M = it.P + 3 * len;
    }
    // groups go round the warps from item to item, and the warp with the last
    // one, often none, prepares the next item (2,000 sightlines: 29.8 ms with a
    // fixed producer, 28.3; one warp alone is always that one)
    const int q0 = (warp - (int)k) & (kGridWarps<L> - 1);
    if (q0 == kGridWarps<L> - 1) {
      const uint32_t nb = b ^ 1u;
      // item k - 1 (the other buffer's) is done by every warp
      if (k > 0) ok = bar_wait(&s_empty[nb], ((k - 1) >> 1) & 1u, A.wait_ms);
      if (!ok) break;
      n_taken += prepare_item<COORD, SMEM, L>(&s_item[nb], &s_next[nb], band_smem + (SMEM ? (size_t)nb * buf_len : 0),
                                                 &s_full[nb], lane);
    }
    for (int q = q0;; q += kGridWarps<L>) {
      if (GAPS) {  // more warps than an item has groups: from a counter
        if (lane == 0) q = atomicAdd(&s_next[b], 1);
        q = __shfl_sync(kFull, q, 0);
      }
      if (q * it.per >= it.bands) break;
      band_group<COORD, MINPOS, GAPS>(A, it, U, it.tf + q * it.per, min(it.per, it.bands - q * it.per), lane, (int)b, stats);
    }
    __syncwarp();
    if (lane == 0) bar_arrive(&s_empty[b]);
  }
  if (!ok && lane == 0) atomicOr(&A.counters[13], GAPS ? kWaitGaps : kWaitGrid);  // a wait ran out: the host reports it
  add_counters(A, lane, stats[0], stats[1], n_taken, GAPS ? 8 : 9);
}

// Two items and (but for short ones, which read few of them) the grid's values.
template <int L>
size_t band_smem_bytes(const PairArgs& a) {
  return 2 * (size_t)(L == kGaps ? 4 : 2) * (a.max_span + 1) * sizeof(double2) +
         (L == kShort ? 0 : (size_t)a.ng * sizeof(float));
}

// Persistent launch: `ctas_per_sm` CTAs per SM (0 or above the occupancy
// limit: as many as fit), or with `max_out` set only that limit.
template <int COORD, bool MINPOS, bool SMEM, int L>
cudaError_t launch_grid(const PairArgs& a, int num_sms, int ctas_per_sm, cudaStream_t stream, int* max_out) {
  constexpr int threads = kGridWarps<L> * 32;
  const size_t smem = SMEM ? band_smem_bytes<L>(a) : 0;
  auto kern = grid_kernel<COORD, MINPOS, SMEM, L>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem);
  if (e != cudaSuccess) return e;
  per_sm = std::max(per_sm, 1);
  if (max_out) {
    *max_out = per_sm;
    return cudaSuccess;
  }
  if (ctas_per_sm > 0 && ctas_per_sm < per_sm) per_sm = ctas_per_sm;
  PairArgs b = a;
  b.claim_max = claim_limit(a.n_items, num_sms * per_sm);
  // (as many as leave each CTA several claims)
  b.short_claim = (int)std::min<unsigned long long>(
      kShortClaim, std::max<unsigned long long>(1, a.n_items / (4ull * num_sms * per_sm)));
  kern<<<num_sms * per_sm, threads, smem, stream>>>(b);
  return cudaGetLastError();
}

// Items and the grid's values are staged in shared memory when two items and
// the values fit a CTA (227 KB), the usual case: 622-pixel forests on 1,800
// values take 47 KB (87 KB with gaps).
constexpr size_t kBandSmem = 224 * 1024;

static_assert(2 * 2 * (kShortPixels + 1) * sizeof(double2) <= kBandSmem / 16, "short items: 16 CTAs an SM");

template <int COORD, bool MINPOS, int L>
cudaError_t launch_grid2(const PairArgs& a, int num_sms, int ctas_per_sm, cudaStream_t stream, int* max_out) {
  if constexpr (L == kShort)
    return launch_grid<COORD, MINPOS, true, L>(a, num_sms, ctas_per_sm, stream, max_out);
  else
    return band_smem_bytes<L>(a) <= kBandSmem
               ? launch_grid<COORD, MINPOS, true, L>(a, num_sms, ctas_per_sm, stream, max_out)
               : launch_grid<COORD, MINPOS, false, L>(a, num_sms, ctas_per_sm, stream, max_out);
}

template <int L>
cudaError_t launch_grid3(const PairArgs& a, int coord, bool minpos, int num_sms, int ctas_per_sm, cudaStream_t stream,
                         int* max_out) {
  if (coord == TOS_CARTESIAN)
    return minpos ? launch_grid2<kCart, true, L>(a, num_sms, ctas_per_sm, stream, max_out)
                  : launch_grid2<kCart, false, L>(a, num_sms, ctas_per_sm, stream, max_out);
  return launch_grid2<kObs, false, L>(a, num_sms, ctas_per_sm, stream, max_out);
}

}  // namespace

cudaError_t launch_grid_kernel(const PairArgs& a, int coord, bool minpos, int num_sms, int ctas_per_sm,
                               cudaStream_t stream, int* max_out) {
  return launch_grid3<kWhole>(a, coord, minpos, num_sms, ctas_per_sm, stream, max_out);
}

cudaError_t launch_short_kernel(const PairArgs& a, int coord, bool minpos, int num_sms, cudaStream_t stream) {
  return launch_grid3<kShort>(a, coord, minpos, num_sms, 0, stream, nullptr);
}

cudaError_t launch_gap_kernel(const PairArgs& a, int coord, bool minpos, int num_sms, cudaStream_t stream) {
  return launch_grid3<kGaps>(a, coord, minpos, num_sms, 0, stream, nullptr);
}

}  // namespace tos
