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
// grid alone and come from prefix tables over the rows.
//
// What bounds it: shared-memory reads.  A step (one row of 32 boundaries)
// takes two 16-byte reads per lane; lanes of neighbouring boundaries sit
// about three rows and three columns apart, so their reads fall in different
// banks, and the seven FP64 instructions of a step issue beside them.
//
// Measured on a B200 against the version that evaluated the r_perp code at
// every boundary of every row and bisected each split run (one warp per item):
// 16,000 sightlines at 16 per square degree, 50 x 50 bins: 970 -> 306 ms;
// 2,000 sightlines on 100 square degrees: 125 -> 39.9 ms; 48 sightlines (one
// wave, where the four warps of a CTA also shorten an item): 1.58 -> 0.17 ms;
// observing coordinates, 500 sightlines: 11.3 -> 7.3 ms.
#include <algorithm>

#include "xi_sweep.cuh"

namespace tos {
namespace {

constexpr int kGridWarps = 4;  // warps per CTA; a CTA takes one item at a time
constexpr int kGridThreads = kGridWarps * 32;
constexpr int kBandsPerWarp = 31;  // 32 boundaries

// Sums of a stretch of rows: w d w d, w d, w d, w w, w, w (didj, di, dj, wgt,
// wi, wj), the centred z sum and the pair count.
struct BandSums {
  double s[6];
  double z;
  uint32_t n;
};

// One item as its warps see it.
template <bool SMEM>
struct BandItem {
  int fi, fj, ni, nj;  // first grid index and pixels of the two sightlines
  const double2* P;    // prefix sums (w*delta, w) of sightline j, by column
  const double2* R;    // (w*delta, w) of sightline i, by row
  const double4* Ri;   // prefix sums of sightline i
  double c;
  float ap;            // Cartesian: 2 (1 - c) inv1^2
  Dest d;
};

// Row constants of the r_perp code of grid row g.
__device__ __forceinline__ RowV code_row(const PairArgs& A, float ap, int g) {
  RowV R;
  R.d1 = A.gU[g];
  const float p = __fmul_rn(R.d1, R.d1);
  const float err = __fmaf_rn(R.d1, R.d1, -p);  // d1*d1 = p + err exactly
  R.A1 = __fmul_rn(R.d1, ap);
  R.dl1 = __fmul_rn(-err, A.inv1sqf);
  return R;
}

// The bounds (lo, hi) of code edge m on u = 2 (1 - c) d1 d2 inv1^2 as computed
// in FP32 without the row's rounding term: a column with u < lo has a code
// below m and one with u >= hi has a code of at least m, for sure.  The margin
// covers the float rounding of d1*d1 (jit_u), four times the width of the
// FP64 re-evaluation window, and the FP32 rounding of u.
__device__ __forceinline__ float2 edge_bounds(const PairArgs& A, int m) {
  const float te = (m == 0) ? -1.0f : (float)m;
  const float se = te - A.off1f;
  if (!(se > 0.f)) return make_float2(-1.f, -1.f);  // below every column
  const float dt = ldexpf(4.f, -A.k1) + 1e-6f * fabsf(A.off1f);
  const float w = A.jit_u + 2.f * se * dt + dt * dt + 4e-6f * se * se;
  return make_float2(se * se - w, se * se + w);
}

// First column in [lo, hi) of row R with code >= m (hi when there is none).
template <bool MINPOS>
__device__ __forceinline__ int edge_column(const PairArgs& A, const RowV& R, const float* colx, double c,
                                           int lo, int hi, int m, unsigned& rech) {
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (perp_code<MINPOS>(A, R, colx[mid], c, rech) >= m) hi = mid; else lo = mid + 1;
  }
  return lo;
}

// The six sums of band t in code c evaluated row by row from differences of
// prefix sums, for a bin whose telescoped sums cancel to rounding level: a
// bin all of whose weights are zero sums to exactly zero this way.
template <int COORD, bool MINPOS>
__device__ __noinline__ void band_by_rows(const PairArgs& A, const double2* P, const double2* R, int fi, int fj,
                                          int nj, double c, float ap, const uint16_t* tt, int g0, int g1, int code,
                                          double* out) {
  double s[6] = {0, 0, 0, 0, 0, 0};
  unsigned rech = 0;
  for (int g = g0; g < g1; ++g) {
    int lo = min(max((int)tt[g] - fj, 0), nj), hi = min(max((int)tt[A.ngp + g] - fj, 0), nj);
    if (COORD == kCart) {
      const RowV V = code_row(A, ap, g);
      const int e = edge_column<MINPOS>(A, V, A.gU + fj, c, lo, hi, code + 1, rech);
      lo = edge_column<MINPOS>(A, V, A.gU + fj, c, lo, e, code, rech);
      hi = e;
    }
    if (hi <= lo) continue;
    const double2 a = P[lo], b = P[hi], r = R[g - fi];
    const double m = (double)(hi - lo), dwd = b.x - a.x, dw = b.y - a.y;
    s[0] += r.x * dwd;
    s[1] += r.x * m;
    s[2] += dwd;
    s[3] += r.y * dw;
    s[4] += r.y * m;
    s[5] += dw;
  }
#pragma unroll
  for (int f = 0; f < 6; ++f) out[f] = s[f];
}

// Bands t0 .. t0 + m - 1 of an item; lane = boundary t0 + lane (lane <= m).
template <int COORD, bool MINPOS, bool SMEM>
__device__ __forceinline__ void band_group(const PairArgs& A, const BandItem<SMEM>& it, int t0, int m, int lane,
                                           unsigned long long* stats) {
  const int n0 = (int)A.g.n0, n1 = (int)A.g.n1;
  const int t = t0 + min(lane, m);
  const bool bound = lane <= m;           // this lane owns a boundary
  const bool owner = lane < m && t != n0; // and a band that is binned
  const int k = (t < n0) ? n0 - 1 - t : t - n0 - 1;
  const int fi = it.fi, fj = it.fj, nj = it.nj, ge = it.fi + it.ni;
  const float ap = it.ap;
  const uint16_t* tt = A.gtab + (size_t)t * A.ngp;         // B_t by grid row
  const uint16_t* inv = A.ginv + (size_t)t * (A.ng + 1);   // first row with B_t >= column
  const double* tz = A.gtz + (size_t)t * (A.ng + 1);       // prefix sums over the rows
  const uint32_t* tb = A.gtb + (size_t)t * (A.ng + 1);
  const double lpj = A.glp[fj], dfj = (double)fj;
  // rows with 0 < b_t < nj: [z, y)
  const int z = bound ? min(max((int)inv[fj + 1], fi), ge) : fi;
  const int y = bound ? min(max((int)inv[fj + nj], fi), ge) : fi;
  const int z1 = __shfl_down_sync(kFull, z, 1), y1 = __shfl_down_sync(kFull, y, 1);
  // codes the bands of the group can hold
  int m0 = 1, mtop = 1;  // edges m0 .. mtop; the last is above every code unless it is n1
  bool top = true;
  if (COORD == kCart) {
    float ulo = 1e30f, uhi = 0.f;
    if (owner && z1 < y) {  // rows of band t: from the first with b_{t+1} > 0 to the last with b_t < nj
      const int c0 = min(max((int)tt[z1] - fj, 0), nj - 1);
      const int c1 = min((int)tt[A.ngp + y - 1] - fj, nj) - 1;
      ulo = __fmul_rn(__fmul_rn(A.gU[z1], ap), A.gU[fj + c0]);
      uhi = __fmul_rn(__fmul_rn(A.gU[y - 1], ap), A.gU[fj + max(c1, 0)]);
    }
    ulo = __uint_as_float(__reduce_min_sync(kFull, __float_as_uint(ulo)));
    uhi = __uint_as_float(__reduce_max_sync(kFull, __float_as_uint(uhi)));
    if (ulo > uhi) return;  // no band of the group has a row
    const float tlo = sqrtf(ulo) + A.off1f, thi = sqrtf(uhi) + A.off1f;
    m0 = max((int)floorf(fminf(tlo, 1e9f)), 0);
    while (m0 <= n1 && !(ulo < edge_bounds(A, m0).y)) ++m0;      // edges below every pair of the group
    while (m0 > 0 && ulo < edge_bounds(A, m0 - 1).y) --m0;
    if (m0 > n1) m0 = n1 + 1;  // every pair is above the axis
    mtop = min(max((int)floorf(fminf(thi, 1e9f)), m0), n1);
    while (mtop < n1 && !(uhi < edge_bounds(A, mtop + 1).x)) ++mtop;  // edges above every pair
    top = mtop < n1;           // the highest codes end with the band, not with an edge
    if (top) ++mtop;
    if (m0 > mtop) m0 = mtop;  // no edge crosses the group
  }
  if (owner && z1 < y) {  // pairs of the band, whatever their code
    const uint32_t nt = (tb[y] - tb[z]) - (uint32_t)fj * (uint32_t)(y - z);
    const uint32_t* tb1 = tb + (A.ng + 1);
    const uint32_t nt1 = (tb1[y1] - tb1[z1]) - (uint32_t)fj * (uint32_t)(y1 - z1) + (uint32_t)nj * (uint32_t)(y - y1);
    stats[0] += nt1 - nt;
  }
  unsigned rech = 0;
  int cur = z;
  BandSums xp;  // X_t of the edge before
#pragma unroll
  for (int f = 0; f < 6; ++f) xp.s[f] = 0.0;
  xp.z = 0.0;
  xp.n = 0;
  const double bias = 4503599627370496.0 + dfj;  // 2^52 + f_j
#pragma unroll 1
  for (int e = m0; e <= mtop; ++e) {
    const bool last = top && e == mtop;
    float2 eb = make_float2(0.f, 0.f);
    int rho = y;
    if (COORD == kCart && !last) {
      eb = edge_bounds(A, e);
      // rho: first row in [cur, y) with u >= eb.x at column b_t
      int lo = cur, hi = y;
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        const float u = __fmul_rn(__fmul_rn(A.gU[mid], ap), A.gU[tt[mid]]);
        if (u >= eb.x) hi = mid; else lo = mid + 1;
      }
      rho = lo;
    }
    // V: rows [cur, rho), four at a time
    double a[6] = {0, 0, 0, 0, 0, 0};
    {
      int g = cur & ~3;
      const uint2* tp = reinterpret_cast<const uint2*>(tt + g);
      const double2* rp = it.R + (g - fi);
      const double2* pj = it.P - fj;
#pragma unroll 1
      for (; g < rho; g += 4, rp += 4) {
        const uint2 w = __ldg(tp++);
        const uint32_t x[4] = {w.x & 0xFFFFu, w.x >> 16, w.y & 0xFFFFu, w.y >> 16};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          if (g + q >= cur && g + q < rho) {
            const double2 p = pj[x[q]], r = rp[q];
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
    // z sum and pair count of the same rows
    double vz = 0.0;
    uint32_t vn = 0;
    if (rho > cur) {
      vz = (tz[rho] - tz[cur]) - 0.5 * (dfj * (A.glp[rho] - A.glp[cur]) + lpj * (double)(rho - cur));
      vn = (tb[rho] - tb[cur]) - (uint32_t)fj * (uint32_t)(rho - cur);
    }
    // band: boundary t + 1 less boundary t
    const int rho1 = __shfl_down_sync(kFull, rho, 1);
    BandSums v;
    {
#pragma unroll
      for (int f = 0; f < 6; ++f) v.s[f] = __shfl_down_sync(kFull, a[f], 1) - a[f];
      v.z = __shfl_down_sync(kFull, vz, 1) - vz;
      v.n = __shfl_down_sync(kFull, vn, 1) - vn;
    }
    // X: rows from rho1 in which the edge crosses the band
    BandSums x;
#pragma unroll
    for (int f = 0; f < 6; ++f) x.s[f] = 0.0;
    x.z = 0.0;
    x.n = 0;
    if (owner) {
      if (COORD == kObs || last) {
        // the band's end: rows [y1, y) with every column from b_t on
        if (y > y1) {
          const double2 p = it.P[nj];
          const double4 ra = it.Ri[y1 - fi], rb = it.Ri[y - fi];
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
      } else {
        const float* colx = A.gU + fj;
        for (int g = rho1; g < y; ++g) {
          const int b0 = min(max((int)tt[g] - fj, 0), nj), b1 = min((int)tt[A.ngp + g] - fj, nj);
          const RowV V = code_row(A, ap, g);
          if (__fmul_rn(V.A1, colx[b0]) >= eb.y) break;  // this row and all after it lie above the edge
          const int q = edge_column<MINPOS>(A, V, colx, it.c, b0, b1, e, rech);
          double2 p = it.P[q];
          const double2 r = it.R[g - fi];
          double bd = (double)q, lz = A.glp[fj + q];
          int bn = q;
          double l0 = lpj;
          if (g >= rho) {  // V_t stopped before this row
            const double2 p0 = it.P[b0];
            p.x -= p0.x;
            p.y -= p0.y;
            bd -= (double)b0;
            bn -= b0;
            l0 = A.glp[fj + b0];
          }
          x.s[0] = __fma_rn(r.x, p.x, x.s[0]);
          x.s[1] = __fma_rn(r.x, bd, x.s[1]);
          x.s[2] += p.x;
          x.s[3] = __fma_rn(r.y, p.y, x.s[3]);
          x.s[4] = __fma_rn(r.y, bd, x.s[4]);
          x.s[5] += p.y;
          x.z = __fma_rn(0.5, __fma_rn((double)A.gl[g] - A.lmid, bd, lz - l0), x.z);
          x.n += (uint32_t)bn;
        }
      }
      // the bin of the codes between this edge and the one before
      const int code = (COORD == kObs) ? 0 : e - 1;
      FAcc F;
      F.n = v.n + x.n - xp.n;
      if (F.n != 0u && code >= 0) {
        const double zc = v.z + x.z - xp.z;
        bool tiny = false;
#pragma unroll
        for (int f = 0; f < 6; ++f) {
          F.s[f] = v.s[f] + x.s[f] - xp.s[f];
          const double mag = fabs(a[f]) + fabs(v.s[f]) + fabs(x.s[f]) + fabs(xp.s[f]);
          tiny = tiny || (F.s[f] != 0.0 && fabs(F.s[f]) < 0x1p-36 * mag);
        }
        if (tiny) {
          double s[6];
          band_by_rows<COORD, MINPOS>(A, it.P, it.R, fi, fj, nj, it.c, ap, tt, z1, y, code, s);
#pragma unroll
          for (int f = 0; f < 6; ++f) F.s[f] = s[f];
        }
        F.s[6] = __fma_rn(A.lmid, (double)F.n, zc);
        F.code = code;
        add_bin<COORD>(A, it.d, k, code, F);
      }
    }
    xp = x;
    cur = rho;
  }
  stats[1] += rech;
}

// The arguments stay in the kernel's parameter space (__grid_constant__):
// the inlined sweep reads them as constant-bank operands.
template <int COORD, bool MINPOS, bool SMEM>
__global__ void __launch_bounds__(kGridThreads, 5) grid_kernel(const __grid_constant__ PairArgs A) {
  extern __shared__ double2 band_smem[];
  __shared__ unsigned long long s_idx;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  unsigned long long stats[2] = {0ull, 0ull};  // pairs in bands, FP64 re-evaluations
  unsigned long long n_taken = 0;
  const int n0 = (int)A.g.n0, nb = 2 * n0 + 1;
  for (;;) {
    __syncthreads();  // the last item's shared data is free
    if (tid == 0) s_idx = atomicAdd(A.next_item, 1ull);
    __syncthreads();
    const unsigned long long idx = s_idx;
    if (idx >= A.n_items) break;
    if (item_owner(A, idx) != kOwnerGrid) continue;  // another kernel's item
    if (warp == 0) ++n_taken;
    const uint32_t i = A.item_i[idx], j = A.item_j[idx];
    BandItem<SMEM> it;
    it.ni = (int)A.npix[i];
    it.nj = (int)A.npix[j];
    it.fi = (int)A.gfirst[i];
    it.fj = (int)A.gfirst[j];
    it.c = A.item_c[idx];
    const double a = 2.0 * dsub(1.0, it.c);
    it.ap = (float)(a * A.g.inv1 * A.g.inv1);
    it.Ri = A.prefix + A.off[i] + i;
    const double2* gP = A.pre2 + A.off[j] + j;
    const double2* gR = A.row2 + A.off[i];
    // bands that hold a pair: b_{t+1} > 0 in the last row, b_t < nj in the first
    int tf = nb, tl = -1;
    {
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
    }
    if (tl < tf) continue;  // the same in every warp
    if (SMEM) {
      double2* sP = band_smem;
      double2* sR = band_smem + A.max_np + 1;
      for (int q = tid; q <= it.nj; q += kGridThreads) sP[q] = gP[q];
      for (int q = tid; q < it.ni; q += kGridThreads) sR[q] = gR[q];
      it.P = sP;
      it.R = sR;
    } else {
      it.P = gP;
      it.R = gR;
    }
    const float4 ri = A.range[i], rj = A.range[j];
    it.d.zb = zbin_of_sum(__fadd_rn(ri.z, rj.z), A.g);
    it.d.cell = dest_row(A, i, j);
    it.d.sep = (COORD == kObs) ? A.item_sep[idx] : 0u;
    __syncthreads();
    const int bands = tl - tf + 1;
    const int groups = (bands + kBandsPerWarp - 1) / kBandsPerWarp;
    const int per = (bands + groups - 1) / groups;
    for (int q = warp; q * per < bands; q += kGridWarps)
      band_group<COORD, MINPOS, SMEM>(A, it, tf + q * per, min(per, bands - q * per), lane, stats);
  }
  add_counters(A, lane, stats[0], stats[1], n_taken, 9);
}

// Persistent launch: `ctas_per_sm` CTAs per SM (0 or above the occupancy
// limit: as many as fit), or with `max_out` set only that limit.
template <int COORD, bool MINPOS, bool SMEM>
cudaError_t launch_grid(const PairArgs& a, int num_sms, int ctas_per_sm, cudaStream_t stream, int* max_out) {
  const size_t smem = SMEM ? (size_t)(2 * a.max_np + 1) * sizeof(double2) : 0;
  auto kern = grid_kernel<COORD, MINPOS, SMEM>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kGridThreads, smem);
  if (e != cudaSuccess) return e;
  per_sm = std::max(per_sm, 1);
  if (max_out) {
    *max_out = per_sm;
    return cudaSuccess;
  }
  if (ctas_per_sm > 0 && ctas_per_sm < per_sm) per_sm = ctas_per_sm;
  kern<<<num_sms * per_sm, kGridThreads, smem, stream>>>(a);
  return cudaGetLastError();
}

// Longest sightline whose prefix sums and row values are staged in shared
// memory: both fit a CTA with at least two CTAs on an SM.
constexpr int kBandSmemPixels = 3400;

template <int COORD, bool MINPOS>
cudaError_t launch_grid2(const PairArgs& a, int num_sms, int ctas_per_sm, cudaStream_t stream, int* max_out) {
  return a.max_np <= kBandSmemPixels ? launch_grid<COORD, MINPOS, true>(a, num_sms, ctas_per_sm, stream, max_out)
                                     : launch_grid<COORD, MINPOS, false>(a, num_sms, ctas_per_sm, stream, max_out);
}

}  // namespace

cudaError_t launch_grid_kernel(const PairArgs& a, int coord, bool minpos, int num_sms, int ctas_per_sm,
                               cudaStream_t stream, int* max_out) {
  if (coord == TOS_CARTESIAN)
    return minpos ? launch_grid2<kCart, true>(a, num_sms, ctas_per_sm, stream, max_out)
                  : launch_grid2<kCart, false>(a, num_sms, ctas_per_sm, stream, max_out);
  return launch_grid2<kObs, false>(a, num_sms, ctas_per_sm, stream, max_out);
}

}  // namespace tos
