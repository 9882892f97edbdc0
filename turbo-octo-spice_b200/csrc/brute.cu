// brute.cu — all-pairs isotropic xi(r) of points (x, y, z, delta, w): the
// computation of bruteGPU / histo_kernel (gpu/brute.cu:7-61, 63-225), redone
// for sm_100a.
//
// Differences from the reference design, all in service of exactness and
// throughput:
//  - points stay resident in HBM (no per-chunk host copies, brute.cu:155-193);
//  - points in lines of P equal steps (a regular grid's lines; found and
//    checked exactly on the device) go through line_kernel: all pairs of two
//    lines with the same offset have one separation, so it is binned once;
//  - other points go through brute_kernel: every unordered pair i < j is
//    visited once, along diagonals: a pair (i, i + delta) lies on diagonal
//    delta, a lane owns K consecutive diagonals of a group of 32 K and walks a
//    segment of rows (i = i0, i0 + 1, ...), so the row's point is a broadcast
//    load and the lane's K columns are a register window that slides by one
//    column per row.  A pair whose separation is that of the row before keeps
//    its bin;
//  - separations are binned in FP32 with an FP64 re-binning of pairs within
//    2^-K bins of an edge, so bins equal those of the FP64 separation
//    sqrt(dx^2+dy^2+dz^2) (the double-precision estimator of bucketxi.cc:79-98);
//  - sums are exact: while a diagonal stays in one bin (or over a pair of
//    lines' offset) the lane adds the FP64 products w_i d_i w_j d_j and w_i w_j
//    in registers; a run that ends goes, rounded once to fixed point, into a
//    per-warp shared-memory window and from there to global 128-bit sums.
//    Integer sums do not depend on the order of the adds and runs do not
//    depend on the launch shape, so the result is the same for every shape.
//
// Measured on a B200 (kernel ms) against the version that walked whole
// diagonals, one group of 32 per warp, and added runs 32 at a time with 64-bit
// shared-memory adds: 64^3 grid, 100 bins: 150 -> 16.3; 20,011 scattered points,
// 50 bins: 42 -> 1.22.  There 625 groups left most warps idle for 20,000 serial
// rows (segments: 42 -> 4.2), the warps' adds met on 16 lines of global sums
// (copies: 4.2 -> 1.4) and window adds on few banks (slot copies).  On the grid
// the diagonal kernel takes 102 ms: 33 of 64 rows change some lane's bin.
// line_kernel is bound by issue and shared-memory adds (58 % and 57 %); its
// 2 FP64 FMAs per pair alone take 3.7 ms.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <limits>
#include <vector>

#include "engine_internal.h"
#include "fixed128.cuh"

namespace tos {
namespace {

constexpr unsigned kFull = 0xFFFFFFFFu;
constexpr int kBruteWarpsMax = 16;  // warps per CTA at most
constexpr int kBWin = 5;            // u64 words per bin of the global sums: dsum lo, hi, wsum lo, hi, count
constexpr int kBWords = 7;          // u32 words per bin of a warp's window (window_add)
constexpr int kBruteAdds = 2016;    // values a window slot takes: 2016 * 2^20 < 2^31
constexpr uint32_t kNoBin = 0xFFFFFFFFu;
constexpr int kBruteAccBins = 4098; // bins of the global sums: copies of nbins + 2 fit in as often as they do
constexpr double kMagic = 6755399441055744.0;  // 1.5 * 2^52

struct BruteArgs {
  const float4* pos;      // (x, y, z, w), n entries
  const double* wd;       // w*delta per point (exact product of the two floats)
  int n;
  int nbins;
  double min, max, spacing;
  float invf, offf, nbf, nbp1f;
  int k;
  float mag;
  int bits;
  double scale_hi[2];     // 2^(F - 42) of fields dsum, wsum: |run sum| * 2^F < 2^62
  int seg;                // rows of a segment: a run has at most that many pairs
  int exact_diff;         // differences of coordinates are exact in FP32
  int wshift;             // log2 of the copies of a window slot (lane l adds to copy l mod 2^wshift)
  int copies;             // copies of the global sums, to spread the adds over (k_brute_finish adds them up)
  int carry;              // the global sums are 128-bit integers with a carry (brute_args)
  // line_kernel: Q lines of P points, step (sx, sy, sz)
  int P, Q, eblocks;      // eblocks: offset blocks per unit
  float sx, sy, sz;
  const double2* val;     // (w*delta, w), point z of line l at z Q + l
  const float4* base;     // first point of each line
  const double* th;       // [nbins + 3] exact-index thresholds on r^2 (brute_thresholds)
  unsigned long long* acc;       // [copies][nbins + 2][kBWin] sums and counts
  unsigned long long* next;      // diagonal-group counter
  unsigned long long* counters;  // [0] FP64 re-binnings
};

__device__ __forceinline__ float sqrt_approx(float x) {
  float r;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// round(c * 2^F) for |c * 2^F| < 2^62, given sh = 2^(F - 42), as w[0] + w[1] 2^21
// + w[2] 2^42 with |w| <= 2^20: each part is rounded off the exact remainder of
// the one above it, and is the low word of its sum with 1.5 * 2^52.
__device__ __forceinline__ void fixed_parts(double c, double sh, int (&w)[3]) {
  const double t2 = __fma_rn(c, sh, kMagic);
  w[2] = __double2loint(t2);
  const double r2 = __fma_rn(c, sh, -__dsub_rn(t2, kMagic));
  const double t1 = __fma_rn(r2, 2097152.0 /* 2^21 */, kMagic);
  w[1] = __double2loint(t1);
  const double r1 = __fma_rn(r2, 2097152.0, -__dsub_rn(t1, kMagic));
  w[0] = __double2loint(__fma_rn(r1, 2097152.0, kMagic));
}

// Histogram index of the FP64 separation, 0 below min, nbins+1 at or above
// max, else floor((r - min) / spacing) + 1 with r = sqrt(dx^2 + dy^2 + dz^2)
// in FP64 (gpu/brute.cu:40-48, bucketxi.cc:79-98).  The index is a
// non-decreasing function of the FP64 r^2, so th[b] (b = 1 .. nbins + 1) is
// the smallest r^2 whose index is at least b (brute_thresholds, with
// th[0] = -1 and th[nbins + 2] = +inf), and an index known to lie within one
// of `near` is decided by two comparisons of r^2.
__device__ __forceinline__ uint32_t exact_index(const BruteArgs& A, float4 a, float4 b, int near) {
  const double dx = dsub((double)a.x, (double)b.x), dy = dsub((double)a.y, (double)b.y),
               dz = dsub((double)a.z, (double)b.z);
  const double r2 = dadd(dadd(dmul(dx, dx), dmul(dy, dy)), dmul(dz, dz));
  const int c = min(max(near, 0), A.nbins + 1);
  return (uint32_t)(c - 1 + (r2 >= A.th[c] ? 1 : 0) + (r2 >= A.th[c + 1] ? 1 : 0));
}

// FP32 histogram index of a separation, and whether it lies within 2^-K bins
// of an edge.
__device__ __forceinline__ int fast_index(const BruteArgs& A, float dx, float dy, float dz, bool& near) {
  const float r2 = __fmaf_rn(dx, dx, __fmaf_rn(dy, dy, __fmul_rn(dz, dz)));
  const float tt = __fmaf_rn(sqrt_approx(r2), A.invf, A.offf);
  const int qq = __float_as_int(__fadd_rz(tt, A.mag)) - A.bits;
  near = (((qq + 1) & ((1 << A.k) - 1)) < 2) && (tt < A.nbp1f) && (tt > -1.f);
  return (tt < 0.f) ? 0 : ((tt >= A.nbf) ? A.nbins + 1 : (qq >> A.k) + 1);
}

// Add a closed run (bin, pairs m, FP64 sums) of this lane to the warp window.
// A window slot is seven 32-bit words, native shared-memory adds: the two sums'
// fixed-point values in three signed parts each (fixed_parts) and the pairs; a
// slot takes kBruteAdds values before a word could overflow.  The
// lanes of a warp often add to the same few bins: a slot has up to eight
// copies in neighbouring banks, one for every 2^wshift-th lane.
__device__ __forceinline__ void window_add(const BruteArgs& A, int* win, int S, int lane, uint32_t bin, uint32_t m,
                                           double dsum, double wsum) {
  int v0[3], v1[3];
  fixed_parts(dsum, A.scale_hi[0], v0);
  fixed_parts(wsum, A.scale_hi[1], v1);
  int* p = win + ((bin << A.wshift) | (lane & ((1u << A.wshift) - 1u)));
  const int step = S << A.wshift;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    atomicAdd(p + k * step, v0[k]);
    atomicAdd(p + (3 + k) * step, v1[k]);
  }
  atomicAdd(p + 6 * step, (int)m);
}

// Add the warp window to the global sums (carry-free: low 32 bits and the
// signed rest of each value; CARRY: 128-bit integers) and clear it.  (A
// template: with the choice made at run time the scattered points' kernel took
// 4 to 10 % longer.)
template <bool CARRY>
__device__ __noinline__ void brute_flush(const BruteArgs& A, int* win, int S, int lane) {
  __syncwarp();
  const int step = S << A.wshift;
  for (int b = lane; b < S; b += 32) {
    unsigned long long cnt = 0;
    long long part[2][3] = {{0, 0, 0}, {0, 0, 0}};
    for (int c = 0; c < (1 << A.wshift); ++c) {
      int* p = win + ((b << A.wshift) | c);
      const uint32_t n = (uint32_t)p[6 * step];
      if (n == 0) continue;  // every run has at least one pair
      cnt += n;
#pragma unroll
      for (int k = 0; k < 6; ++k) part[k / 3][k % 3] += p[k * step];
#pragma unroll
      for (int w = 0; w < kBWords; ++w) p[w * step] = 0;
    }
    if (cnt == 0) continue;
    unsigned long long* g = A.acc + ((size_t)(blockIdx.x % A.copies) * S + b) * kBWin;
#pragma unroll
    for (int f = 0; f < 2; ++f) {
      const __int128 v = ((__int128)part[f][2] << 42) + ((__int128)part[f][1] << 21) + (__int128)part[f][0];
      const unsigned long long lo = CARRY ? (unsigned long long)v : (unsigned long long)v & 0xFFFFFFFFull;
      long long h = (long long)(v >> (CARRY ? 64 : 32));
      if (CARRY)
        h += atomicAdd(&g[2 * f], lo) > ~lo;  // the low word's carry
      else
        atomicAdd(&g[2 * f], lo);
      if (h != 0) atomicAdd(&g[2 * f + 1], (unsigned long long)h);
    }
    atomicAdd(&g[4], cnt);
  }
  __syncwarp();
}

// Units: diagonal group g x row segment s, claimed in order of g.  Group g
// holds diagonals 1 + g * 32K .. 1 + (g + 1) * 32K - 1; lane L owns
// 1 + g * 32K + K L + m, m = 0 .. K-1; segment s is the rows [s seg, (s + 1) seg).
// A diagonal's runs end at a segment's end, whatever K is, so that the sums
// do not depend on the launch shape.
template <int K, bool CARRY>
__global__ void __launch_bounds__(kBruteWarpsMax * 32, K == 1 ? 2 : 1) brute_kernel(const __grid_constant__ BruteArgs A) {
  extern __shared__ int bsm[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int S = A.nbins + 2;
  int* win = bsm + (size_t)warp * ((kBWords * S) << A.wshift);
  for (int k = lane; k < (kBWords * S) << A.wshift; k += 32) win[k] = 0;
  __syncwarp();
  const int span = 32 * K;
  const int ngroups = (A.n - 1 + span - 1) / span, nseg = (A.n - 1 + A.seg - 1) / A.seg;
  const unsigned long long units = (unsigned long long)ngroups * nseg;
  unsigned long long n_recheck = 0;
  const int per = 32 >> A.wshift;  // values a slot can receive when every lane adds one
  int adds = 0;                    // values a window slot can have received
  for (;;) {
    unsigned long long u = 0;
    if (lane == 0) u = atomicAdd(A.next, 1ull);
    u = __shfl_sync(kFull, u, 0);
    if (u >= units) break;
    const int dg = 1 + (int)(u / nseg) * span;      // the group's first diagonal
    const int t0 = (int)(u % nseg) * A.seg;         // the segment's rows [t0, t1)
    const int t1 = min(t0 + A.seg, A.n - dg);       // rows with a pair on the group's first diagonal
    if (t0 >= t1) continue;
    const int d0 = dg + K * lane;      // this lane's first diagonal
    uint32_t cur[K], pbin[K], pm[K];   // bin of the open run; a closed run, not added yet (pm pairs)
    int s0[K];
    bool edge[K];                      // the pair lies near a bin edge
    double ds[K], ws[K], pd[K], pw[K];
    float ex[K], ey[K], ez[K];         // the last separation
    float4 cp[K];
    double cwd[K];
#pragma unroll
    for (int m = 0; m < K; ++m) {
      cur[m] = kNoBin;
      pbin[m] = pm[m] = 0u;
      s0[m] = t0;
      edge[m] = false;
      ds[m] = ws[m] = pd[m] = pw[m] = 0.0;
      ex[m] = ey[m] = ez[m] = __int_as_float(0x7FC00000);  // NaN: unlike every separation
    }
    // the lane's newest column (t + d0 + K - 1), walked by pointer; j_end: the first row without one
    const float4* pj = A.pos + (d0 + K - 1);
    const double* wdj = A.wd + (d0 + K - 1);
    const int j_end = A.n - (d0 + K - 1);
#pragma unroll
    for (int m = 0; m < K; ++m) {  // columns of row t0
      cp[m] = make_float4(0.f, 0.f, 0.f, 0.f);
      cwd[m] = 0.0;
      if (t0 + d0 + m < A.n) {
        cp[m] = A.pos[t0 + d0 + m];
        cwd[m] = A.wd[t0 + d0 + m];
      }
    }
    float4 pi = A.pos[t0];
    double wdi = A.wd[t0];
#pragma unroll 1
    for (int t = t0; t < t1; ++t) {
      // the next row and column load while this row is worked on
      const float4 npi = A.pos[t + 1];  // t + 1 < n: diagonals start at 1
      const double nwdi = A.wd[t + 1];
      float4 ncp = cp[K - 1];
      double ncwd = 0.0;
      if (t + 1 < j_end) {
        ncp = pj[t + 1];
        ncwd = wdj[t + 1];
      }
      const double wi = (double)pi.w;
#pragma unroll
      for (int m = 0; m < K; ++m) {
        const bool in = t < j_end + (K - 1 - m);  // t + d0 + m < n
        const float dx = __fsub_rn(pi.x, cp[m].x), dy = __fsub_rn(pi.y, cp[m].y),
                    dz = __fsub_rn(pi.z, cp[m].z);
        // An unchanged separation keeps its bin: for points on a grid it
        // changes only where the row or the column wraps to the next line.
        // (A pair near an edge is decided by the FP64 separation, which can
        // change under equal FP32 differences unless those are exact.)
        const bool fresh = in && (dx != ex[m] || dy != ey[m] || dz != ez[m] || (edge[m] && !A.exact_diff));
        if (__any_sync(kFull, fresh)) {
          bool near;
          const int b = fast_index(A, dx, dy, dz, near);
          uint32_t key = cur[m];
          if (fresh) {
            key = (uint32_t)b;
            if (near) {
              key = exact_index(A, pi, cp[m], b);
              ++n_recheck;
            }
            edge[m] = near;
            ex[m] = dx;
            ey[m] = dy;
            ez[m] = dz;
          }
          const bool change = key != cur[m];
          const bool close = change && cur[m] != kNoBin;
          // a lane keeps one closed run; when one closes its second, every
          // lane adds the run it keeps (scattered points: 32 runs a row)
          if (__any_sync(kFull, close && pm[m] != 0u)) {
            if (adds + per > kBruteAdds) {
              brute_flush<CARRY>(A, win, S, lane);
              adds = 0;
            }
            if (pm[m] != 0u) window_add(A, win, S, lane, pbin[m], pm[m], pd[m], pw[m]);
            adds += per;
            pm[m] = 0u;
          }
          if (close) {
            pbin[m] = cur[m];
            pm[m] = (uint32_t)(t - s0[m]);
            pd[m] = ds[m];
            pw[m] = ws[m];
          }
          if (change) {
            cur[m] = key;
            s0[m] = t;
            ds[m] = 0.0;
            ws[m] = 0.0;
          }
        }
        if (in) {
          ds[m] = __fma_rn(wdi, cwd[m], ds[m]);
          ws[m] = __fma_rn(wi, (double)cp[m].w, ws[m]);
        }
      }
#pragma unroll
      for (int m = 0; m + 1 < K; ++m) {
        cp[m] = cp[m + 1];
        cwd[m] = cwd[m + 1];
      }
      cp[K - 1] = ncp;
      cwd[K - 1] = ncwd;
      pi = npi;
      wdi = nwdi;
    }
    // the runs kept and the runs still open: a diagonal's last pair is at row
    // n - 1 - diagonal or at the segment's end
#pragma unroll
    for (int m = 0; m < K; ++m) {
      if (adds + 2 * per > kBruteAdds) {
        brute_flush<CARRY>(A, win, S, lane);
        adds = 0;
      }
      if (pm[m] != 0u) window_add(A, win, S, lane, pbin[m], pm[m], pd[m], pw[m]);
      const int e = min(t1, j_end + (K - 1 - m));
      if (cur[m] != kNoBin && e > s0[m]) window_add(A, win, S, lane, cur[m], (uint32_t)(e - s0[m]), ds[m], ws[m]);
      adds += 2 * per;
    }
  }
  brute_flush<CARRY>(A, win, S, lane);
  for (int o = 16; o > 0; o >>= 1) n_recheck += __shfl_xor_sync(kFull, n_recheck, o);
  if (lane == 0) atomicAdd(&A.counters[0], n_recheck);
}

// Over the points: out[0], out[1] the largest |w * delta| and |w| (bit patterns
// of non-negative doubles), out[2] whether a value is not finite, out[3] the
// largest |coordinate| (float bits) and out[4] 1024 less the smallest exponent
// of a coordinate's lowest set bit: the coordinates are multiples of
// 2^(1024 - out[4]).
__global__ void k_brute_bounds(const float* pts, int n, unsigned long long* out) {
  double mwd = 0, mw = 0;
  bool nonfinite = false;
  unsigned top = 0u, low = 0u;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    const float* p = pts + 5 * (size_t)k;
    if (!isfinite(p[0]) || !isfinite(p[1]) || !isfinite(p[2]) || !isfinite(p[3]) || !isfinite(p[4]))
      nonfinite = true;
    mwd = fmax(mwd, fabs((double)p[4] * (double)p[3]));
    mw = fmax(mw, fabs((double)p[4]));
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const unsigned u = __float_as_uint(p[a]) & 0x7FFFFFFFu;
      if (u == 0u) continue;
      top = max(top, u);
      const unsigned ex = u >> 23, man = ex ? (u & 0x7FFFFFu) | 0x800000u : u;
      const int bit = (int)max(ex, 1u) - 150 + (__ffs((int)man) - 1);
      low = max(low, (unsigned)(1024 - bit));
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    mwd = fmax(mwd, __shfl_xor_sync(kFull, mwd, o));
    mw = fmax(mw, __shfl_xor_sync(kFull, mw, o));
  }
  top = __reduce_max_sync(kFull, top);
  low = __reduce_max_sync(kFull, low);
  nonfinite = __any_sync(kFull, nonfinite);
  if ((threadIdx.x & 31) == 0) {
    atomicMax(&out[0], (unsigned long long)__double_as_longlong(mwd));
    atomicMax(&out[1], (unsigned long long)__double_as_longlong(mw));
    if (nonfinite) atomicOr(&out[2], 1ull);
    atomicMax(&out[3], (unsigned long long)top);
    atomicMax(&out[4], (unsigned long long)low);
  }
}

// Points in lines of P equal steps (a regular grid's lines): with line a's
// point z at base_a + z step, the pairs of two lines a <= b with z' - z = e all
// have one separation, so a lane (line b) bins an offset e once and adds
// P - |e| products.  A warp takes line a and 32 lines b; per block of kLineE
// offsets a window of kLineE points of line b slides along line a, so a step
// costs one 16-byte read per lane and a broadcast for 2 kLineE FP64 FMAs.
// Values are stored by z, then line.
constexpr int kLineE = 8;
template <bool CARRY>
__global__ void __launch_bounds__(kBruteWarpsMax * 32) line_kernel(const __grid_constant__ BruteArgs A) {
  extern __shared__ int bsm[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int S = A.nbins + 2;
  int* win = bsm + (size_t)warp * ((kBWords * S) << A.wshift);
  for (int k = lane; k < (kBWords * S) << A.wshift; k += 32) win[k] = 0;
  __syncwarp();
  const int P = A.P, Q = A.Q;
  const int groups = (Q + 31) >> 5, blocks = (2 * P - 1 + kLineE - 1) / kLineE;
  const int parts = (blocks + A.eblocks - 1) / A.eblocks;  // units per (line, group)
  const unsigned long long units = (unsigned long long)Q * groups * parts;
  unsigned long long n_recheck = 0;
  const int per = (32 >> A.wshift) * kLineE;
  int adds = 0;
  for (;;) {
    unsigned long long u = 0;
    if (lane == 0) u = atomicAdd(A.next, 1ull);
    u = __shfl_sync(kFull, u, 0);
    if (u >= units) break;
    const int part = (int)(u % parts);
    const int a = (int)((u / parts) / groups), g = (int)((u / parts) % groups);
    if (g * 32 + 31 < a) continue;  // every line of the group comes before line a
    const int b = g * 32 + lane;
    const bool in = b >= a && b < Q;
    const double2* row = A.val + a;
    const double2* col = A.val + min(b, Q - 1);
    const float4 pa = A.base[a], pb = A.base[min(b, Q - 1)];
    const int eb1 = min(blocks, (part + 1) * A.eblocks);
    for (int eb = part * A.eblocks; eb < eb1; ++eb) {
      const int e0 = -(P - 1) + eb * kLineE;  // offsets e0 .. e0 + kLineE - 1
      const int zlo = max(0, -(e0 + kLineE - 1)), zhi = min(P, P - e0);
      double ds[kLineE], ws[kLineE];
      double2 c[kLineE];
#pragma unroll
      for (int m = 0; m < kLineE; ++m) {
        ds[m] = ws[m] = 0.0;
        const int z = zlo + e0 + m - 1;  // shifted in by one at the first step
        c[m] = (z >= 0 && z < P) ? col[(size_t)z * Q] : make_double2(0.0, 0.0);
      }
#pragma unroll kLineE
      for (int z = zlo; z < zhi; ++z) {
        const double2 r = row[(size_t)z * Q];
        const int zc = z + e0 + kLineE - 1;
#pragma unroll
        for (int m = 0; m + 1 < kLineE; ++m) c[m] = c[m + 1];
        c[kLineE - 1] = zc < P ? col[(size_t)zc * Q] : make_double2(0.0, 0.0);
#pragma unroll
        for (int m = 0; m < kLineE; ++m) {
          ds[m] = __fma_rn(r.x, c[m].x, ds[m]);
          ws[m] = __fma_rn(r.y, c[m].y, ws[m]);
        }
      }
      if (adds + per > kBruteAdds) {
        brute_flush<CARRY>(A, win, S, lane);
        adds = 0;
      }
      adds += per;
#pragma unroll
      for (int m = 0; m < kLineE; ++m) {
        const int e = e0 + m;
        if (e < P && in && (b > a || e > 0)) {
          // the offset's first pair: every position is a float, so the sums are exact
          const float za = (float)max(0, -e), zb = (float)(max(0, -e) + e);
          const float4 p = make_float4(__fmaf_rn(za, A.sx, pa.x), __fmaf_rn(za, A.sy, pa.y), __fmaf_rn(za, A.sz, pa.z), 0.f);
          const float4 q = make_float4(__fmaf_rn(zb, A.sx, pb.x), __fmaf_rn(zb, A.sy, pb.y), __fmaf_rn(zb, A.sz, pb.z), 0.f);
          bool near;
          int bin = fast_index(A, __fsub_rn(p.x, q.x), __fsub_rn(p.y, q.y), __fsub_rn(p.z, q.z), near);
          if (near) {
            bin = (int)exact_index(A, p, q, bin);
            ++n_recheck;
          }
          window_add(A, win, S, lane, (uint32_t)bin, (uint32_t)(P - abs(e)), ds[m], ws[m]);
        }
      }
    }
  }
  brute_flush<CARRY>(A, win, S, lane);
  for (int o = 16; o > 0; o >>= 1) n_recheck += __shfl_xor_sync(kFull, n_recheck, o);
  if (lane == 0) atomicAdd(&A.counters[0], n_recheck);
}

// Line structure of the points (before the bounds are read): pass 0 finds the
// first step that differs from step 0 (out[0] = n less its index; 0: none),
// pass 1 counts the points off the pattern of lines of that length (out[1]).
__device__ __forceinline__ bool same_step(const float* p, float sx, float sy, float sz) {
  return __fsub_rn(p[5], p[0]) == sx && __fsub_rn(p[6], p[1]) == sy && __fsub_rn(p[7], p[2]) == sz;
}
__global__ void k_brute_lines(const float* pts, int n, int pass, unsigned long long* out) {
  const float sx = __fsub_rn(pts[5], pts[0]), sy = __fsub_rn(pts[6], pts[1]), sz = __fsub_rn(pts[7], pts[2]);
  const int P = pass ? n - (int)out[0] + 1 : 1;
  unsigned v = 0u;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t + 1 < n; t += gridDim.x * blockDim.x) {
    const bool same = same_step(pts + 5 * (size_t)t, sx, sy, sz);
    if (pass == 0) {
      if (!same) v = max(v, (unsigned)(n - t));
    } else if (!same && (t + 1) % P != 0) {
      ++v;
    }
  }
  if (pass == 0) {
    v = __reduce_max_sync(kFull, v);
    if ((threadIdx.x & 31) == 0 && v) atomicMax(&out[0], (unsigned long long)v);
  } else {
    v = __reduce_add_sync(kFull, v);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(&out[1], (unsigned long long)v);
  }
}

// (w*delta, w) by z, then line; line starts.
__global__ void k_line_prep(const float* pts, int n, int P, int Q, double2* val, float4* base) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    const float* p = pts + 5 * (size_t)k;
    const int line = k / P, z = k % P;
    val[(size_t)z * Q + line] = make_double2((double)p[4] * (double)p[3], (double)p[4]);
    if (z == 0) base[line] = make_float4(p[0], p[1], p[2], 0.f);
  }
}

__global__ void k_brute_prep(const float* pts, int n, float4* pos, double* wd) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    const float* p = pts + 5 * (size_t)k;
    pos[k] = make_float4(p[0], p[1], p[2], p[4]);
    wd[k] = (double)p[4] * (double)p[3];
  }
}

// 128-bit sums -> the caller's dsum, wsum (FP64) and counts.
__device__ __forceinline__ __int128 brute_sum(const unsigned long long* g, int carry) {
  return carry ? (__int128)(((unsigned __int128)g[1] << 64) | g[0])
               : (__int128)(long long)g[1] * (__int128)4294967296ll + (__int128)g[0];
}
__global__ void k_brute_finish(const unsigned long long* acc, int nb2, int copies, int carry, double inv0, double inv1,
                               double* dsum, double* wsum, uint64_t* counts) {
  for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < nb2; b += gridDim.x * blockDim.x) {
    __int128 v0 = 0, v1 = 0;
    uint64_t m = 0;
    for (int c = 0; c < copies; ++c) {
      const unsigned long long* g = acc + ((size_t)c * nb2 + b) * kBWin;
      v0 += brute_sum(g, carry);
      v1 += brute_sum(g + 2, carry);
      m += g[4];
    }
    dsum[b] = i128_double(v0) * inv0;
    wsum[b] = i128_double(v1) * inv1;
    counts[b] = m;
  }
}

// Bounds of a call's points: largest |w * delta| and |w|, and whether every
// difference of coordinates is exact in FP32.
struct BruteBounds {
  double mwd, mw;
  int exact_diff;
  int P;  // points per line of equal steps, 0 when the points are not in such lines
};

// The kernel's variants, by diagonals per lane.
struct BruteVariant {
  int k;
  void (*fn[2])(BruteArgs);  // by BruteArgs::carry
};
const BruteVariant kVariants[] = {{1, {brute_kernel<1, false>, brute_kernel<1, true>}},
                                  {2, {brute_kernel<2, false>, brute_kernel<2, true>}},
                                  {4, {brute_kernel<4, false>, brute_kernel<4, true>}}};
const BruteVariant kLineVariant = {1, {line_kernel<false>, line_kernel<true>}};

// Copies of window slots are made while a block stays below this much shared
// memory, so that three blocks share an SM.
constexpr size_t kBruteCopySmem = 72 * 1024;

// Launch shape: per warp a window of kBWords u32 words for each of the nbins +
// 2 bins, so as many warps (up to `warps_max`) as
// the block's opt-in shared memory holds.  Fails only if not even one warp fits.
tos_status brute_shape(const tos_engine* e, int nbins, int warps_max, int* warps, int* wshift, size_t* smem) {
  const size_t per_warp = (size_t)kBWords * (nbins + 2) * 4;
  const size_t fit = e->smem_optin / per_warp;
  if (fit < 1)
    return fail(TOS_ERR_UNSUPPORTED, "nbins too large for one warp's shared-memory window on this device");
  *warps = (int)std::min<size_t>((size_t)warps_max, fit);
  *wshift = 0;
  while (*wshift < 3 && ((size_t)*warps * per_warp << (*wshift + 1)) <= kBruteCopySmem) ++*wshift;
  *smem = (size_t)*warps * per_warp << *wshift;
  return TOS_OK;
}

// Fill the kernel arguments shared by both entry points (binning, FP32
// fast-path constants and the fixed-point scales from the bounds of |w d|
// and |w|: a run holds at most A.seg pairs).  Segments of rows: enough units
// for every warp several times over (about 2^15 where the pairs allow it, a
// unit of at least 32 x 32 pairs), chosen from n alone.
void brute_args(BruteArgs& A, int n, int nbins, double min, double max, const BruteBounds& B) {
  const double mwd = B.mwd, mw = B.mw;
  A.exact_diff = B.exact_diff;
  A.seg = 32;
  while (A.seg < 8192 && (double)n * n / 64.0 > 32768.0 * A.seg) A.seg *= 2;
  A.P = B.P;
  if (A.P) {
    A.Q = n / A.P;
    A.seg = A.P;  // a run's most pairs
    // units of one (line, 32 lines) where there are many, else of one offset block
    A.eblocks = (double)A.Q * A.Q >= 1e6 ? 1 << 20 : 1;
  }
  // Carry-free sums hold a bin that takes every pair while its values, below
  // 2^62 for A.seg pairs, add up to less than 2^94 and its flushes (at least
  // 2^11 pairs each, but for the last ones) to less than 2^32.  Beyond that the
  // low word's add returns its carry.
  const double pairs = 0.5 * n * ((double)n - 1.0);
  A.carry = pairs > 4294967296.0 * A.seg || pairs > 1099511627776.0 /* 2^40 */ ? 1 : 0;
  A.copies = std::max(1, std::min(64, kBruteAccBins / (nbins + 2)));
  A.n = n;
  A.nbins = nbins;
  A.min = min;
  A.max = max;
  A.spacing = (max - min) / nbins;
  A.invf = (float)(1.0 / A.spacing);
  A.offf = (float)(-min / A.spacing);
  A.nbf = (float)nbins;
  A.nbp1f = (float)nbins + 1.0f;
  int bl = 0;
  for (uint32_t v = (uint32_t)nbins + 2; v; v >>= 1) ++bl;
  A.k = std::max(0, std::min(13, 21 - bl));
  A.mag = std::ldexp(1.5f, 23 - A.k);
  std::memcpy(&A.bits, &A.mag, 4);
  const double per[2] = {mwd * mwd * (double)A.seg, mw * mw * (double)A.seg};
  for (int f = 0; f < 2; ++f) {
    int F = (int)std::floor(62.0 - std::log2(std::max(per[f], 1e-300)));
    F = std::max(-60, std::min(F, 200));
    A.scale_hi[f] = std::ldexp(1.0, F - 42);
  }
}

// k_brute_bounds' five words and k_brute_lines' two as bounds (false: a value is not finite).
// Differences of multiples of 2^e below 2^(e + 24) in magnitude are floats.
bool brute_bounds(const unsigned long long* h, int n, BruteBounds* B) {
  if (h[2]) return false;
  std::memcpy(&B->mwd, &h[0], 8);
  std::memcpy(&B->mw, &h[1], 8);
  B->mwd = std::max(B->mwd, 1e-300);
  B->mw = std::max(B->mw, 1e-300);
  const uint32_t u = (uint32_t)h[3];
  float top;
  std::memcpy(&top, &u, 4);
  const int low = 1024 - (int)h[4];
  B->exact_diff = h[4] == 0 || (low >= -126 && 2.0 * (double)top <= std::ldexp(1.0, low + 24)) ? 1 : 0;
  // lines: whole ones, long enough to bin an offset once for several pairs,
  // short and many enough to fill the warps.  Kernel ms as lines | as scattered
  // points, 50 bins: at the shortest, 2,500 lines of 8 0.42 | 0.93, 8,000 of 8
  // 4.1 | 9.3 (of 4 they are scattered: 10.3 for 16,000); at the fewest, 32 of
  // 1,024 0.36 | 1.19, 64 of 64 0.022 | 0.051 (16 of 64: 0.027 scattered).
  const int P = h[5] ? n - (int)h[5] + 1 : n;
  B->P = (B->exact_diff && h[6] == 0 && P >= 8 && P <= 1024 && n % P == 0 && n / P >= 32) ? P : 0;
  return true;
}

// Bounds and line structure of the device points (misc: seven cleared words).
tos_status brute_look(const float* pts, int n, unsigned long long* misc, cudaStream_t st, BruteBounds* B) {
  const int blocks = std::min(1024, (n + 255) / 256);
  k_brute_bounds<<<blocks, 256, 0, st>>>(pts, n, misc);
  k_brute_lines<<<blocks, 256, 0, st>>>(pts, n, 0, misc + 5);
  k_brute_lines<<<blocks, 256, 0, st>>>(pts, n, 1, misc + 5);
  TOS_CUDA_TRY(cudaGetLastError());
  unsigned long long h[7];
  TOS_CUDA_TRY(cudaMemcpyAsync(h, misc, sizeof(h), cudaMemcpyDeviceToHost, st));
  TOS_CUDA_TRY(cudaStreamSynchronize(st));
  if (!brute_bounds(h, n, B)) return fail(TOS_ERR_INVALID_ARG, "points must be finite");
  return TOS_OK;
}

// The kernel's arrays from the device points: n float4 and n doubles of
// scratch hold the positions and w*delta, or in the line layout (w*delta, w)
// and the lines' first points.
tos_status brute_prepare(BruteArgs* A, const float* pts, float4* pos, double* wd, cudaStream_t st) {
  const int n = A->n, blocks = std::min(4096, (n + 255) / 256);
  if (A->P) {
    float p[8];
    TOS_CUDA_TRY(cudaMemcpyAsync(p, pts, sizeof(p), cudaMemcpyDeviceToHost, st));
    TOS_CUDA_TRY(cudaStreamSynchronize(st));
    A->sx = p[5] - p[0], A->sy = p[6] - p[1], A->sz = p[7] - p[2];
    A->val = reinterpret_cast<double2*>(pos);
    A->base = reinterpret_cast<float4*>(wd);
    k_line_prep<<<blocks, 256, 0, st>>>(pts, n, A->P, A->Q, reinterpret_cast<double2*>(pos),
                                        reinterpret_cast<float4*>(wd));
  } else {
    A->pos = pos;
    A->wd = wd;
    k_brute_prep<<<blocks, 256, 0, st>>>(pts, n, pos, wd);
  }
  TOS_CUDA_TRY(cudaGetLastError());
  return TOS_OK;
}

double brute_inv_scale(const BruteArgs& A, int f) { return 1.0 / (A.scale_hi[f] * 4398046511104.0 /* 2^42 */); }

// The histogram index of an FP64 squared separation r2, computed as the
// reference's double-precision estimator does from r = sqrt(r2).
int brute_index_of_r2(double r2, double min, double max, double spacing, int nbins) {
  const double r = std::sqrt(r2);
  if (r < min) return 0;
  if (r >= max) return nbins + 1;
  double k = std::floor(tos::ddiv(tos::dsub(r, min), spacing));
  if (k > (double)(nbins - 1)) k = (double)(nbins - 1);
  return (int)k + 1;
}

// th[b], b = 1 .. nbins + 1: the smallest double r2 >= 0 whose index is at
// least b (the index is non-decreasing in r2), th[0] = -1, th[nbins + 2] = +inf.
// IEEE sqrt, subtraction and division round the same on the host and the
// device, so the device's comparisons reproduce the FP64 index exactly.
std::vector<double> brute_thresholds(double min, double max, int nbins) {
  std::vector<double> th((size_t)nbins + 3);
  th[0] = -1.0;
  th[(size_t)nbins + 2] = std::numeric_limits<double>::infinity();
  const double spacing = (max - min) / nbins;
  for (int b = 1; b <= nbins + 1; ++b) {
    const double r = std::max(min + (b - 1) * spacing, 0.0);
    th[b] = first_double(r * r, [&](double r2) { return brute_index_of_r2(r2, min, max, spacing, nbins) >= b; });
  }
  return th;
}

// Launch variant `vi` with up to `warps_max` warps per CTA, persistent (as
// many CTAs as fit on the SMs), between events ev[4] and ev[5].
tos_status brute_launch_shape(tos_engine* e, BruteArgs A, cudaStream_t st, int vi, int warps_max) {
  int warps = 0;
  size_t smem = 0;
  TOS_TRY(brute_shape(e, A.nbins, warps_max, &warps, &A.wshift, &smem));
  const auto fn = (A.P ? kLineVariant : kVariants[vi]).fn[A.carry];
  TOS_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int per_sm = 0;
  TOS_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, warps * 32, smem));
  e->brute_last[0] = A.P, e->brute_last[1] = A.P ? 1 : kVariants[vi].k, e->brute_last[2] = warps;
  TOS_CUDA_TRY(cudaEventRecord(e->ev[4], st));
  fn<<<e->num_sms * std::max(1, per_sm), warps * 32, smem, st>>>(A);
  TOS_CUDA_TRY(cudaGetLastError());
  TOS_CUDA_TRY(cudaEventRecord(e->ev[5], st));
  return TOS_OK;
}

// The default shape, or the one tos_brute_tune picked for this bin count and
// kernel (points in lines or not).
constexpr int kBruteDefaultVariant = 0, kBruteDefaultWarps = 8;

tos_status brute_launch(tos_engine* e, const BruteArgs& A, cudaStream_t st) {
  int vi = kBruteDefaultVariant, warps_max = kBruteDefaultWarps;
  {
    std::lock_guard<std::mutex> lk(e->tune_mu);
    auto it = e->brute_tuned.find({A.nbins, A.P != 0});
    if (it != e->brute_tuned.end()) {
      vi = it->second.first;
      warps_max = it->second.second;
    }
  }
  return brute_launch_shape(e, A, st, vi, warps_max);
}

}  // namespace
}  // namespace tos

using namespace tos;

namespace tos {
namespace {

// Scratch kept on the engine between calls is at most this large.
constexpr size_t kBruteKeep = 64u << 20;

struct DevScope {
  int prev = 0;
  explicit DevScope(int d) {
    cudaGetDevice(&prev);
    cudaSetDevice(d);
  }
  ~DevScope() { cudaSetDevice(prev); }
};

tos_status brute_check(const void* points, size_t n_points, double min, double max, int nbins) {
  if (!points) return fail(TOS_ERR_INVALID_ARG, "null argument");
  if (n_points < 2 || n_points > (1u << 24)) return fail(TOS_ERR_INVALID_ARG, "need 2 <= n <= 2^24 points");
  if (nbins <= 0 || nbins > 4096) return fail(TOS_ERR_INVALID_ARG, "nbins must be in [1, 4096]");
  if (!(max > min) || !std::isfinite(min) || !std::isfinite(max))
    return fail(TOS_ERR_INVALID_ARG, "need finite min < max");
  return TOS_OK;
}

// Upload the points and thresholds, check and prepare them, and set up the
// kernel arguments on the engine's scratch (its lock held), for the first
// `limit` points or whole lines of them.
tos_status brute_setup(tos_engine* e, const float* points, int n, double min, double max, int nbins, BruteArgs* A,
                       int limit = 1 << 30) {
  BruteScratch& W = e->brute;
  cudaStream_t st = e->stream;
  const int nb2 = nbins + 2;
  const std::vector<double> th = brute_thresholds(min, max, nbins);  // kept until the stream sync below
  TOS_TRY(W.th.alloc(th.size()));
  TOS_TRY(W.pts.alloc((size_t)n * 5));
  TOS_TRY(W.pos.alloc(n));
  TOS_TRY(W.wd.alloc(n));
  TOS_TRY(W.acc.alloc((size_t)kBruteAccBins * kBWin));
  TOS_TRY(W.out.alloc((size_t)nb2 * 3));
  TOS_TRY(W.misc.alloc(9));  // [0] unit counter [1] rechecks [2..8] bounds, lines
  TOS_CUDA_TRY(cudaMemcpyAsync(W.pts.p, points, (size_t)n * 5 * sizeof(float), cudaMemcpyHostToDevice, st));
  TOS_CUDA_TRY(cudaMemcpyAsync(W.th.p, th.data(), th.size() * sizeof(double), cudaMemcpyHostToDevice, st));
  TOS_CUDA_TRY(cudaMemsetAsync(W.acc.p, 0, (size_t)kBruteAccBins * kBWin * 8, st));
  TOS_CUDA_TRY(cudaMemsetAsync(W.misc.p, 0, 9 * 8, st));
  BruteBounds B;
  TOS_TRY(brute_look(W.pts.p, n, W.misc.p + 2, st, &B));
  if (n > limit) n = B.P ? limit / B.P * B.P : limit;
  brute_args(*A, n, nbins, min, max, B);
  TOS_TRY(brute_prepare(A, W.pts.p, W.pos.p, W.wd.p, st));
  A->th = W.th.p;
  A->acc = W.acc.p;
  A->next = W.misc.p;
  A->counters = W.misc.p + 1;
  return TOS_OK;
}

// Gives the scratch back when it is large (after the stream has been waited for).
struct BruteKeep {
  tos_engine* e;
  ~BruteKeep() {
    if (e->brute.bytes() > kBruteKeep) {
      cudaStreamSynchronize(e->stream);
      e->brute.release();
    }
  }
};

}  // namespace
}  // namespace tos

extern "C" tos_status tos_brute_run(tos_engine* e, const float* points, size_t n_points, double min,
                                    double max, int nbins, double* dsum, double* wsum,
                                    uint64_t* counts, double* ms_kernel) {
  if (!e || !points || !dsum || !wsum || !counts) return fail(TOS_ERR_INVALID_ARG, "null argument");
  TOS_TRY(brute_check(points, n_points, min, max, nbins));
  std::lock_guard<std::mutex> lock(e->mu);
  DevScope dev(e->device);
  BruteKeep keep{e};
  const int n = (int)n_points, nb2 = nbins + 2;
  cudaStream_t st = e->stream;
  BruteArgs A{};
  TOS_TRY(brute_setup(e, points, n, min, max, nbins, &A));
  TOS_TRY(brute_launch(e, A, st));
  double* out = e->brute.out.p;  // dsum, wsum, counts
  k_brute_finish<<<(nb2 + 127) / 128, 128, 0, st>>>(A.acc, nb2, A.copies, A.carry, brute_inv_scale(A, 0),
                                                   brute_inv_scale(A, 1), out, out + nb2, reinterpret_cast<uint64_t*>(out + 2 * nb2));
  TOS_CUDA_TRY(cudaGetLastError());
  std::vector<double> h((size_t)3 * nb2);
  TOS_CUDA_TRY(cudaMemcpyAsync(h.data(), out, h.size() * 8, cudaMemcpyDeviceToHost, st));
  TOS_CUDA_TRY(cudaStreamSynchronize(st));
  std::memcpy(dsum, h.data(), (size_t)nb2 * 8);
  std::memcpy(wsum, h.data() + nb2, (size_t)nb2 * 8);
  std::memcpy(counts, h.data() + 2 * (size_t)nb2, (size_t)nb2 * 8);
  if (ms_kernel) {
    float ms = 0;
    cudaEventElapsedTime(&ms, e->ev[4], e->ev[5]);
    *ms_kernel = ms;
  }
  return TOS_OK;
}

// Autotuner of the brute-force kernel's launch shape: every variant (1, 2 or
// 4 diagonals per lane; one for points in lines, whose kernel has no such
// choice) with 4, 8 and 16 warps per CTA, timed on the first 131,072 points (or
// as many whole lines), best of two timed launches after a warm-up.
extern "C" tos_status tos_brute_tune(tos_engine* e, const float* points, size_t n_points, double min,
                                     double max, int nbins, int* diagonals_per_lane, int* warps_per_cta) {
  if (!e) return fail(TOS_ERR_INVALID_ARG, "null argument");
  TOS_TRY(brute_check(points, n_points, min, max, nbins));
  std::lock_guard<std::mutex> lock(e->mu);
  DevScope dev(e->device);
  BruteKeep keep{e};
  cudaStream_t st = e->stream;
  BruteArgs A{};
  TOS_TRY(brute_setup(e, points, (int)n_points, min, max, nbins, &A, 131072));
  const int warp_opts[3] = {4, 8, 16};
  float best = 0.f;
  int best_v = kBruteDefaultVariant, best_w = kBruteDefaultWarps;
  const int variants = A.P ? 1 : (int)(sizeof(kVariants) / sizeof(kVariants[0]));
  for (int vi = 0; vi < variants; ++vi) {
    for (int wo : warp_opts) {
      float t_min = 0.f;
      for (int rep = 0; rep < 3; ++rep) {
        TOS_CUDA_TRY(cudaMemsetAsync(A.acc, 0, (size_t)kBruteAccBins * kBWin * 8, st));
        TOS_CUDA_TRY(cudaMemsetAsync(A.next, 0, 16, st));
        TOS_TRY(brute_launch_shape(e, A, st, vi, wo));
        TOS_CUDA_TRY(cudaEventSynchronize(e->ev[5]));
        float ms = 0.f;
        TOS_CUDA_TRY(cudaEventElapsedTime(&ms, e->ev[4], e->ev[5]));
        if (rep > 0 && (rep == 1 || ms < t_min)) t_min = ms;
      }
      if (best == 0.f || t_min < best) {
        best = t_min;
        best_v = vi;
        best_w = wo;
      }
    }
  }
  {
    std::lock_guard<std::mutex> lk(e->tune_mu);
    e->brute_tuned[{nbins, A.P != 0}] = std::make_pair(best_v, best_w);
  }
  if (diagonals_per_lane) *diagonals_per_lane = kVariants[best_v].k;
  if (warps_per_cta) *warps_per_cta = best_w;
  return TOS_OK;
}

extern "C" tos_status tos_brute_last_shape(tos_engine* e, int* points_per_line, int* diagonals_per_lane,
                                           int* warps_per_cta) {
  if (!e) return fail(TOS_ERR_INVALID_ARG, "null argument");
  std::lock_guard<std::mutex> lock(e->mu);
  if (points_per_line) *points_per_line = e->brute_last[0];
  if (diagonals_per_lane) *diagonals_per_lane = e->brute_last[1];
  if (warps_per_cta) *warps_per_cta = e->brute_last[2];
  return TOS_OK;
}

// ============================================================================
// Allocation-free variant of tos_brute_run.
//
// Some callers cannot allocate device memory while they count pairs: code
// that manages every byte of the GPU through its own pool, code that runs
// where a cudaMalloc would synchronise the device or is not allowed, or
// service loops that must not touch the allocator at all.  tos_brute_run keeps its
// scratch with the engine and grows it; tos_brute_run_noalloc takes its inputs and outputs
// in device memory and keeps all scratch in one statically sized device
// array that the library reserves on every GPU that loads it, until exit.
// ============================================================================

namespace tos {
namespace {

constexpr size_t kNoAllocMaxPoints = size_t(1) << 18;  // 262,144 points (a 64^3 grid)
constexpr int kNoAllocMaxBins = 4096;

constexpr size_t round256(size_t b) { return (b + 255) & ~size_t(255); }
// scratch layout (byte offsets, each 256-byte aligned)
constexpr size_t kNaPos = 0;                                                  // float4[n]
constexpr size_t kNaWd = kNaPos + round256(16 * kNoAllocMaxPoints);           // double[n]
constexpr size_t kNaAcc = kNaWd + round256(8 * kNoAllocMaxPoints);            // u64[nbins + 2][kBWin]
constexpr size_t kNaTh = kNaAcc + round256(8 * kBWin * (kNoAllocMaxBins + 2));  // double[nbins + 3]
constexpr size_t kNaMisc = kNaTh + round256(8 * (kNoAllocMaxBins + 3));         // u64[8]
constexpr size_t kNoAllocBytes = kNaMisc + 256;                               // ~6.5 MB

// The scratch.  Host code must not pass this name to a kernel: on the host
// it stands for a host-side shadow, not for the device memory; the device
// address comes from cudaGetSymbolAddress (noalloc_scratch below).
static __device__ __align__(256) unsigned char g_brute_scratch[kNoAllocBytes];

// Device address of g_brute_scratch on `device` (current): looked up once per
// device; the lookup may load the module on that device.
tos_status noalloc_scratch(int device, unsigned char** out) {
  static std::mutex mu;
  static std::vector<unsigned char*> addr;
  std::lock_guard<std::mutex> lock(mu);
  if ((size_t)device >= addr.size()) addr.resize(device + 1, nullptr);
  if (!addr[device]) {
    void* p = nullptr;
    const cudaError_t err = cudaGetSymbolAddress(&p, g_brute_scratch);
    if (err != cudaSuccess || !p)
      return fail(TOS_ERR_CUDA, std::string("cudaGetSymbolAddress of the brute scratch: ") +
                                    cudaGetErrorString(err));
    addr[device] = (unsigned char*)p;
  }
  *out = addr[device];
  return TOS_OK;
}

}  // namespace
}  // namespace tos

extern "C" tos_status tos_brute_run_noalloc(tos_engine* e, const float* d_points, size_t n_points,
                                            double min, double max, int nbins, double* d_dsum,
                                            double* d_wsum, uint64_t* d_counts, double* ms_kernel) {
  if (!e || !d_points || !d_dsum || !d_wsum || !d_counts) return fail(TOS_ERR_INVALID_ARG, "null argument");
  if (n_points < 2) return fail(TOS_ERR_INVALID_ARG, "need at least 2 points");
  if (n_points > kNoAllocMaxPoints)
    return fail(TOS_ERR_INVALID_ARG, "tos_brute_run_noalloc takes at most " +
                                         std::to_string(kNoAllocMaxPoints) + " points (got " +
                                         std::to_string(n_points) + "); use tos_brute_run");
  if (nbins <= 0 || nbins > kNoAllocMaxBins)
    return fail(TOS_ERR_INVALID_ARG, "nbins must be in [1, " + std::to_string(kNoAllocMaxBins) + "]");
  if (!(max > min) || !std::isfinite(min) || !std::isfinite(max))
    return fail(TOS_ERR_INVALID_ARG, "need finite min < max");
  std::lock_guard<std::mutex> lock(e->mu);
  int prev = 0;
  cudaGetDevice(&prev);
  cudaSetDevice(e->device);
  struct Restore {
    int d;
    ~Restore() { cudaSetDevice(d); }
  } restore{prev};
  unsigned char* S = nullptr;
  TOS_TRY(noalloc_scratch(e->device, &S));
  const int n = (int)n_points;
  const int nb2 = nbins + 2;
  cudaStream_t st = e->stream;
  float4* pos = (float4*)(S + kNaPos);
  double* wd = (double*)(S + kNaWd);
  unsigned long long* acc = (unsigned long long*)(S + kNaAcc);
  double* thr = (double*)(S + kNaTh);
  unsigned long long* misc = (unsigned long long*)(S + kNaMisc);  // [0] unit counter [1] rechecks [2..8] bounds, lines
  const std::vector<double> th = brute_thresholds(min, max, nbins);  // kept until the stream sync
  TOS_CUDA_TRY(cudaMemcpyAsync(thr, th.data(), th.size() * sizeof(double), cudaMemcpyHostToDevice, st));
  // the scratch keeps the previous call's contents: clear what accumulates
  TOS_CUDA_TRY(cudaMemsetAsync(acc, 0, (size_t)kBruteAccBins * kBWin * sizeof(unsigned long long), st));
  TOS_CUDA_TRY(cudaMemsetAsync(misc, 0, 9 * sizeof(unsigned long long), st));
  BruteBounds B;
  TOS_TRY(brute_look(d_points, n, misc + 2, st, &B));
  // the same kernel and arguments as tos_brute_run, pointing into the scratch
  BruteArgs A{};
  brute_args(A, n, nbins, min, max, B);
  TOS_TRY(brute_prepare(&A, d_points, pos, wd, st));
  A.th = thr;
  A.acc = acc;
  A.next = misc;
  A.counters = misc + 1;
  TOS_TRY(brute_launch(e, A, st));
  k_brute_finish<<<(nb2 + 127) / 128, 128, 0, st>>>(acc, nb2, A.copies, A.carry, brute_inv_scale(A, 0),
                                                   brute_inv_scale(A, 1), d_dsum, d_wsum, d_counts);
  TOS_CUDA_TRY(cudaGetLastError());
  TOS_CUDA_TRY(cudaStreamSynchronize(st));
  if (ms_kernel) {
    float ms = 0;
    cudaEventElapsedTime(&ms, e->ev[4], e->ev[5]);
    *ms_kernel = ms;
  }
  return TOS_OK;
}
