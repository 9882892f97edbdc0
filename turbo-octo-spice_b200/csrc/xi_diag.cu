// xi_diag.cu — diagonal-sweep kernels of the XiEstimator pair count for Polar
// (r, mu) coordinates (XiEstimator.cc:168-225), items whose z index is
// constant: in blocks (below), or pair by pair where blocks do not pay
// (diag_pairs_kernel).
//
// Along a row of the pixel-pair matrix the Polar key (r bin, mu bin) changes
// every few columns, so runs along rows are short.  Along a diagonal
// (p1 + s, p2 + s) both distances grow together: r_par = d2 - d1 stays nearly
// constant and r_perp grows slowly, so the key stays the same for tens to
// hundreds of pairs.  A lane owns two neighbouring diagonals p2 - p1 = delta
// and walks them in blocks of 16 rows without binning the pairs: it adds the
// products w_i d_i w_j d_j and w_i w_j of the block in FP64 and keeps the
// extremes of |d2 - d1| and of the FP32 r^2.  With them r and mu of every pair
// of the block lie between bounds; when the bounds, widened by a margin over
// every rounding of the reference's expression, fall into one key the block
// has that key.  The other blocks (a key changes inside, about a tenth) are
// queued per warp and swept pair by pair, 32 blocks at a time, one per lane,
// each pair binned as in the pixel-pair kernel (FP32, FP64 near an edge).
//
// While the key stays the same a diagonal only adds its block sums.  The other
// XiBin sums of a run of rows [s0, s1) are differences of the two sightlines'
// FP64 prefix sums:
//   di = P_i[s1] - P_i[s0],  dj = P_j[s1 + delta] - P_j[s0 + delta]  (w d, w, loglam).
// Closed runs go through a per-warp queue, 32 at a time; eight lanes add a
// run's eight sums to its 128-byte entry of the per-cell sums (one lane per
// run would touch 32 lines with every add).
//
// A lane's two diagonals share each column (the second's column is the first's
// one row later), and a sightline's pixels lie even ones first, then odd ones,
// so that the lanes of a warp, two diagonals apart, read neighbouring entries.
//
// What bounds it: issue (53 % of cycles) and the shared-memory pipe (64 %);
// about a third of the instructions are the block sums, a fifth each the block
// keys and the pair-by-pair blocks (6.6 % of the pairs).
//
// Measured on a B200 against the version that binned every pair (one warp per
// item): 7,000 sightlines at 16/deg^2, 50 x 20 bins: 486 -> 261 ms; five mocks
// of 5,000 sightlines in all: 292 -> 153 ms; jackknife of 2,500 sightlines (its
// few rows once went to the pixel-pair kernel: low words of 32 bits could have
// wrapped after 2^32 adds): 363 -> 97 ms with its covariance.  Block bounds from the extremes of
// d1 d2 instead of r^2 sent twice the blocks pair by pair; functions that are
// not inlined and read the arguments through the kernel's parameters cost 6 %;
// one lane per run with its own 15 adds touched 32 lines an add and took 30 of
// 46 shared-memory and L1 cycles a step.
#include <algorithm>

#include "bulk_pipeline.cuh"
#include "xi_device.cuh"

namespace tos {
namespace {

constexpr int kDiagWarps = 8;  // warps per CTA; a CTA has two items in flight
constexpr int kDiagThreads = kDiagWarps * 32;
constexpr int kDiagRows = 16;  // rows of a block
constexpr int kDiagSpan = 64;  // diagonals of a warp's group
constexpr int kQueue = 64;     // runs or blocks a warp holds (taken 32 at a time)

// A warp's queues and the staging of the sums of 32 runs.
struct WarpQ {
  unsigned long long rech;  // FP64 re-evaluations
  double didj[kQueue], wgt[kQueue];
  double val[8][34];  // (rows longer by two: eight fields of two runs lie in different banks)
  uint32_t key[kQueue];
  int s0[kQueue], s1[kQueue], delta[kQueue];
  // blocks to sweep pair by pair (first row, diagonal), each with the run its
  // diagonal had open before it
  int2 block[kQueue];
  uint32_t bkey[kQueue];
  int bs0[kQueue];
  double bdidj[kQueue], bwgt[kQueue];
};

// Per-item constants.
struct DItem {
  uint32_t cell, zb;
  int ni, nj;
  int dlo, groups;       // first diagonal and number of 64-diagonal groups (0: the end)
  float ap;              // 2(1 - c)
  double c;
  uint64_t prei, prej;   // the two sightlines' first prefix sums
  const PixPack* rows;   // padded pixels of sightline i, even ones first
  const PixPack* cols;   // padded pixels of sightline j, even ones first
};

// The CTA's two items (pair by pair: one a warp) and the launch's arguments for the functions that are
// not inlined: through a reference to the kernel's parameters they would read
// them by generic loads.
__shared__ DItem s_item[kDiagWarps];
__shared__ PairArgs s_args;
__shared__ Claim s_claim;  // of the warp that prepares an item

// Row values of the pixel-pair kernel's Polar fast path (xi_kernels.cu
// fast_bin): x1 = d1, A1 = d1 * 2(1 - c), dl1 = -(d1*d1 - fl(d1*d1)).
struct DRow {
  float x1, d1, A1, dl1;
};

// FP32 Polar key of one pixel pair (packed b0 << 16 | b1, or kInvalidKey) and
// whether it lies within 2^-K bins of an edge (or r^2 is tiny) and must be
// re-binned in FP64.  The same decision as xi_kernels.cu fast_bin.  c0, c1: its
// codes, or kNoCode in c0 below r2_small, where they are no guide.
constexpr int kNoCode = -0x40000000;
template <bool MINPOS>
__device__ __forceinline__ uint32_t polar_key(const PairArgs& A, const DRow& R, float x2, bool& recheck, int& c0,
                                              int& c1) {
  const float s = __fsub_rn(x2, R.x1);
  const float r2 = __fmaf_rn(s, s, __fmaf_rn(R.A1, x2, R.dl1));
  const float rs = rsqrt_approx(r2);
  const float t0 = __fmaf_rn(__fmul_rn(r2, rs), A.inv0f, A.off0f);
  const float t1 = __fmaf_rn(__fmul_rn(fabsf(s), rs), A.inv1f, A.off1f);
  const bool small = !(r2 >= A.r2_small);
  const int q0 = __float_as_int(__fadd_rz(t0, A.mag0)) - A.bits0;
  const int q1 = __float_as_int(__fadd_rz(t1, A.mag1)) - A.bits1;
  bool valid = (t0 < A.n0f) && (t1 < A.n1f);
  bool coarse = (t0 < A.n0p1f) && (t1 < A.n1p1f);
  if (MINPOS) {
    valid = valid && (t0 > -1.0f) && (t1 > -1.0f);
    coarse = coarse && (t0 > -2.0f) && (t1 > -2.0f);
  }
  int b0 = q0 >> A.k0, b1 = q1 >> A.k1;
  c0 = small ? kNoCode : b0;
  c1 = b1;
  if (MINPOS) {
    b0 = max(b0, 0);
    b1 = max(b1, 0);
  }
  const bool edge = (((q1 + 1) & ((1 << A.k1) - 1)) < 2) || (((q0 + 1) & ((1 << A.k0) - 1)) < 2);
  recheck = (coarse && edge) || small;
  return valid ? (((uint32_t)b0 << 16) | (uint32_t)b1) : kInvalidKey;
}

// Exact key of a pair near an edge whose FP32 codes are b0, b1 (each within
// one of the exact code): the reference's r^2 against the smallest r^2 of each
// r code (thr_r2), and |d2 - d1|^2 against thr_mu^2 r^2, where mu's rounding
// cannot matter beyond 1e-14 relative; closer than that, or without codes
// (kNoCode: a tiny r), the reference's own expression decides.
__device__ __noinline__ uint32_t polar_key_exact(const PairArgs& A, float d1, float d2, double c, int b0, int b1) {
  const double r1_sq = (double)fmul(d1, d1);
  const double two_r1_cos12 = dmul((double)fmul(2.0f, d1), c);
  const double r_sq = dadd(r1_sq, dmul(dsub((double)d2, two_r1_cos12), (double)d2));
  const double s = (double)fabsf(fsub(d1, d2)), s2 = s * s;
  const int n0 = (int)A.g.n0, n1 = (int)A.g.n1;
  const int a0 = min(max(b0, 0), n0), a1 = min(max(b1, 0), n1);
  const int e0 = a0 - 1 + (r_sq >= A.thr_r2[a0] ? 1 : 0) + (r_sq >= A.thr_r2[a0 + 1] ? 1 : 0);
  const double ma = A.thr_mu2[a1] * r_sq, mb = A.thr_mu2[a1 + 1] * r_sq;
  const bool close = fabs(s2 - ma) <= 1e-14 * s2 || fabs(s2 - mb) <= 1e-14 * s2;
  if (close || b0 == kNoCode) {
    uint32_t p0 = 0, p1 = 0;
    return exact_polar(d1, d2, c, A.g, &p0, &p1) ? ((p0 << 16) | p1) : kInvalidKey;
  }
  const int e1 = a1 - 1 + (s2 >= ma ? 1 : 0) + (s2 >= mb ? 1 : 0);
  return (unsigned)e0 < (unsigned)n0 && (unsigned)e1 < (unsigned)n1 ? (((uint32_t)e0 << 16) | (uint32_t)e1)
                                                                     : kInvalidKey;
}

// Key of every pair with slo <= |d2 - d1| <= shi and r2lo <= r^2 <= r2hi, r^2 =
// (d2 - d1)^2 + 2(1 - c) d1 d2 in FP32: the packed key, kInvalidKey when no such
// pair is binned, or kMixedKey when the bounds do not settle it.  The
// reference's r^2 differs by the float rounding of d1*d1 (at most A.jit2);
// 3e-6 relative and A.eps0, A.eps1 bins cover the FP32 evaluation here and the
// rounding of the reference's.
constexpr uint32_t kMixedKey = 0xFFFFFFFEu;
template <bool MINPOS>
__device__ __forceinline__ uint32_t block_key(const PairArgs& A, float slo, float shi, float r2lo, float r2hi) {
  r2lo = __fmaf_rn(r2lo, 1.f - 3e-6f, -A.jit2);
  r2hi = __fmaf_rn(r2hi, 1.f + 3e-6f, A.jit2);
  if (!(r2lo >= A.r2_small)) return kMixedKey;
  const float ia = rsqrt_approx(r2lo), ib = rsqrt_approx(r2hi);
  const float t0a = __fmaf_rn(r2lo * ia, A.inv0f, A.off0f - A.eps0);
  const float t0b = __fmaf_rn(r2hi * ib, A.inv0f, A.off0f + A.eps0);
  if (t0a >= A.n0f) return kInvalidKey;
  const float t1a = __fmaf_rn(slo * ib, A.inv1f, A.off1f - A.eps1);
  const float t1b = __fmaf_rn(shi * ia, A.inv1f, A.off1f + A.eps1);
  if (t1a >= A.n1f) return kInvalidKey;
  bool ok = (t0b < A.n0f) && (t1b < A.n1f);
  if (MINPOS) {
    if (t0b <= -1.f || t1b <= -1.f) return kInvalidKey;
    ok = ok && t0a > -1.f && t1a > -1.f;
  }
  const int b0 = (int)t0a, b1 = (int)t1a;  // toward zero: (-1, 0) is bin 0
  ok = ok && b0 == (int)t0b && b1 == (int)t1b;
  return ok ? (((uint32_t)b0 << 16) | (uint32_t)b1) : kMixedKey;
}

// Warp-sum the kernel's counters into A.counters[0] (evaluated pairs), [1]
// (FP64 re-evaluations) and [12] (items taken).
__device__ __forceinline__ void add_counters_diag(const PairArgs& A, int lane, unsigned long long n_eval,
                                                  unsigned long long n_recheck, unsigned long long n_taken) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    n_eval += __shfl_xor_sync(kFull, n_eval, o);
    n_recheck += __shfl_xor_sync(kFull, n_recheck, o);
  }
  if (lane == 0) {
    atomicAdd(&A.counters[0], n_eval);
    atomicAdd(&A.counters[1], n_recheck);
    atomicAdd(&A.counters[12], n_taken);
  }
}

// Add the queue entries [first, first + n) of the warp to the item's row: a
// lane works out the sums of one run, then eight lanes take a run, a field
// each, so that the adds of a run fall into its one 128-byte entry.
__device__ __noinline__ void drain(int buf, WarpQ& Q, int first, int n, int lane) {
  const PairArgs& A = s_args;
  const DItem& it = s_item[buf];
  __syncwarp();
  uint32_t at = 0xFFFFFFFFu;  // flat bin of the run
  if (lane < n) {
    const int e = first + lane;
    const int delta = Q.delta[e];
    const uint32_t key = Q.key[e];
    // the rows of the run inside the matrix
    const int s0 = max(Q.s0[e], -delta), s1 = min(min(Q.s1[e], it.ni), it.nj - delta);
    if (s1 > s0) {
      const double2 *pi = A.pre2 + it.prei, *pj = A.pre2 + it.prej + delta;
      const double *li = A.prel + it.prei, *lj = A.prel + it.prej + delta;
      const double2 ia = pi[s0], ib = pi[s1], ja = pj[s0], jb = pj[s1];
      const double lz = (li[s1] - li[s0]) + (lj[s1] - lj[s0]);
      const uint32_t b0 = key >> 16, b1 = key & 0xFFFFu;
      const uint32_t idx = it.zb + (b1 + b0 * A.g.n1) * A.g.n2;  // as XiEstimator.cc:196-201
      if (idx < A.g.ntotal)
        at = idx;
      else
        atomicAdd(&A.counters[2], (unsigned long long)(s1 - s0));
      Q.val[0][lane] = Q.didj[e];
      Q.val[1][lane] = ib.x - ia.x;
      Q.val[2][lane] = jb.x - ja.x;
      Q.val[3][lane] = Q.wgt[e];
      Q.val[4][lane] = ib.y - ia.y;
      Q.val[5][lane] = jb.y - ja.y;
      Q.val[6][lane] = 0.5 * lz;
      Q.val[7][lane] = __longlong_as_double((long long)(s1 - s0));
    }
  }
  __syncwarp();
  const int f = lane & 7;
  const double sh = A.scale_hi[min(f, 6)];
  unsigned long long* row = A.acc + (size_t)it.cell * A.g.ntotal * kAccWords;
#pragma unroll 2
  for (int q = 0; q < 8; ++q) {
    const int e = q * 4 + (lane >> 3);
    const uint32_t idx = __shfl_sync(kFull, at, e);
    if (idx == 0xFFFFFFFFu) continue;
    unsigned long long* base = row + (size_t)idx * kAccWords;
    const double v = Q.val[f][e];
    if (f == 7)
      red_add(base + 14, (unsigned long long)__double_as_longlong(v));
    else
      add128(base + f, base + 7 + f, to_fixed_wide(v, sh));
  }
  __syncwarp();
}

// Queue the runs of the lanes that close one; 32 waiting runs are added.
__device__ __forceinline__ void push_run(int buf, WarpQ& Q, int& qn, bool close,
                                         uint32_t key, int s0, int s1, int delta, double didj, double wgt, int lane) {
  const unsigned cm = __ballot_sync(kFull, close);
  if (cm == 0) return;
  if (close) {
    const int e = qn + __popc(cm & ((1u << lane) - 1u));
    Q.key[e] = key;
    Q.s0[e] = s0;
    Q.s1[e] = s1;
    Q.delta[e] = delta;
    Q.didj[e] = didj;
    Q.wgt[e] = wgt;
  }
  qn += __popc(cm);
  if (qn >= 32) {
    qn -= 32;
    drain(buf, Q, qn, 32, lane);
  }
}

// Sweep the queued blocks [first, first + n) pair by pair, one per lane.  A
// block usually closes one run: it is kept until the end of the block, when
// the lanes' closed runs are queued together.  Returns the runs in the queue.
template <bool MINPOS>
__device__ __noinline__ int sweep_blocks(int buf, WarpQ& Q, int first, int n, int qn, int lane) {
  const PairArgs& A = s_args;
  const DItem& it = s_item[buf];
  unsigned rech = 0;
  __syncwarp();
  int delta = 0, lo = 0, hi = 0, s0 = 0;
  uint32_t cur = kInvalidKey;  // the run open before the block goes on in it
  double didj = 0.0, wgt = 0.0;
  if (lane < n) {
    const int2 b = Q.block[first + lane];
    delta = b.y;
    lo = max(b.x, -delta);
    hi = min(min(b.x + kDiagRows, it.ni), it.nj - delta);
    cur = Q.bkey[first + lane];
    s0 = Q.bs0[first + lane];
    didj = Q.bdidj[first + lane];
    wgt = Q.bwgt[first + lane];
  }
  const float ap = it.ap;
  // rows lo, lo + 1, ... and columns lo + delta, ... alternate between the halves
  const int oi = kParityPad + ((it.ni + 1) >> 1), oj = kParityPad + ((it.nj + 1) >> 1);
  const PixPack* re = it.rows + kParityPad + (lo >> 1);
  const PixPack* r0 = re + ((lo & 1) ? oi : 0);
  const PixPack* r1 = re + ((lo & 1) ? 1 : oi);
  const int c = lo + delta;
  const PixPack* ce = it.cols + kParityPad + (c >> 1);
  const PixPack* c0 = ce + ((c & 1) ? oj : 0);
  const PixPack* c1 = ce + ((c & 1) ? 1 : oj);
  uint32_t pkey = kInvalidKey;  // a closed run, not queued yet
  int ps0 = 0, ps1 = 0;
  double pd = 0.0, pw = 0.0;
#pragma unroll 2
  for (int k = 0; k < kDiagRows; ++k) {
    const int s = lo + k;
    const PixPack rp = (k & 1) ? r1[k >> 1] : r0[k >> 1];  // past `hi`: padding or the next pixels, not used
    const PixPack cp = (k & 1) ? c1[k >> 1] : c0[k >> 1];
    DRow R;
    R.x1 = R.d1 = rp.d;
    const float p = __fmul_rn(R.d1, R.d1);
    R.dl1 = -__fmaf_rn(R.d1, R.d1, -p);  // -(d1*d1 - fl(d1*d1)), exact
    R.A1 = __fmul_rn(R.d1, ap);
    bool recheck;
    int b0, b1;
    uint32_t key = polar_key<MINPOS>(A, R, cp.d, recheck, b0, b1);
    const bool in = s < hi;
    if (recheck && in) {
      key = polar_key_exact(A, R.d1, cp.d, it.c, b0, b1);
      ++rech;
    }
    const bool change = in && key != cur;
    const bool close = change && cur != kInvalidKey;
    // a second run closed by this block: the first one is queued now
    if (__any_sync(kFull, close && pkey != kInvalidKey))
      push_run(buf, Q, qn, close && pkey != kInvalidKey, pkey, ps0, ps1, delta, pd, pw, lane);
    if (close) {
      pkey = cur;
      ps0 = s0;
      ps1 = s;
      pd = didj;
      pw = wgt;
    }
    if (change) {
      cur = key;
      s0 = s;
      didj = 0.0;
      wgt = 0.0;
    }
    if (in) {
      didj = __fma_rn(rp.wd, cp.wd, didj);
      wgt = __fma_rn((double)rp.w, (double)cp.w, wgt);
    }
  }
  push_run(buf, Q, qn, pkey != kInvalidKey, pkey, ps0, ps1, delta, pd, pw, lane);
  push_run(buf, Q, qn, cur != kInvalidKey, cur, s0, hi, delta, didj, wgt, lane);
  rech = __reduce_add_sync(kFull, rech);
  if (lane == 0) Q.rech += rech;
  return qn;
}

__device__ __forceinline__ float fmin3(float a, float b, float c) {
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float fmax3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// The sums and bounds of one block of kDiagRows rows (from row sb, column c of
// the lane's first diagonal) of a lane's two diagonals; MASKED: bit k of
// mask[m] is set where row sb + k of diagonal m lies in the matrix (the others
// read padding of zero weight).
struct BlockSums {
  double bd[2], bw[2];
  float slo[2], shi[2], r2lo[2], r2hi[2];
};
template <bool MASKED>
__device__ __forceinline__ void block_sums(const DItem& it, int sb, int c, const unsigned (&mask)[2], BlockSums& B) {
  const int oi = kParityPad + ((it.ni + 1) >> 1), oj = kParityPad + ((it.nj + 1) >> 1);  // odd half after even
  // rows sb + k and columns c + k + 1 by parity: one pointer each, a step per two rows
  const PixPack* re = it.rows + kParityPad + (sb >> 1);
  const PixPack* r0 = re + ((sb & 1) ? oi : 0);
  const PixPack* r1 = re + ((sb & 1) ? 1 : oi);
  const PixPack* ce = it.cols + kParityPad + (c >> 1);
  const PixPack* c0 = ce + ((c & 1) ? 1 : oj);
  const PixPack* c1 = ce + ((c & 1) ? oj + 1 : 1);
  PixPack ca = ce[(c & 1) ? oj : 0];
  double wa = (double)ca.w;
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    B.bd[m] = B.bw[m] = 0.0;
    B.slo[m] = B.r2lo[m] = 3e38f;
    B.shi[m] = B.r2hi[m] = 0.f;
  }
  float sp[2], rp[2];  // |d2 - d1| and r^2 of the even row, taken with the odd row's
  // (a loop of four rows: fully unrolled, the kernel's code outgrows the instruction cache)
#pragma unroll 1
  for (int kk = 0; kk < kDiagRows; kk += 4, r0 += 2, r1 += 2, c0 += 2, c1 += 2)
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const PixPack r = (k & 1) ? r1[k >> 1] : r0[k >> 1];
    const PixPack cb = (k & 1) ? c1[k >> 1] : c0[k >> 1];
    const double w1 = (double)r.w, wb = (double)cb.w;
    const float A1 = __fmul_rn(it.ap, r.d);
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      const float x2 = m ? cb.d : ca.d;
      const float s = fabsf(__fsub_rn(x2, r.d));
      const float r2 = __fmaf_rn(s, s, __fmul_rn(A1, x2));
      if (MASKED) {
        if ((mask[m] >> (kk + k)) & 1u) {
          B.slo[m] = fminf(B.slo[m], s);
          B.shi[m] = fmaxf(B.shi[m], s);
          B.r2lo[m] = fminf(B.r2lo[m], r2);
          B.r2hi[m] = fmaxf(B.r2hi[m], r2);
        }
      } else if (k & 1) {
        B.slo[m] = fmin3(B.slo[m], sp[m], s);
        B.shi[m] = fmax3(B.shi[m], sp[m], s);
        B.r2lo[m] = fmin3(B.r2lo[m], rp[m], r2);
        B.r2hi[m] = fmax3(B.r2hi[m], rp[m], r2);
      } else {
        sp[m] = s;
        rp[m] = r2;
      }
      B.bd[m] = __fma_rn(r.wd, m ? cb.wd : ca.wd, B.bd[m]);
      B.bw[m] = __fma_rn(w1, m ? wb : wa, B.bw[m]);
    }
    ca = cb;
    wa = wb;
  }
}

// One diagonal of a lane: the open run.
struct DiagRun {
  uint32_t cur;
  int s0;
  double didj, wgt;
};

// Sweep diagonals d0 .. d0 + 63 of an item: lane L takes d0 + 2 L and the next.
// `it` is s_item[buf] in registers.
template <bool MINPOS>
__device__ __forceinline__ void diag_group(const PairArgs& A, const DItem& it, int buf, int d0, int lane, WarpQ& Q,
                                           unsigned long long& n_eval_sum) {
  const int ni = it.ni, nj = it.nj;
  const int da = d0 + 2 * lane;  // diagonals da and da + 1
  const int s_lo = max(0, -(d0 + kDiagSpan - 1));
  const int s_hi = min(ni, nj - d0);
  DiagRun run[2];
#pragma unroll
  for (int m = 0; m < 2; ++m) run[m] = DiagRun{kInvalidKey, 0, 0.0, 0.0};
  int qn = 0, bn = 0;  // queued runs and blocks (the same in every lane)
  unsigned n_eval = 0;
#pragma unroll 1
  for (int sb = s_lo; sb < s_hi; sb += kDiagRows) {
    BlockSums B;
    unsigned mask[2] = {0xFFFFu, 0xFFFFu};
    if (sb + kDiagRows <= ni && sb + d0 >= 0 && sb + kDiagRows + d0 + kDiagSpan - 1 <= nj) {
      block_sums<false>(it, sb, sb + da, mask, B);  // every pair of the 64 diagonals lies in the matrix
      n_eval += 2 * kDiagRows;
    } else {
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const int lo = max(0, -(da + m) - sb), hi = min(kDiagRows, min(ni, nj - (da + m)) - sb);
        mask[m] = hi > lo ? (1u << hi) - (1u << lo) : 0u;
        n_eval += __popc(mask[m]);
      }
      block_sums<true>(it, sb, sb + da, mask, B);
    }
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      const uint32_t key =
          mask[m] ? block_key<MINPOS>(A, B.slo[m], B.shi[m], B.r2lo[m], B.r2hi[m]) : kInvalidKey;
      // blocks to sweep pair by pair take the open run along
      const bool mixed = key == kMixedKey;
      const bool change = key != run[m].cur;
      push_run(buf, Q, qn, change && !mixed && run[m].cur != kInvalidKey, run[m].cur, run[m].s0, sb, da + m,
               run[m].didj, run[m].wgt, lane);
      const unsigned xm = __ballot_sync(kFull, mixed);
      if (mixed) {
        const int e = bn + __popc(xm & ((1u << lane) - 1u));
        Q.block[e] = make_int2(sb, da + m);
        Q.bkey[e] = run[m].cur;
        Q.bs0[e] = run[m].s0;
        Q.bdidj[e] = run[m].didj;
        Q.bwgt[e] = run[m].wgt;
      }
      if (change) {
        run[m].cur = mixed ? kInvalidKey : key;
        run[m].s0 = sb;
        run[m].didj = 0.0;
        run[m].wgt = 0.0;
      }
      run[m].didj += B.bd[m];
      run[m].wgt += B.bw[m];
      if (xm) {
        bn += __popc(xm);
        if (bn >= 32) {
          bn -= 32;
          qn = sweep_blocks<MINPOS>(buf, Q, bn, 32, qn, lane);
        }
      }
    }
  }
  // runs still open at the last row, then the queues
#pragma unroll
  for (int m = 0; m < 2; ++m)
    push_run(buf, Q, qn, run[m].cur != kInvalidKey, run[m].cur, run[m].s0, s_hi, da + m, run[m].didj, run[m].wgt,
             lane);
  if (bn) qn = sweep_blocks<MINPOS>(buf, Q, 0, bn, qn, lane);
  drain(buf, Q, 0, qn, lane);
  n_eval_sum += n_eval;
}

// The constants of item idx (sightlines i, j) and its diagonals [dlo, dhi];
// false when none reaches the grid (all lanes of one warp).
__device__ __forceinline__ bool diag_window(const PairArgs& A, unsigned long long idx, uint32_t i, uint32_t j, int lane,
                                            DItem& it, int& dlo, int& dhi) {
  it.ni = (int)A.npix[i];
  it.nj = (int)A.npix[j];
  it.c = A.item_c[idx];
  const double a = 2.0 * dsub(1.0, it.c);
  it.ap = (float)a;
  const float4 ri = A.range[i], rj = A.range[j];
  it.zb = zbin_of_sum(__fadd_rn(ri.z, rj.z), A.g);
  it.cell = dest_row(A, i, j);
  it.prei = A.off[i] + i;
  it.prej = A.off[j] + j;
  // Column window |d1 - d2| < lim of every row (the pixel-pair kernel's
  // Polar bound: r^2 >= (d2 - d1)^2 + 2(1 - c) dmin_i dmin_j - err), and
  // from it the diagonals that reach it.
  dlo = -(it.ni - 1);
  dhi = it.nj - 1;
  if (A.prune) {
    float lim = A.win_lim;
    if (ri.x > 0.f && rj.x > 0.f) {
      const double q = A.polar_r2 - fmax(a, 0.0) * (double)ri.x * (double)rj.x * (1.0 - 1e-6) + A.polar_e2;
      lim = fminf(lim, (float)(sqrt(fmax(q, 0.0)) * (1.0 + 1e-6) + 1e-3));
    }
    const float* rowd = A.dist_pad + A.off[i] + (uint64_t)kPad * (i + 1);
    const float* cold = A.dist_pad + A.off[j] + (uint64_t)kPad * (j + 1);
    // over stretches of rows: the window's ends grow with the row, so the
    // first row's lower end and the last row's upper end bound a stretch
    const int step = (it.ni + 63) >> 6;
    dlo = 0x7FFFFFFF;
    dhi = -0x7FFFFFFF;
    for (int r = lane * step; r < it.ni; r += 32 * step) {
      const int re = min(r + step, it.ni) - 1;
      const float xa = rowd[r], xb = rowd[re];
      int lo = 0, hi = it.nj;  // first column with fl(xa - x2) < lim
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (__fsub_rn(xa, cold[mid]) < lim) hi = mid; else lo = mid + 1;
      }
      int lo2 = lo, hi2 = it.nj;  // first column with x2 >= xb and fl(x2 - xb) >= lim
      while (lo2 < hi2) {
        const int mid = (lo2 + hi2) >> 1;
        const float x2 = cold[mid];
        if (x2 >= xb && __fsub_rn(x2, xb) >= lim) hi2 = mid; else lo2 = mid + 1;
      }
      if (lo2 > lo) {
        dlo = min(dlo, lo - re);
        dhi = max(dhi, lo2 - 1 - r);
      }
    }
    dlo = __reduce_min_sync(kFull, dlo);
    dhi = __reduce_max_sync(kFull, dhi);
    if (dhi < dlo) return false;
    dlo = max(dlo, -(it.ni - 1));
    dhi = min(dhi, it.nj - 1);
  }
  return true;
}

// Prepare the next owned item into `h` (all lanes of one warp; SMEM: its
// pixels into buf), arriving on `full`.  Returns the items taken.
template <bool SMEM>
__device__ __noinline__ int prepare_diag(DItem* h, int* next, PixPack* buf, unsigned long long* full, int lane) {
  const PairArgs& A = s_args;
  int taken = 0;
  DItem it;
  it.groups = 0;
  for (;;) {
    unsigned long long idx = 0;
    if (!claim_item(A, kOwnerDiag, s_claim, lane, idx)) break;
    ++taken;
    const uint32_t i = A.item_i[idx], j = A.item_j[idx];
    int dlo, dhi;
    if (!diag_window(A, idx, i, j, lane, it, dlo, dhi)) continue;
    it.dlo = dlo;
    it.groups = (dhi - dlo) / kDiagSpan + 1;
    const PixPack *gi = A.pix2 + A.off[i] + (uint64_t)(2 * kParityPad) * i,
                  *gj = A.pix2 + A.off[j] + (uint64_t)(2 * kParityPad) * j;
    const int len = A.max_np + 3 * kParityPad;
    it.rows = SMEM ? buf : gi;
    it.cols = SMEM ? buf + len : gj;
    if (lane == 0) {
      *h = it;
      *next = 0;
      if (SMEM) {
        const uint32_t bi = (uint32_t)(it.ni + 3 * kParityPad) * 16u, bj = (uint32_t)(it.nj + 3 * kParityPad) * 16u;
        bar_arrive_tx(full, bi + bj);
        bulk_load(buf, gi, bi, full);
        bulk_load(buf + len, gj, bj, full);
      } else {
        bar_arrive(full);
      }
    }
    __syncwarp();
    return taken;
  }
  if (lane == 0) {  // no item left
    it.groups = 0;
    *h = it;
    bar_arrive(full);
  }
  __syncwarp();
  return taken;
}

// The arguments stay in the kernel's parameter space (__grid_constant__):
// the inlined sweep reads them as constant-bank operands.  Two item buffers
// per CTA, as in the band sweep (xi_grid.cu): the warps take turns to prepare the
// next item before their share of this one, and each warp takes the item's groups from a
// counter and goes on to the next item by itself.
template <bool MINPOS, bool SMEM>
__global__ void __launch_bounds__(kDiagThreads, 2) diag_kernel(const __grid_constant__ PairArgs A) {
  extern __shared__ PixPack diag_smem[];  // the item buffers, then the warps' queues
  __shared__ int s_next[2];
  __shared__ unsigned long long s_full[2], s_empty[2];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int buf_len = 2 * (A.max_np + 3 * kParityPad);
  WarpQ& Q = reinterpret_cast<WarpQ*>(diag_smem + (SMEM ? 2 * (size_t)buf_len : 0))[warp];
  if (lane == 0) Q.rech = 0ull;
  if (tid == 0) {
    s_args = A;
    s_claim.todo = 0u;
    for (int b = 0; b < 2; ++b) {
      bar_init(&s_full[b], 1);
      bar_init(&s_empty[b], kDiagWarps);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  unsigned long long n_eval = 0;
  unsigned long long n_taken = 0;
  bool ok = true;
  if (warp == 0) n_taken += prepare_diag<SMEM>(&s_item[0], &s_next[0], diag_smem, &s_full[0], lane);
  for (uint32_t k = 0;; ++k) {
    const uint32_t b = k & 1u;
    ok = bar_wait(&s_full[b], (k >> 1) & 1u, A.wait_ms);
    if (!ok) {
      // the copies that this warp started must land before it ends
      if (k == 0 ? warp == 0 : ((warp - (int)(k - 1)) & (kDiagWarps - 1)) == 0)
        bar_wait(&s_full[b], (k >> 1) & 1u, kWaitMs);
      break;
    }
    DItem it = s_item[b];
    if (it.groups == 0) break;
    if (SMEM) {  // the same pointers, known to be in shared memory
      it.rows = diag_smem + (size_t)b * buf_len;
      it.cols = it.rows + A.max_np + 3 * kParityPad;
    }
    if (((warp - (int)k) & (kDiagWarps - 1)) == 0) {  // the warps take turns
      const uint32_t nb = b ^ 1u;
      if (k > 0) ok = bar_wait(&s_empty[nb], ((k - 1) >> 1) & 1u, A.wait_ms);  // item k - 1 is done by every warp
      if (!ok) break;
      n_taken += prepare_diag<SMEM>(&s_item[nb], &s_next[nb], diag_smem + (SMEM ? (size_t)nb * buf_len : 0),
                                    &s_full[nb], lane);
    }
    for (;;) {
      int q = 0;
      if (lane == 0) q = atomicAdd(&s_next[b], 1);
      q = __shfl_sync(kFull, q, 0);
      if (q >= it.groups) break;
      diag_group<MINPOS>(A, it, (int)b, it.dlo + q * kDiagSpan, lane, Q, n_eval);
    }
    __syncwarp();
    if (lane == 0) bar_arrive(&s_empty[b]);
  }
  if (!ok && lane == 0) atomicOr(&A.counters[13], kWaitDiag);  // a wait ran out: the host reports it
  __syncwarp();
  add_counters_diag(A, lane, n_eval, lane == 0 ? Q.rech : 0ull, n_taken);
}

// ---- pair by pair -----------------------------------------------------------
// Items for which blocks do not pay: in short sightlines most of a block's 16
// rows and a group's 64 diagonals lie outside the matrix, and a CTA an item is
// bound by the chain of reads that prepares it; missing pixels or unlike steps
// change |d2 - d1| inside the blocks, and fine bins leave few of one key.  Each
// such item has a warp, whose lanes walk a diagonal each, row by row, and bin
// every pair.  Bound by issue (80 % of cycles, 125 instructions a step).
//
// Measured on a B200 (ms): all items in blocks | pair by pair | the sweep before
// the blocks, which binned every pair.  50 x 20 bins to 200:
//   328,000 items of 16 pixels                       3.81 | 0.76 | 0.78
//   of 64                                            7.48 | 4.52 | 4.15
//   of 128                                           13.1 | 13.0 | 12.4
//   of 256                                           26.6 | 41.0 | 40.2
//   73,000 of 560, none masked                       13.1 | 26.6 | 26.5
//   8 % masked (windows and single pixels)           20.5 | 26.0 | 25.8
//   222,000 of 128 in 150, scattered                 19.6 | 10.9 | 13.4
//   54,000 of 560, every sightline its own step      31.1 | 32.6 | 32.7
// 200 x 100 bins, 73,000 of 560: none masked 27.3 | 30.1 | 29.3, 8 % masked
// 37.7 | 30.5 | 31.6; 100 x 50: 18.1 | 27.8 | 27.6, 27.9 | 27.7 | 27.7; 25 x 4
// to 150 (the blocks' runs meet on its 100 bins): 6.7 | 13.9 | 13.7, 16.7 | 13.4
// | 15.6.

// One item's arrays: distances (padded by sentinels) and (w*delta, w).
struct PairsItem {
  const float *rowd, *cold;
  const double2 *row2, *col2;
};

// Diagonals d0 .. d0 + 31 (lane = diagonal - d0, up to dhi) of the warp's item.
template <bool MINPOS>
__device__ __forceinline__ void pairs_group(const PairArgs& A, const PairsItem& p, int ni, int nj, float ap, int buf,
                                            int d0, int dhi, int lane, WarpQ& Q, unsigned& n_eval, unsigned& rech) {
  const int delta = d0 + lane;
  const int s_lo = max(0, -(d0 + 31)), s_hi = min(ni, nj - d0);
  const int lo = max(0, -delta);
  const int rows = delta <= dhi ? max(min(ni, nj - delta) - lo, 0) : 0;  // of the lane, from lo
  n_eval += rows;
  // column s + delta: -31 .. nj + 31, within the padding of the distances
  const float *rd = p.rowd + s_lo, *cd = p.cold + (s_lo + delta);
  const double2 *rw = p.row2 + s_lo, *cw = p.col2 + (s_lo + delta);
  uint32_t cur = kInvalidKey;
  int s0 = 0, qn = 0;
  double didj = 0.0, wgt = 0.0;
#pragma unroll 1
  for (int s = s_lo; s < s_hi; ++s, ++rd, ++cd, ++rw, ++cw) {
    const bool in = (unsigned)(s - lo) < (unsigned)rows;
    const float x2 = *cd;
    const double2 r = *rw;
    double2 q = make_double2(0.0, 0.0);
    if (in) q = *cw;
    DRow R;
    R.x1 = R.d1 = *rd;
    const float d2 = __fmul_rn(R.d1, R.d1);
    R.dl1 = -__fmaf_rn(R.d1, R.d1, -d2);  // -(d1*d1 - fl(d1*d1)), exact
    R.A1 = __fmul_rn(R.d1, ap);
    bool recheck;
    int b0, b1;
    uint32_t key = polar_key<MINPOS>(A, R, x2, recheck, b0, b1);
    recheck = recheck && in;
    if (__any_sync(kFull, recheck)) {
      if (recheck) {
        key = polar_key_exact(s_args, R.d1, x2, s_item[buf].c, b0, b1);
        ++rech;
      }
    }
    if (!in) key = kInvalidKey;
    const bool change = key != cur;
    push_run(buf, Q, qn, change && cur != kInvalidKey, cur, s0, s, delta, didj, wgt, lane);
    if (change) {
      cur = key;
      s0 = s;
      didj = 0.0;
      wgt = 0.0;
    }
    didj = __fma_rn(r.x, q.x, didj);  // (no bin: the run's sums are dropped)
    wgt = __fma_rn(r.y, q.y, wgt);
  }
  push_run(buf, Q, qn, cur != kInvalidKey, cur, s0, s_hi, delta, didj, wgt, lane);
  drain(buf, Q, 0, qn, lane);
}

template <bool MINPOS>
__global__ void __launch_bounds__(kDiagThreads, 3) diag_pairs_kernel(const __grid_constant__ PairArgs A) {
  extern __shared__ PixPack diag_smem[];  // the warps' queues
  __shared__ Claim s_claims[kDiagWarps];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  WarpQ& Q = reinterpret_cast<WarpQ*>(diag_smem)[warp];
  if (tid == 0) s_args = A;
  if (lane == 0) s_claims[warp].todo = 0u;
  __syncthreads();
  unsigned long long n_eval = 0, n_rech = 0, n_taken = 0, idx = 0;
  while (claim_item(A, kOwnerDiagPairs, s_claims[warp], lane, idx, A.short_claim)) {
    ++n_taken;
    const uint32_t i = A.item_i[idx], j = A.item_j[idx];
    DItem it;
    int dlo, dhi;
    if (!diag_window(A, idx, i, j, lane, it, dlo, dhi)) continue;
    __syncwarp();  // the last item's sums are added
    if (lane == 0) s_item[warp] = it;
    __syncwarp();
    const PairsItem p = {A.dist_pad + A.off[i] + (uint64_t)kPad * (i + 1), A.dist_pad + A.off[j] + (uint64_t)kPad * (j + 1),
                         A.row2 + A.off[i], A.row2 + A.off[j]};
    const int ni = it.ni, nj = it.nj;
    const float ap = it.ap;
    unsigned ev = 0, re = 0;
    for (int d0 = dlo; d0 <= dhi; d0 += 32) pairs_group<MINPOS>(A, p, ni, nj, ap, warp, d0, dhi, lane, Q, ev, re);
    n_eval += ev;
    n_rech += re;
  }
  add_counters_diag(A, lane, n_eval, n_rech, n_taken);
}

// Two items of two padded sightlines.
size_t diag_smem_bytes(const PairArgs& a) { return (size_t)4 * (a.max_np + 3 * kParityPad) * sizeof(PixPack); }

// Persistent launch: `ctas_per_sm` CTAs per SM (0 or above the occupancy
// limit: as many as fit), or with `max_out` set only that limit.
template <bool MINPOS, bool SMEM>
cudaError_t launch_diag(const PairArgs& a, int num_sms, int ctas_per_sm, cudaStream_t stream, int* max_out) {
  const size_t smem = kDiagWarps * sizeof(WarpQ) + (SMEM ? diag_smem_bytes(a) : 0);  // two items of two sightlines
  auto kern = diag_kernel<MINPOS, SMEM>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kDiagThreads, smem);
  if (e != cudaSuccess) return e;
  per_sm = per_sm > 0 ? per_sm : 1;
  if (max_out) {
    *max_out = per_sm;
    return cudaSuccess;
  }
  if (ctas_per_sm > 0 && ctas_per_sm < per_sm) per_sm = ctas_per_sm;
  PairArgs b = a;
  b.claim_max = claim_limit(a.n_items, num_sms * per_sm);
  kern<<<num_sms * per_sm, kDiagThreads, smem, stream>>>(b);
  return cudaGetLastError();
}

// Items are staged in shared memory when two fit a CTA beside its queues.
constexpr size_t kDiagSmem = 224 * 1024 - kDiagWarps * sizeof(WarpQ);

template <bool MINPOS>
cudaError_t launch_diag2(const PairArgs& a, int num_sms, int ctas_per_sm, cudaStream_t stream, int* max_out) {
  return diag_smem_bytes(a) <= kDiagSmem
             ? launch_diag<MINPOS, true>(a, num_sms, ctas_per_sm, stream, max_out)
             : launch_diag<MINPOS, false>(a, num_sms, ctas_per_sm, stream, max_out);
}

template <bool MINPOS>
cudaError_t launch_pairs(const PairArgs& a, int num_sms, cudaStream_t stream) {
  constexpr size_t smem = kDiagWarps * sizeof(WarpQ);
  auto kern = diag_pairs_kernel<MINPOS>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kDiagThreads, smem);
  if (e != cudaSuccess) return e;
  const int ctas = num_sms * (per_sm > 0 ? per_sm : 1);
  PairArgs b = a;
  b.claim_max = claim_limit(a.n_items, ctas * kDiagWarps);
  // short items several at a time (16 of 32 pixels), as many as leave each warp several claims
  b.short_claim = (int)std::min<unsigned long long>(
      std::max(1, std::min(16, 512 / std::max(a.max_np, 1))),
      std::max<unsigned long long>(1, a.n_items / (4ull * ctas * kDiagWarps)));
  kern<<<ctas, kDiagThreads, smem, stream>>>(b);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_diag_pairs_kernel(const PairArgs& a, bool minpos, int num_sms, cudaStream_t stream) {
  return minpos ? launch_pairs<true>(a, num_sms, stream) : launch_pairs<false>(a, num_sms, stream);
}

cudaError_t launch_diag_kernel(const PairArgs& a, bool minpos, int num_sms, int ctas_per_sm, cudaStream_t stream,
                               int* max_out) {
  return minpos ? launch_diag2<true>(a, num_sms, ctas_per_sm, stream, max_out)
                : launch_diag2<false>(a, num_sms, ctas_per_sm, stream, max_out);
}

}  // namespace tos
