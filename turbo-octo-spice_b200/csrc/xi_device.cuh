// xi_device.cuh — device helpers shared by the pixel-pair kernel
// (xi_kernels.cu) and the run-sweep kernel (xi_runs.cu): FP32 approximations,
// fixed-point conversion, 128-bit accumulation, and the exact re-binning that
// follows the reference's FP64 expression order.
#pragma once

#include "xi_kernels.cuh"

namespace tos {
namespace {

constexpr unsigned kFull = 0xFFFFFFFFu;
enum { kPolar = TOS_POLAR, kCart = TOS_CARTESIAN, kObs = TOS_OBSERVING };

__device__ __forceinline__ float sqrt_approx(float x) {
  float r;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float rsqrt_approx(float x) {
  float r;
  asm("rsqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// Fixed-point image round(c * scale) of a contribution, |c*scale| < 2^51.
__device__ __forceinline__ long long to_fixed(double c, double scale) {
  return __double_as_longlong(__fma_rn(c, scale, kMagic52)) - kMagic52Bits;
}

// round(c * 2^F) for |c * 2^F| < 2^62, given sh = 2^(F-44): the high part is
// rounded first and the exact remainder carries the low 44 bits.
__device__ __forceinline__ long long to_fixed_wide(double c, double sh) {
  const double v = c * sh;
  const double r = __dadd_rn(v, kMagic52);
  const long long qh = __double_as_longlong(r) - kMagic52Bits;
  const double rem = v - __dsub_rn(r, kMagic52);  // r - magic is qh exactly; |rem| <= 0.5
  return (qh << 44) + to_fixed(rem, 17592186044416.0 /* 2^44 */);
}

// Window word of field k, part p (0 = low).
__device__ __forceinline__ int wword(int k, int p) {
  return (k < kSigned) ? 3 * k + p : 3 * kSigned + 2 * (k - kSigned) + p;
}
constexpr int kWordCount = 3 * kSigned + 2 * (7 - kSigned);      // 17
constexpr int kWordContrib = kWordCount + 1;                     // 18

// Global reduction add with no returned value (red, not atom): nothing in
// the thread waits for it.
__device__ __forceinline__ void red_add(unsigned long long* p, unsigned long long v) {
  asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Add a signed value v (|v| < 2^89) to one field's sums {lo, hi} in the
// carry-free format of kAccWords: lo += v mod 2^26, hi += floor(v / 2^26).
__device__ __forceinline__ void add_wide(unsigned long long* lo, unsigned long long* hi, __int128 v) {
  red_add(lo, (unsigned long long)v & kAccMask);
  const long long h = (long long)(v >> kAccShift);
  if (h != 0) red_add(hi, (unsigned long long)h);
}
__device__ __forceinline__ void add128(unsigned long long* lo, unsigned long long* hi, long long q) {
  red_add(lo, (unsigned long long)q & kAccMask);
  const long long h = q >> kAccShift;
  if (h != 0) red_add(hi, (unsigned long long)h);
}

// ---- exact re-binning (reference expression order) returning the two axis
// indices; z is handled per item.  Mirrors ref_bin_* in tos_common.h.
__device__ __forceinline__ bool exact_cart(float d1, float d2, double c, const RefGrid& g,
                                           uint32_t* b0, uint32_t* b1) {
  const double r1_sq = (double)fmul(d1, d1);
  const double two_r1_cos12 = dmul((double)fmul(2.0f, d1), c);
  const double r_para = (double)fabsf(fsub(d1, d2));
  const uint32_t p = ref_u32(dmul(dsub(r_para, g.min0), g.inv0));
  if (p >= g.n0) return false;
  const double r_sq = dadd(r1_sq, dmul(dsub((double)d2, two_r1_cos12), (double)d2));
  const double x = fabs(dsub(r_sq, dmul(r_para, r_para)));
  const uint32_t q = ref_u32(dmul(dsub(dsqrt(x), g.min1), g.inv1));
  if (q >= g.n1) return false;
  *b0 = p;
  *b1 = q;
  return true;
}

__device__ __forceinline__ bool exact_polar(float d1, float d2, double c, const RefGrid& g,
                                            uint32_t* b0, uint32_t* b1) {
  const double r1_sq = (double)fmul(d1, d1);
  const double two_r1_cos12 = dmul((double)fmul(2.0f, d1), c);
  const double r_sq = dadd(r1_sq, dmul(dsub((double)d2, two_r1_cos12), (double)d2));
  const double r = dsqrt(r_sq);
  const uint32_t p = ref_u32(dmul(dsub(r, g.min0), g.inv0));
  if (p >= g.n0) return false;
  if (r == 0) return false;
  const double mu = ddiv((double)fabsf(fsub(d1, d2)), r);
  const uint32_t q = ref_u32(dmul(dsub(mu, g.min1), g.inv1));
  if (q >= g.n1) return false;
  *b0 = p;
  *b1 = q;
  return true;
}

__device__ __forceinline__ bool exact_obs(float l1, float l2, const RefGrid& g, uint32_t* b0) {
  const uint32_t p = ref_u32(dmul(dsub((double)fabsf(fsub(l1, l2)), g.min0), g.inv0));
  if (p >= g.n0) return false;
  *b0 = p;
  return true;
}

// Prefix sums of sightline i.
__device__ __forceinline__ Prefix prefix_of(const PairArgs& A, uint32_t i) {
  return Prefix{A.pre2 + A.off[i] + i, A.prel + A.off[i] + i};
}

// Items of the run-sweep kernel when A.run_split is set: z index constant
// over the item and (Cartesian) 2(1 - cos theta) large enough for the
// reference's r_perp expression to grow with the column distance along every
// row.  Both kernels evaluate this same predicate.
__device__ __forceinline__ bool run_item(const PairArgs& A, double c, bool zconst) {
  return zconst && dmul(2.0, dsub(1.0, c)) >= A.run_amin;
}

__device__ __forceinline__ uint32_t zbin_of_sum(float lsum, const RefGrid& g) {
  return ref_u32(dmul(dsub(dmul(0.5, (double)lsum), g.min2), g.invn2));
}

// Items of the diagonal-sweep kernel when A.diag_split is set (Polar): the z
// index is constant over the item (from the z codes zlo, zhi of the smallest
// and largest loglam sums and their indices).  Both the diagonal-sweep and
// the pixel-pair kernel evaluate this same predicate.
__device__ __forceinline__ bool diag_item(const PairArgs& A, double zlo, double zhi, uint32_t zb_lo,
                                          uint32_t zb_hi) {
  return A.diag_split && zlo > -1.0 && zhi < 2147483648.0 && zb_lo == zb_hi;
}

// The kernel that takes item idx, from the predicates above as each kernel
// applies them (load_item for the pointer sweep, the pixel-pair kernel's own
// test): one lane per item, so that a kernel can claim a batch of items and skip
// the others' without loading each one warp-wide.
enum ItemOwner { kOwnerNone = 0, kOwnerGrid, kOwnerShort, kOwnerGaps, kOwnerRun, kOwnerDiag, kOwnerDiagPairs, kOwnerPair };
__device__ __forceinline__ int item_owner(const PairArgs& A, unsigned long long idx) {
  const uint32_t i = A.item_i[idx], j = A.item_j[idx];
  if (A.npix[i] == 0 || A.npix[j] == 0) return kOwnerNone;
  const float4 ri = A.range[i], rj = A.range[j];
  const float lsum_lo = __fadd_rn(ri.z, rj.z), lsum_hi = __fadd_rn(ri.w, rj.w);
  const double zlo = dmul(dsub(dmul(0.5, (double)lsum_lo), A.g.min2), A.g.invn2);
  const double zhi = dmul(dsub(dmul(0.5, (double)lsum_hi), A.g.min2), A.g.invn2);
  const uint32_t zb_lo = zbin_of_sum(lsum_lo, A.g), zb_hi = zbin_of_sum(lsum_hi, A.g);
  const bool zconst = zlo > -1.0 && zhi < 2147483648.0 && zb_lo == zb_hi;
  if (A.run_split && run_item(A, A.item_c[idx], zconst)) {
    if ((A.grid_split || A.gap_split) && A.gfirst[i] != kNoGrid && A.gfirst[j] != kNoGrid) {
      if (A.grid_split && A.gspan[i] == A.npix[i] && A.gspan[j] == A.npix[j])
        return max(A.npix[i], A.npix[j]) <= kShortPixels ? kOwnerShort : kOwnerGrid;
      if (A.gap_split) return kOwnerGaps;
    }
    return kOwnerRun;
  }
  if (diag_item(A, zlo, zhi, zb_lo, zb_hi))
    return max(A.npix[i], A.npix[j]) > (uint32_t)A.diag_len ? kOwnerDiag : kOwnerDiagPairs;
  return kOwnerPair;
}

// Items per claim of a kernel that takes few of the items (the run sweep and
// the pixel-pair kernel beside the grid or diagonal sweep): a warp claims 32
// with one atomic and keeps its own.
constexpr int kClaimItems = 32;

// The claims of a CTA that prepares one item at a time (the band and diagonal
// sweeps): items base + k, k a set bit of `todo`, are its own still to do.
struct Claim {
  unsigned long long base;
  unsigned todo;
};

// The next item of kernel `owner` (one warp; false: none left).  A claim takes
// one item, so that long items spread over the CTAs (`size` items, up to
// kClaimItems, where they are short); after those of another kernel it takes
// twice as many, up to A.claim_max, until it holds one of its own: a sweep that
// owns few of the items goes through the others up to 32 at a time.  (8.0e6 items
// of 4,000 contiguous sightlines, one of them masked: the gap sweep scanned them
// in 52 ms one by one, now in 2.)
__device__ __forceinline__ bool claim_item(const PairArgs& A, int owner, Claim& C, int lane, unsigned long long& idx,
                                           int size = 1) {
  unsigned todo = C.todo;
  if (todo == 0u) {
    idx = 0;
    if (size == 1) {
      if (lane == 0) idx = atomicAdd(A.next_item, 1ull);
      idx = __shfl_sync(kFull, idx, 0);
      if (idx >= A.n_items) return false;
      if (item_owner(A, idx) == owner) return true;
      size = 2;
    }
    for (; todo == 0u; size = min(2 * size, max(size, A.claim_max))) {
      if (lane == 0) idx = atomicAdd(A.next_item, (unsigned long long)size);
      idx = __shfl_sync(kFull, idx, 0);
      if (idx >= A.n_items) return false;
      const unsigned long long mine = idx + lane;
      todo = __ballot_sync(kFull, lane < size && mine < A.n_items && item_owner(A, mine) == owner);
    }
    if (lane == 0) C.base = idx;
  } else {
    idx = C.base;
  }
  idx += __ffs(todo) - 1;
  __syncwarp();  // every lane has read C
  if (lane == 0) C.todo = todo & (todo - 1u);
  __syncwarp();
  return true;
}

}  // namespace
}  // namespace tos
