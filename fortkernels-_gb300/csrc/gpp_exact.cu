// Operand passes of the exact GPP contractions (gpp_exact.cuh).
//
// Y[iw][g][ig] = G (c + i b) / (c^2 + b^2), G = I_eps wtilde, c = wx - Re
// wtilde, b = Im wtilde, 0 where the pole guard drops the term
// (BGW-Kernels/gppKer.cpp:394-404, conj(aqsm) and vcoul moved to the
// epilogue); the half sum keeps the terms the guard drops
// (gppKerSeq.cpp:206-242).  Row iw * ng + g of the contraction is one
// frequency of one column; the occupied bands' ssx factors (gppKer.cpp:38-58)
// are a second group of rows.
//
// gx_max_kernel bounds the factors per row (the digits' exponent) from FP32
// values, one pass over the inputs at memory speed.
// gx_ff_kernel forms them from FP64 numerators in float-float arithmetic (FP32
// pairs: ~2^-48 rms), cuts them into
// digits with paired FP32 operations and writes each row's digits as 16-byte
// chunks: 16 columns x 32 g-vectors staged in shared memory, four CTAs per SM.
// Bound by issue slots (69 % issuing, FP64 pipe 53 %, FMA 49 %): 2.42 ms at
// 1638 x 32768 with the occupied bands' factors (2.38 ms with the reciprocal's
// first-order correction and an exponent bit to spare, whose band sums' errors
// were 7.4e-15 instead of 4.8e-15; 2.74 ms with digits of one
// value per instruction, the general FP64 split and all large factors counted).
// Factors of two elements per instruction need 80 registers or spill at two
// or three CTAs per SM: 3.13 and 3.35 ms.
// (The factors in FP64, 34 operations per column and g-vector, ran at the FP64
// pipe's 2 per clock per SM: 3.54 ms at 1638 x 32768, with the occupied bands'
// own pass another 3.86 ms.)  The half sum's factors, FP64 before, stay in FP64
// (gx_f64_kernel): poles inside the guard, and occupied bands' sums that
// cancel (2.3e-14 with float-float factors, 2e-15 so).
#include <algorithm>

#include "gpp_exact.cuh"
#include "floatfloat.cuh"
#include "runtime.h"

namespace sigma {
namespace {

constexpr int kGxThreads = 256;
constexpr int kGxCols = 16;  // columns per CTA
constexpr int kIgBlk = 512;  // g-vector block of the half sum's reference loop
// Half sum: poles inside the guard make a few factors of a row much larger
// than the rest, so a count of large ones says little, and the row's exponent
// serves the rest badly: its operands take seven digits.  Its check sums, over
// the row's own range, the factors' squares times those of the least element
// that any band has there (ExactPrep::band_min): no row pair's sum of squares
// is below that.  From 2^-38 K on (units of the rows' largest elements) the
// error of 2^-61 sqrt(K) is at most 2^-42 of the root mean square.  Uniform
// inputs with the nearest of 5e7 poles at 7e-5 lie at 2^-32 or above.  (Segment
// sums of squares of row and bands, multiplied as if unrelated, let a factor of
// 2^30 through that met zeros: errors of 6e-10.)
constexpr float kHalfPower = 1.f / 274877906944.f;

template <int kForm>
struct Form {
  static constexpr bool kReal = kForm == kGxReal || kForm == kGxRealOcc, kRealOcc = kForm == kGxRealOcc;
  static constexpr bool kHalf = kForm == kGxHalf, kHalfOcc = kForm == kGxHalfOcc;
  static constexpr bool kLeast = kHalf || kHalfOcc;  // checked against band_min
  static constexpr bool kF64 = kRealOcc || kHalf || kHalfOcc;  // factors in FP64, seven digits
  static constexpr int kSlabs = kHalf ? 4 : kReal ? kNW : 2 * kNW, kParts = kReal ? 1 : 2;  // the most slabs
};

template <int kForm>
__device__ __forceinline__ double2 gx_load(const double* a, size_t off) {
  if (Form<kForm>::kReal) return make_double2(a[off], 0.0);
  return reinterpret_cast<const double2*>(a)[off];
}
// End of a slab's g-vectors in column g.
template <int kForm>
__device__ __forceinline__ int gx_limit(const GxDev& p, int g, int slab) {
  if (!Form<kForm>::kHalf && !Form<kForm>::kHalfOcc) return p.nc;
  const int igp = p.igp_of[g];
  if (igp < 0) return 0;
  if (Form<kForm>::kHalfOcc) return min(igp, p.brk[g]);
  return slab < kNW ? max(igp - 1, 0) : igp;
}
// Row of a slab's column, and the end of its group's row blocks.
__device__ __forceinline__ int gx_row(const ExactPrep& ex, int ng, int nf, int slab, int g) {
  return slab < nf ? slab * ng + g : ex.n_main_blocks * kExRows + (slab - nf) * ng + g;
}
__device__ __forceinline__ int gx_rows_end(const ExactPrep& ex, int nf, int slab) {
  return (slab < nf ? ex.n_main_blocks : ex.n_row_blocks) * kExRows;
}

// The leading 24 bits of a double as FP32 (integer pipe).
__device__ __forceinline__ float f32_lead(double x) { return ff_of(x).hi; }
__device__ __forceinline__ bool any_bits(double2 v) {
  return ((unsigned)__double2hiint(v.x) << 1 | (unsigned)__double2loint(v.x) | (unsigned)__double2hiint(v.y) << 1 |
          (unsigned)__double2loint(v.y)) != 0;
}

// One CTA per column: exponents of its rows.  Squared magnitudes from FP32
// values (c from exact FP32 halves), the guard taken somewhat wide on both
// sides, with a 2^-8 margin; what FP32 cannot bound raises the flag.  Squares
// below 1e-36 count as 1e-36: an upper bound, so that no element exceeds its
// row's exponent (one far above its row fails the overlap check).
constexpr float kTinySq = 1e-36f;
template <int kForm>
__global__ void __launch_bounds__(kGxThreads) gx_max_kernel(GxDev p, ExactPrep ex, int nf, int nf2) {
  using F = Form<kForm>;
  __shared__ unsigned s_m[F::kSlabs][kGxThreads / 32];
  chain_begin();
  ex_begin_counts(ex);  // the first kernel of an execution
  const int g = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool occ = F::kHalfOcc || F::kRealOcc || nf2 > 0;
  FF wx[kNW];
  float iwx4[kNW];
  // |wtilde| or |I_eps| above 1e15 or not finite, |wx| outside 1e-9 .. 1e9:
  // reciprocals and their squares may flush to 0
  bool huge = false;
#pragma unroll
  for (int iw = 0; iw < kNW; ++iw) {
    wx[iw] = ff_of(p.wx[iw]);
    huge = huge || !(fabsf(wx[iw].hi) < 1e9f && fabsf(wx[iw].hi) > 1e-9f);
    const float i2 = rcp_approx(wx[iw].hi * wx[iw].hi);
    iwx4[iw] = i2 * i2;
  }
  unsigned m[F::kSlabs];  // bits of non-negative floats; infinite and NaN are the largest
#pragma unroll
  for (int i = 0; i < F::kSlabs; ++i) m[i] = 0u;
  auto top = [](unsigned& v, float y) { v = max(v, __float_as_uint(y)); };
  bool bad = false, bad_e = false;  // a nonzero factor, I_eps value below 1e-18
  const int k_end = gx_limit<kForm>(p, g, F::kSlabs - 1), k_freq = gx_limit<kForm>(p, g, 0);
  auto element = [&](int k, double2 w, double2 e) {
    const float er = f32_lead(e.x), ei = F::kReal ? 0.f : f32_lead(e.y);
    const float e2 = fmaf(er, er, ei * ei);
    const bool any_e = any_bits(e);
    if (F::kHalf) {
      top(m[F::kSlabs - 1], e2);
      bad_e = bad_e || (any_e && !(e2 > kTinySq));
      if (k >= k_freq || k % kIgBlk == kIgBlk - 1) return;
    }
    const FF a = ff_of(w.x);
    const float b = F::kReal ? 0.f : f32_lead(w.y), b2 = b * b;
    const float s2 = fmaf(a.hi, a.hi, b2);  // |wtilde|^2
    huge = huge || !(s2 + e2 < 1e30f);
    const bool any = any_bits(w) && any_e;
    const float g2 = any ? fmaxf(s2, kTinySq) * fmaxf(e2, kTinySq) : 0.f;  // |G|^2
    const float least = fminf(s2, e2) > kTinySq ? kTinySq : INFINITY;       // factors from here on are not small ones
    // the guard's threshold, somewhat above and below
    const float up = fmaxf(0.2501f, s2 * 4.001e-6f), low = 0.2499f;
#pragma unroll
    for (int iw = 0; iw < kNW; ++iw) {
      const float c = (wx[iw].hi - a.hi) + (wx[iw].lo - a.lo);
      const float w2 = fmaf(c, c, b2), r = rcp_approx(w2);
      if (!F::kRealOcc && (F::kHalf ? !(w2 > up) : !(w2 <= low))) {  // also NaN
        const float y = g2 * r;
        top(m[iw], y);
        bad = bad || (any && !(y > least));
      }
      if (!F::kHalf && (!F::kReal || F::kRealOcc) && occ) {
        const float z = (wx[iw].hi + a.hi) + (wx[iw].lo + a.lo);
        const float rz = rcp_approx(fmaf(z, z, b2));
        float y = w2 > up ? 0.f : 0.25f * g2 * rz;  // |G / (2 (wx + wtilde))|^2
        // |Omega2 / (wx^2 - wtilde^2)|^2, |Omega2 / wx^2|^2
        if (!(w2 <= low)) y = fmaxf(y, s2 * g2 * (F::kHalfOcc ? r * rz : iwx4[iw]));
        top(m[F::kSlabs > kNW ? kNW + iw < F::kSlabs ? kNW + iw : 0 : iw], y);
        bad = bad || (any && !(y > least));
      }
    }
  };
  // four elements' loads in flight per thread
  for (int k0 = tid; k0 < k_end; k0 += 4 * kGxThreads) {
    double2 w[4], e[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int k = min(k0 + q * kGxThreads, k_end - 1);
      w[q] = gx_load<kForm>(p.wt, (size_t)g * p.nc + k);
      e[q] = gx_load<kForm>(p.ieps, (size_t)g * p.nc + k);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (k0 + q * kGxThreads < k_end) element(k0 + q * kGxThreads, w[q], e[q]);
  }
  bad = __syncthreads_or(bad);
  if (F::kHalf) bad_e = __syncthreads_or(bad_e);
  huge = __syncthreads_or(huge);
#pragma unroll
  for (int i = 0; i < F::kSlabs; ++i) {
    const unsigned v = __reduce_max_sync(0xffffffffu, m[i]);
    if (lane == 0) s_m[i][warp] = v;
  }
  __syncthreads();
  if (tid < nf + nf2) {
    unsigned v = 0;
    for (int q = 0; q < kGxThreads / 32; ++q) v = max(v, s_m[tid][q]);
    const float f = sqrtf(__uint_as_float(v)) * (1.f + 1.f / 256.f);
    // a factor too small for FP32 may only be ignored beside large ones
    const bool small = F::kHalf && tid == F::kSlabs - 1 ? bad_e : bad;
    if (huge || !(f < 1e18f) || (small && !(f > 1e-6f)) || (v && f < 1e-18f)) ex_raise(ex);
    ex.ea[gx_row(ex, p.ng, nf, tid, g)] = v ? (int)(__float_as_uint(f) >> 23) - 126 : kExZeroRow;
  }
}

// ---------------------------------------------------------------- float-float factors
// Decisions in the FP64 path's expressions: bit 0 the guard keeps the term,
// bit 1 the second occupied-band branch.
static __device__ __noinline__ unsigned gx_decide(double wx, double a, double b) {
  const double b2 = guard_b2(b), wv = guard_w(wx, a, b2);
  if (keep_nonneg(wv, guard_thr(a, b2))) return 1u;
  return gt_nonneg(wv, 0.0) && gt_nonneg(guard_thr2(a, b2), wv) ? 2u : 0u;
}

__device__ __forceinline__ FF gx_norm(FF x) { return ff_norm(x.hi, x.lo); }

struct Factors {
  double2 y, s;  // Y and ssx
};
// One frequency's factors in FP64, for elements or frequencies outside the
// float-float range.
static __device__ __noinline__ Factors gx_wide(double wx, double2 wt, double2 ie) {
  const double a = wt.x, b = wt.y, b2 = guard_b2(b), c = __dsub_rn(wx, a), dr = wx + a;
  const double gx = fma(ie.x, a, -(ie.y * b)), gy = fma(ie.x, b, ie.y * a);
  const unsigned mask = gx_decide(wx, a, b);
  Factors f{make_double2(0.0, 0.0), make_double2(0.0, 0.0)};
  if (mask & 1u) {
    const double r = rcp_f64(fma(c, c, b2)), i2 = rcp_f64(wx * wx);
    f.y = make_double2(fma(gx, c, -(gy * b)) * r, fma(gy, c, gx * b) * r);
    f.s = make_double2(fma(a, gx, -(b * gy)) * i2, fma(a, gy, b * gx) * i2);  // Omega2 / wx^2
  } else if (mask & 2u) {
    const double q = -0.5 * rcp_f64(fma(dr, dr, b2));
    f.s = make_double2(fma(gx, dr, gy * b) * q, fma(gy, dr, -(gx * b)) * q);
  }
  return f;
}

// The three frequencies' factors of one element: put(slab, re, im) takes Y in
// slabs 0-2 and ssx in 3-5 as normalised pairs.
template <int kForm, bool kOcc, class Put>
__device__ __forceinline__ void gx_factors(const FF (&wx)[kNW], const FF (&iwx2)[kNW], const double* wxd,
                                           bool wx_wide, double2 wt, double2 ie, Put put) {
  using F = Form<kForm>;
  if (wx_wide || !ff_range(wt.x, wt.y) || !ff_range(ie.x, ie.y)) {
#pragma unroll
    for (int iw = 0; iw < kNW; ++iw) {
      const Factors f = gx_wide(wxd[iw], wt, ie);
      put(iw, ff_of_rn(f.y.x), ff_of_rn(f.y.y));
      if (kOcc) put(kNW + iw, ff_of_rn(f.s.x), ff_of_rn(f.s.y));
    }
    return;
  }
  // G, c and |wdiff|^2 in FP64 (11 operations, 5.5 clocks per SM, beside ~10
  // clocks of FP32 work): exact decisions, and the factor's error is that of
  // the float-float reciprocal and products alone (G and c in float-float put
  // a strongly cancelling band sum at 2.3e-12)
  const FF zero{0.f, 0.f};
  const double b2d = guard_b2(wt.y);
  FF gx, gy = zero, b = zero, b2 = zero, a = zero, ox = zero, oy = zero;
  if (F::kReal) {
    gx = ff_split_in_range(__dmul_rn(ie.x, wt.x));
  } else {
    gx = ff_split_in_range(fma(ie.x, wt.x, -__dmul_rn(ie.y, wt.y)));
    gy = ff_split_in_range(fma(ie.x, wt.y, __dmul_rn(ie.y, wt.x)));
    b = ff_split_in_range(wt.y);
  }
  if (kOcc) {
    a = ff_split_in_range(wt.x);
    b2 = ff_mul(b, b);
    ox = gx_norm(ff_dot2_raw(a, gx, b, gy));  // Omega2 = wtilde G
    oy = gx_norm(ff_dot2_raw(a, gy, ff_neg(b), gx));
  }
  // the guard's second condition binds from |wtilde|^2 = 62500 on; dropped
  // terms with |wtilde|^2 well above the second branch's bound take it
  const float af = __double2float_rn(wt.x), bf = __double2float_rn(wt.y), s2 = fmaf(af, af, bf * bf);
  const bool binds = s2 >= 62000.f, big = s2 > 1.01e-6f;
#pragma unroll
  for (int iw = 0; iw < kNW; ++iw) {
    const double cd = __dsub_rn(wxd[iw], wt.x), wv = fma(cd, cd, b2d);
    bool keep = keep_nonneg(wv, kLimitTwo), second = !keep && gt_nonneg(wv, 0.0);
    if (binds || (kOcc && !keep && !big)) {
      const unsigned mask = gx_decide(wxd[iw], wt.x, wt.y);
      keep = mask & 1u;
      second = mask & 2u;
    }
    const FF c = ff_split_in_range(cd);
    if (F::kReal) {
      const FF y = ff_mul(gx, gx_norm(ff_rcp2_raw(c)));
      put(iw, keep ? y : zero, zero);
    } else {
      const FF r = gx_norm(ff_rcp2_raw(ff_split_in_range(wv)));
      const FF yx = ff_mul(gx_norm(ff_dot2_raw(gx, c, gy, b)), r);
      const FF yy = ff_mul(gx_norm(ff_dot2_raw(gy, c, ff_neg(gx), b)), r);
      put(iw, keep ? yx : zero, keep ? yy : zero);
      if (kOcc) {
        // Omega2 / wx^2 or -G conj(z) / (2 |z|^2), z = wx + wtilde
        const FF z = ff_add(wx[iw], a);
        const FF rz = gx_norm(ff_rcp2_raw(ff_sq_add(z, b2)));
        const FF tx = gx_norm(ff_dot2_raw(gx, z, gy, ff_neg(b))), ty = gx_norm(ff_dot2_raw(gy, z, gx, b));
        const FF m = keep ? iwx2[iw] : FF{-0.5f * rz.hi, -0.5f * rz.lo};
        const FF sx = ff_mul(keep ? ox : tx, m), sy = ff_mul(keep ? oy : ty, m);
        const bool on = keep || second;
        put(kNW + iw, on ? sx : zero, on ? sy : zero);
      }
    }
  }
}

constexpr int kFfK = 32;  // g-vectors per staged tile
template <int kForm, bool kOcc>
struct FfPlanes {
  static constexpr int kSlabs = kOcc ? 6 : 3;
  // high and low halves; conflict-free along g-vectors, and for pairs of them along columns
  float hi[Form<kForm>::kParts][kSlabs][kGxCols][kFfK + 2], lo[Form<kForm>::kParts][kSlabs][kGxCols][kFfK + 2];
};

// Items (column block, run of `run` g-vectors).  Column blocks run past ng to
// cover the padding rows of each group's last row block (zero digits).
template <int kForm, bool kOcc>
__global__ void __launch_bounds__(kGxThreads, 4) gx_ff_kernel(GxDev p, ExactPrep ex, float* stat, int nf, int run) {
  using F = Form<kForm>;
  constexpr int kSlabs = FfPlanes<kForm, kOcc>::kSlabs;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  FfPlanes<kForm, kOcc>& sm = *reinterpret_cast<FfPlanes<kForm, kOcc>*>(smem_raw);
  __shared__ float s_scale[kSlabs][kGxCols], s_thr[kSlabs][kGxCols];
  __shared__ int s_lim[kGxCols], s_need;
  __shared__ FF s_wx[kNW], s_iwx2[kNW];
  __shared__ bool s_wide;
  chain_begin();
  if (*ex.flag) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int p0 = blockIdx.x * kGxCols;
  if (tid == 0) {
    s_need = 0;
    bool wide = false;
    for (int iw = 0; iw < kNW; ++iw) {
      const double w = p.wx[iw];
      wide = wide || !ff_freq_range(w);
      s_wx[iw] = ff_of_rn(w);
      s_iwx2[iw] = ff_of_rn(rcp_f64(w * w));
    }
    s_wide = wide;
  }
  __syncthreads();
  if (tid < kSlabs * kGxCols) {
    const int i = tid / kGxCols, pl = tid % kGxCols, g = p0 + pl, R = gx_row(ex, p.ng, nf, i, g);
    const int e = g < p.ng ? ex.ea[R] : kExZeroRow;
    // -2^(7 - e) and 2^(e - 1 - slack) (|e| < 64 unless flagged; a zero row's values are zero)
    s_scale[i][pl] = e == kExZeroRow ? 0.f : -__uint_as_float((unsigned)(134 - e) << 23);
    s_thr[i][pl] = e == kExZeroRow ? INFINITY : __uint_as_float((unsigned)(126 - kExSlackA + e) << 23);
    if (i == 0) s_lim[pl] = g < p.ng ? gx_limit<kForm>(p, g, 0) : 0;
    const bool last = i == nf - 1 || i == kSlabs - 1;
    if ((g < p.ng || last) && R < gx_rows_end(ex, nf, i)) atomicMax(&s_need, ex.kt_lim[R / kExRows] * kExKTile);
  }
  __syncthreads();
  const int k_begin = blockIdx.y * run, k_end = min(s_need, k_begin + run);  // tiles the contraction reads
  float acc[2][kSlabs];  // large factors per column of this warp
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int i = 0; i < kSlabs; ++i) acc[j][i] = 0.f;
  for (int k0 = k_begin; k0 < k_end; k0 += kFfK) {
    const FF wx[kNW] = {s_wx[0], s_wx[1], s_wx[2]}, iwx2[kNW] = {s_iwx2[0], s_iwx2[1], s_iwx2[2]};
    const bool counted = k0 % kExSeg < kExCount;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int pl = warp + 8 * j, g = p0 + pl, ig = k0 + lane;
      if (ig < s_lim[pl]) {
        const double2 wt = gx_load<kForm>(p.wt, (size_t)g * p.nc + ig);
        const double2 ie = gx_load<kForm>(p.ieps, (size_t)g * p.nc + ig);
        if (ig + kFfK < s_lim[pl]) {
          const size_t next = ((size_t)g * p.nc + ig + kFfK) * (F::kReal ? 1 : 2);
          prefetch_l2(p.wt + next);
          prefetch_l2(p.ieps + next);
        }
        gx_factors<kForm, kOcc>(wx, iwx2, p.wx, s_wide, wt, ie, [&](int i, FF re, FF im) {
          sm.hi[0][i][pl][lane] = re.hi;
          sm.lo[0][i][pl][lane] = re.lo;
          if (!F::kReal) {
            sm.hi[F::kParts - 1][i][pl][lane] = im.hi;
            sm.lo[F::kParts - 1][i][pl][lane] = im.lo;
          }
        });
      } else {
#pragma unroll
        for (int i = 0; i < kSlabs; ++i)
#pragma unroll
          for (int q = 0; q < F::kParts; ++q) sm.hi[q][i][pl][lane] = sm.lo[q][i][pl][lane] = 0.f;
      }
      if (counted)
#pragma unroll
        for (int i = 0; i < kSlabs; ++i)
          acc[j][i] += fmaxf(fabsf(sm.hi[0][i][pl][lane]), fabsf(sm.hi[F::kParts - 1][i][pl][lane])) >= s_thr[i][pl]
                           ? 1.f : 0.f;
    }
    __syncthreads();
    // digits: a warp takes one (slab, part, K tile), its lanes the 16
    // columns x 2 chunks (512 contiguous bytes per slice)
#pragma unroll 1
    for (int t = warp; t < kSlabs * F::kParts * 2; t += kGxThreads / 32) {
      const int q = t & 1, part = (t >> 1) % F::kParts, i = (t >> 1) / F::kParts;
      const int pl = lane & 15, ch = lane >> 4, g = p0 + pl, R = gx_row(ex, p.ng, nf, i, g);
      const int tile = k0 / kExKTile + q;
      // padding rows follow the group's last slab's columns
      if (g >= p.ng && i != nf - 1 && i != kSlabs - 1) continue;
      if (R >= gx_rows_end(ex, nf, i) || tile >= ex.kt_lim[R / kExRows]) continue;
      unsigned char* dst =
          ex.a_tiles + ((size_t)(R / kExRows) * F::kParts * ex.kt + part * ex.kt + tile) * ex_a_bytes(6);
      const int k = q * kExKTile + ch * 8;
      ex_put_ff(dst, R % kExRows, ch, reinterpret_cast<const float2*>(&sm.hi[part][i][pl][k]),
                reinterpret_cast<const float2*>(&sm.lo[part][i][pl][k]), s_scale[i][pl]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int i = 0; i < kSlabs; ++i) {
      float a = acc[j][i];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
      const int g = p0 + warp + 8 * j;
      if (lane == 0 && g < p.ng) stat[(size_t)gx_row(ex, p.ng, nf, i, g) * gridDim.y + blockIdx.y] = a;
    }
}

// ---------------------------------------------------------------- half-sum factors
// kGxHalf and kGxHalfOcc (sch and ssx, gppKerSeq.cpp:96-139): least sums of
// squares per run; kGxRealOcc (gppKer_real.cpp:20-60): large factors per
// segment.
template <int kForm>
struct F64 {
  static constexpr bool kOcc = kForm != kGxHalf, kReal = kForm == kGxRealOcc;
  static constexpr int S = 7, kSlabs = Form<kForm>::kSlabs, kParts = Form<kForm>::kParts;
  static constexpr int kK = kForm == kGxHalfOcc ? 32 : 64;  // g-vectors per staged tile
  struct Planes {
    double v[kParts][kSlabs][kGxCols][kK + 1];
  };
};
// 1 / x for either sign.
__device__ __forceinline__ double rcp_signed(double x) {
  const double r = rcp_f64(fabs(x));
  return __hiloint2double(__double2hiint(r) | (__double2hiint(x) & 0x80000000), __double2loint(r));
}

// The factors of one element, FP64; in_freq: within the frequencies' range.
template <int kForm>
__device__ __forceinline__ void gx_f64_factors(const double (&wx)[kNW], const double (&iwx2)[kNW],
                                               const FF (&wxf)[kNW], double2 wt, double2 ie, bool in_freq,
                                               double2 (&y)[Form<kForm>::kSlabs]) {
  constexpr bool kOcc = F64<kForm>::kOcc;
  if (!kOcc) y[F64<kForm>::kSlabs - 1] = make_double2(-ie.x, -ie.y);
  if (!in_freq) return;
  const double a = wt.x, b = wt.y;
  if (F64<kForm>::kReal) {
    // kept: Omega2 / wx^2, second branch: -G / (2 (wx + wtilde)): 17 FP64
    // operations.  For |wtilde| in the usual range the guard is |c| > 1/2, c =
    // wx - wtilde: taken in FP32 from the exact halves, in FP64 within 2^-20
    // of its bounds (2.83 -> 2.24 ms at 1638 x 32768).
    const double g = __dmul_rn(ie.x, a), om = __dmul_rn(g, a);
    const FF as = ff_split_in_range(a);
    const float af = fabsf(as.hi);
    const bool plain = af < 240.f && af > 1.01e-3f;
#pragma unroll
    for (int iw = 0; iw < kNW; ++iw) {
      const float c = fabsf((wxf[iw].hi - as.hi) + (wxf[iw].lo - as.lo));
      bool keep = c > 0.5f, second = !keep;
      if (!plain || fabsf(c - 0.5f) < 9.5e-7f || !(c > 9.5e-7f)) {
        const unsigned mask = gx_decide(wx[iw], a, 0.0);
        keep = mask & 1u;
        second = mask & 2u;
      }
      const double r = rcp_signed(__dadd_rn(wx[iw], a));
      // -r / 2 (r normal: |wx + wtilde| is far from the overflow threshold here)
      const double h = __hiloint2double((__double2hiint(r) - 0x100000) ^ 0x80000000, __double2loint(r));
      const double v = __dmul_rn(keep ? om : g, keep ? iwx2[iw] : h);
      y[iw].x = keep || second ? v : 0.0;
    }
    return;
  }
  const double gx = fma(ie.x, a, -__dmul_rn(ie.y, b)), gy = fma(ie.x, b, __dmul_rn(ie.y, a));
  const double gbx = __dmul_rn(gx, b), gby = __dmul_rn(gy, b);
  const double b2 = guard_b2(b);
  // the guard's second condition binds only for |wtilde|^2 >= 62500
  const float af = fabsf(__double2float_rn(a)), bf = fabsf(__double2float_rn(b));
  const double thr = af < 170.f && bf < 170.f ? kLimitTwo : guard_thr(a, b2);
  const bool some = !kOcc || fmaxf(af, bf) > 1.1e-6f || fma(a, a, b2) > kTo1 * kTo1;
#pragma unroll
  for (int iw = 0; iw < kNW; ++iw) {
    const double c = __dsub_rn(wx[iw], a);
    const double wv = fma(c, c, b2);
    const double r = rcp_f64(wv);
    const double yx = __dmul_rn(fma(gx, c, -gby), r), yy = __dmul_rn(fma(gy, c, gbx), r);
    const bool low = gt_nonneg(thr, wv);
    if (low != kOcc) y[iw] = make_double2(yx, yy);
    if (kForm == kGxHalfOcc) {
      // kept: Omega2 / (wx^2 - wtilde^2) = sch wtilde / z, else -G / (2 z), z = wx + wtilde
      const double z = __dadd_rn(wx[iw], a), rz = rcp_f64(fma(z, z, b2));
      const double qx = low ? __dmul_rn(gx, -0.5) : fma(yx, a, -__dmul_rn(yy, b));
      const double qy = low ? __dmul_rn(gy, -0.5) : fma(yx, b, __dmul_rn(yy, a));
      const double sx = __dmul_rn(fma(qx, z, __dmul_rn(qy, b)), rz), sy = __dmul_rn(fma(qy, z, -__dmul_rn(qx, b)), rz);
      if (!low || some) y[(kNW + iw) % F64<kForm>::kSlabs] = make_double2(sx, sy);
    }
  }
}

template <int kForm>
__global__ void __launch_bounds__(kGxThreads, F64<kForm>::kK == 64 && !F64<kForm>::kReal ? 3 : 4)
    gx_f64_kernel(GxDev p, ExactPrep ex, float* stat, int nf, int run) {
  using H = F64<kForm>;
  constexpr int kSlabs = H::kSlabs, kK = H::kK;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  typename H::Planes& sm = *reinterpret_cast<typename H::Planes*>(smem_raw);
  __shared__ int s_e[kSlabs][kGxCols], s_lim[2][kGxCols], s_need;
  chain_begin();
  if (*ex.flag) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int p0 = blockIdx.x * kGxCols;
  const int rows_pad = ex.n_row_blocks * kExRows;
  const double wx[kNW] = {p.wx[0], p.wx[1], p.wx[2]};
  double iwx2[kNW];
#pragma unroll
  for (int iw = 0; iw < kNW; ++iw) iwx2[iw] = H::kReal ? rcp_f64(__dmul_rn(wx[iw], wx[iw])) : 0.0;
  FF wxf[kNW];
#pragma unroll
  for (int iw = 0; iw < kNW; ++iw) wxf[iw] = H::kReal ? ff_of_rn(wx[iw]) : FF{0.f, 0.f};
  if (tid == 0) s_need = 0;
  __syncthreads();
  if (tid < nf * kGxCols) {
    const int i = tid / kGxCols, pl = tid % kGxCols, g = p0 + pl, R = i * p.ng + g;
    s_e[i][pl] = g < p.ng ? ex.ea[R] : kExZeroRow;
    if (i < 2) s_lim[i][pl] = g < p.ng ? gx_limit<kForm>(p, g, i ? kSlabs - 1 : 0) : 0;
    if (R < rows_pad && (g < p.ng || i == nf - 1)) atomicMax(&s_need, ex.kt_lim[R / kExRows] * kExKTile);
  }
  __syncthreads();
  const int k_begin = blockIdx.y * run, k_end = min(s_need, k_begin + run);  // tiles the contraction reads
  float acc[2][kSlabs] = {};  // per column of this warp
  for (int k0 = k_begin; k0 < k_end; k0 += kK) {
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int pl = warp + 8 * j, g = p0 + pl;
#pragma unroll
      for (int h = 0; h < kK / 32; ++h) {
        const int k = h * 32 + lane, ig = k0 + k;
        float least = 0.f;  // of any band at this g-vector, relative to its largest
        if (Form<kForm>::kLeast && ig < s_lim[1][pl]) least = fminf(ex.band_min[ig], 1.f);
        double2 y[kSlabs];
#pragma unroll
        for (int i = 0; i < kSlabs; ++i) y[i] = make_double2(0.0, 0.0);
        if (ig < s_lim[1][pl]) {
          const double2 wt = gx_load<kForm>(p.wt, (size_t)g * p.nc + ig);
          const double2 ie = gx_load<kForm>(p.ieps, (size_t)g * p.nc + ig);
          if (H::kReal && ig + kK < s_lim[1][pl]) {
            const size_t next = (size_t)g * p.nc + ig + kK;
            prefetch_l2(p.wt + next);
            prefetch_l2(p.ieps + next);
          }
          const bool in_freq = ig < s_lim[0][pl] && (H::kOcc || ig % kIgBlk != kIgBlk - 1);
          gx_f64_factors<kForm>(wx, iwx2, wxf, wt, ie, in_freq, y);
        }
#pragma unroll
        for (int i = 0; i < kSlabs; ++i) {
          sm.v[0][i][pl][k] = y[i].x;
          if (!H::kReal) sm.v[H::kParts - 1][i][pl][k] = y[i].y;
          const int e = s_e[min(i, nf - 1)][pl];  // |e| < 64 unless flagged; a zero row is not checked
          if (!Form<kForm>::kLeast) {
            const int big = max(__double2hiint(y[i].x) & 0x7FFFFFFF, __double2hiint(y[i].y) & 0x7FFFFFFF);
            acc[j][i] += ig % kExSeg < kExCount && big >= (min(e, 1000) + 1022 - kExSlackA) << 20 ? 1.f : 0.f;
          } else {
            const float a = ex_rel_mag(y[i].x, y[i].y, e) * least;
            acc[j][i] = fmaf(a, a, acc[j][i]);
          }
        }
      }
    }
    __syncthreads();
    constexpr int kTiles = kK / kExKTile;
#pragma unroll 1
    for (int t = warp; t < nf * H::kParts * kTiles; t += kGxThreads / 32) {
      const int q = t % kTiles, part = t / kTiles % H::kParts, i = t / (kTiles * H::kParts);
      const int pl = lane & 15, ch = lane >> 4, g = p0 + pl, R = i * p.ng + g;
      const int tile = k0 / kExKTile + q;
      if ((g >= p.ng && i < nf - 1) || R >= rows_pad || tile >= ex.kt_lim[R / kExRows]) continue;
      unsigned char* dst =
          ex.a_tiles + ((size_t)(R / kExRows) * H::kParts * ex.kt + part * ex.kt + tile) * ex_a_bytes(H::S);
      ex_put<H::S>(dst, kExASlice, R % kExRows, ch, &sm.v[part][i][pl][q * kExKTile + ch * 8], s_e[i][pl]);
    }
  }
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int i = 0; i < kSlabs; ++i) {
      float a = acc[j][i];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
      const int g = p0 + warp + 8 * j;
      if (lane == 0 && i < nf && g < p.ng) stat[(size_t)(i * p.ng + g) * gridDim.y + blockIdx.y] = a;
    }
}

// One warp per row: the large factors that must coincide with large elements
// of every band (see exact_stats_kernel); half sum: the least sum of squares
// with any band (kHalfPower).
template <int kForm>
__global__ void gx_check_kernel(GxDev p, ExactPrep ex, const float* stat, int nf, int slabs, int per_seg) {
  chain_begin();
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (i >= slabs * p.ng) return;
  const int g = i % p.ng, row = gx_row(ex, p.ng, nf, i / p.ng, g);
  if (ex.ea[row] == kExZeroRow) return;
  // a segment's value: the sum of its runs'
  auto st = [&](int s) {
    const float* v = stat + ((size_t)row * ex.n_kseg + s) * per_seg;
    float sum = 0.f;
    for (int q = 0; q < per_seg; ++q) sum += v[q];
    return sum;
  };
  if (Form<kForm>::kLeast) {
    const int k = gx_limit<kForm>(p, g, Form<kForm>::kHalf ? i / p.ng : 0);
    float sum = 0.f;
    for (int s = lane; s * kExSeg < k; s += 32) sum += st(s);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0 && !(sum >= (float)k * kHalfPower)) ex_raise(ex);
  } else {
    int sum = 0;
    for (int s = lane; s * kExSeg < p.nc; s += 32)
      sum += max(0, (int)st(s) + min(ex.seg_min[s], kExCount) - min(kExCount, p.nc - s * kExSeg));
    sum = __reduce_add_sync(0xffffffffu, sum);
    if (lane == 0 && (long long)sum * kExOverlap < p.nc) ex_raise(ex);
  }
}

// Row limits of the half sum and the contraction's shape.
void gx_size(ExactPrep& ex, const GxShape& q, const std::vector<int>& igp_of, int sms, int& nf, int& nf2,
             std::vector<int>& kend, ExactTables* t) {
  const bool half = q.form == kGxHalf, half_occ = q.form == kGxHalfOcc;
  nf = half_occ ? 2 * kNW : half && q.with_static ? kNW + 1 : kNW;
  nf2 = q.form == kGxGpp && q.nvband > 0 ? kNW : 0;
  kend.clear();
  if (half || half_occ) {
    kend.resize((size_t)nf * q.ng);
    for (int f = 0; f < nf; ++f)
      for (int g = 0; g < q.ng; ++g)
        kend[(size_t)f * q.ng + g] = igp_of[g] < 0 ? 0 : std::max(igp_of[g] - (half && f < kNW ? 1 : 0), 0);
  }
  const bool real = q.form == kGxReal || q.form == kGxRealOcc;
  exact_size(ex, q.form == kGxGpp || q.form == kGxReal ? 6 : 7, half || half_occ ? 2 * q.nb : q.nb, q.nc, q.ng, nf, !real, sms,
             kend.empty() ? nullptr : kend.data(), t, nf2, nf2 ? q.nvband : 0);
}
// g-vectors per factor item: a segment, or less where the columns are too few
// to give every SM its four CTAs twice (409 x 8192: 64 or 512 ... at 128); at
// least one staged tile.
int gx_run(const ExactPrep& ex, int ng, int sms) {
  int run = kExSeg;
  while (run > (ex.slices == 6 ? kFfK : 64) && (long long)((ng + kGxCols - 1) / kGxCols) * ex.n_kseg * (kExSeg / run) < 8LL * sms) run /= 2;
  return run;
}
size_t gx_stat_bytes(const ExactPrep& ex, int run) {
  return sizeof(float) * (size_t)ex.n_row_blocks * kExRows * ex.n_kseg * (kExSeg / run);
}

template <int kForm, bool kOcc>
cudaError_t launch_ff(const GppExact& g, const GxDev& p, dim3 grid, cudaStream_t s) {
  constexpr int smem = sizeof(FfPlanes<kForm, kOcc>);
  cudaError_t e =
      cudaFuncSetAttribute(gx_ff_kernel<kForm, kOcc>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  return launch_chained(gx_ff_kernel<kForm, kOcc>, grid, kGxThreads, smem, s, true, p, g.ex, g.stat, g.nf, g.run);
}

template <int kForm>
cudaError_t launch_operands(const GppExact& g, const GxDev& p, cudaStream_t s, bool begin) {
  using F = Form<kForm>;
  const ExactPrep& ex = g.ex;
  cudaError_t e = begin ? exact_begin_flag(ex, s) : cudaSuccess;
  if (e != cudaSuccess) return e;
  e = launch_chained(gx_max_kernel<kForm>, p.ng, kGxThreads, 0, s, true, p, ex, g.nf, g.nf2);
  if (e != cudaSuccess) return e;
  const int nb = F::kHalfOcc || F::kRealOcc ? p.nvband : p.nb;
  e = launch_exact_b(ex, p.aqsn, nb, p.aqsm, F::kHalf || F::kHalfOcc ? nb : 0, p.nc, s);
  if (e != cudaSuccess) return e;
  const int slabs = g.nf + g.nf2;
  const int pad = std::max(ex.n_main_blocks * kExRows - g.nf * p.ng,
                           (ex.n_row_blocks - ex.n_main_blocks) * kExRows - g.nf2 * p.ng);
  const dim3 grid((p.ng + pad + kGxCols - 1) / kGxCols, ex.n_kseg * (kExSeg / g.run));
  if constexpr (F::kF64) {
    constexpr int smem = sizeof(typename F64<kForm>::Planes);
    e = cudaFuncSetAttribute(gx_f64_kernel<kForm>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    e = launch_chained(gx_f64_kernel<kForm>, grid, kGxThreads, smem, s, true, p, ex, g.stat, g.nf, g.run);
  } else if (kForm == kGxGpp && g.nf2) {
    e = launch_ff<kGxGpp, true>(g, p, grid, s);
  } else {
    e = launch_ff<kForm, false>(g, p, grid, s);
  }
  if (e != cudaSuccess) return e;
  return launch_chained(gx_check_kernel<kForm>, (slabs * p.ng * 32 + 255) / 256, 256, 0, s, true, p, ex, g.stat, g.nf,
                        slabs, kExSeg / g.run);
}

}  // namespace

// From these products on (3 x columns x bands x g-vectors) the contraction beats
// the float-float passes, whose time stays flat below (one CTA's latency):
// measured us, contraction against passes, at 8 x 12 x 256 (74 k) 58 / 158 with
// occupied bands and 50 / 66 without, real 16 x 20 x 512 (0.5 M) 105 / 138 and
// 52 / 56; the half sum's two contractions 221 / 187 at 24 x 40 x 1024 (2.9 M),
// 230 / 229 at 60 x 60 x 1024 (11 M), 315 / 372 at 60 x 60 x 2048.
bool gpp_exact_pays(const GxShape& q) {
  const double products = (double)kNW * q.ng * q.nb * q.nc;
  switch (q.form) {
    case kGxReal: return products >= 1 << 18;
    case kGxHalf: return products >= 1 << 23;
    default: return products >= 1 << 16;
  }
}

bool gpp_exact_fits(const GxShape& q) {
  return gpp_exact_pays(q) && exact_holds(q.nc, q.form != kGxReal && q.form != kGxRealOcc);
}

size_t gpp_exact_work_bytes(const GxShape& q, const std::vector<int>& igp_of, int sms, size_t* own) {
  ExactPrep ex{};
  std::vector<int> kend;
  int nf, nf2;
  gx_size(ex, q, igp_of, sms, nf, nf2, kend, nullptr);
  if (own) *own = exact_own_bytes(ex);
  return exact_work_bytes(ex) + gx_stat_bytes(ex, gx_run(ex, q.ng, sms));
}

namespace {

// Sizes g; returns its tables.
ExactTables gx_plan(GppExact& g, const GxShape& q, const std::vector<int>& igp_of, int sms) {
  g = GppExact();
  ExactTables t;
  std::vector<int> kend;
  gx_size(g.ex, q, igp_of, sms, g.nf, g.nf2, kend, &t);
  g.run = gx_run(g.ex, q.ng, sms);
  g.form = q.form;
  g.grid = sms;
  return t;
}
void gx_bind(GppExact& g, void* work, void* own) {
  exact_bind(g.ex, work, own);
  g.stat = reinterpret_cast<float*>(static_cast<char*>(work) + exact_work_bytes(g.ex));
}

}  // namespace

bool gpp_exact_create(GppExact& g, const GxShape& q, const std::vector<int>& igp_of, int sms, int arena_slot) {
  const ExactTables t = gx_plan(g, q, igp_of, sms);
  const size_t work = (exact_work_bytes(g.ex) + gx_stat_bytes(g.ex, g.run) + 255) / 256 * 256;
  const size_t all = work + exact_own_bytes(g.ex);
  void* block = arena_slot >= 0 ? arena_optional(arena_slot, all) : nullptr;
  if (!block) {
    if (!room_for_optional(all) || cudaMalloc(&g.block, all) != cudaSuccess) {
      cudaGetLastError();
      g = GppExact();
      return false;
    }
    block = g.block;
  }
  gx_bind(g, block, static_cast<char*>(block) + work);
  if (exact_upload_tables(g.ex, t) != cudaSuccess) {
    cudaGetLastError();
    gpp_exact_destroy(g);
    return false;
  }
  g.ready = true;
  return true;
}

void gpp_exact_create(GppExact& g, const GxShape& q, const std::vector<int>& igp_of, int sms, const GxShared& m) {
  const ExactTables t = gx_plan(g, q, igp_of, sms);
  gx_bind(g, m.work, m.own);
  exact_pack_own(g.ex, t, m.own_host);
  g.ready = true;
}

void gpp_exact_destroy(GppExact& g) {
  if (g.block) cudaFree(g.block);
  g = GppExact();
}

cudaError_t launch_gpp_exact_operands(const GppExact& g, const GxDev& p, cudaStream_t s, bool begin) {
  switch (g.form) {
    case kGxReal: return launch_operands<kGxReal>(g, p, s, begin);
    case kGxRealOcc: return launch_operands<kGxRealOcc>(g, p, s, begin);
    case kGxHalf: return launch_operands<kGxHalf>(g, p, s, begin);
    case kGxHalfOcc: return launch_operands<kGxHalfOcc>(g, p, s, begin);
    default: return launch_operands<kGxGpp>(g, p, s, begin);
  }
}

cudaError_t launch_gpp_exact_sums(const GppExact& g, const GxDev& p, int* status, double2* out, double2* occ_out,
                                  cudaStream_t s) {
  cudaError_t e = launch_exact_gemm(g.ex, g.grid, status, s);
  if (e != cudaSuccess) return e;
  const int nb = g.form == kGxHalfOcc || g.form == kGxRealOcc ? p.nvband : p.nb;
  const bool pair = g.form == kGxHalf || g.form == kGxHalfOcc;
  FfDev d{};
  d.nb = pair ? 2 * nb : nb;
  d.nc = p.nc;
  d.ng = p.ng;
  d.nf = g.nf;
  d.aqsm = reinterpret_cast<const double2*>(p.aqsm);
  d.aqsn = reinterpret_cast<const double2*>(p.aqsn);
  d.igp_of = p.igp_of;
  d.vcoul = p.vcoul;
  d.vfac = g.form == kGxRealOcc ? p.occ : 0.5;
  d.pair_bands = pair ? nb : 0;
  d.pair_static = g.form == kGxHalf && g.nf > kNW;
  return launch_exact_finish(d, g.ex, out, nullptr, s,
                             ExSecond{p.nvband, g.nf2, p.occ, g.nf2 ? occ_out : nullptr});
}

}  // namespace sigma
