// Operand passes of the exact GPP contractions (gpp_exact.cuh).
//
// Y[iw][g][ig] = G (c + i b) / (c^2 + b^2), G = I_eps wtilde, c = wx - Re
// wtilde, b = Im wtilde, 0 where the pole guard drops the term
// (BGW-Kernels/gppKer.cpp:394-404, conj(aqsm) and vcoul moved to the
// epilogue); the half sum keeps the terms the guard drops
// (gppKerSeq.cpp:206-242).  Row iw * ng + g of the contraction is one
// frequency of one column.
//
// gx_max_kernel bounds |Y| per row (the digits' exponent) from FP32 factors,
// one pass over the inputs at memory speed.
// gx_factor_kernel forms Y in FP64 (34 FP64 operations per column and
// g-vector for the three frequencies, bound by the FP64 pipe's 2 per clock per
// SM; the digits run on the integer pipe beside them), stages 16 columns x 64
// g-vectors in shared memory and writes each row's digits as 16-byte chunks.
#include <algorithm>

#include "gpp_exact.cuh"
#include "floatfloat.cuh"

namespace sigma {
namespace {

constexpr int kGxThreads = 256;
constexpr int kGxCols = 16;  // columns per CTA
constexpr int kGxK = 64;     // g-vectors per staged tile
constexpr int kGxPad = 1;    // conflict-free planes: lanes run along g-vectors, then along columns
constexpr int kIgBlk = 512;  // g-vector block of the half sum's reference loop
// Half sum: poles inside the guard make a few factors of a row much larger
// than the rest, so a count of large ones says little, and the row's exponent
// serves the rest badly: its operands take seven digits.  Its check compares
// the sum of squares that each row and the least band share per segment with
// K: at 2^-30 the estimated error is 2^-48 of the sum's root mean square
// (taking elements within a segment as unrelated), below the float-float
// terms', whose factors come from a 2^-45 reciprocal.
constexpr float kHalfPower = 1.f / 1073741824.f;

template <int kForm>
struct Form {
  static constexpr bool kReal = kForm == kGxReal, kHalf = kForm == kGxHalf;
  static constexpr int kSlabs = kHalf ? 4 : kNW, kParts = kReal ? 1 : 2;
  static constexpr int kSlices = kHalf ? 7 : 6;
};
template <int kForm>
struct FactorPlanes {
  double v[Form<kForm>::kParts][Form<kForm>::kSlabs][kGxCols][kGxK + kGxPad];
};

template <int kForm>
__device__ __forceinline__ double2 gx_load(const double* a, size_t off) {
  if (Form<kForm>::kReal) return make_double2(a[off], 0.0);
  return reinterpret_cast<const double2*>(a)[off];
}
// End of a slab's g-vectors in column igp.
template <int kForm>
__device__ __forceinline__ int gx_limit(int igp, int slab, int nc) {
  if (!Form<kForm>::kHalf) return nc;
  return igp < 0 ? 0 : (slab < kNW ? max(igp - 1, 0) : igp);
}

// One CTA per column: exponents of its rows.  |Y| from FP32 values (c from
// exact FP32 halves), the guard taken somewhat wide, with a 2^-8 margin;
// what FP32 cannot bound raises the flag.
template <int kForm>
__global__ void __launch_bounds__(kGxThreads) gx_max_kernel(GxDev p, ExactPrep ex, int nf) {
  using F = Form<kForm>;
  __shared__ unsigned s_m[F::kSlabs][kGxThreads / 32];
  const int g = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int igp = p.igp_of[g];
  FF wx[kNW];
#pragma unroll
  for (int iw = 0; iw < kNW; ++iw) wx[iw] = ff_of(p.wx[iw]);
  unsigned m[F::kSlabs];  // bits of non-negative floats; NaN is the largest
#pragma unroll
  for (int i = 0; i < F::kSlabs; ++i) m[i] = 0u;
  bool bad = false;
  const int k_end = gx_limit<kForm>(igp, F::kSlabs - 1, p.nc), k_freq = gx_limit<kForm>(igp, 0, p.nc);
#pragma unroll 4
  for (int k = tid; k < k_end; k += kGxThreads) {
    const double2 w = gx_load<kForm>(p.wt, (size_t)g * p.nc + k), e = gx_load<kForm>(p.ieps, (size_t)g * p.nc + k);
    const FF a = ff_of(w.x);
    const float b = __double2float_rn(w.y), er = __double2float_rn(e.x), ei = __double2float_rn(e.y);
    if (F::kHalf) {
      m[F::kSlabs - 1] = max(m[F::kSlabs - 1], __float_as_uint(fmaxf(fabsf(er), fabsf(ei))));
      if (er != er || ei != ei) m[F::kSlabs - 1] = 0x7F800000u;
      if (k >= k_freq || k % kIgBlk == kIgBlk - 1) continue;
    }
    const float gx = er * a.hi - ei * b, gy = er * b + ei * a.hi;
    const float lim = F::kHalf ? fmaxf(0.2501f, fmaf(a.hi, a.hi, b * b) * 4.001e-6f) : 0.f;
    const bool any = (e.x != 0.0 || e.y != 0.0) && (w.x != 0.0 || w.y != 0.0);
#pragma unroll
    for (int iw = 0; iw < kNW; ++iw) {
      const float c = (wx[iw].hi - a.hi) + (wx[iw].lo - a.lo);
      const float w2 = fmaf(c, c, b * b);
      if (F::kHalf ? !(w2 > lim) : !(w2 <= 0.2499f)) {  // also NaN
        const float r = __frcp_rn(w2);
        const float y = fmaxf(fabsf(gx * c - gy * b), fabsf(gy * c + gx * b)) * r;
        m[iw] = max(m[iw], __float_as_uint(y != y ? INFINITY : y));
        if (w2 > 1e30f) m[iw] = 0x7F800000u;  // the FP32 reciprocal may be 0: flagged below
        bad = bad || (any && !(y > 1e-18f));
      }
    }
  }
  bad = __syncthreads_or(bad);
#pragma unroll
  for (int i = 0; i < F::kSlabs; ++i) {
    const unsigned v = __reduce_max_sync(0xffffffffu, m[i]);
    if (lane == 0) s_m[i][warp] = v;
  }
  __syncthreads();
  if (tid < nf) {
    unsigned v = 0;
    for (int q = 0; q < kGxThreads / 32; ++q) v = max(v, s_m[tid][q]);
    const float f = __uint_as_float(v) * (1.f + 1.f / 256.f);
    // a factor too small for FP32 may only be ignored beside large ones
    if (!(f < 1e18f) || (bad && !(f > 1e-6f)) || (v && f < 1e-18f)) ex_raise(ex);
    ex.ea[tid * p.ng + g] = v ? (int)(__float_as_uint(f) >> 23) - 126 : kExZeroRow;
  }
}

// Items (column block, 512-g-vector segment).  Column blocks run past ng to
// cover the padding rows of the last row block (zero digits).
template <int kForm>
__global__ void __launch_bounds__(kGxThreads, Form<kForm>::kHalf ? 3 : 4)
    gx_factor_kernel(GxDev p, ExactPrep ex, float* stat, int nf) {
  using F = Form<kForm>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  FactorPlanes<kForm>& sm = *reinterpret_cast<FactorPlanes<kForm>*>(smem_raw);
  __shared__ int s_e[F::kSlabs][kGxCols], s_igp[kGxCols];
  if (*ex.flag) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int p0 = blockIdx.x * kGxCols, seg = blockIdx.y;
  const int rows_pad = ex.n_row_blocks * kExRows;
  const double wx[kNW] = {p.wx[0], p.wx[1], p.wx[2]};
  // K tiles of the item's rows that the contraction reads
  int need = 0;
  if (tid < nf * kGxCols) {
    const int iw = tid / kGxCols, g = p0 + tid % kGxCols, R = iw * p.ng + g;
    s_e[iw][tid % kGxCols] = g < p.ng ? ex.ea[R] : kExZeroRow;
    if (iw == 0) s_igp[tid % kGxCols] = g < p.ng ? p.igp_of[g] : -1;
    if (R < rows_pad && (g < p.ng || iw == nf - 1)) need = ex.kt_lim[R / kExRows] * kExKTile;
  }
  const int k_begin = seg * kExSeg;
  int k_end = min(ex.kt * kExKTile, k_begin + kExSeg);
  if (F::kHalf) {
    __shared__ int s_need;
    if (tid == 0) s_need = 0;
    __syncthreads();
    if (need) atomicMax(&s_need, need);
    __syncthreads();
    k_end = min(k_end, s_need);
  }
  float acc[2][F::kSlabs];  // large factors, or sums of squares, per column of this warp
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int i = 0; i < F::kSlabs; ++i) acc[j][i] = 0.f;
  for (int k0 = k_begin; k0 < k_end; k0 += kGxK) {
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int pl = warp + 8 * j, g = p0 + pl;
#pragma unroll
      for (int h = 0; h < kGxK / 32; ++h) {
        const int k = h * 32 + lane, ig = k0 + k;
        double2 y[F::kSlabs];
#pragma unroll
        for (int i = 0; i < F::kSlabs; ++i) y[i] = make_double2(0.0, 0.0);
        const int igp = F::kHalf ? s_igp[pl] : 0;
        if (g < p.ng && ig < gx_limit<kForm>(igp, F::kSlabs - 1, p.nc)) {
          const double2 wt = gx_load<kForm>(p.wt, (size_t)g * p.nc + ig);
          const double2 ie = gx_load<kForm>(p.ieps, (size_t)g * p.nc + ig);
          if (F::kHalf) y[F::kSlabs - 1] = make_double2(-ie.x, -ie.y);
          // the guard's second condition binds only for |wtilde|^2 >= 62500
          const bool plain =
              fabsf(__double2float_rn(wt.x)) < 170.f && fabsf(__double2float_rn(wt.y)) < 170.f;
          if (F::kReal) {
            const double gr = __dmul_rn(ie.x, wt.x);
            const double thr = plain ? kLimitTwo : guard_thr(wt.x, 0.0);
#pragma unroll
            for (int iw = 0; iw < kNW; ++iw) {
              const double c = __dsub_rn(wx[iw], wt.x);
              const double wv = __dmul_rn(c, c);
              const double v = __dmul_rn(gr, __dmul_rn(c, rcp_f64(wv)));
              y[iw].x = keep_nonneg(wv, thr) ? v : 0.0;
            }
          } else if (!F::kHalf || (ig < gx_limit<kForm>(igp, 0, p.nc) && ig % kIgBlk != kIgBlk - 1)) {
            const double gx = fma(ie.x, wt.x, -__dmul_rn(ie.y, wt.y)), gy = fma(ie.x, wt.y, __dmul_rn(ie.y, wt.x));
            const double gbx = __dmul_rn(gx, wt.y), gby = __dmul_rn(gy, wt.y);
            const double b2 = guard_b2(wt.y);
            const double thr = plain ? kLimitTwo : guard_thr(wt.x, b2);
#pragma unroll
            for (int iw = 0; iw < kNW; ++iw) {
              const double c = __dsub_rn(wx[iw], wt.x);
              const double wv = fma(c, c, b2);
              const double r = rcp_f64(wv);
              const double yx = __dmul_rn(fma(gx, c, -gby), r), yy = __dmul_rn(fma(gy, c, gbx), r);
              const bool keep = F::kHalf ? gt_nonneg(thr, wv) : keep_nonneg(wv, thr);
              y[iw] = make_double2(keep ? yx : 0.0, keep ? yy : 0.0);
            }
          }
        }
#pragma unroll
        for (int i = 0; i < F::kSlabs; ++i) {
          sm.v[0][i][pl][k] = y[i].x;
          if (!F::kReal) sm.v[F::kParts - 1][i][pl][k] = y[i].y;
          const int e = min(s_e[min(i, nf - 1)][pl], 1000);
          if (F::kHalf) {
            const float u = __uint_as_float((unsigned)(127 - e) << 23);  // 2^-e, |e| < 61 unless flagged
            const float a = __double2float_rn(y[i].x) * u, b = __double2float_rn(y[i].y) * u;
            acc[j][i] = fmaf(a, a, fmaf(b, b, acc[j][i]));
          } else {
            const int big = max(__double2hiint(y[i].x) & 0x7FFFFFFF, __double2hiint(y[i].y) & 0x7FFFFFFF);
            acc[j][i] += big >= (e + 1022 - kExSlackA) << 20 ? 1.f : 0.f;
          }
        }
      }
    }
    __syncthreads();
    // digits: a warp takes one (slab, part, K tile), its lanes the 16
    // columns x 2 chunks (512 contiguous bytes per slice)
    constexpr int kTiles = kGxK / kExKTile;
#pragma unroll 1
    for (int t = warp; t < nf * F::kParts * kTiles; t += kGxThreads / 32) {
      const int q = t % kTiles, part = t / kTiles % F::kParts, iw = t / (kTiles * F::kParts);
      const int pl = lane & 15, ch = lane >> 4, g = p0 + pl, R = iw * p.ng + g;
      const int tile = k0 / kExKTile + q;
      // padding rows follow the last slab's columns
      if ((g >= p.ng && iw < nf - 1) || R >= rows_pad || tile >= ex.kt_lim[R / kExRows]) continue;
      unsigned char* dst =
          ex.a_tiles + ((size_t)(R / kExRows) * F::kParts * ex.kt + part * ex.kt + tile) * ex_a_bytes(F::kSlices);
      ex_put<F::kSlices>(dst, kExASlice, R % kExRows, ch, &sm.v[part][iw][pl][q * kExKTile + ch * 8], s_e[iw][pl]);
    }
  }
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int i = 0; i < F::kSlabs; ++i) {
      float a = acc[j][i];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
      const int g = p0 + warp + 8 * j;
      if (lane == 0 && i < nf && g < p.ng) stat[(size_t)(i * p.ng + g) * ex.n_kseg + seg] = a;
    }
}

// One warp per row: the large factors that must coincide with large elements
// of every band (see exact_stats_kernel); half sum: the power shared with the
// least band (kHalfPower).
template <int kForm>
__global__ void gx_check_kernel(ExactPrep ex, const float* stat, const int* kend, int rows, int nc) {
  const int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (row >= rows || ex.ea[row] == kExZeroRow) return;
  const float* st = stat + (size_t)row * ex.n_kseg;
  if (Form<kForm>::kHalf) {
    const int k = kend[row];
    float sum = 0.f;
    for (int s = lane; s * kExSeg < k; s += 32)
      sum += st[s] * fminf(__int_as_float(ex.seg_pow[s]), (float)kExSeg) / (float)min(kExSeg, nc - s * kExSeg);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0 && !(sum >= (float)k * kHalfPower)) ex_raise(ex);
  } else {
    int sum = 0;
    for (int s = lane; s < ex.n_kseg; s += 32)
      sum += max(0, (int)st[s] + min(ex.seg_min[s], kExSeg) - min(kExSeg, nc - s * kExSeg));
    sum = __reduce_add_sync(0xffffffffu, sum);
    if (lane == 0 && (long long)sum * kExOverlap < nc) ex_raise(ex);
  }
}

// Row limits of the half sum and the contraction's shape.
void gx_size(ExactPrep& ex, GxForm form, int nb, int nc, int ng, int nf, const std::vector<int>& igp_of, int sms,
             std::vector<int>& kend, ExactTables* t) {
  kend.clear();
  if (form == kGxHalf) {
    kend.resize((size_t)nf * ng);
    for (int f = 0; f < nf; ++f)
      for (int g = 0; g < ng; ++g)
        kend[(size_t)f * ng + g] = igp_of[g] < 0 ? 0 : std::max(igp_of[g] - (f < kNW ? 1 : 0), 0);
  }
  exact_size(ex, form == kGxHalf ? 7 : 6, form == kGxHalf ? 2 * nb : nb, nc, ng, nf, form != kGxReal, sms,
             form == kGxHalf ? kend.data() : nullptr, t);
}
size_t gx_stat_bytes(const ExactPrep& ex, int ng, int nf) { return sizeof(float) * (size_t)nf * ng * ex.n_kseg; }

template <int kForm>
cudaError_t launch_operands(const GppExact& g, const GxDev& p, cudaStream_t s) {
  const ExactPrep& ex = g.ex;
  cudaError_t e = exact_begin(ex, s);
  if (e != cudaSuccess) return e;
  e = launch_exact_b(ex, p.aqsn, p.nb, p.aqsm, Form<kForm>::kHalf ? p.nb : 0, p.nc, s);
  if (e != cudaSuccess) return e;
  gx_max_kernel<kForm><<<p.ng, kGxThreads, 0, s>>>(p, ex, g.nf);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  constexpr int smem = sizeof(FactorPlanes<kForm>);
  e = cudaFuncSetAttribute(gx_factor_kernel<kForm>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  const int cols = p.ng + ex.n_row_blocks * kExRows - g.nf * p.ng;
  gx_factor_kernel<kForm>
      <<<dim3((cols + kGxCols - 1) / kGxCols, ex.n_kseg), kGxThreads, smem, s>>>(p, ex, g.stat, g.nf);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  const int rows = g.nf * p.ng;
  gx_check_kernel<kForm><<<(rows * 32 + 255) / 256, 256, 0, s>>>(ex, g.stat, g.kend, rows, p.nc);
  return cudaGetLastError();
}

}  // namespace

size_t gpp_exact_work_bytes(GxForm form, int nb, int nc, int ng, int nf, const std::vector<int>& igp_of, int sms) {
  ExactPrep ex{};
  std::vector<int> kend;
  gx_size(ex, form, nb, nc, ng, nf, igp_of, sms, kend, nullptr);
  return exact_work_bytes(ex) + gx_stat_bytes(ex, ng, nf);
}

bool gpp_exact_create(GppExact& g, GxForm form, int nb, int nc, int ng, int nf, const std::vector<int>& igp_of,
                      int sms, void* shared_work) {
  g = GppExact();
  if ((double)nf * ng * nb * nc < kExactMin) return false;
  ExactTables t;
  std::vector<int> kend;
  gx_size(g.ex, form, nb, nc, ng, nf, igp_of, sms, kend, &t);
  const size_t work = exact_work_bytes(g.ex), own = exact_own_bytes(g.ex);
  if (cudaMalloc(&g.own, own + sizeof(int) * kend.size()) != cudaSuccess) g.own = nullptr;
  if (g.own && !shared_work && cudaMalloc(&g.work, work + gx_stat_bytes(g.ex, ng, nf)) != cudaSuccess) {
    cudaFree(g.own);
    g.own = g.work = nullptr;
  }
  if (!g.own) {
    cudaGetLastError();
    g = GppExact();
    return false;
  }
  void* w = shared_work ? shared_work : g.work;
  exact_bind(g.ex, w, g.own);
  g.form = form;
  g.nf = nf;
  g.stat = reinterpret_cast<float*>(static_cast<char*>(w) + work);
  g.grid = sms;
  cudaError_t e = exact_upload_tables(g.ex, t);
  if (e == cudaSuccess && !kend.empty()) {
    g.kend = reinterpret_cast<int*>(static_cast<char*>(g.own) + own);
    e = cudaMemcpy(g.kend, kend.data(), sizeof(int) * kend.size(), cudaMemcpyHostToDevice);
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    gpp_exact_destroy(g);
    return false;
  }
  return true;
}

void gpp_exact_destroy(GppExact& g) {
  if (g.own) cudaFree(g.own);
  if (g.work) cudaFree(g.work);
  g = GppExact();
}

cudaError_t launch_gpp_exact_operands(const GppExact& g, const GxDev& p, cudaStream_t s) {
  if (g.form == kGxHalf) return launch_operands<kGxHalf>(g, p, s);
  if (g.form == kGxReal) return launch_operands<kGxReal>(g, p, s);
  return launch_operands<kGxGpp>(g, p, s);
}

cudaError_t launch_gpp_exact_sums(const GppExact& g, const GxDev& p, int* status, double2* out, cudaStream_t s) {
  cudaError_t e = launch_exact_gemm(g.ex, g.grid, status, s);
  if (e != cudaSuccess) return e;
  FfDev d{};
  d.nb = g.form == kGxHalf ? 2 * p.nb : p.nb;
  d.nc = p.nc;
  d.ng = p.ng;
  d.nf = g.nf;
  d.aqsm = reinterpret_cast<const double2*>(p.aqsm);
  d.aqsn = reinterpret_cast<const double2*>(p.aqsn);
  d.igp_of = p.igp_of;
  d.vcoul = p.vcoul;
  d.vfac = 0.5;
  d.pair_bands = g.form == kGxHalf ? p.nb : 0;
  d.pair_static = g.nf > kNW;
  return launch_exact_finish(d, g.ex, out, nullptr, s);
}

}  // namespace sigma
