// Operand passes of the exact GPP contraction (gpp_exact.cuh).
//
// Y[iw][g][ig] = G (c + i b) / (c^2 + b^2), G = I_eps wtilde, c = wx - Re
// wtilde, b = Im wtilde, 0 where the pole guard drops the term
// (BGW-Kernels/gppKer.cpp:394-404, conj(aqsm) and vcoul moved to the
// epilogue).  Row iw * ng + g of the contraction is one frequency of one
// column.
//
// gpp_exact_max_kernel bounds |Y| per row (the digits' exponent) from FP32
// factors, one pass over the inputs at memory speed.
// gpp_exact_factor_kernel forms Y in FP64 (34 FP64 operations per column and
// g-vector for the three frequencies, bound by the FP64 pipe's 2 per clock per
// SM; the digits run on the integer pipe beside them), stages 16 columns x 64
// g-vectors in shared memory and writes each row's digits as 16-byte chunks.
#include <algorithm>
#include <vector>

#include "gpp_exact.cuh"
#include "floatfloat.cuh"

namespace sigma {
namespace {

constexpr int kGxThreads = 256;
constexpr int kGxCols = 16;  // columns per CTA
constexpr int kGxK = 64;     // g-vectors per staged tile
constexpr int kGxPad = 1;    // conflict-free planes: lanes run along g-vectors, then along columns

struct FactorPlanes {
  double r[kNW][kGxCols][kGxK + kGxPad], i[kNW][kGxCols][kGxK + kGxPad];
};

// One CTA per column: exponents of its three rows.  |Y| from FP32 values (c
// from exact FP32 halves), kept somewhat below the guard's threshold, with a
// 2^-8 margin; what FP32 cannot bound raises the flag.
__global__ void __launch_bounds__(kGxThreads) gpp_exact_max_kernel(GppDev p, ExactPrep ex) {
  __shared__ unsigned s_m[kNW][kGxThreads / 32];
  const int g = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  FF wx[kNW];
#pragma unroll
  for (int iw = 0; iw < kNW; ++iw) wx[iw] = ff_of(p.wx[iw]);
  const double2* wt = p.wt + (size_t)g * p.nc;
  const double2* ie = p.ieps + (size_t)g * p.nc;
  unsigned m[kNW] = {0u, 0u, 0u};  // bits of non-negative floats; NaN is the largest
  bool bad = false;
#pragma unroll 4
  for (int k = tid; k < p.nc; k += kGxThreads) {
    const double2 w = wt[k], e = ie[k];
    const FF a = ff_of(w.x);
    const float b = __double2float_rn(w.y), er = __double2float_rn(e.x), ei = __double2float_rn(e.y);
    const float gx = er * a.hi - ei * b, gy = er * b + ei * a.hi;
    const bool any = (e.x != 0.0 || e.y != 0.0) && (w.x != 0.0 || w.y != 0.0);
#pragma unroll
    for (int iw = 0; iw < kNW; ++iw) {
      const float c = (wx[iw].hi - a.hi) + (wx[iw].lo - a.lo);
      const float w2 = fmaf(c, c, b * b);
      if (!(w2 <= 0.2499f)) {  // also NaN
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
  for (int iw = 0; iw < kNW; ++iw) {
    const unsigned v = __reduce_max_sync(0xffffffffu, m[iw]);
    if (lane == 0) s_m[iw][warp] = v;
  }
  __syncthreads();
  if (tid < kNW) {
    unsigned v = 0;
    for (int q = 0; q < kGxThreads / 32; ++q) v = max(v, s_m[tid][q]);
    const float f = __uint_as_float(v) * (1.f + 1.f / 256.f);
    // a factor too small for FP32 may only be ignored beside large ones
    if (!(f < 1e18f) || (bad && !(f > 1e-6f))) *ex.flag = 1;
    ex.ea[tid * p.ng + g] = v ? (int)(__float_as_uint(f) >> 23) - 126 : kExZeroRow;
  }
}

// Items (column block, 512-g-vector segment).  Column blocks run past ng to
// cover the padding rows of the last row block (zero digits).
__global__ void __launch_bounds__(kGxThreads, 4) gpp_exact_factor_kernel(GppDev p, ExactPrep ex, int* counts) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  FactorPlanes& sm = *reinterpret_cast<FactorPlanes*>(smem_raw);
  __shared__ int s_e[kNW][kGxCols];
  if (*ex.flag) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int p0 = blockIdx.x * kGxCols, seg = blockIdx.y;
  const int rows_pad = ex.n_row_blocks * kExRows;
  const double wx[kNW] = {p.wx[0], p.wx[1], p.wx[2]};
  if (tid < kNW * kGxCols) {
    const int iw = tid / kGxCols, g = p0 + tid % kGxCols;
    s_e[iw][tid % kGxCols] = g < p.ng ? ex.ea[iw * p.ng + g] : kExZeroRow;
  }
  const int k_begin = seg * kExSeg, k_end = min(ex.kt * kExKTile, k_begin + kExSeg);
  int cnt[2][kNW] = {{0, 0, 0}, {0, 0, 0}};
  for (int k0 = k_begin; k0 < k_end; k0 += kGxK) {
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int pl = warp + 8 * j, g = p0 + pl;
#pragma unroll
      for (int h = 0; h < kGxK / 32; ++h) {
        const int k = h * 32 + lane, ig = k0 + k;
        double2 y[kNW] = {make_double2(0.0, 0.0), make_double2(0.0, 0.0), make_double2(0.0, 0.0)};
        if (g < p.ng && ig < p.nc) {
          const double2 wt = p.wt[(size_t)g * p.nc + ig], ie = p.ieps[(size_t)g * p.nc + ig];
          const double gx = fma(ie.x, wt.x, -__dmul_rn(ie.y, wt.y)), gy = fma(ie.x, wt.y, __dmul_rn(ie.y, wt.x));
          const double gbx = __dmul_rn(gx, wt.y), gby = __dmul_rn(gy, wt.y);
          const double b2 = guard_b2(wt.y);
          // the guard's second condition binds only for |wtilde|^2 >= 62500
          double thr = kLimitTwo;
          if (!(fabsf(__double2float_rn(wt.x)) < 170.f && fabsf(__double2float_rn(wt.y)) < 170.f))
            thr = guard_thr(wt.x, b2);
#pragma unroll
          for (int iw = 0; iw < kNW; ++iw) {
            const double c = __dsub_rn(wx[iw], wt.x);
            const double wv = fma(c, c, b2);
            const double r = rcp_f64(wv);
            const double yx = __dmul_rn(fma(gx, c, -gby), r), yy = __dmul_rn(fma(gy, c, gbx), r);
            const bool keep = keep_nonneg(wv, thr);
            y[iw] = make_double2(keep ? yx : 0.0, keep ? yy : 0.0);
          }
        }
#pragma unroll
        for (int iw = 0; iw < kNW; ++iw) {
          sm.r[iw][pl][k] = y[iw].x;
          sm.i[iw][pl][k] = y[iw].y;
          const int thr = (min(s_e[iw][pl], 1000) + 1022 - kExSlackA) << 20;
          const int big = max(__double2hiint(y[iw].x) & 0x7FFFFFFF, __double2hiint(y[iw].y) & 0x7FFFFFFF);
          cnt[j][iw] += __popc(__ballot_sync(0xffffffffu, big >= thr));
        }
      }
    }
    __syncthreads();
    // digits: a warp takes one (frequency, part, K tile), its lanes the 16
    // columns x 2 chunks (512 contiguous bytes per slice)
#pragma unroll 1
    for (int t = warp; t < kNW * 2 * (kGxK / kExKTile); t += kGxThreads / 32) {
      const int q = t % (kGxK / kExKTile), part = t / (kGxK / kExKTile) % 2, iw = t / (2 * (kGxK / kExKTile));
      const int pl = lane & 15, ch = lane >> 4, g = p0 + pl, R = iw * p.ng + g;
      const int tile = k0 / kExKTile + q;
      // padding rows follow the last frequency's columns
      if (tile >= ex.kt || (g >= p.ng && (iw < kNW - 1 || R >= rows_pad))) continue;
      unsigned char* dst =
          ex.a_tiles + ((size_t)(R / kExRows) * 2 * ex.kt + part * ex.kt + tile) * kExABytes;
      ex_put(dst, kExASlice, R % kExRows, ch, &(part ? sm.i : sm.r)[iw][pl][q * kExKTile + ch * 8], s_e[iw][pl]);
    }
  }
  if (lane == 0)
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int iw = 0; iw < kNW; ++iw) {
        const int g = p0 + warp + 8 * j;
        if (g < p.ng) counts[(size_t)(iw * p.ng + g) * ex.n_kseg + seg] = cnt[j][iw];
      }
}

// One warp per row: the large factors that must coincide with large elements
// of every band (see exact_stats_kernel).
__global__ void gpp_exact_check_kernel(ExactPrep ex, const int* counts, int rows, int nc) {
  const int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (row >= rows || ex.ea[row] == kExZeroRow) return;
  int sum = 0;
  for (int s = lane; s < ex.n_kseg; s += 32)
    sum += max(0, counts[(size_t)row * ex.n_kseg + s] + min(ex.seg_min[s], kExSeg) - min(kExSeg, nc - s * kExSeg));
  sum = __reduce_add_sync(0xffffffffu, sum);
  if (lane == 0 && (long long)sum * kExOverlap < nc) *ex.flag = 1;
}

}  // namespace

bool gpp_exact_create(GppExact& g, int nb, int nc, int ng, int sms) {
  g = GppExact();
  if ((double)kNW * ng * nb * nc < kExactMin) return false;
  ExactTables t;
  exact_size(g.ex, nb, nc, ng, kNW, true, sms, nullptr, &t);
  const size_t bytes = exact_bytes(g.ex);
  if (cudaMalloc(&g.block, bytes + sizeof(int) * (size_t)kNW * ng * g.ex.n_kseg) != cudaSuccess) {
    cudaGetLastError();
    g.block = nullptr;
    return false;
  }
  exact_bind(g.ex, g.block);
  g.counts = reinterpret_cast<int*>(static_cast<char*>(g.block) + bytes);
  g.grid = sms;
  if (exact_upload_tables(g.ex, t) != cudaSuccess) {
    cudaGetLastError();
    gpp_exact_destroy(g);
    return false;
  }
  return true;
}

void gpp_exact_destroy(GppExact& g) {
  if (g.block) cudaFree(g.block);
  g = GppExact();
}

cudaError_t launch_gpp_exact_operands(const GppExact& g, const GppDev& p, cudaStream_t s) {
  const ExactPrep& ex = g.ex;
  cudaError_t e = exact_begin(ex, s);
  if (e != cudaSuccess) return e;
  e = launch_exact_b(ex, p.aqsn, p.nb, p.nc, s);
  if (e != cudaSuccess) return e;
  gpp_exact_max_kernel<<<p.ng, kGxThreads, 0, s>>>(p, ex);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  constexpr int smem = sizeof(FactorPlanes);
  e = cudaFuncSetAttribute(gpp_exact_factor_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  const int cols = p.ng + ex.n_row_blocks * kExRows - kNW * p.ng;
  gpp_exact_factor_kernel<<<dim3((cols + kGxCols - 1) / kGxCols, ex.n_kseg), kGxThreads, smem, s>>>(p, ex, g.counts);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  const int rows = kNW * p.ng;
  gpp_exact_check_kernel<<<(rows * 32 + 255) / 256, 256, 0, s>>>(ex, g.counts, rows, p.nc);
  return cudaGetLastError();
}

cudaError_t launch_gpp_exact_sums(const GppExact& g, const GppDev& p, int* status, double2* acht_n1, cudaStream_t s) {
  cudaError_t e = launch_exact_gemm(g.ex, g.grid, status, s);
  if (e != cudaSuccess) return e;
  FfDev d{};
  d.nb = p.nb;
  d.nc = p.nc;
  d.ng = p.ng;
  d.nf = kNW;
  d.aqsm = p.aqsm;
  d.igp_of = p.igp_of;
  d.vcoul = p.vcoul;
  d.vfac = 0.5;
  return launch_exact_finish(d, g.ex, acht_n1, nullptr, s);
}

}  // namespace sigma
