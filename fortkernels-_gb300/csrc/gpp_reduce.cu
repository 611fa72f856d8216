// Deterministic cross-block reduction of the GPP partial sums.
//
// The reference sums per-thread partial arrays after its band loop
// (BGW-Kernels/gppKer.cpp:431-439) in an order that changes with OpenMP's
// dynamic schedule.  Here every partial has a fixed slot, and the sums run in
// a fixed order with Neumaier-compensated FP64 accumulation: one block per
// (band, frequency) sums the column blocks and g-vector splits (each thread
// a fixed strided subset, then a fixed butterfly per warp and the warps in
// order), then one warp per frequency sums the bands.  Results are
// identical run to run.
#include <algorithm>

#include "sigma_internal.cuh"

namespace sigma {
namespace {


// Threads per row: two warps where the rows fill the chip and are short (eight
// spend most of the time in their butterflies, 80 FP64 operations each at two
// lanes per clock per SM: 100 -> 41 us at the FP32 form's 1542 rows), else
// eight, whose loads overlap (the tensor form's six long rows: 43 us, 73 us
// with two).
constexpr int kRowWarps = 8;
int row_threads(int rows, int count) { return rows >= 304 && count <= 1024 ? 64 : 32 * kRowWarps; }
int row_count(const ReduceArgs& a) {
  return std::max(a.sch_rows > 0 ? a.sch_ncb * a.sch_splits : 0, a.nvband > 0 ? a.ssx_ncb * a.ssx_splits : 0);
}

// Row `row` of the band-sum stage (one block).
__device__ __forceinline__ void reduce_bands_row(const ReduceArgs& a, int row) {
  __shared__ double s_x[kRowWarps], s_y[kRowWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n_sch = a.sch_rows * kNW;
  const bool is_sch = row < n_sch;
  const int* run_if = is_sch ? a.sch_run_if : a.ssx_run_if;
  if (run_if && !*run_if) return;
  const int e = is_sch ? row : row - n_sch;
  const int n1 = e / kNW, iw = e % kNW;
  const int bn = is_sch ? a.sch_bn : kSsxBN;
  const int ncb = is_sch ? a.sch_ncb : a.ssx_ncb;
  const int ns = is_sch ? a.sch_splits : a.ssx_splits;
  const double2* part = is_sch ? a.sch_partial : a.ssx_partial;
  const int bb = n1 / bn, bl = n1 % bn;
  Comp sx, sy;
  const int count = ncb * ns;
#pragma unroll 4
  for (int q = threadIdx.x; q < count; q += blockDim.x) {
    const size_t item = (size_t)bb * count + q;  // (bb * ncb + cb) * ns + s
    const double2 v = part[item * bn * kNW + bl * kNW + iw];
    sx.add(v.x);
    sy.add(v.y);
  }
  const double rx = warp_sum_comp(sx), ry = warp_sum_comp(sy);
  if (lane == 0) {
    s_x[warp] = rx;
    s_y[warp] = ry;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    Comp tx, ty;
    for (int w = 0; w < (int)blockDim.x / 32; ++w) {
      tx.add(s_x[w]);
      ty.add(s_y[w]);
    }
    if (is_sch)
      a.acht_n1[e] = make_double2(tx.value(), ty.value());
    else
      a.asx_n1[e] = make_double2(tx.value(), ty.value());
  }
}

__global__ void __launch_bounds__(32 * kRowWarps) reduce_bands_kernel(ReduceArgs a) {
  chain_begin();
  reduce_bands_row(a, blockIdx.x);
}

// One warp per frequency and sum (blocks 0-5), each on an SM of its own: six
// warps of one SM share its two FP64 lanes per clock (15.5 -> 13.4 us at
// 512 bands).  Block 6: the band sums of the last frequency.
constexpr int kTotalBlocks = 2 * kNW + 1;
__device__ __forceinline__ void reduce_total_block(int block, const double2* acht_n1, const double2* asx_n1, int nb,
                                                   int nvband, double2* achtemp, double2* asxtemp,
                                                   double2* acht_n1_loc) {
  const int lane = threadIdx.x;
  if (block == 2 * kNW) {
    if (acht_n1_loc)
      for (int n1 = lane; n1 < nb; n1 += 32) acht_n1_loc[n1] = acht_n1[n1 * kNW + 2];
    return;
  }
  const bool ach = block < kNW;
  const int iw = ach ? block : block - kNW;
  const double2* src = ach ? acht_n1 : asx_n1;
  const int n = ach ? nb : nvband;
  Comp sx, sy;
#pragma unroll 8
  for (int n1 = lane; n1 < n; n1 += 32) {
    const double2 v = src[n1 * kNW + iw];
    sx.add(v.x);
    sy.add(v.y);
  }
  const double rx = warp_sum_comp(sx), ry = warp_sum_comp(sy);
  if (lane == 0) (ach ? achtemp : asxtemp)[iw] = make_double2(rx, ry);
}

__global__ void reduce_total_kernel(const double2* acht_n1, const double2* asx_n1, int nb,
                                    int nvband, double2* achtemp, double2* asxtemp,
                                    double2* acht_n1_loc) {
  chain_begin();
  reduce_total_block(blockIdx.x, acht_n1, asx_n1, nb, nvband, achtemp, asxtemp, acht_n1_loc);
}

// Group forms over many instances: blocks row_off .. + (sch_rows + nvband) * 3
// of each job, then one block per job.
__global__ void __launch_bounds__(32 * kRowWarps) reduce_bands_group_kernel(const ReduceJob* jobs, int n) {
  chain_begin();
  const int row = blockIdx.x;
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (jobs[mid].row_off <= row) lo = mid; else hi = mid - 1;
  }
  reduce_bands_row(jobs[lo].a, row - jobs[lo].row_off);
}

__global__ void reduce_total_group_kernel(const ReduceJob* jobs) {
  chain_begin();
  const ReduceJob& j = jobs[blockIdx.x / kTotalBlocks];
  reduce_total_block(blockIdx.x % kTotalBlocks, j.a.acht_n1, j.a.asx_n1, j.a.nb, j.a.nvband, j.achtemp, j.asxtemp, j.acht_n1_loc);
}

}  // namespace

ReduceJob gpp_reduce_job(const GppWork& sch, const GppWork& ssx, int nb, double2* acht_n1, double2* achtemp,
                         double2* asxtemp, double2* acht_n1_loc, int row_off) {
  ReduceJob j{};
  ReduceArgs& a = j.a;
  a.sch_rows = sch.partial ? nb : 0;
  a.sch_partial = sch.partial;
  a.sch_run_if = sch.run_if;
  a.ssx_run_if = ssx.run_if;
  a.sch_ncb = sch.n_col_blocks;
  a.sch_splits = sch.n_splits;
  a.sch_bn = sch.bn;
  a.ssx_partial = ssx.partial;
  a.ssx_ncb = ssx.n_col_blocks;
  a.ssx_splits = ssx.n_splits;
  a.nb = nb;
  a.nvband = ssx.band_count;
  a.acht_n1 = acht_n1;
  a.asx_n1 = acht_n1 + (size_t)nb * kNW;
  j.achtemp = achtemp;
  j.asxtemp = asxtemp;
  j.acht_n1_loc = acht_n1_loc;
  j.row_off = row_off;
  return j;
}

int gpp_reduce_job_count(const ReduceJob& j) { return row_count(j.a); }
int gpp_reduce_job_rows(const ReduceJob& j) { return (j.a.sch_rows + j.a.nvband) * kNW; }

cudaError_t launch_gpp_reduce_group(const ReduceJob* jobs, int n, int total_rows, int max_count, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  if (total_rows > 0) {
    cudaError_t e = launch_chained(reduce_bands_group_kernel, total_rows, row_threads(total_rows, max_count), 0, s, true, jobs, n);
    if (e != cudaSuccess) return e;
  }
  return launch_chained(reduce_total_group_kernel, n * kTotalBlocks, 32, 0, s, true, jobs);
}

cudaError_t launch_gpp_reduce(const GppWork& sch, const GppWork& ssx, int nb, double2* acht_n1,
                              double2* achtemp, double2* asxtemp, double2* acht_n1_loc,
                              cudaStream_t s) {
  ReduceArgs a;
  a.sch_rows = sch.partial ? nb : 0;
  a.sch_partial = sch.partial;
  a.sch_run_if = sch.run_if;
  a.ssx_run_if = ssx.run_if;
  a.sch_ncb = sch.n_col_blocks;
  a.sch_splits = sch.n_splits;
  a.sch_bn = sch.bn;
  a.ssx_partial = ssx.partial;
  a.ssx_ncb = ssx.n_col_blocks;
  a.ssx_splits = ssx.n_splits;
  a.nb = nb;
  a.nvband = ssx.band_count;
  a.acht_n1 = acht_n1;
  a.asx_n1 = acht_n1 + (size_t)nb * kNW;
  const int rows = (a.sch_rows + a.nvband) * kNW;
  if (rows > 0) {
    cudaError_t e = launch_chained(reduce_bands_kernel, rows, row_threads(rows, row_count(a)), 0, s, true, a);
    if (e != cudaSuccess) return e;
  }
  return launch_chained(reduce_total_kernel, kTotalBlocks, 32, 0, s, true, acht_n1, a.asx_n1, nb, a.nvband, achtemp, asxtemp,
                        acht_n1_loc);
}

}  // namespace sigma
