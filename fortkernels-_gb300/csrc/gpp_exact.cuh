// FP64 GPP band sums with one frequency set for every band, as an exact digit
// contraction on the tensor cores (exact_gemm.cuh): the complex sum, the
// gppsum = 1 half sum and the real-valued sum.
#pragma once

#include <vector>

#include "exact_gemm.cuh"

namespace sigma {

// The band sums are acht_n1[n][iw] = sum_g 0.5 vcoul conj(aqsm) sum_ig aqsn Y
// with the band-independent factors Y[iw][g][ig], formed in FP64 once per
// (column, g-vector) and written as the contraction's A digits.  512 bands x
// 1638 columns x 32768 g-vectors: 17.5 ms with the occupied bands, 150 ms with
// float-float terms (sch_fp64y_kernel); 128 x 409 x 8192: 1.12 ms, 3.40 ms.
enum GxForm {
  kGxGpp,   // complex, three frequencies, all g-vectors
  kGxHalf,  // gppsum = 1: three frequencies below igp - 1 and, with four
            // slabs, -I_eps below igp (the static remainder); the bands are
            // aqsn's, then aqsm's (the sums T and U)
  kGxReal   // real arrays
};

// One instance; arrays complex (interleaved) or real.
struct GxDev {
  int nb, nc, ng;
  const double *aqsm, *aqsn, *ieps, *wt, *vcoul, *wx;
  const int* igp_of;
};

struct GppExact {
  ExactPrep ex{};
  GxForm form = kGxGpp;
  int nf = kNW;           // row slabs of ng columns
  int* kend = nullptr;    // [nf ng] first zero K of each row (half sum)
  float* stat = nullptr;  // [nf ng][n_kseg] large factors per segment (half sum: sums of squares)
  int grid = 0;
  void *own = nullptr, *work = nullptr;  // work null when the caller's is used
  explicit operator bool() const { return own != nullptr; }
};

// Sizes, allocates and fills the contraction of one instance; false (with
// nothing allocated) when the problem is below kExactMin products or the
// device has no room: the FP64 kernel keeps the work.  nf: kNW, or 4 for the
// half sum with its static remainder.  With shared_work set (at least
// gpp_exact_work_bytes) the instance has no workspace of its own.
bool gpp_exact_create(GppExact& g, GxForm form, int nb, int nc, int ng, int nf, const std::vector<int>& igp_of,
                      int sms, void* shared_work = nullptr);
size_t gpp_exact_work_bytes(GxForm form, int nb, int nc, int ng, int nf, const std::vector<int>& igp_of, int sms);
void gpp_exact_destroy(GppExact& g);

// launch_gpp_exact_operands forms the operands and raises g.ex.flag for
// values outside the split's range; unless it is raised, launch_gpp_exact_sums
// leaves the sums in out: [nb][3] (half sum: [2 nb][nf], T then U).
cudaError_t launch_gpp_exact_operands(const GppExact& g, const GxDev& p, cudaStream_t s);
cudaError_t launch_gpp_exact_sums(const GppExact& g, const GxDev& p, int* status, double2* out, cudaStream_t s);

// Kernels of one execution: two for the bands, three for the factors, the
// contraction and two for its epilogue.
constexpr int kGxLaunches = 8;

inline GxDev gx_dev(const GppDev& p) {
  auto d = [](const double2* x) { return reinterpret_cast<const double*>(x); };
  return GxDev{p.nb, p.nc, p.ng, d(p.aqsm), d(p.aqsn), d(p.ieps), d(p.wt), p.vcoul, p.wx, p.igp_of};
}

}  // namespace sigma
