// FP64 GPP band sums with one frequency set for every band, as an exact digit
// contraction on the tensor cores (exact_gemm.cuh).
#pragma once

#include "exact_gemm.cuh"

namespace sigma {

// The band sums are acht_n1[n][iw] = sum_g 0.5 vcoul conj(aqsm) sum_ig aqsn Y
// with the band-independent factors Y[iw][g][ig], formed in FP64 once per
// (column, g-vector) and written as the contraction's A digits.  512 bands x
// 1638 columns x 32768 g-vectors: 17.5 ms with the occupied bands, 150 ms with
// float-float terms (sch_fp64y_kernel); 128 x 409 x 8192: 1.12 ms, 3.40 ms.
struct GppExact {
  ExactPrep ex{};
  int* counts = nullptr;  // [3 ng][n_kseg] large factors per segment
  int grid = 0;
  void* block = nullptr;
};

// Sizes, allocates and fills the contraction of one instance; false (with
// nothing allocated) when the problem is below kExactMin products or the
// device has no room: the FP64 kernel keeps the work.
bool gpp_exact_create(GppExact& g, int nb, int nc, int ng, int sms);
void gpp_exact_destroy(GppExact& g);
// The main pass: acht_n1[nb][3] unless g.ex.flag is raised.
// launch_gpp_exact_operands forms the operands and raises the flag for
// values outside the split's range; the contraction and its epilogue follow.
cudaError_t launch_gpp_exact_operands(const GppExact& g, const GppDev& p, cudaStream_t s);
cudaError_t launch_gpp_exact_sums(const GppExact& g, const GppDev& p, int* status, double2* acht_n1, cudaStream_t s);

}  // namespace sigma
