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
// 1638 columns x 32768 g-vectors: 11.8 ms with the occupied bands, 150 ms with
// float-float terms (sch_fp64y_kernel); 128 x 409 x 8192: 0.46 ms, 3.40 ms.
// The occupied bands' sums (asxtemp) are the same contraction with other
// factors, of the first bands only: further rows of it, or, where the kernel
// they replace was FP64 throughout, a contraction of their own with seven
// digits (six put the half sum's and the real asxtemp at 2 to 4 times the FP64
// kernels' error).
enum GxForm {
  kGxGpp,     // complex, three frequencies, all g-vectors; occupied rows: ssx
  kGxReal,    // real arrays
  kGxRealOcc, // real arrays, the occupied bands' ssx
  kGxHalf,    // gppsum = 1: three frequencies below igp - 1 and, with four
              // slabs, -I_eps below igp (the static remainder); the bands are
              // aqsn's, then aqsm's (the sums T and U)
  kGxHalfOcc  // gppsum = 1, occupied bands: sch and ssx of three frequencies
              // below min(igp, brk); bands as kGxHalf
};

// One instance; arrays complex (interleaved) or real.
struct GxDev {
  int nb, nvband, nc, ng;
  double occ;
  const double *aqsm, *aqsn, *ieps, *wt, *vcoul, *wx;
  const int* igp_of;
  const int* brk = nullptr;  // kGxHalfOcc: [ng] first g-vector of the cut
};

struct GppExact {
  ExactPrep ex{};
  GxForm form = kGxGpp;
  int nf = kNW, nf2 = 0;  // row slabs of ng columns: all bands', occupied bands'
  float* stat = nullptr;  // [rows][runs] large factors per run (half sum: least sums of squares with any band)
  int run = 0;            // g-vectors per factor item (a segment or a power-of-two part of it)
  int grid = 0;
  void* block = nullptr;  // its allocation; null when the caller's memory is used
  bool ready = false;
  explicit operator bool() const { return ready; }
};

// Memory of a caller that runs several contractions one after another on one
// stream: one workspace (at least gpp_exact_work_bytes of each), and tables
// (gpp_exact_own_bytes each), packed into host memory for one copy.
struct GxShared {
  void *work, *own;  // device
  char* own_host;
};

// The contraction's shape: nb bands (kGxRealOcc, kGxHalfOcc: the occupied ones),
// nvband of them occupied, with_static for kGxHalf's fourth slab.
struct GxShape {
  GxForm form;
  int nb, nvband, nc, ng;
  bool with_static;
};

// Sizes, allocates and fills the contraction of one instance; false (with
// nothing allocated) when the device has no room, or the workspace would take
// more than half of its free memory: the FP64 kernels keep the
// work, as for problems too small for it (gpp_exact_fits).
// A plan that lives for one host call takes its memory from an arena slot
// (ArenaSlot) where it may.
bool gpp_exact_create(GppExact& g, const GxShape& q, const std::vector<int>& igp_of, int sms, int arena_slot = -1);
void gpp_exact_create(GppExact& g, const GxShape& q, const std::vector<int>& igp_of, int sms, const GxShared& m);
bool gpp_exact_fits(const GxShape& q);
bool gpp_exact_pays(const GxShape& q);  // large enough, whatever the sums' length
size_t gpp_exact_work_bytes(const GxShape& q, const std::vector<int>& igp_of, int sms, size_t* own = nullptr);
void gpp_exact_destroy(GppExact& g);

// launch_gpp_exact_operands forms the operands and raises g.ex.flag for
// values outside the split's range (begin: clears the flag first, else the
// caller has); unless it
// is raised, launch_gpp_exact_sums leaves the sums in out: [nb][3] (kGxHalf:
// [2 nb][nf], T then U; kGxHalfOcc: [2 nvband][6], sch then ssx, both
// weighted 0.5 vcoul; kGxRealOcc: [nvband][3], weighted occ vcoul) and
// kGxGpp's occupied bands' in occ_out [nvband][3].
cudaError_t launch_gpp_exact_operands(const GppExact& g, const GxDev& p, cudaStream_t s, bool begin = true);
cudaError_t launch_gpp_exact_sums(const GppExact& g, const GxDev& p, int* status, double2* out, double2* occ_out,
                                  cudaStream_t s);

// Kernels of one execution: two for the bands, three for the factors, the
// contraction and two for the epilogue.
inline int gpp_exact_launches(const GppExact& g) { return g ? 8 : 0; }

inline GxDev gx_dev(const GppDev& p) {
  auto d = [](const double2* x) { return reinterpret_cast<const double*>(x); };
  return GxDev{p.nb, p.nvband, p.nc, p.ng, p.occ, d(p.aqsm), d(p.aqsn), d(p.ieps), d(p.wt), p.vcoul, p.wx, p.igp_of};
}

}  // namespace sigma
