// Column-weighted FP64 contractions on the tcgen05 tensor cores: operands cut
// into fixed-point BF16 digits, digit products summed exactly.
//
//   out[n][f] = sum_g w(g) conj(m[n][igp(g)]) * sum_k A[f][g][k] b[n][k]
//
// is the sum behind the FP64 forms of the FF contraction, the static
// remainders and the GPP band sums.  GB300 runs FP64 multiply-adds at 1/64 of
// the FP32 rate (1.25 TFLOP/s) and BF16 products at 1.9 PFLOP/s, so 21 exact
// BF16 products per FP64 product are ~70 times faster.
//
// Splitting.  Row r of an operand gets one exponent e with |x| < 2^e for every
// element, and x 2^(52 - e) is rounded to an integer of at most 53 bits,
// written as six digits (8 bits, then 5 x 9 bits, balanced: |d0| <= 128,
// |d1..5| <= 256).  Every digit is exact in BF16's 8 significant bits.
// Digit products i + j = s share the weight 2^-9s: the 21 products with
// s <= 5 go to six FP32 accumulators, one per s.  Over 128 K values the sums
// stay below 2^24 (s <= 2: 128 (2 2^15 + 2^16) = 2^24 at most), so the FP32
// accumulation is exact whatever the data; s = 3 .. 5 carry weights of 2^-41
// and below of the row maxima and may round in the all-equal worst case only.
// Dropped products (s >= 6) and the digits' own rounding are 2^-53 of the
// product of the row maxima.
//
// That error is relative to the rows' largest elements.  exact_stats checks
// that large elements of every row pair coincide often enough for it to stay
// below the float-float terms' error (ExactPrep::flag); rows that fail, and
// values that are not finite, raise the flag, and the callers' FP64 kernels
// run instead.
#pragma once

#include <vector>

#include "ff_internal.cuh"
#include "sigma_tma.cuh"

namespace sigma {

constexpr int kExSlices = 6;
constexpr int kExKTile = 16;     // K elements per staged tile (one 32-byte swizzle row)
constexpr int kExRows = 128;     // A rows per tile
constexpr int kExCols = 80;      // B' rows per slice: 40 complex bands (Re, Im interleaved) or 80 real ones
constexpr int kExSeg = 512;      // K values per segment of the overlap check
constexpr uint32_t kExASlice = kExRows * kExKTile * 2;          // 4 KB
constexpr uint32_t kExABytes = kExSlices * kExASlice;           // 24 KB
constexpr uint32_t kExBSlice = kExCols * kExKTile * 2;          // 2.5 KB
constexpr uint32_t kExBBytes = kExSlices * kExBSlice;           // 15 KB
// Exponent slack of the overlap check: an element counts as large when its
// larger part is within 2^-slack of its row's maximum.
constexpr int kExSlackA = 5, kExSlackB = 3;
constexpr int kExOverlap = 16;   // a row pair needs K / kExOverlap coinciding large elements
constexpr int kExZeroRow = 4096; // exponent of a row without a nonzero value (its digits are zero)

// Operand layout.  halves = 2: complex, the real and imaginary parts laid
// along K' as in the split-BF16 form,
//   A'[R][k'] = Re A[R][k] (k' < K), Im A[R][k] (k' >= K)
//   B'[2n][k'] = Re b, -Im b;   B'[2n + 1][k'] = Im b, Re b
// halves = 1: real operands, 80 bands per tile.
struct ExactPrep {
  unsigned char* a_tiles;   // [n_row_blocks][halves*kt][6][128][16] bf16
  unsigned char* b_tiles;   // [n_col_blocks][halves*kt][6][80][16] bf16
  int halves, kt;           // K tiles per half (K padded to 32: an even count)
  int bands;                // bands per column block (40 complex, 80 real)
  int n_row_blocks, n_col_blocks;
  int n_splits, split_tiles;
  int n_entries, n_items, max_pieces;
  const int4* entries;      // [n_entries]: row block, piece, first K' tile, tiles (even)
  const int* pieces;        // [n_row_blocks]
  const int* kt_lim;        // [n_row_blocks]: K tiles per half that can be nonzero (even)
  int max_seg;              // frequencies one row block can touch
  int n_kseg;               // ceil(K / kExSeg)
  int* ea;                  // [n_row_blocks * 128] exponents of the A rows
  int* eb;                  // [n_col_blocks * bands] exponents of the bands
  int* seg_min;             // [n_kseg] over the bands: large elements per segment
  int* flag;                // nonzero: the operands are outside the split's range
  long long* raw_hi;        // [row block][col block][piece][80][128] sums of s <= 3, unit 2^(ea+eb-41)
  float* raw_lo;            // the same shape: sums of s = 4, 5 in that unit
  double2* partial;         // [row block][col block][max_seg][bands]
  double2* partial2;        // second output (FfDev::vcoul2)
};

struct ExactTables {
  std::vector<int4> entries;
  std::vector<int> pieces, kt_lim;
};

// Shape of a contraction: rows = nf * ng A rows over K = nc.  row_kend as in
// ozaki_size.
void exact_size(ExactPrep& ex, int nb, int nc, int ng, int nf, bool cplx, int grid, const int* row_kend,
                ExactTables* tables);
size_t exact_bytes(const ExactPrep& ex);
void exact_bind(ExactPrep& ex, void* base);
cudaError_t exact_upload_tables(const ExactPrep& ex, const ExactTables& t);

// Plans take the exact form from this many products on (rows x bands x K): below it
// its ten launches cost more than the FP64 kernel.
constexpr double kExactMin = 1 << 22;

// One contraction, in order:
//   exact_begin       clears the flag and the overlap counts
//   launch_exact_b    band exponents, overlap counts and the B digits
//   launch_exact_a    row exponents, overlap check and the A digits of
//                     complex rows (or the caller's own producer of both)
//   launch_exact_gemm the digit products
//   launch_exact_finish  FP64 sums of the rows per band, into out[n][nf]
cudaError_t exact_begin(const ExactPrep& ex, cudaStream_t s);
cudaError_t launch_exact_b(const ExactPrep& ex, const double2* b, int nb, int nc, cudaStream_t s);
cudaError_t launch_exact_a(const ExactPrep& ex, const double2* a, int rows, int nc, const int* row_kend,
                           cudaStream_t s);
cudaError_t launch_exact_gemm(const ExactPrep& ex, int grid, int* status, cudaStream_t s);
cudaError_t launch_exact_finish(const FfDev& d, const ExactPrep& ex, double2* out, double2* out2, cudaStream_t s);

// ---------------------------------------------------------------- device helpers
// Byte offset of element (row r, k) inside a K-major 32-byte-swizzled tile of
// 16-element rows: 16-byte chunk c of row r is stored at chunk c ^ (r / 4 % 2).
__host__ __device__ __forceinline__ uint32_t sw32_offset(int r, int ch) {
  return (uint32_t)(r * 32 + ((ch ^ ((r >> 2) & 1)) << 4));
}

// The six digits of x 2^(52 - e) as 9-bit fields of one word, field i + 256
// being digit i shifted by 9 (5 - i): the balanced digits need no carries.
// Round to nearest on the integer pipe (the FP64 pipe is 1/64 rate).
constexpr unsigned long long kExBias = 256ull * (1ull + (1ull << 9) + (1ull << 18) + (1ull << 27) + (1ull << 36) +
                                                 (1ull << 45));
__device__ __forceinline__ unsigned long long ex_fields(double x, int e) {
  const unsigned long long bits = (unsigned long long)__double_as_longlong(x);
  const int ex = (int)(bits >> 52) & 0x7FF;
  const int sh = 1023 + e - ex;  // >= 1 as |x| < 2^e
  unsigned long long m = (bits & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull;
  m = sh > 54 || ex == 0 ? 0ull : ((m >> (sh - 1)) + 1) >> 1;
  const long long v = (long long)bits < 0 ? -(long long)m : (long long)m;
  return (unsigned long long)v + kExBias;
}
// Digit i of a field word as FP32 (exact).
__device__ __forceinline__ float ex_digit(unsigned long long f, int i) {
  const unsigned d = (unsigned)(f >> (9 * (5 - i))) & 511u;
  return __uint_as_float(0x4B000000u | d) - 8388864.f;  // 2^23 + 256
}
// Digits i of two values as a BF16 pair (each exact in the upper half of FP32).
__device__ __forceinline__ uint32_t ex_pair(unsigned long long f0, unsigned long long f1, int i) {
  return __byte_perm(__float_as_uint(ex_digit(f0, i)), __float_as_uint(ex_digit(f1, i)), 0x7632);
}

// 16-byte digit chunks (8 K values of one row) of the six slices.
struct ExChunk {
  uint4 s[kExSlices];
};
__device__ __forceinline__ ExChunk ex_chunk(const double (&v)[8], int e) {
  ExChunk c;
  unsigned long long f[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) f[j] = ex_fields(v[j], e);
#pragma unroll
  for (int i = 0; i < kExSlices; ++i)
    c.s[i] = make_uint4(ex_pair(f[0], f[1], i), ex_pair(f[2], f[3], i), ex_pair(f[4], f[5], i), ex_pair(f[6], f[7], i));
  return c;
}
__device__ __forceinline__ ExChunk ex_negate(const ExChunk& c) {
  ExChunk n;
#pragma unroll
  for (int i = 0; i < kExSlices; ++i)
    n.s[i] = make_uint4(c.s[i].x ^ 0x80008000u, c.s[i].y ^ 0x80008000u, c.s[i].z ^ 0x80008000u, c.s[i].w ^ 0x80008000u);
  return n;
}
__device__ __forceinline__ void ex_store(unsigned char* tile, uint32_t slice_bytes, int r, int ch, const ExChunk& c) {
  unsigned char* p = tile + sw32_offset(r, ch);
#pragma unroll
  for (int i = 0; i < kExSlices; ++i) *reinterpret_cast<uint4*>(p + i * slice_bytes) = c.s[i];
}

// The same for 8 values whose digits come from a plane of doubles in shared
// memory (a factor pass's staging).
__device__ __forceinline__ void ex_put(unsigned char* tile, uint32_t slice_bytes, int r, int ch, const double* v, int e) {
  double x[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) x[j] = v[j];
  ex_store(tile, slice_bytes, r, ch, ex_chunk(x, e));
}

}  // namespace sigma
