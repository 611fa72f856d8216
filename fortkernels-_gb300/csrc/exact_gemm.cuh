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
// and below of the row maxima and may round where the data are all alike.
// Dropped products (s >= 6) come to 2^-52 rms of the product of the row maxima,
// the digits' own rounding to 2^-54.
//
// Seven digits (28 products) serve operands whose rows hold a few elements
// far above the rest: the half sum's factors near poles.
//
// Over random digits a product's error is 2^-52 (six digits) or 2^-61 (seven)
// rms of the product of its rows' largest elements, and that of a sum of K
// products sqrt(K) times it, whatever the elements' own size.  So every row
// pair is checked for a sum of squares that is large enough beside it.  The
// statistics passes count that elements within 2^-5 (A) and 2^-4 (B) of their
// rows' largest meet in at least K / 128 places of every row pair: if all others
// were zero, the error would be 2^-39.5 of the sum's root mean square with six
// digits and 2^-48 with seven (uniform inputs: 2^-51 with six).  Rows that fail,
// and values that are not finite, raise ExactPrep::flag, and the callers' FP64
// kernels run instead.  The half sum's rows end at their igp and may hold few
// large elements (factors near poles); they are checked against band_min, the
// least element of any band at each K value (gx_check_kernel).
//
// The splitting is the error-free transformation of matrix products of Ozaki,
// Ogita, Oishi and Rump (Numerical Algorithms 59, 2012), here with one exponent
// per row, digits fixed by BF16's significand and integer sums.
#pragma once

#include <vector>

#include "ff_internal.cuh"
#include "sigma_tma.cuh"

namespace sigma {

constexpr int kExKTile = 16;     // K elements per staged tile (one 32-byte swizzle row)
constexpr int kExRows = 128;     // A rows per tile
constexpr int kExSeg = 512;      // K values per segment of the overlap check,
constexpr int kExCount = 128;    // of which the first are counted (a lower bound, at a quarter of the work)
constexpr uint32_t kExASlice = kExRows * kExKTile * 2;  // 4 KB
// S slices (digits) per value and at most so many B' rows per slice, such that
// the S accumulators fit tensor memory's 512 columns: 6 x 80 (40 complex bands,
// Re and Im interleaved, or 80 real ones) or 7 x 64.  ex_pick_cols takes fewer (48
// or 64) where they pad the bands less.
constexpr int ex_max_cols(int S) { return S == 6 ? 80 : 64; }
int ex_pick_cols(int S, int b_rows);
constexpr uint32_t ex_a_bytes(int S) { return S * kExASlice; }                                 // 24 / 28 KB
constexpr uint32_t ex_b_slice(int cols) { return (uint32_t)cols * kExKTile * 2; }              // 1.5 to 2.5 KB
constexpr uint32_t ex_b_bytes(int S, int cols) { return S * ex_b_slice(cols); }                // 9 to 15 KB
// Exponent slack of the overlap check: an element counts as large when its
// larger part is within 2^-slack of its row's maximum.
constexpr int kExSlackA = 4, kExSlackB = 3;
constexpr int kExOverlap = 128;  // a row pair needs K / kExOverlap coinciding large elements
constexpr int kExZeroRow = 4096; // exponent of a row without a nonzero value (its digits are zero)

// Operand layout.  halves = 2: complex, the real and imaginary parts laid
// along K' as in the split-BF16 form,
//   A'[R][k'] = Re A[R][k] (k' < K), Im A[R][k] (k' >= K)
//   B'[2n][k'] = Re b, -Im b;   B'[2n + 1][k'] = Im b, Re b
// halves = 1: real operands, one B' row per band.
struct ExactPrep {
  unsigned char* a_tiles;   // [n_row_blocks][halves*kt][slices][128][16] bf16
  unsigned char* b_tiles;   // [n_col_blocks][halves*kt][slices][cols][16] bf16
  int slices, cols;         // 6 and 48, 64 or 80, or 7 and 64
  int halves, kt;           // K tiles per half (K padded to 32: an even count)
  int bands;                // bands per column block (cols / 2 complex, cols real)
  int n_row_blocks, n_col_blocks;
  // Row blocks from n_main_blocks on (a second group of rows, from row
  // n_main_blocks * 128: the occupied bands' factors) meet the first
  // n_col_blocks2 band blocks only.
  int n_main_blocks, n_col_blocks2;
  int n_splits, split_tiles;
  int n_entries, n_main_entries, n_items, max_pieces;
  const int4* entries;      // [n_entries]: row block, piece, first K' tile, tiles (even)
  const int* pieces;        // [n_row_blocks]
  const int* kt_lim;        // [n_row_blocks]: K tiles per half that can be nonzero (even)
  int max_seg;              // frequencies one row block can touch
  int n_kseg;               // ceil(K / kExSeg)
  int* ea;                  // [n_row_blocks * 128] exponents of the A rows
  int* eb;                  // [n_col_blocks * bands] exponents of the bands
  int* seg_min;             // [n_kseg] over the bands: large elements per segment
  float* band_min;          // [16 kt] least magnitude of the bands per K value, unit 2^eb (complex, seven slices)
  int* flag;                // nonzero: the operands are outside the split's range
  int* any;                 // nullable: raised with flag (one word for a batch)
  long long* raw_hi;        // [row block][col block][piece][cols][128] sums of s <= 3, unit 2^(ea+eb-41)
  float* raw_lo;            // the same shape: sums of s >= 4 in that unit
  double2* partial;         // [row block][col block][max_seg][bands]
  double2* partial2;        // second output (FfDev::vcoul2)
};

struct ExactTables {
  std::vector<int4> entries;
  std::vector<int> pieces, kt_lim;
};

// Complex contractions of seven digits keep band_min, after seg_min.
__host__ __device__ __forceinline__ bool ex_has_band_min(const ExactPrep& ex) {
  return ex.slices == 7 && ex.halves == 2;
}
__host__ __device__ __forceinline__ int ex_count_words(const ExactPrep& ex) {
  return ex.n_kseg + (ex_has_band_min(ex) ? ex.kt * kExKTile : 0);
}

// Index of a (row block, band block) pair in the raw sums and partials.
__host__ __device__ __forceinline__ size_t ex_block_index(const ExactPrep& ex, int rb, int cb) {
  return rb < ex.n_main_blocks
             ? (size_t)rb * ex.n_col_blocks + cb
             : (size_t)ex.n_main_blocks * ex.n_col_blocks + (size_t)(rb - ex.n_main_blocks) * ex.n_col_blocks2 + cb;
}

// Shape of a contraction: nf * ng A rows over K = nc with nb bands, and nf2 *
// ng further rows with the first nb2 bands.  row_kend as in ozaki_size (rows
// of the first group).
void exact_size(ExactPrep& ex, int slices, int nb, int nc, int ng, int nf, bool cplx, int grid, const int* row_kend,
                ExactTables* tables, int nf2 = 0, int nb2 = 0);
// Buffers: `work` (digits, exponents, raw sums) may be shared by contractions
// that run one after another on one stream; `own` (flag and tables; from a
// 256-byte boundary) may not.  exact_pack_own writes own's contents, the flag
// down, into host memory; exact_upload_tables copies them.
size_t exact_work_bytes(const ExactPrep& ex);
size_t exact_own_bytes(const ExactPrep& ex);
void exact_bind(ExactPrep& ex, void* work, void* own);
void exact_pack_own(const ExactPrep& ex, const ExactTables& t, char* host);
cudaError_t exact_upload_tables(const ExactPrep& ex, const ExactTables& t);

// FF plans take the exact form from this many products on (rows x bands x K):
// 8 x (5 x 12) x 256 = 0.12 M takes 42 us, 67 us on the FP64 pipe.
constexpr double kExactMin = 1 << 16;

// The 64-bit integer sums hold K' products of the rows' largest elements (2^41
// each) below K' = 2^22; longer sums stay with the FP64 kernels.
constexpr bool exact_holds(int nc, bool cplx) { return (cplx ? 2LL : 1LL) * nc <= 1 << 21; }

// One contraction, in order:
//   exact_begin       clears the flag and the overlap counts
//   launch_exact_b    band exponents, overlap counts and the B digits of bands
//                     b0[nb0][nc] and, after them, b1[nb1][nc] (complex, or
//                     real with halves = 1)
//   launch_exact_a    row exponents, overlap check and the A digits of
//                     complex rows (or the caller's own producer of both)
//   launch_exact_gemm the digit products; a wait that gives up also raises
//                     the flag (the status word records it)
//   launch_exact_finish  FP64 sums of the row groups per band, into out[n][f]
//                     (complex; halves = 1: FfDev::aqsm holds real values and
//                     the imaginary parts are zero); FfDev::nf, nb and vfac
//                     are the first group's
cudaError_t exact_begin(const ExactPrep& ex, cudaStream_t s);
cudaError_t exact_begin_flag(const ExactPrep& ex, cudaStream_t s);  // the flag alone (the caller's first kernel
                                                                     // calls ex_begin_counts)
cudaError_t launch_exact_b(const ExactPrep& ex, const void* b0, int nb0, const void* b1, int nb1, int nc,
                           cudaStream_t s);
cudaError_t launch_exact_a(const ExactPrep& ex, const double2* a, int rows, int nc, cudaStream_t s);
cudaError_t launch_exact_gemm(const ExactPrep& ex, int grid, int* status, cudaStream_t s);
// The second row group's epilogue, and its sums.
struct ExSecond {
  int nb, nf;
  double vfac;
  double2* out;  // [nb][nf]; null: no such group
};
cudaError_t launch_exact_finish(const FfDev& d, const ExactPrep& ex, double2* out, double2* out2, cudaStream_t s,
                                const ExSecond& second = ExSecond{0, 0, 0.0, nullptr});

// ---------------------------------------------------------------- device helpers
// Byte offset of element (row r, k) inside a K-major 32-byte-swizzled tile of
// 16-element rows: 16-byte chunk c of row r is stored at chunk c ^ (r / 4 % 2).
__host__ __device__ __forceinline__ uint32_t sw32_offset(int r, int ch) {
  return (uint32_t)(r * 32 + ((ch ^ ((r >> 2) & 1)) << 4));
}

// The overlap counts' start values, by the threads of a grid that precedes
// launch_exact_b.
__device__ __forceinline__ void ex_begin_counts(const ExactPrep& ex) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < ex_count_words(ex); i += gridDim.x * blockDim.x)
    ex.seg_min[i] = 0x7f7f7f7f;  // band_min follows it
}
__device__ __forceinline__ void ex_raise(const ExactPrep& ex) {
  *ex.flag = 1;
  if (ex.any) *ex.any = 1;
}

// The larger part of (re, im) over 2^e, rounded towards zero to 20 bits (|x| < 2^e;
// integer pipe).
__device__ __forceinline__ float ex_rel_mag(double re, double im, int e) {
  const int d = max(__double2hiint(re) & 0x7FFFFFFF, __double2hiint(im) & 0x7FFFFFFF);
  const int sh = 1023 + e - (d >> 20);
  return sh < 100 ? __uint_as_float(((unsigned)(127 - sh) << 23) | ((unsigned)(d & 0xFFFFF) << 3)) : 0.f;
}

// The S digits of x (|x| < 2^e; S = 6: of x 2^(52 - e), 7: x 2^(61 - e)) as
// 9-bit fields of one word, the field 9 (S - 1 - i) being digit i + 256: the
// balanced digits need no carries.  Round to nearest on the integer pipe (the
// FP64 pipe is 1/64 rate).
template <int S>
__device__ __forceinline__ unsigned long long ex_fields(double x, int e) {
  const unsigned long long bits = (unsigned long long)__double_as_longlong(x);
  const int ex = (int)(bits >> 52) & 0x7FF;
  const int sh = 1023 + e - ex;  // >= 1 as |x| < 2^e
  unsigned long long m = ((bits & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull) << (9 * (S - 6));
  m = sh > 63 || ex == 0 ? 0ull : ((m >> (sh - 1)) + 1) >> 1;
  const long long v = (long long)bits < 0 ? -(long long)m : (long long)m;
  constexpr unsigned long long kBias = 256ull * (((1ull << (9 * (S - 1))) - 1) / 511 + (1ull << (9 * (S - 1))));
  return (unsigned long long)v + kBias;
}
// Digit i of a field word as FP32 (exact).
template <int S>
__device__ __forceinline__ float ex_digit(unsigned long long f, int i) {
  const unsigned d = (unsigned)(f >> (9 * (S - 1 - i))) & 511u;
  return __uint_as_float(0x4B000000u | d) - 8388864.f;  // 2^23 + 256
}
// Digits i of two values as a BF16 pair (each exact in the upper half of FP32).
template <int S>
__device__ __forceinline__ uint32_t ex_pair(unsigned long long f0, unsigned long long f1, int i) {
  return __byte_perm(__float_as_uint(ex_digit<S>(f0, i)), __float_as_uint(ex_digit<S>(f1, i)), 0x7632);
}

// 16-byte digit chunks (8 K values of one row) of the slices.
template <int S>
struct ExChunk {
  uint4 s[S];
};
template <int S>
__device__ __forceinline__ ExChunk<S> ex_chunk(const double (&v)[8], int e) {
  ExChunk<S> c;
  unsigned long long f[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) f[j] = ex_fields<S>(v[j], e);
#pragma unroll
  for (int i = 0; i < S; ++i)
    c.s[i] = make_uint4(ex_pair<S>(f[0], f[1], i), ex_pair<S>(f[2], f[3], i), ex_pair<S>(f[4], f[5], i),
                        ex_pair<S>(f[6], f[7], i));
  return c;
}
template <int S>
__device__ __forceinline__ ExChunk<S> ex_negate(const ExChunk<S>& c) {
  ExChunk<S> n;
#pragma unroll
  for (int i = 0; i < S; ++i)
    n.s[i] = make_uint4(c.s[i].x ^ 0x80008000u, c.s[i].y ^ 0x80008000u, c.s[i].z ^ 0x80008000u, c.s[i].w ^ 0x80008000u);
  return n;
}
template <int S>
__device__ __forceinline__ void ex_store(unsigned char* tile, uint32_t slice_bytes, int r, int ch, const ExChunk<S>& c) {
  unsigned char* p = tile + sw32_offset(r, ch);
#pragma unroll
  for (int i = 0; i < S; ++i) *reinterpret_cast<uint4*>(p + i * slice_bytes) = c.s[i];
}
// The same for 8 values from a plane of doubles in shared memory (a factor
// pass's staging).
template <int S>
__device__ __forceinline__ void ex_put(unsigned char* tile, uint32_t slice_bytes, int r, int ch, const double* v, int e) {
  double x[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) x[j] = v[j];
  ex_store<S>(tile, slice_bytes, r, ch, ex_chunk<S>(x, e));
}

// The six digits of two values hi + lo (|lo| at most half an ulp of hi) in
// units of 2^(7 - e), for |hi| < 2^e: FP32 operations on both lanes of
// paired instructions.  Every step is exact but the last addition, which
// rounds at 2^-60 of 2^e (lo joins the third remainder by TwoSum; its
// rounding error, 2^-51, joins the fourth).  The second digit is rounded with lo
// in the remainder: beside a remainder of 1/2 lo would put the third at 257,
// which BF16 does not hold (a bit more room in e avoids that too, at twice the
// error of every product).  neg_scale = -2^(7 - e): the
// digits of the negated value come out negated, kM - (x + kM), without an
// instruction of their own.
__device__ __forceinline__ void ex_ff_digits(float2 hi, float2 lo, float neg_scale, float2 (&d)[6]) {
  const float2 kM = make_float2(12582912.f, 12582912.f);  // 1.5 * 2^23: adding it rounds to an integer
  const float2 k512 = make_float2(512.f, 512.f), m1 = make_float2(-1.f, -1.f);
  const float w0 = neg_scale * 262144.f;
  const float2 u = __fmul2_rn(hi, make_float2(neg_scale, neg_scale)), w = __fmul2_rn(lo, make_float2(w0, w0));
  d[0] = __ffma2_rn(__fadd2_rn(u, kM), m1, kM);
  float2 r = __fadd2_rn(u, d[0]);
  const float2 rw = __ffma2_rn(w, make_float2(1.f / 262144.f, 1.f / 262144.f), r);
  d[1] = __ffma2_rn(__ffma2_rn(rw, k512, kM), m1, kM);
  r = __ffma2_rn(r, k512, d[1]);
  d[2] = __ffma2_rn(__fadd2_rn(__ffma2_rn(r, k512, w), kM), m1, kM);
  r = __ffma2_rn(r, k512, d[2]);
  const float2 s = __fadd2_rn(r, w);
  const float2 bv = __ffma2_rn(r, m1, s), av = __ffma2_rn(bv, m1, s);
  const float2 e = __fadd2_rn(__ffma2_rn(av, m1, r), __ffma2_rn(bv, m1, w));
  d[3] = __ffma2_rn(__ffma2_rn(s, k512, kM), m1, kM);
  r = __ffma2_rn(e, k512, __ffma2_rn(s, k512, d[3]));
  d[4] = __ffma2_rn(__ffma2_rn(r, k512, kM), m1, kM);
  r = __ffma2_rn(r, k512, d[4]);
  d[5] = __ffma2_rn(__ffma2_rn(r, k512, kM), m1, kM);
}
__device__ __forceinline__ void ex_put_ff(unsigned char* tile, int r, int ch, const float2* hi, const float2* lo,
                                          float neg_scale) {
  unsigned char* p = tile + sw32_offset(r, ch);
  uint32_t w[6][4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float2 d[6];
    ex_ff_digits(hi[j], lo[j], neg_scale, d);
#pragma unroll
    for (int i = 0; i < 6; ++i) w[i][j] = __byte_perm(__float_as_uint(d[i].x), __float_as_uint(d[i].y), 0x7632);
  }
#pragma unroll
  for (int i = 0; i < 6; ++i)
    *reinterpret_cast<uint4*>(p + i * kExASlice) = make_uint4(w[i][0], w[i][1], w[i][2], w[i][3]);
}

}  // namespace sigma
