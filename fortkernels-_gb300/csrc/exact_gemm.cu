// Exact digit contraction (exact_gemm.cuh): operand checks and digits, the
// tcgen05 kernel, and the FP64 epilogue.
//
// The contraction kernel.  A CTA takes one (128 rows x 80 B' rows x K range; 64
// or 48 B' rows where they pad the bands less) item at a time.  Per 16-K tile
// the 21 digit products run as nine MMAs: the B slices are stacked along N, so
// A_i times [B_j .. B_k] fills the adjacent accumulators s = i + j .. i + k in
// one instruction (N up to 240), which reads A from shared memory once for up
// to three products (107 bytes per clock of the 128 available; one MMA per
// product would need 166).  TMEM holds the six accumulators (480 of 512
// columns).  They live 128 K values; the nine MMAs are issued as two groups (s
// = 0..2, then s = 3..5) over three, two and three tiles, so that one group's
// accumulators are read while the other group's products run: reading them
// costs 18 % of the kernel with pairs of tiles and eight reading warps, whose
// windows (the first group's products over two tiles) are too short, 15 % so.
// Sixteen drain warps convert the FP32 integers and add them to 64-bit integer
// sums (s <= 3) and FP32 sums (s = 4, 5) in registers, no FP64 operation (2 per
// clock per SM on this part); an item ends with its raw sums written out, and
// exact_finish_kernel forms the weighted FP64 sums.
//
// Measured: the kernel at 512 bands x 4914 rows x 65536 K' with the occupied
// rows 9.31 -> 8.93 ms with the longer windows, 8.45 ms with a
// leaner issue loop; the FF contraction of 512 x (15
// x 820) x 16384 in 12.4 ms, 555 ms with FP64 multiply-adds (ff_fp64.cu);
// normwise error 2.8e-15 (5e-15).
//
// Roles (608 threads): warps 0-15 drain, warp 16 streams 39 KB tiles (one bulk
// copy per operand) into a ring of five or six stages, warp 18 waits for the
// stages and the accumulators and releases warp 17, which issues the MMAs (the
// issuing thread polls no shared memory, which would stall the tensor pipe).
#include <algorithm>
#include <climits>
#include <cstring>

#include "exact_gemm.cuh"

namespace sigma {
namespace {

using namespace tma;

constexpr int kDrainWarps = 16;
constexpr int kCopyWarp = kDrainWarps, kIssueWarp = kDrainWarps + 1, kGateWarpEx = kDrainWarps + 2;
constexpr int kThreadsEx = (kDrainWarps + 3) * 32;
constexpr uint32_t ex_stage(int S, int cols) { return ex_a_bytes(S) + ex_b_bytes(S, cols); }  // 33 to 42 KB
// Stages of the ring: five, or six where they fit 227 KB (48 and 64 columns of six slices).
constexpr int ex_stages(int S, int cols) { return 6 * ex_stage(S, cols) + 1024 <= 227 * 1024 ? 6 : 5; }
constexpr uint32_t ex_smem(int S, int cols) { return ex_stages(S, cols) * ex_stage(S, cols) + 1024; }
constexpr int kBlockTiles = 8;  // K tiles per accumulator lifetime (128 K values),
// taken in groups of three, two and three tiles from tile s of an item on, or,
// where the ring holds too few for that (seven slices), in pairs
template <int S>
__device__ __forceinline__ int ex_group(int s, int nst) {
  const int n = S == 7 || s % kBlockTiles == 3 ? 2 : 3;
  return min(n, nst - s);
}

// 32-byte swizzle: rows of 16 elements (32 B), 8-row groups of 256 B (layout
// code 6 in bits 61-63).
__device__ __forceinline__ uint64_t sw32_desc(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr >> 4) & 0x3FFFu);
  d |= (uint64_t)1u << 16;
  d |= (uint64_t)(256u >> 4) << 32;
  d |= (uint64_t)1u << 46;
  d |= (uint64_t)6u << 61;
  return d;
}

__device__ __forceinline__ void arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// The gate and the issuing warp meet; the gate's failure flag is passed on.
__device__ __forceinline__ bool gate_sync(bool flag) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 q, %1, 0;\n\t"
      "bar.red.or.pred p, 2, 64, q;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(r)
      : "r"((uint32_t)flag)
      : "memory");
  return r != 0;
}

// W (8 or 4) consecutive TMEM columns of this warp's 32 lanes (no wait).
template <int W>
__device__ __forceinline__ void tmem_ld(uint32_t taddr, float (&v)[W]) {
  static_assert(W == 8 || W == 4, "columns per load");
  uint32_t r[W];
  if constexpr (W == 8)
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
  else
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(taddr)
                 : "memory");
#pragma unroll
  for (int i = 0; i < W; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

struct ExItem {
  int rb, cb, t0, nst;
  size_t pidx;
};
// Band blocks vary fastest (the CTAs of one time share A tiles), then the row
// blocks of one K split, the splits slowest.
__device__ __forceinline__ ExItem ex_decode(const ExactPrep& ex, int item) {
  ExItem t;
  const int main_items = ex.n_main_entries * ex.n_col_blocks;
  const bool main = item < main_items;
  const int i = main ? item : item - main_items, n = main ? ex.n_col_blocks : ex.n_col_blocks2;
  t.cb = i % n;
  const int4 e = ex.entries[(main ? 0 : ex.n_main_entries) + i / n];
  t.rb = e.x;
  t.t0 = e.z;
  t.nst = e.w;
  t.pidx = ex_block_index(ex, t.rb, t.cb) * ex.max_pieces + e.y;
  return t;
}

constexpr uint32_t idesc_n(int n) { return idesc_bf16_f32(128, n); }

// Columns Q .. Q + W of a drain: the lo accumulators (s = 0 .. 2) into the 64-bit
// sums, the hi ones (s = 3 on) into those and the FP32 sums.
template <int kCols, int Q, int W, int N>
__device__ __forceinline__ void drain_lo(uint32_t t, long long (&hi)[N]) {
  float v0[W], v1[W], v2[W];
  tmem_ld<W>(t + Q, v0);
  tmem_ld<W>(t + kCols + Q, v1);
  tmem_ld<W>(t + 2 * kCols + Q, v2);
  tmem_wait_ld();
#pragma unroll
  for (int i = 0; i < W; ++i) {
    // |v0| <= 2^21: its integer from the bits of v0 + 1.5 * 2^23 (a conversion
    // takes three to four issue slots' time)
    const int i0 = __float_as_int(v0[i] + 12582912.f) - 0x4B400000;
    const int u = i0 * 512 + __float2int_rn(v1[i]);  // below 2^31
    hi[Q + i] += (long long)u * (1 << 18) + (long long)__float2int_rn(v2[i]) * 512;
  }
}
template <int kHi, int kCols, int Q, int W, int N>
__device__ __forceinline__ void drain_hi(uint32_t t, long long (&hi)[N], float (&lo)[N]) {
  float v[kHi][W];
#pragma unroll
  for (int d = 0; d < kHi; ++d) tmem_ld<W>(t + (3 + d) * kCols + Q, v[d]);
  tmem_wait_ld();
#pragma unroll
  for (int i = 0; i < W; ++i) {
    hi[Q + i] += __float2int_rn(v[0][i]);
    float f = v[kHi - 1][i];
#pragma unroll
    for (int d = kHi - 2; d >= 1; --d) f = fmaf(f, 1.f / 512.f, v[d][i]);
    lo[Q + i] = fmaf(f, 1.f / 512.f, lo[Q + i]);
  }
}

template <int S, int kCols>
__global__ void __launch_bounds__(kThreadsEx, 1) exact_gemm_kernel(ExactPrep ex, int* status) {
  constexpr int kColsQ = kCols / 4, kStagesEx = ex_stages(S, kCols);
  constexpr int kHi = S - 3;                // accumulators from s = 3 on
  constexpr int kGroup = S == 7 ? 2 : 3;    // most tiles of ex_group (seven slices: always two)
  constexpr uint32_t kStage = ex_stage(S, kCols), kABytes = ex_a_bytes(S), kBBytes = ex_b_bytes(S, kCols),
                     kBSlice = ex_b_slice(kCols);
  static_assert(kCols % 16 == 0 && kColsQ >= 8 && kColsQ <= 20 && S * kCols <= 512 && kHi * kCols <= 256,
                "tensor memory and one MMA's width");
  extern __shared__ unsigned char smem_raw[];
  // full[5], empty[5], lo full, hi full, lo empty, hi empty, done
  __shared__ __align__(8) unsigned long long bars[2 * kStagesEx + 5];
  __shared__ uint32_t tmem_slot;
  chain_begin();
  // operands outside the split's range: the FP64 kernel runs instead (one
  // read for the CTA: another CTA may raise the flag below)
  if (__syncthreads_or(threadIdx.x == 0 && *ex.flag)) return;

  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t sbase = (raw + 1023u) & ~1023u;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t full0 = smem_u32(&bars[0]), empty0 = smem_u32(&bars[kStagesEx]);
  const uint32_t accf = smem_u32(&bars[2 * kStagesEx]), acce = smem_u32(&bars[2 * kStagesEx + 2]);
  const uint32_t done0 = smem_u32(&bars[2 * kStagesEx + 4]);

  if (warp == 0) tmem_alloc(smem_u32(&tmem_slot), 512);
  if (tid == 0) {
    for (int i = 0; i < 2 * kStagesEx + 2; ++i) mbar_init(smem_u32(&bars[i]), 1);
    mbar_init(acce, kDrainWarps);
    mbar_init(acce + 8u, kDrainWarps);
    mbar_init(done0, 1);
    fence_mbar_init();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;

  if (warp == kCopyWarp) {
    if (lane == 0) {
      uint32_t g = 0;  // tiles issued by this CTA
      bool ok = true;
      for (int item = blockIdx.x; ok && item < ex.n_items; item += gridDim.x) {
        const ExItem it = ex_decode(ex, item);
        const size_t kts = (size_t)ex.halves * ex.kt;
        const unsigned char* a = ex.a_tiles + ((size_t)it.rb * kts + it.t0) * kABytes;
        const unsigned char* b = ex.b_tiles + ((size_t)it.cb * kts + it.t0) * kBBytes;
        for (int s = 0; s < it.nst; ++s, ++g) {
          const uint32_t st = g % kStagesEx, use = g / kStagesEx;
          if (use > 0 && !mbar_wait(empty0 + 8u * st, (use - 1) & 1u, status)) {
            ok = false;
            break;
          }
          const uint32_t bar = full0 + 8u * st, dst = sbase + st * kStage;
          mbar_expect_tx(bar, kStage);
          bulk_load(dst, a + (size_t)s * kABytes, kABytes, bar);
          bulk_load(dst + kABytes, b + (size_t)s * kBBytes, kBBytes, bar);
        }
      }
      // the last copies land before the CTA ends, also when another warp's wait
      // gave up and nothing consumes them
      for (uint32_t t = g > (uint32_t)kStagesEx ? g - kStagesEx : 0u; t < g; ++t)
        mbar_wait_own(full0 + 8u * (t % kStagesEx), (t / kStagesEx) & 1u);
    }
    __syncwarp();
  } else if (warp == kGateWarpEx) {
    // per group of tiles: its stages full; at a block's first group also the
    // lo accumulators drained, and (second meeting) the hi accumulators
    bool failed = false;
    uint32_t g = 0, blk = 0;  // tiles and accumulator lifetimes so far
    for (int item = blockIdx.x; item < ex.n_items; item += gridDim.x) {
      const int nst = ex_decode(ex, item).nst;
      for (int s = 0, n; s < nst; s += n, g += n) {
        n = ex_group<S>(s, nst);
        const bool first = s % kBlockTiles == 0;
        if (lane == 0 && !failed) {
          if (first && blk > 0) failed = !mbar_wait(acce, (blk - 1) & 1u, status);
          for (uint32_t t = g; t < g + n && !failed; ++t)
            failed = !mbar_wait(full0 + 8u * (t % kStagesEx), (t / kStagesEx) & 1u, status);
        }
        __syncwarp();
        gate_sync(failed);
        if (first) {
          if (lane == 0 && !failed && blk > 0) failed = !mbar_wait(acce + 8u, (blk - 1) & 1u, status);
          __syncwarp();
          gate_sync(failed);
          ++blk;
        }
      }
    }
    // the last lifetime drained
    if (lane == 0 && !failed && blk > 0) {
      mbar_wait(acce, (blk - 1) & 1u, status);
      mbar_wait(acce + 8u, (blk - 1) & 1u, status);
    }
    __syncwarp();
  } else if (warp == kIssueWarp) {
    uint32_t st0 = 0;  // ring stage of the next tile
    bool failed = false;
    for (int item = blockIdx.x; item < ex.n_items; item += gridDim.x) {
      const int nst = ex_decode(ex, item).nst;
      for (int s = 0, n; s < nst; s += n) {
        n = ex_group<S>(s, nst);
        const bool first = s % kBlockTiles == 0;
        const bool last = (s + n) % kBlockTiles == 0 || s + n >= nst;
        failed = gate_sync(false) || failed;
        // the group's tiles: stage and descriptors of the first slices (slices
        // follow at constant distances in the address field), formed by the
        // whole warp: inside the single lane's branch they are not uniform
        // and each instruction waits for its operands' moves (8.80 -> 8.45 ms
        // at 512 bands, seven slices 16.5 -> 15.4 ms)
        uint32_t st[kGroup];
        uint64_t da[kGroup], db[kGroup];
#pragma unroll
        for (int q = 0; q < kGroup; ++q) {
          st[q] = st0 + q < (uint32_t)kStagesEx ? st0 + q : st0 + q - kStagesEx;
          da[q] = sw32_desc(sbase + st[q] * kStage);
          db[q] = da[q] + (kABytes >> 4);
        }
        st0 += n;
        if (st0 >= (uint32_t)kStagesEx) st0 -= kStagesEx;
        if (lane == 0 && !failed) {
          tc_fence_after();
#pragma unroll
          for (int q = 0; q < kGroup; ++q) {
            if (kGroup > 2 && q >= n) break;
            mma_f16(tmem, da[q], db[q], idesc_n(3 * kCols), first && q == 0 ? 0u : 1u);
            mma_f16(tmem + kCols, da[q] + (kExASlice >> 4), db[q], idesc_n(2 * kCols), 1u);
            mma_f16(tmem + 2 * kCols, da[q] + (2 * kExASlice >> 4), db[q], idesc_n(kCols), 1u);
          }
          if (last) mma_commit(accf);
        }
        __syncwarp();
        if (first) failed = gate_sync(false) || failed;
        if (lane == 0 && !failed) {
          tc_fence_after();
          const uint32_t d = tmem + 3 * kCols;
#pragma unroll
          for (int q = 0; q < kGroup; ++q) {
            if (kGroup > 2 && q >= n) break;
            // A_i times the B slices j with 3 <= i + j < S
#pragma unroll
            for (int i = 0; i < S; ++i) {
              const int j0 = i < 3 ? 3 - i : 0, w = S - i - j0;
              mma_f16(d + (i + j0 - 3) * kCols, da[q] + (i * kExASlice >> 4), db[q] + (j0 * kBSlice >> 4),
                      idesc_n(w * kCols), first && q == 0 && i == 0 ? 0u : 1u);
            }
            mma_commit(empty0 + 8u * st[q]);
          }
          if (last) mma_commit(accf + 8u);
        }
        __syncwarp();
      }
    }
    // the MMAs issued end before the tensor memory is released, also when the
    // wait of a warp that reads them gave up
    if (lane == 0) {
      mma_commit(done0);
      mbar_wait_own(done0, 0);
    }
    __syncwarp();
  } else {
    const int quarter = warp >> 2, row = (warp & 3) * 32 + lane;
    const uint32_t tl = tmem + ((uint32_t)((warp & 3) * 32) << 16) + quarter * kColsQ;
    uint32_t blk = 0;
    for (int item = blockIdx.x; item < ex.n_items; item += gridDim.x) {
      const ExItem it = ex_decode(ex, item);
      long long hi[kColsQ];
      float lo[kColsQ];
#pragma unroll
      for (int i = 0; i < kColsQ; ++i) {
        hi[i] = 0;
        lo[i] = 0.f;
      }
      const int nblk = (it.nst + kBlockTiles - 1) / kBlockTiles;
#pragma unroll 1
      for (int c = 0; c < nblk; ++c, ++blk) {
        mbar_wait(accf, blk & 1u, status);
        tc_fence_after();
        drain_lo<kCols, 0, 8>(tl, hi);
        if constexpr (kColsQ >= 16) drain_lo<kCols, 8, 8>(tl, hi);
        if constexpr (kColsQ % 8 == 4) drain_lo<kCols, kColsQ - 4, 4>(tl, hi);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) arrive(acce);
        mbar_wait(accf + 8u, blk & 1u, status);
        tc_fence_after();
        drain_hi<kHi, kCols, 0, 8>(tl, hi, lo);
        if constexpr (kColsQ >= 16) drain_hi<kHi, kCols, 8, 8>(tl, hi, lo);
        if constexpr (kColsQ % 8 == 4) drain_hi<kHi, kCols, kColsQ - 4, 4>(tl, hi, lo);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) arrive(acce + 8u);
      }
      const size_t base = (it.pidx * kCols + quarter * kColsQ) * kExRows + row;
#pragma unroll
      for (int i = 0; i < kColsQ; ++i) {
        ex.raw_hi[base + (size_t)i * kExRows] = hi[i];
        ex.raw_lo[base + (size_t)i * kExRows] = lo[i];
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  // a wait gave up: the sums are incomplete, the FP64 kernels form them
  if (tid == 0 && status_set(status)) ex_raise(ex);
  if (warp == 0) tmem_dealloc(tmem, 512);
}

// ---------------------------------------------------------------- operand checks
// Magnitude bits (upper word without sign) of a value's larger part.
template <bool kReal>
__device__ __forceinline__ unsigned ex_mag(const int2* v, size_t k, unsigned& low) {
  if (kReal) {
    const int2 d = v[k];
    low = (unsigned)d.x;
    return (unsigned)d.y & 0x7FFFFFFFu;
  }
  const int4 d = reinterpret_cast<const int4*>(v)[k];
  low = (unsigned)(d.x | d.z);
  return max((unsigned)d.y & 0x7FFFFFFFu, (unsigned)d.w & 0x7FFFFFFFu);
}

// One CTA per row of values: its exponent (largest part below 2^e) and, per
// 512-value segment, how many of its first 128 elements are large.  Bands (kB)
// lower seg_min to their counts;
// A rows add up how many large elements must coincide with large elements of
// every band and raise the flag when they are too few.  Zero rows are exact
// and pass.
template <bool kB, bool kReal>
__global__ void __launch_bounds__(256) exact_stats_kernel(ExactPrep ex, const void* x0, int n0, const void* x1,
                                                          int nc) {
  __shared__ unsigned s_max[8];
  __shared__ int s_sum[8];
  chain_begin();
  const int row = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int2* v = static_cast<const int2*>(row < n0 ? x0 : x1) + (size_t)(row < n0 ? row : row - n0) * nc * (kReal ? 1 : 2);
  unsigned m = 0, any = 0;
  for (int k = tid; k < nc; k += 256) {
    unsigned low;
    m = max(m, ex_mag<kReal>(v, k, low));
    any |= low;
  }
  if (any) m = max(m, 1u);
  m = __reduce_max_sync(0xffffffffu, m);
  if (lane == 0) s_max[warp] = m;
  __syncthreads();
  m = s_max[0];
#pragma unroll
  for (int i = 1; i < 8; ++i) m = max(m, s_max[i]);
  const int exm = (int)(m >> 20);
  if (tid == 0) {
    (kB ? ex.eb : ex.ea)[row] = m ? exm - 1022 : kExZeroRow;
    if (m && (exm < 1023 - 400 || exm > 1023 + 400)) ex_raise(ex);
  }
  if (m == 0) return;
  const unsigned thr = (unsigned)max(exm - (kB ? kExSlackB : kExSlackA), 1) << 20;
  int sum = 0;
  for (int s = warp; s < ex.n_kseg; s += 8) {
    int c = 0;
    const int k1 = min(nc, s * kExSeg + kExCount);  // the counted part
    for (int k = s * kExSeg + lane; k < k1; k += 32) {
      unsigned low;
      c += ex_mag<kReal>(v, k, low) >= thr ? 1 : 0;
    }
    c = __reduce_add_sync(0xffffffffu, c);
    if (lane == 0) {
      if (kB) {
        atomicMin(&ex.seg_min[s], c);
      } else {
        sum += max(0, c + min(ex.seg_min[s], kExCount) - min(kExCount, nc - s * kExSeg));
      }
    }
  }
  if (kB) return;
  if (lane == 0) s_sum[warp] = sum;
  __syncthreads();
  if (tid == 0) {
    int t = 0;
    for (int i = 0; i < 8; ++i) t += s_sum[i];
    if ((long long)t * kExOverlap < nc) ex_raise(ex);
  }
}

// ---------------------------------------------------------------- digits
// Element t: (row block, K tile pair, row, 8-value chunk of the 32 K values).
__global__ void __launch_bounds__(256) exact_slice_a_kernel(ExactPrep ex, const double2* a, int rows, int nc) {
  constexpr int S = 6;
  chain_begin();
  if (*ex.flag) return;
  const int pairs = ex.kt / 2;
  const long long total = (long long)ex.n_row_blocks * pairs * kExRows * 4;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    const int ch = (int)(t & 3), r = (int)(t >> 2) & (kExRows - 1);
    const long long rest = t / (4 * kExRows);
    const int kp = (int)(rest % pairs), rb = (int)(rest / pairs);
    if (2 * kp >= ex.kt_lim[rb]) continue;  // zero tiles, not read by the contraction
    const int R = rb * kExRows + r, k0 = kp * 32 + ch * 8;
    double re[8], im[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const double2 d = R < rows && k0 + j < nc ? a[(size_t)R * nc + k0 + j] : make_double2(0.0, 0.0);
      re[j] = d.x;
      im[j] = d.y;
    }
    const int e = R < rows ? ex.ea[R] : kExZeroRow;
    unsigned char* tile = ex.a_tiles + ((size_t)rb * 2 * ex.kt + 2 * kp + (ch >> 1)) * ex_a_bytes(S);
    ex_store<S>(tile, kExASlice, r, ch & 1, ex_chunk<S>(re, e));
    ex_store<S>(tile + (size_t)ex.kt * ex_a_bytes(S), kExASlice, r, ch & 1, ex_chunk<S>(im, e));
  }
}

template <int S, int kCols, bool kReal>
__global__ void __launch_bounds__(256) exact_slice_b_kernel(ExactPrep ex, const void* b0, int nb0, const void* b1,
                                                            int nb, int nc) {
  chain_begin();
  if (*ex.flag) return;
  constexpr int kW = kReal ? 1 : 2, kBands = kReal ? kCols : kCols / 2;
  constexpr uint32_t kSlice = ex_b_slice(kCols), kBytes = ex_b_bytes(S, kCols);
  const int pairs = ex.kt / 2;
  const long long total = (long long)ex.n_col_blocks * pairs * kBands * 4;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    const int ch = (int)(t & 3), nl = (int)((t >> 2) % kBands);
    const long long rest = t / (4 * kBands);
    const int kp = (int)(rest % pairs), cb = (int)(rest / pairs);
    const int n = cb * kBands + nl, k0 = kp * 32 + ch * 8;
    const double* src =
        static_cast<const double*>(n < nb0 ? b0 : b1) + ((size_t)(n < nb0 ? n : n - nb0) * nc + k0) * kW;
    double re[8], im[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      re[j] = im[j] = 0.0;
      if (n < nb && k0 + j < nc) {
        if (kReal) {
          re[j] = src[j];
        } else {
          const double2 d = reinterpret_cast<const double2*>(src)[j];
          re[j] = d.x;
          im[j] = d.y;
        }
      }
    }
    const int e = n < nb ? ex.eb[n] : kExZeroRow;
    if constexpr (S == 7 && !kReal) {
      // band_min: the warp's eight bands first (its lanes are 4 chunks x 8
      // bands of one band block and K tile pair); a band of zeros is exact
      static_assert(kBands % 8 == 0, "whole warps in a band block");
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float m = e == kExZeroRow ? INFINITY : ex_rel_mag(re[j], im[j], e);
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) m = fminf(m, __shfl_xor_sync(0xffffffffu, m, o));
        if ((threadIdx.x & 31) < 4) atomicMin(reinterpret_cast<int*>(&ex.band_min[k0 + j]), __float_as_int(m));
      }
    }
    unsigned char* tile = ex.b_tiles + ((size_t)cb * ex.halves * ex.kt + 2 * kp + (ch >> 1)) * kBytes;
    const ExChunk<S> cr = ex_chunk<S>(re, e);
    if (kReal) {
      ex_store<S>(tile, kSlice, nl, ch & 1, cr);
      continue;
    }
    unsigned char* upper = tile + (size_t)ex.kt * kBytes;  // K' >= K
    const ExChunk<S> ci = ex_chunk<S>(im, e);
    ex_store<S>(tile, kSlice, 2 * nl, ch & 1, cr);
    ex_store<S>(tile, kSlice, 2 * nl + 1, ch & 1, ci);
    ex_store<S>(upper, kSlice, 2 * nl, ch & 1, ex_negate<S>(ci));
    ex_store<S>(upper, kSlice, 2 * nl + 1, ch & 1, cr);
  }
}

// ---------------------------------------------------------------- epilogue
// (hi + lo) 2^(e - 41): the 64-bit sum and the FP32 tail in FP64.
__device__ __forceinline__ double ex_value(long long hi, double lo, int e) {
  return scalbn((double)hi + lo, e - 41);
}

// Epilogue weights: conj(aqsm[n][igp]) times the column weight.  With
// pair_bands set (the half sum's second band set), bands from pair_bands on
// take band n - pair_bands, and in the last frequency aqsn's.
__device__ __forceinline__ double2 ex_weight(const FfDev& p, int n, int f, int igp) {
  const bool second = p.pair_bands > 0 && n >= p.pair_bands;
  const double2* m = second && f == p.nf - 1 && p.pair_static ? p.aqsn : p.aqsm;
  return m[(size_t)(second ? n - p.pair_bands : n) * p.nc + igp];
}

// One CTA per (row block, pair of bands): tempz of 128 rows x 2 bands from the
// pieces' raw sums (added as integers, so their order does not matter), times weight * conj(aqsm[n1][igp]), summed over the rows of each
// frequency in a fixed order.
constexpr int kFinRow = kExRows + 1, kFinThreads = 256, kFinBands = 2;
template <bool kReal>
__global__ void __launch_bounds__(kFinThreads) exact_finish_kernel(FfDev p, ExactPrep ex, ExSecond p2) {
  constexpr int kBands = kFinBands;
  const int kCols = ex.cols, b0 = blockIdx.z * kBands;  // bands b0 and b0 + 1 of the block
  __shared__ double2 s_prod[kBands * kFinRow];  // complex, or real
  double* s_real = reinterpret_cast<double*>(s_prod);
  chain_begin();
  if (*ex.flag) return;
  // row block rb of the group whose row blocks start at rb0
  const bool first = (int)blockIdx.x < ex.n_main_blocks;
  const int rb0 = first ? 0 : ex.n_main_blocks, nf = first ? p.nf : p2.nf, nb = first ? p.nb : p2.nb;
  const int rb = (int)blockIdx.x - rb0, cb = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (!first && cb >= ex.n_col_blocks2) return;
  if (!first) p.vfac = p2.vfac;
  const int rows = nf * p.ng, r = tid & (kExRows - 1), R = rb * kExRows + r;
  const size_t block = ex_block_index(ex, rb0 + rb, cb);
  const int f = R / p.ng, igp = R < rows ? p.igp_of[R % p.ng] : -1;
  const double wgt = ff_column_weight(p, igp);
  const int e_row = R < rows ? ex.ea[rb0 * kExRows + R] : 0, np = ex.pieces[rb0 + rb];
  const size_t base = block * ex.max_pieces * kCols * kExRows + r;
  static_assert(kFinThreads == kBands * kExRows, "one thread per row and band");
  {
    const int b = tid >> 7;
    const int n = cb * ex.bands + b0 + b;
    double2 v = make_double2(0.0, 0.0);
    if (igp >= 0 && n < nb) {
      long long hr = 0, hi = 0;
      double lr = 0.0, li = 0.0;
#pragma unroll 8
      for (int q = 0; q < np; ++q) {
        const size_t o = base + ((size_t)q * kCols + (kReal ? b0 + b : 2 * (b0 + b))) * kExRows;
        hr += ex.raw_hi[o];
        lr += ex.raw_lo[o];
        if (!kReal) {
          hi += ex.raw_hi[o + kExRows];
          li += ex.raw_lo[o + kExRows];
        }
      }
      const int e = e_row + ex.eb[n];
      const double zr = ex_value(hr, lr, e);
      if (kReal) {
        v.x = zr * reinterpret_cast<const double*>(p.aqsm)[(size_t)n * p.nc + igp] * wgt;
      } else {
        const double zi = ex_value(hi, li, e);
        const double2 m = ex_weight(p, n, f, igp);
        v = make_double2((zr * m.x + zi * m.y) * wgt, (zi * m.x - zr * m.y) * wgt);
      }
    }
    if (kReal)
      s_real[b * kFinRow + r] = v.x;
    else
      s_prod[b * kFinRow + r] = v;
  }
  __syncthreads();
  const int f0 = rb * kExRows / p.ng, f1 = (min((rb + 1) * kExRows, rows) - 1) / p.ng;
  for (int o = warp; o < kBands * (f1 - f0 + 1); o += kFinThreads / 32) {
    const int b = o % kBands, fo = f0 + o / kBands;
    const int lo = max(fo * p.ng - rb * kExRows, 0), hi = min((fo + 1) * p.ng - rb * kExRows, kExRows);
    double sx = 0.0, sy = 0.0, tx = 0.0, ty = 0.0;
    for (int q = lo + lane; q < hi; q += 32) {
      const double2 v = kReal ? make_double2(s_real[b * kFinRow + q], 0.0) : s_prod[b * kFinRow + q];
      sx += v.x;
      sy += v.y;
      if (p.vcoul2) {
        const int ig2 = p.igp_of[(rb * kExRows + q) % p.ng];
        const double w2 = ig2 >= 0 ? p.vfac2 * p.vcoul2[ig2] : 0.0;
        tx += v.x * w2;
        ty += v.y * w2;
      }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
      sx += __shfl_xor_sync(0xffffffffu, sx, d);
      sy += __shfl_xor_sync(0xffffffffu, sy, d);
      if (p.vcoul2) {
        tx += __shfl_xor_sync(0xffffffffu, tx, d);
        ty += __shfl_xor_sync(0xffffffffu, ty, d);
      }
    }
    if (lane == 0) {
      const size_t i = (block * ex.max_seg + (fo - f0)) * ex.bands + b0 + b;
      ex.partial[i] = make_double2(sx, sy);
      if (p.vcoul2) ex.partial2[i] = make_double2(tx, ty);
    }
  }
}

// out[n][f], then out2, then the second group's: eight lanes per entry,
// fixed-order compensated sum over the row blocks (a warp per entry took 8 us
// even for a few hundred entries: 80 FP64 operations a warp, at two lanes per
// clock).
constexpr int kRedThreads = 64, kRedLanes = 8;
__global__ void __launch_bounds__(kRedThreads) exact_reduce_kernel(FfDev p, ExactPrep ex, ExSecond p2, double2* out,
                                                                   double2* out2) {
  chain_begin();
  if (*ex.flag) return;
  const int lane = threadIdx.x % kRedLanes, w = (blockIdx.x * kRedThreads + threadIdx.x) / kRedLanes;
  const int n1 = p.nb * p.nf, n2 = out2 ? n1 : 0, n3 = p2.out ? p2.nb * p2.nf : 0;
  const bool second = w >= n1 + n2, extra = !second && w >= n1;
  const int e = second ? w - n1 - n2 : extra ? w - n1 : w, nf = second ? p2.nf : p.nf;
  const int n = e / nf, f = e % nf, cb = n / ex.bands, b = n % ex.bands, rb0 = second ? ex.n_main_blocks : 0;
  const int lo = f * p.ng / kExRows, hi = w < n1 + n2 + n3 ? ((f + 1) * p.ng - 1) / kExRows : -1;
  const double2* partial = extra ? ex.partial2 : ex.partial;
  Comp sx, sy;
  for (int rb = lo + lane; rb <= hi; rb += kRedLanes) {
    const double2 v = partial[(ex_block_index(ex, rb0 + rb, cb) * ex.max_seg + (f - rb * kExRows / p.ng)) * ex.bands + b];
    sx.add(v.x);
    sy.add(v.y);
  }
  const double x = lanes_sum_comp<kRedLanes>(sx), y = lanes_sum_comp<kRedLanes>(sy);
  if (lane == 0 && hi >= 0) (second ? p2.out : extra ? out2 : out)[(size_t)n * nf + f] = make_double2(x, y);
}

size_t up256(size_t v) { return (v + 255) / 256 * 256; }

struct ExSizes {
  size_t a, b, ea, eb, seg, hi, lo, part;  // work
  size_t flag, ent, pcs;                   // own
};
ExSizes ex_sizes(const ExactPrep& ex) {
  ExSizes z;
  const size_t kts = (size_t)ex.halves * ex.kt;
  const size_t blocks = ex_block_index(ex, ex.n_row_blocks, 0);
  const size_t slots = blocks * ex.max_pieces * ex.cols * kExRows;
  z.a = up256((size_t)ex.n_row_blocks * kts * ex_a_bytes(ex.slices));
  z.b = up256((size_t)ex.n_col_blocks * kts * ex_b_bytes(ex.slices, ex.cols));
  z.ea = up256(sizeof(int) * (size_t)ex.n_row_blocks * kExRows);
  z.eb = up256(sizeof(int) * (size_t)ex.n_col_blocks * ex.bands);
  z.seg = up256(sizeof(int) * (size_t)ex_count_words(ex));
  z.hi = up256(sizeof(long long) * slots);
  z.lo = up256(sizeof(float) * slots);
  z.part = up256(sizeof(double2) * blocks * ex.max_seg * ex.bands);
  z.flag = 256;
  z.ent = up256(sizeof(int4) * (size_t)std::max(ex.n_entries, 1));
  z.pcs = up256(sizeof(int) * (size_t)ex.n_row_blocks);
  return z;
}

}  // namespace

// B' rows per column block.  A narrower block's MMAs take less time but read A
// from shared memory as often: 620, 530 and 480 us per block of 80, 64 and
// 48 rows at 4914 A rows x 65536 K' (DRAM-bound below).  The fewest padded rows
// win mostly where the number of blocks stays: 128 bands take four blocks of
// 64, 2.11 ms there, 2.5 in four of 80; 72 bands two of 80, 1.24 ms, 1.44 in
// three of 48.
int ex_pick_cols(int S, int b_rows) {
  if (S != 6) return ex_max_cols(S);
  int best = 80;
  long long cost = LLONG_MAX;
  for (const int c : {80, 64, 48}) {
    const long long t = (long long)((b_rows + c - 1) / c) * (c == 80 ? 620 : c == 64 ? 530 : 480);
    if (t < cost) {
      cost = t;
      best = c;
    }
  }
  return best;
}

void exact_size(ExactPrep& ex, int slices, int nb, int nc, int ng, int nf, bool cplx, int grid, const int* row_kend,
                ExactTables* tables, int nf2, int nb2) {
  const int rows = nf * ng;
  ex.halves = cplx ? 2 : 1;
  ex.slices = slices;
  ex.cols = ex_pick_cols(slices, (cplx ? 2 : 1) * nb);
  ex.bands = cplx ? ex.cols / 2 : ex.cols;
  ex.kt = (nc + 31) / 32 * 2;
  ex.n_main_blocks = (rows + kExRows - 1) / kExRows;
  ex.n_row_blocks = ex.n_main_blocks + (nf2 * ng + kExRows - 1) / kExRows;
  ex.n_col_blocks = (nb + ex.bands - 1) / ex.bands;
  ex.n_col_blocks2 = (nb2 + ex.bands - 1) / ex.bands;
  ex.max_seg = (kExRows + ng - 2) / ng + 1;
  ex.n_kseg = (nc + kExSeg - 1) / kExSeg;
  std::vector<int> kl(ex.n_row_blocks, ex.kt);
  for (int rb = 0; rb < ex.n_main_blocks && row_kend; ++rb) {
    int k = 0;
    for (int r = rb * kExRows; r < std::min(rows, (rb + 1) * kExRows); ++r) k = std::max(k, std::min(row_kend[r], nc));
    kl[rb] = (k + 31) / 32 * 2;
  }
  // K splits: the count whose slowest CTA is done first.  An item costs its
  // tiles plus about 6 tiles' time for its raw sums and the ring's refill, a
  // piece about one tile's time in the epilogue.  Items of one length take
  // ceil(items / grid) turns; ragged ones (row limits) are dealt out as the
  // kernel's static schedule does.
  const int all = ex.halves * ex.kt;
  const long long blocks = (long long)ex_block_index(ex, ex.n_row_blocks, 0);
  long long best = LLONG_MAX;
  int splits = 1;
  for (int s = 1; s <= std::min(all / 2, 96); s += row_kend && s >= 8 ? s / 4 : 1) {
    const int len = (all / 2 + s - 1) / s * 2;
    long long cost = 0;
    if (!row_kend) {
      cost = (blocks * s + grid - 1) / grid * (len + 6LL) + s;
    } else {
      std::vector<int4> ent;
      std::vector<int> pieces;
      k_entries(ex.n_main_blocks, ex.halves, ex.kt, len, (all + len - 1) / len, kl, ent, pieces);
      std::vector<long long> load(grid, 0);
      long long i = 0;
      for (const int4& e : ent)
        for (int c = 0; c < ex.n_col_blocks; ++c, ++i) load[i % grid] += e.w + 6;
      cost = *std::max_element(load.begin(), load.end()) + *std::max_element(pieces.begin(), pieces.end());
    }
    if (cost < best) {
      best = cost;
      splits = s;
    }
  }
  ex.split_tiles = (all / 2 + splits - 1) / splits * 2;
  ex.n_splits = (all + ex.split_tiles - 1) / ex.split_tiles;
  std::vector<int4> ent, ent2;
  std::vector<int> pieces, pieces2;
  k_entries(ex.n_main_blocks, ex.halves, ex.kt, ex.split_tiles, ex.n_splits, kl, ent, pieces);
  k_entries(ex.n_row_blocks - ex.n_main_blocks, ex.halves, ex.kt, ex.split_tiles, ex.n_splits,
            std::vector<int>(kl.begin() + ex.n_main_blocks, kl.end()), ent2, pieces2);
  ex.n_main_entries = (int)ent.size();
  for (int4 e : ent2) ent.push_back(make_int4(e.x + ex.n_main_blocks, e.y, e.z, e.w));
  pieces.insert(pieces.end(), pieces2.begin(), pieces2.end());
  ex.n_entries = (int)ent.size();
  ex.n_items = ex.n_main_entries * ex.n_col_blocks + (ex.n_entries - ex.n_main_entries) * ex.n_col_blocks2;
  ex.max_pieces = std::max(1, *std::max_element(pieces.begin(), pieces.end()));
  if (tables) {
    tables->entries = std::move(ent);
    tables->pieces = std::move(pieces);
    tables->kt_lim = std::move(kl);
  }
}

size_t exact_work_bytes(const ExactPrep& ex) {
  const ExSizes z = ex_sizes(ex);
  return z.a + z.b + z.ea + z.eb + z.seg + z.hi + z.lo + 2 * z.part + 1024;
}
size_t exact_own_bytes(const ExactPrep& ex) {
  const ExSizes z = ex_sizes(ex);
  return z.flag + z.ent + 2 * z.pcs;
}

void exact_bind(ExactPrep& ex, void* work, void* own) {
  const ExSizes z = ex_sizes(ex);
  char* p = nullptr;
  auto from = [&](void* base, uintptr_t align) {
    p = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(base) + align - 1) & ~(align - 1));
  };
  auto take = [&](size_t bytes) {
    char* q = p;
    p += bytes;
    return q;
  };
  from(work, 1024);
  ex.a_tiles = reinterpret_cast<unsigned char*>(take(z.a));
  ex.b_tiles = reinterpret_cast<unsigned char*>(take(z.b));
  ex.ea = reinterpret_cast<int*>(take(z.ea));
  ex.eb = reinterpret_cast<int*>(take(z.eb));
  ex.seg_min = reinterpret_cast<int*>(take(z.seg));
  ex.band_min = reinterpret_cast<float*>(ex.seg_min + ex.n_kseg);
  ex.raw_hi = reinterpret_cast<long long*>(take(z.hi));
  ex.raw_lo = reinterpret_cast<float*>(take(z.lo));
  ex.partial = reinterpret_cast<double2*>(take(z.part));
  ex.partial2 = reinterpret_cast<double2*>(take(z.part));
  from(own, 256);
  ex.flag = reinterpret_cast<int*>(take(z.flag));
  ex.entries = reinterpret_cast<const int4*>(take(z.ent));
  ex.pieces = reinterpret_cast<const int*>(take(z.pcs));
  ex.kt_lim = reinterpret_cast<const int*>(take(z.pcs));
  ex.any = nullptr;
}

void exact_pack_own(const ExactPrep& ex, const ExactTables& t, char* host) {
  const ExSizes z = ex_sizes(ex);
  std::memset(host, 0, z.flag);
  host += z.flag;
  if (!t.entries.empty()) std::memcpy(host, t.entries.data(), sizeof(int4) * t.entries.size());
  std::memcpy(host + z.ent, t.pieces.data(), sizeof(int) * t.pieces.size());
  std::memcpy(host + z.ent + z.pcs, t.kt_lim.data(), sizeof(int) * t.kt_lim.size());
}
cudaError_t exact_upload_tables(const ExactPrep& ex, const ExactTables& t) {
  std::vector<char> host(exact_own_bytes(ex));
  exact_pack_own(ex, t, host.data());
  // own begins 256 bytes, the flag's, before its first table
  return cudaMemcpy(const_cast<char*>(reinterpret_cast<const char*>(ex.entries)) - 256, host.data(), host.size(),
                    cudaMemcpyHostToDevice);
}

cudaError_t exact_begin_flag(const ExactPrep& ex, cudaStream_t s) {
  return cudaMemsetAsync(ex.flag, 0, sizeof(int), s);
}
cudaError_t exact_begin(const ExactPrep& ex, cudaStream_t s) {
  cudaError_t e = exact_begin_flag(ex, s);
  if (e != cudaSuccess) return e;
  return cudaMemsetAsync(ex.seg_min, 0x7f, sizeof(int) * (size_t)ex_count_words(ex), s);
}

cudaError_t launch_exact_b(const ExactPrep& ex, const void* b0, int nb0, const void* b1, int nb1, int nc,
                           cudaStream_t s) {
  const int nb = nb0 + nb1;
  const bool real = ex.halves == 1;
  auto* stats = real ? exact_stats_kernel<true, true> : exact_stats_kernel<true, false>;
  cudaError_t e = launch_chained(stats, nb, 256, 0, s, true, ex, b0, nb0, b1, nc);
  if (e != cudaSuccess) return e;
  auto* slice = exact_slice_b_kernel<6, 80, false>;
  if (ex.slices == 7)
    slice = real ? exact_slice_b_kernel<7, 64, true> : exact_slice_b_kernel<7, 64, false>;
  else if (ex.cols == 80)
    slice = real ? exact_slice_b_kernel<6, 80, true> : exact_slice_b_kernel<6, 80, false>;
  else if (ex.cols == 64)
    slice = real ? exact_slice_b_kernel<6, 64, true> : exact_slice_b_kernel<6, 64, false>;
  else
    slice = real ? exact_slice_b_kernel<6, 48, true> : exact_slice_b_kernel<6, 48, false>;
  return launch_chained(slice, 152 * 8, 256, 0, s, true, ex, b0, nb0, b1, nb, nc);
}

cudaError_t launch_exact_a(const ExactPrep& ex, const double2* a, int rows, int nc, cudaStream_t s) {
  cudaError_t e = launch_chained(exact_stats_kernel<false, false>, rows, 256, 0, s, true, ex, a, rows, nullptr, nc);
  if (e != cudaSuccess) return e;
  return launch_chained(exact_slice_a_kernel, 152 * 16, 256, 0, s, true, ex, a, rows, nc);
}

cudaError_t launch_exact_gemm(const ExactPrep& ex, int grid, int* status, cudaStream_t s) {
  if (ex.n_items == 0) return cudaSuccess;  // every row is zero: the epilogue sums no pieces
  auto* kernel = ex.slices == 7    ? exact_gemm_kernel<7, 64>
                 : ex.cols == 80 ? exact_gemm_kernel<6, 80>
                 : ex.cols == 64 ? exact_gemm_kernel<6, 64>
                                 : exact_gemm_kernel<6, 48>;
  const uint32_t smem = ex_smem(ex.slices, ex.cols);
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  return launch_chained(kernel, std::min(grid, ex.n_items), kThreadsEx, smem, s, true, ex, status);
}

cudaError_t launch_exact_finish(const FfDev& d, const ExactPrep& ex, double2* out, double2* out2, cudaStream_t s,
                                const ExSecond& second) {
  auto* kernel = ex.halves == 1 ? exact_finish_kernel<true> : exact_finish_kernel<false>;
  cudaError_t e = launch_chained(kernel, dim3(ex.n_row_blocks, ex.n_col_blocks, ex.bands / kFinBands), kFinThreads, 0,
                                 s, true, d, ex, second);
  if (e != cudaSuccess) return e;
  const int entries = d.nb * d.nf * (out2 ? 2 : 1) + (second.out ? second.nb * second.nf : 0);
  return launch_chained(exact_reduce_kernel, (entries * kRedLanes + kRedThreads - 1) / kRedThreads, kRedThreads, 0, s,
                        true, d, ex, second, out, out2);
}

}  // namespace sigma
