// FP64 trailing update of the plain LU on the BF16 tensor cores (the PDGEMM
// step of SRC/pdgetrf.f:288-290, C <- C + alpha * A * B with FP64 A, B, C):
// sm_103a's tcgen05.mma has no FP64 kind, so the product is formed exactly
// from integer slices (the error-free splitting of Ozaki, Ogita and Oishi,
// "Error-free transformations of matrix multiplication by using fast routines
// of matrix multiplication and its applications", Numer. Algorithms 59, 2012).
//
// Splitting. Row i of A is scaled by 2^-e_i (e_i the exponent of its largest
// magnitude, so |A(i,k)| 2^-e_i < 1), rounded to a multiple of 2^-55 and cut into
// S = 7 balanced base-256 digits:
//   A(i,k) 2^-e_i = sum_{s=1..7} a_s(i,k) 2^(1-8s),  a_s integer, |a_s| <= 128;
// column j of B likewise with 2^-f_j and b_t. BF16 holds every such digit exactly
// (8 significant bits). Balanced digits carry 8 bits a slice where truncated ones
// of the same exactness carry 7: 7 slices and 28 products instead of 8 and 36,
// with the same 2^-56 of the scale kept.
//
// Exact products. For K <= 256, sum_k a_s b_t is an integer of magnitude at
// most 256 * 128^2 = 2^22: up to four such products sum exactly in FP32, in
// any order and with any alignment the tensor core uses, because every partial
// sum is an integer of magnitude at most 2^24. With d = s + t, the update is
//   (A B)(i,j) = 2^(e_i + f_j) sum_d 2^(2-8d) P_d,   P_d = sum_{s+t=d} sum_k a_s b_t.
// Each diagonal d = 2..8 has its own TMEM accumulator (7 x 64 columns). d <= 5
// holds at most 4 products: exact; d = 6..8 hold 5 to 7, exact unless their sum
// passes 2^24, which takes most of the 1280 to 1792 terms at full magnitude with
// one sign (constant rows of 254/255 do that; the FP32 rounding is then 2^-24 of terms
// 2^-40 below the scales' largest sum); d >= 9 is dropped: at most 6 256 128^2 2^-70,
// 2^-45.4, of 2^(e_i + f_j). 28 slice products, issued as 10 instructions per 16-wide
// k step: A slice s against B slices t = 0..6-s (consecutive in shared memory)
// into accumulators s..6 (consecutive in TMEM) in groups of up to 4 (N up to
// 256).
//
// Epilogue. P_2..P_6 are read back as exact integers and combined with the
// rounded P_7 + P_8/256 into one 64-bit integer I = sum_d P_d 2^(56-8d) (|I| <
// 2^63), rounded to 53 bits once and scaled by 2^(e_i+f_j-54) with integer
// arithmetic; C(i,j) then takes it by one FP64 addition (alpha = +-1; otherwise
// by an fma with alpha). This GPU converts 64-bit integers and adds or
// multiplies doubles at 2 lanes per cycle and SM, so a conversion, a
// multiplication and an fma per element would take as long as the tile's
// products, and a 64-bit conversion before the accumulators are released would
// hold the products up. The result is within 2^-45.4 of 2^(e_i + f_j) of the exact
// product (about K/1.3 units of 2^-53, as an FP64 GEMM's bound of K units), reached
// where all low digits have one sign: 2^-46.1 for constant operands of 0.1, 2^-45.4
// for one large entry among small ones with that pattern, where a GEMM's actual error
// is below 2^-50; on operands without a pattern it is a few units of 2^-53. (8
// truncated slices and 36 products: 2^-45.2.) It is independent of the accumulation
// order (run to run identical). Rows or columns holding Inf or NaN give NaN in their
// row or column of C.
//
// Balancing along k. A B = (A 2^-d)(2^d B) for any integers d_k, so the
// scales are taken after an exact power-of-two balancing (ex x: |x| < 2^ex x,
// over the k whose column of A and row of B are both nonzero):
//   e_i = max_k (ex A(i,k) - d_k),   f_j = max_k (ex B(k,j) + d_k).
// The shift goes into the slicing's shift counts; no scaled value is ever
// formed. Side A (the default): d_k = c_k, the exponent of the largest
// magnitude in column k of A. In the LU A = L21 (|L| <= 1, so c_k ~ 0 and
// nothing moves on well-scaled data); on a row-graded matrix a block's pivots
// differ widely in size, column k of L21 is ~2^-(s_pk) and row k of U12
// ~2^(s_pk), and without the balancing the largest L21 and U12 entries of a
// pair (i, j) sit at different k, so 2^(e_i + f_j) would exceed every term of
// the product by the pivots' spread. Side B: d_k = -h_k, h_k the exponent of
// the largest magnitude in row k of B -- for the U12 solve's product
// (inv(L_bb) - I) A12_b, whose rows of B carry the pivots' scales while the
// columns of the inverse do not.
//
// Error budget. With G = max_k (c_k + h_k), side A compares each row's error
// bound 2^(e_i + G) with F_i = max_k (ex A(i,k) + h_k), the exponent of a
// lower bound of max_j (|A| |B|)(i,j) (an FP64 GEMM's bound for that row);
// side B compares each column's 2^(f_j + G) with F_j = max_k (c_k +
// ex B(k,j)). Where any row (column) is more than OZ_BUDGET bits above it (a
// row of A small exactly where a row of B holds an entry far above the rest),
// or a scale leaves the normal FP64 range, the whole pass is computed in FP64
// arithmetic instead (fixed order, every product an FMA; side B: by substitution
// with L_bb) by the same launches. Accuracy model: each row's (column's) error is within about
// 2^OZ_BUDGET of the FP64 GEMM's error bound for its largest |A||B| term
// (normwise per row or column); for inputs that are diagonal scalings of
// well-scaled data that is the componentwise level. Operands whose large
// entries cross (row i large at k1 only, column j large at k2 only) keep the
// normwise bound but not a componentwise one.
//
// Structure (one CTA per SM, a few 128 x 64 tiles of C per CTA, 18 warps):
//   * warp 0 allocates all 512 TMEM columns (7 accumulators x 64 columns);
//   * one thread issues TMA loads: for each 64-wide k block, the seven 128x64
//     A slices one at a time through a 7-deep ring and the seven 64x64 B
//     slices into one half of a double buffer, half a block ahead (128-byte
//     swizzle);
//   * one thread issues tcgen05.mma.kind::f16 (M=128, N=64..256, K=16): A
//     slice s against B slices t <= 8 - s into accumulators s+t-2;
//   * 16 epilogue warps load their part of C while the tile's products run, read
//     the accumulators with tcgen05.ld (warp w owns lanes 32(w%4).. = tile rows,
//     and a quarter of the columns), combine them into integers, hand the TMEM
//     back to the MMA thread, and update C in place (coalesced per column)
//     while the next tile's products run.
// Every mbarrier wait is bounded; on timeout the CTA records kFlagTimeout,
// drains what it issued, frees its TMEM and returns.
//
// Bound: a tile's products take 14300 cycles of the tensor pipe; it takes 30000 (m =
// n = 6144 .. 16384, k = 256), 3000 of them the read-out of the accumulators, which
// is not overlapped; the rest is no throughput (L2 at 9.9 TB/s, but a third less of
// it by multicast to two CTAs takes as long; shared-memory banks 39 %). Measured, m =
// n = 16384: 3.3 ms, 42 TFLOP/s FP64-equivalent; with 36 products of 7-bit slices,
// three FP64-rate operations per element and descriptors computed per instruction,
// 5.0 ms. 128 x 64 tiles of 8192 x 256 x 256: 47 us (72 before).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>
#include <climits>

#include "common.cuh"
#include "sl_internal.h"
#include "tc_common.cuh"

namespace sl {
namespace {
using namespace tc;

constexpr int OZ_S = 7;          // slices per operand: balanced base-256 digits
constexpr int OZ_KMAX = 256;     // exactness bound on K per pass
constexpr int OBM = 128, OBN = 64, OBK = 64;
constexpr int A_SLICE_BYTES = OBM * OBK * 2;          // 16 KB
constexpr int B_SLICE_BYTES = OBN * OBK * 2;          // 8 KB
constexpr int B_CHUNK_BYTES = OZ_S * B_SLICE_BYTES;   // 56 KB per k block
constexpr int A_RING = 7;
constexpr int OZ_TMEM_COLS = 512;
constexpr int GROUP_M = 8;       // tile raster: 8 row tiles sweep the columns together

// Balancing / budget area at the start of the scratch: h keys [256] (rows of
// B), c keys [256] (columns of A), the FP64-route flag. Each word is
// (epoch << 12) | (exponent + OZ_EBIAS), so a pass ignores what earlier passes
// left (epochs only grow) and nothing has to be cleared between passes.
constexpr int OZ_KINFO_BYTES = kOzKinfoBytes;
constexpr int OZ_KI_H = 0, OZ_KI_C = OZ_KMAX, OZ_KI_FLAG = 2 * OZ_KMAX;
constexpr int OZ_EBIAS = kOzEbias;
constexpr int OZ_BUDGET = 8;     // bits above the FP64 GEMM's row (column) bound
constexpr int OZ_NOEXP = INT_MIN / 4;

__device__ unsigned long long g_oz_fp64_routes;  // passes that took the FP64 route

struct __align__(8) OzBars {
  uint64_t afull[A_RING], aempty[A_RING];
  uint64_t bfull[2], bempty[2];
  uint64_t tfull, tempty;  // accumulators complete / drained
  uint32_t tmem_base;
};

constexpr int OZ_EPI_WARPS = 16;  // four per TMEM lane quadrant
constexpr int OZ_EC = OBN / (OZ_EPI_WARPS / 4);  // columns of an epilogue warp: 16
constexpr int OZ_THREADS = 64 + 32 * OZ_EPI_WARPS;  // warp 0 TMA, warp 1 MMA, the rest epilogue

size_t oz_smem_bytes() {
  return 1024 + (size_t)A_RING * A_SLICE_BYTES + 2 * (size_t)B_CHUNK_BYTES + sizeof(OzBars) + 64;
}

// kind::f16 instruction descriptor, M = 128, N = nn (a multiple of 64 <= 256)
__host__ __device__ constexpr uint32_t oz_idesc(int nn) {
  return (1u << 4)                       // D format: F32
         | (1u << 7) | (1u << 10)        // A, B: BF16
         | ((uint32_t)(nn >> 3) << 17)   // N / 8
         | ((uint32_t)(OBM >> 4) << 24); // M / 16
}

__device__ __forceinline__ void touch16(uint32_t* r) {
  asm volatile(""
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]),
                 "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]),
                 "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]));
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// Tile t of the grouped raster: (m0, n0).
__device__ __forceinline__ void oz_tile(int t, int tiles_m, int tiles_n, int& m0, int& n0) {
  const int per_group = GROUP_M * tiles_n;
  const int gid = t / per_group, first_m = gid * GROUP_M;
  const int gsize = min(tiles_m - first_m, GROUP_M);
  const int in_group = t % per_group;
  m0 = (first_m + in_group % gsize) * OBM;
  n0 = (in_group / gsize) * OBN;
}

// The B slices of chunk c (tile first + c / nkc, k block c % nkc) into
// half c & 1 of the B double buffer, once chunk c-2 has released it.
__device__ __forceinline__ bool oz_issue_b(int c, int first, int nkc, int tiles_m, int tiles_n,
                                           int n_pad, unsigned char* sB, const CUtensorMap* tmB,
                                           OzBars* bars, int* issued) {
  const int hb = c & 1;
  if (c >= 2 && !mbar_wait(&bars->bempty[hb], ((c >> 1) - 1) & 1)) return false;
  int m0, n0;
  oz_tile(first + c / nkc, tiles_m, tiles_n, m0, n0);
  const int kc = c % nkc;
  mbar_expect_tx(&bars->bfull[hb], B_CHUNK_BYTES);
  for (int t = 0; t < OZ_S; ++t)
    tma_load_2d(sB + hb * B_CHUNK_BYTES + t * B_SLICE_BYTES, tmB, &bars->bfull[hb], kc * OBK,
                t * n_pad + n0);
  *issued = c + 1;
  return true;
}

// The unit-lower factor of a side-B pass: the pass is B <- B + N B with N = inv(L) - I,
// flags nonzero where N is not to be used.
struct OzUnitLower {
  const double* L = nullptr;
  long long ldl = 0;
  const int* flags = nullptr;
  int nflags = 0;
};

// B <- inv(L) B by forward substitution: the FP64 route of a side-B pass. A CTA
// takes 64 columns of B (kb <= 256 rows, 128 KB) into shared memory; thread t
// has column t % 64 and every ninth row below the one that is final. Bound: the
// FP64 unit: a 256-wide block that goes this way adds 0.65 ms (two such passes) to a
// factorization of N = 4096 (13.1 ms).
__device__ __noinline__ void oz_substitute(unsigned char* smem, int n, int kb, OzUnitLower ul, double* B,
                                           long long ldb, int tiles_n) {
  double* sB = reinterpret_cast<double*>(smem);  // [kb][64]
  const int tid = threadIdx.x, c = tid & (OBN - 1), g = tid / OBN;
  for (int t = blockIdx.x; t < tiles_n; t += gridDim.x) {
    const int n0 = t * OBN;
    __syncthreads();
    for (int idx = tid; idx < kb * OBN; idx += OZ_THREADS) {
      const int cc = idx / kb, k = idx - cc * kb;
      sB[k * OBN + cc] = (n0 + cc < n) ? B[k + (long long)(n0 + cc) * ldb] : 0.0;
    }
    __syncthreads();
    for (int q = 0; q < kb; ++q) {
      const double x = sB[q * OBN + c];
      const double* l = ul.L + (long long)q * ul.ldl;
#pragma unroll 4
      for (int r = q + 1 + g; r < kb; r += OZ_THREADS / OBN) sB[r * OBN + c] = fma(-l[r], x, sB[r * OBN + c]);
      __syncthreads();
    }
    for (int idx = tid; idx < kb * OBN; idx += OZ_THREADS) {
      const int cc = idx / kb, k = idx - cc * kb;
      if (n0 + cc < n) B[k + (long long)(n0 + cc) * ldb] = sB[k * OBN + cc];
    }
  }
}

// The FP64 route of a pass whose slices would exceed the error budget: the
// CTA's tiles computed directly from the FP64 operands. B's 64 columns of a
// tile (kb <= 256 rows, 128 KB) are staged in shared memory before any of
// them is written. When B aliases C (whole_cols) a CTA takes whole column
// blocks instead -- tile t of the CTA is column block t with every row tile --
// so no other CTA writes the columns it reads. Threads 64.. own one row and
// OZ_EC columns each; products accumulate in k order with one FMA each, then
// C = fma(alpha, acc, C).
__device__ __noinline__ void oz_fp64_tiles(unsigned char* smem, int m, int n, int kb,
                                           const double* __restrict__ A, long long lda,
                                           const double* B, long long ldb, double alpha,
                                           double* C, long long ldc, int first_tile,
                                           int my_tiles, int tiles_m, int tiles_n,
                                           int whole_cols) {
  double* sB = reinterpret_cast<double*>(smem);  // [kb][64]
  const int tid = threadIdx.x;
  const int nsub = whole_cols ? tiles_m : 1;
  for (int it = 0; it < my_tiles * nsub; ++it) {
    int m0, n0;
    if (whole_cols) {
      const int t = first_tile + it / nsub;
      if (t >= tiles_n) break;
      n0 = t * OBN;
      m0 = (it % nsub) * OBM;
    } else {
      oz_tile(first_tile + it, tiles_m, tiles_n, m0, n0);
    }
    __syncthreads();
    if (!whole_cols || (it % nsub) == 0)
      for (int idx = tid; idx < kb * OBN; idx += OZ_THREADS) {
        const int c = idx / kb, k = idx - c * kb;
        sB[k * OBN + c] = (n0 + c < n) ? B[k + (long long)(n0 + c) * ldb] : 0.0;
      }
    __syncthreads();
    if (tid >= 64) {
      const int t = tid - 64, row = m0 + (t & (OBM - 1)), h = t >> 7;
      if (row < m) {
        double acc[OZ_EC];
#pragma unroll
        for (int j = 0; j < OZ_EC; ++j) acc[j] = 0.0;
        const double* arow = A + row;
        for (int k = 0; k < kb; ++k) {
          const double a = arow[(long long)k * lda];
          const double* bk = sB + k * OBN + h * OZ_EC;
#pragma unroll
          for (int j = 0; j < OZ_EC; ++j) acc[j] = fma(a, bk[j], acc[j]);
        }
#pragma unroll
        for (int j = 0; j < OZ_EC; ++j) {
          const int col = n0 + h * OZ_EC + j;
          if (col < n) {
            double* cp = C + row + (long long)col * ldc;
            *cp = fma(alpha, acc[j], *cp);
          }
        }
      }
    }
  }
}

// An integer |x| <= 2^24 held in FP32, plus 5 kMagicBits modulo 2^32: the addition
// of 1.5 2^23 leaves an integer of up to 22 bits in the low bits, so x is taken in
// two parts, x = 4 h + l. Four FP32 operations at 128 lanes a cycle, where the
// conversion instruction takes 16.
constexpr float kMagic = 12582912.0f;
constexpr unsigned kMagicBits = 0x4B400000u;
__device__ __forceinline__ unsigned oz_int24(float x) {
  const float h = fmaf(x, 0.25f, kMagic);
  const float l = fmaf(h - kMagic, -4.0f, x) + kMagic;
  return 4u * __float_as_uint(h) + __float_as_uint(l);
}
// Exponent of a power of two (-1023 for zero, beyond any sum's range for NaN).
__device__ __forceinline__ int oz_exp_field(double x) {
  const int f = (__double2hiint(x) >> 20) & 0x7ff;
  return f == 0x7ff ? 1 << 14 : f - 1023;
}
// v 2^E rounded to nearest once, E in [-1022, 960], on the integer pipe.
__device__ __forceinline__ double oz_ldexp(long long v, int E) {
  const unsigned long long u = (unsigned long long)(v < 0 ? -v : v);
  const int lz = __clzll((long long)u);
  const unsigned long long w = u << (lz & 63);
  unsigned long long m = w >> 11;
  m += ((unsigned)(w & 2047) + (unsigned)(m & 1)) > 1024u ? 1 : 0;
  // the significand's leading bit adds one to the exponent below it
  const unsigned long long bits = ((unsigned long long)(unsigned)(E + 63 - lz + 1022) << 52) + m;
  return u == 0 ? 0.0 : __longlong_as_double((long long)(bits | ((unsigned long long)v & (1ULL << 63))));
}

// An epilogue warp's part of the accumulators as integers I = sum_d P_d 2^(56-8d),
// trow its TMEM address; release() once everything is in registers.
template <class F>
__device__ __forceinline__ void oz_read_sums(uint32_t trow, long long* I, F release) {
  // two accumulators at a time keep the register count down; P_2 <= 2^22
  // converts by an addition (1.5 * 2^23, whose bits are taken off again), the
  // next ones by two or by the conversion instruction, turn about
  uint32_t r[2][16];
  auto get2 = [&](int a, bool both) {
    tmem_ld16_nowait(trow + (uint32_t)(a * OBN), r[0]);
    if (both) tmem_ld16_nowait(trow + (uint32_t)((a + 1) * OBN), r[1]);
    tmem_ld_wait();
    touch16(r[0]);
    if (both) touch16(r[1]);
  };
  get2(0, true);
#pragma unroll
  for (int j = 0; j < OZ_EC; ++j) {
    const unsigned p2 = __float_as_uint(__uint_as_float(r[0][j]) + kMagic);
    const unsigned p3 = oz_int24(__uint_as_float(r[1][j]));
    const unsigned hi = (p2 << 8) + p3 - 261u * kMagicBits;  // (modulo 2^32, as the sum's high half)
    I[j] = (long long)((unsigned long long)hi << 32);
  }
  get2(2, true);
#pragma unroll
  for (int j = 0; j < OZ_EC; ++j) {
    const long long p4 = __float2int_rn(__uint_as_float(r[0][j]));
    const long long p5 = (int)(oz_int24(__uint_as_float(r[1][j])) - 5u * kMagicBits);
    I[j] += (p4 << 24) + (p5 << 16);
  }
  get2(4, false);
#pragma unroll
  for (int j = 0; j < OZ_EC; ++j) I[j] += (long long)__float2int_rn(__uint_as_float(r[0][j])) << 8;
  get2(5, true);
  release();
#pragma unroll
  for (int j = 0; j < OZ_EC; ++j)
    I[j] += __float2int_rn(fmaf(__uint_as_float(r[1][j]), 0.00390625f, __uint_as_float(r[0][j])));
}
// C(row, 16 columns) = cv + alpha 2^(e_i + f_j - 54) I, rsc and sc the scales.
__device__ __forceinline__ void oz_update_c(const long long* I, const double* cv, double* crow,
                                            long long ldc, int ncol, double alpha, double rsc,
                                            const double* sc) {
  // one FP64 addition per element, unless some element of the warp needs
  // the general form: general alpha, scales near the range's ends, zero and
  // non-finite ones (a vote, so that the compiler does not compute both)
  const int er = oz_exp_field(rsc);
  const bool unit = alpha == 1.0 || alpha == -1.0, neg = alpha < 0.0;
  bool plain = unit;
#pragma unroll
  for (int j = 0; j < OZ_EC; ++j) {
    plain = plain && (j >= ncol || (unsigned)(er + oz_exp_field(sc[j]) + 1022) <= 1982u);
  }
  if (__all_sync(0xffffffffu, plain)) {
#pragma unroll
    for (int j = 0; j < OZ_EC; ++j)
      if (j < ncol)
        crow[(long long)j * ldc] = cv[j] + oz_ldexp(neg ? -I[j] : I[j], er + oz_exp_field(sc[j]));
  } else {
#pragma unroll
    for (int j = 0; j < OZ_EC; ++j)
      if (j < ncol) crow[(long long)j * ldc] = fma(alpha * rsc * sc[j], __ll2double_rn(I[j]), cv[j]);
  }
}

// CTA b takes tiles b tpc .. b tpc + tpc - 1 of the raster (a few, so that
// SMs turn over and the panel's kernels on the high-priority stream find
// room between them). The TMA thread runs
// ahead through a flat sequence of k blocks ("chunks", nkc per tile): for
// chunk c it loads the A slices through the ring, and after the fourth of
// them the B slices of chunk c+1 into the other half of the B double
// buffer. The MMA thread starts a tile once the epilogue has drained the
// previous tile's accumulators (tempty); the epilogue warps drain them into
// 16 combined integers per thread (tmem -> registers), release the TMEM, and
// update C from registers while the next tile's products run.
__global__ void __launch_bounds__(OZ_THREADS, 1)
ozgemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
              int m, int n, int kpad, int m_pad, int n_pad, const double* __restrict__ rs,
              const double* __restrict__ cs, double alpha, double* C, long long ldc, int tpc,
              int* status, const double* __restrict__ A64, long long lda, const double* B64,
              long long ldb, int kb, const unsigned long long* kinfo, unsigned long long epoch, OzUnitLower ul) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* base = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  unsigned char* sA = base;                                   // A_RING x 16 KB
  unsigned char* sB = base + A_RING * A_SLICE_BYTES;          // 2 x 56 KB
  OzBars* bars = (OzBars*)(sB + 2 * B_CHUNK_BYTES);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles_m = m_pad / OBM, tiles_n = n_pad / OBN;
  const int tiles = tiles_m * tiles_n;
  const int first_tile = (int)blockIdx.x * tpc;
  const int my_tiles = max(0, min(tpc, tiles - first_tile));
  const int nkc = kpad / OBK;
  const int total = my_tiles * nkc;  // chunks of this CTA
  __shared__ int s_fail, s_aiss, s_acons, s_biss, s_bcons;
  // a CTA that timed out already marked the launch failed: skip the work (the word may
  // be written meanwhile, by the other stream too: the block decides as one)
  if (__syncthreads_or(*(volatile int*)status != 0)) return;
  // the slicing found the pass outside the error budget: FP64 route
  if (*(volatile const unsigned long long*)(kinfo + OZ_KI_FLAG) == epoch) {
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(&g_oz_fp64_routes, 1ULL);
    if (ul.L)
      oz_substitute(base, n, kb, ul, C, ldc, tiles_n);
    else
      oz_fp64_tiles(base, m, n, kb, A64, lda, B64, ldb, alpha, C, ldc, first_tile, my_tiles,
                    tiles_m, tiles_n, B64 == C ? 1 : 0);
    return;
  }

  if (threadIdx.x == 0) {
    s_fail = 0;
    s_aiss = s_acons = s_biss = s_bcons = 0;
    for (int i = 0; i < A_RING; ++i) {
      mbar_init(&bars->afull[i], 1);
      mbar_init(&bars->aempty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars->bfull[i], 1);
      mbar_init(&bars->bempty[i], 1);
    }
    mbar_init(&bars->tfull, 1);
    mbar_init(&bars->tempty, OZ_EPI_WARPS);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&bars->tmem_base)),
                 "r"(OZ_TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = bars->tmem_base;

  if (warp == 0) {
    if (lane == 0) {
      // ---- TMA producer ----
      asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmA)) : "memory");
      asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmB)) : "memory");
      bool ok = total == 0 ||
                oz_issue_b(0, first_tile, nkc, tiles_m, tiles_n, n_pad, sB, &tmB, bars, &s_biss);
      for (int c = 0; ok && c < total; ++c) {
        int m0, n0;
        oz_tile(first_tile + c / nkc, tiles_m, tiles_n, m0, n0);
        const int kc = c % nkc;
        for (int sl = 0; ok && sl < OZ_S; ++sl) {
          const int g = c * OZ_S + sl, st = g % A_RING;
          if (g >= A_RING && !mbar_wait(&bars->aempty[st], ((g / A_RING) - 1) & 1)) {
            ok = false;
            break;
          }
          mbar_expect_tx(&bars->afull[st], A_SLICE_BYTES);
          tma_load_2d(sA + st * A_SLICE_BYTES, &tmA, &bars->afull[st], kc * OBK, sl * m_pad + m0);
          s_aiss = g + 1;
          if (sl == 3 && c + 1 < total &&
              !oz_issue_b(c + 1, first_tile, nkc, tiles_m, tiles_n, n_pad, sB, &tmB, bars, &s_biss))
            ok = false;
        }
        if (s_fail) ok = false;
      }
      if (!ok) {
        atomicExch(status, (int)kFlagTimeout);
        s_fail = 1;
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // ---- MMA issuer ----
      // A slice s against B slices t = 0 .. 6-s lands in accumulators s .. 6:
      // consecutive TMEM columns and, in the B buffer, consecutive slices, so
      // one instruction covers up to 4 of them (N up to 256).
      bool ok = true;
      const uint64_t adesc = smem_desc_sw128(sA), bdesc = smem_desc_sw128(sB);
      for (int it = 0; ok && it < my_tiles; ++it) {
        if (it >= 1 && !mbar_wait(&bars->tempty, (it - 1) & 1)) { ok = false; break; }
        asm volatile("tcgen05.fence::after_thread_sync;");
        for (int kc = 0; ok && kc < nkc; ++kc) {
          const int c = it * nkc + kc, hb = c & 1;
          if (!mbar_wait(&bars->bfull[hb], (c >> 1) & 1)) { ok = false; break; }
          s_bcons = c + 1;
          // A slice sl of a chunk always stands in ring slot sl, so that every
          // operand's place is a constant added to two descriptors: computed
          // anew per instruction they took the one issuing thread 170 cycles an
          // instruction, where the products take 90.
          static_assert(A_RING == OZ_S, "slot of a slice");
          const uint64_t b0 = bdesc + (uint64_t)((hb * B_CHUNK_BYTES) >> 4);
#pragma unroll
          for (int sl = 0; sl < OZ_S; ++sl) {
            if (!mbar_wait(&bars->afull[sl], c & 1)) { ok = false; break; }
            asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll
            for (int kk = 0; kk < OBK / 16; ++kk) {
              // the very first products write every accumulator (s = 0 covers
              // them all); every later one adds
              const uint32_t accum = (sl > 0 || kk > 0) ? 1u : (kc > 0 ? 1u : 0u);
#pragma unroll
              for (int t0 = 0; t0 + sl < OZ_S; t0 += 4) {
                const int cnt = OZ_S - sl - t0 < 4 ? OZ_S - sl - t0 : 4;
                umma_f16(tmem + (uint32_t)((sl + t0) * OBN),
                         adesc + (uint64_t)((sl * A_SLICE_BYTES + kk * 32) >> 4),
                         b0 + (uint64_t)((t0 * B_SLICE_BYTES + kk * 32) >> 4), oz_idesc(cnt * OBN), accum);
              }
            }
            umma_commit(&bars->aempty[sl]);
            s_acons = c * OZ_S + sl + 1;
          }
          if (!ok) break;
          umma_commit(&bars->bempty[hb]);
        }
        if (ok) umma_commit(&bars->tfull);  // arrives when the tile's products are complete
        if (s_fail) ok = false;
      }
      if (!ok) {
        atomicExch(status, (int)kFlagTimeout);
        s_fail = 1;
      }
    }
  } else {
    // ---- epilogue: warp w reads TMEM lanes 32 (w % 4) .. +31 = tile rows,
    // columns EC g .. EC g + EC - 1 with g = (w - 2) / 4 ----
    constexpr int EC = OZ_EC;
    const int quad = warp & 3, cg = (warp - 2) >> 2;
    const uint32_t trow = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(cg * EC);
    for (int it = 0; it < my_tiles; ++it) {
      int m0, n0;
      oz_tile(first_tile + it, tiles_m, tiles_n, m0, n0);
      // this tile's part of C on its way while the products run
      const int row = m0 + quad * 32 + lane, nb0 = n0 + cg * EC;
      const int ncol = row < m ? min(EC, n - nb0) : 0;
      double* crow = C + (long long)row + (long long)nb0 * ldc;
      double cv[EC];
#pragma unroll
      for (int j = 0; j < EC; ++j) cv[j] = j < ncol ? crow[(long long)j * ldc] : 0.0;
      const double rsc = ncol > 0 ? rs[row] : 0.0;
      if (!mbar_wait(&bars->tfull, it & 1)) {
        if (lane == 0) {
          atomicExch(status, (int)kFlagTimeout);
          s_fail = 1;
        }
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;");
      long long I[EC];
      oz_read_sums(trow, I, [&]() {
        // the accumulators are in registers: the next tile's products may start
        asm volatile("tcgen05.fence::before_thread_sync;");
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->tempty);
      });
      double sc[EC];
#pragma unroll
      for (int j = 0; j < EC; ++j) sc[j] = __ldg(cs + min(nb0 + j, n - 1));
      oz_update_c(I, cv, crow, ldc, ncol, alpha, rsc, sc);
      if (s_fail) break;
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (s_fail && threadIdx.x == 0) {
    // Drain copies that were issued but never consumed (bounded waits).
    for (int g = s_acons; g < s_aiss; ++g) mbar_wait(&bars->afull[g % A_RING], (g / A_RING) & 1);
    for (int c = s_bcons; c < s_biss; ++c) mbar_wait(&bars->bfull[c & 1], (c >> 1) & 1);
  }
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(OZ_TMEM_COLS));
  }
}

// ---- slicing (integer arithmetic on the FP64 bit patterns) ----------------
//
// With x = +-m 2^q (m the significand as an integer, 53 bits for normal x)
// and a scale exponent e with |x| < 2^e, V = +-round(|x| 2^(55-e)) is m shifted
// left by at most 2 bits, or right with rounding. Adding 128 to its six low
// digits' places turns V's balanced base-256 digits into bytes: digit s (1-based)
// is byte 7-s of the sum less 128, the first one what stands above them (-128 ..
// 128). With the balancing, A(i,k) is cut against e_i + d_k and B(k,j) against
// f_j - d_k.
constexpr unsigned long long kMagMask = 0x7fffffffffffffffULL;
constexpr unsigned long long kInfBits = 0x7ff0000000000000ULL;

// the sum V + 128 (1 + 256 + .. + 256^5) of x with the given bits
constexpr unsigned long long kDigitBias = 0x0000808080808080ULL;
__device__ __forceinline__ unsigned long long oz_digits(unsigned long long bits, int e) {
  const int bexp = (int)((bits >> 52) & 0x7ff);
  unsigned long long m = bits & 0xfffffffffffffULL;
  int q = -1074;
  if (bexp != 0) {
    m |= 1ULL << 52;
    q = bexp - 1075;
  }
  const int sh = q - e + 55;
  unsigned long long U;
  if (sh >= 0) U = m << sh;
  else U = sh < -54 ? 0ULL : (m + (1ULL << (-sh - 1))) >> -sh;
  return ((bits >> 63) ? 0ULL - U : U) + kDigitBias;
}

// frexp exponent of a magnitude given by its bit pattern (finite, nonzero):
// 2^(ex-1) <= |x| < 2^ex
__device__ __forceinline__ int oz_scale_exp(unsigned long long kmax) {
  const int bexp = (int)(kmax >> 52);
  if (bexp != 0) return bexp - 1022;
  return (63 - __clzll((long long)kmax)) - 1073;  // subnormal
}

// 2^(e - 27) as a double (the epilogue's scale factor half), NaN for a
// non-finite row or column, 0 for a zero one; the caller has checked that
// e - 27 is a normal exponent
__device__ __forceinline__ double oz_scale_value(int e, bool bad) {
  if (bad) return __longlong_as_double(0x7ff8000000000000LL);
  if (e == OZ_NOEXP) return 0.0;
  return __longlong_as_double((long long)((unsigned long long)(e - 27 + 1023) << 52));
}
__device__ __forceinline__ bool oz_scale_in_range(int e) {
  return e == OZ_NOEXP || (e - 27 >= -1022 && e - 27 <= 1023);
}

// Slice s (0-based) of two digit sums as a pair of BF16: each byte becomes the
// low mantissa bits of 2^23, whose exact difference to 2^23 + 128 is the digit
// (its upper 16 bits are its BF16); the first digit is the sum's signed top.
__device__ __forceinline__ uint32_t oz_slice2(unsigned long long w0, unsigned long long w1, int s) {
  const uint32_t hi0 = (uint32_t)(w0 >> 32), lo0 = (uint32_t)w0, hi1 = (uint32_t)(w1 >> 32), lo1 = (uint32_t)w1;
  float f0, f1;
  if (s == 0) {
    f0 = (float)((int)hi0 >> 16);
    f1 = (float)((int)hi1 >> 16);
  } else {
    const int byte = 6 - s;  // of the 64-bit sum
    const uint32_t a0 = byte >= 4 ? hi0 : lo0, a1 = byte >= 4 ? hi1 : lo1;
    const uint32_t sel = 0x7650u | (uint32_t)(byte & 3);
    f0 = __uint_as_float(__byte_perm(a0, 0x4B000000u, sel)) - 8388736.0f;
    f1 = __uint_as_float(__byte_perm(a1, 0x4B000000u, sel)) - 8388736.0f;
  }
  return __byte_perm(__float_as_uint(f0), __float_as_uint(f1), 0x7632);
}

__device__ __forceinline__ int oz_warp_imax(int v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, off));
  return v;
}
// biased exponent of a finite nonzero value (1 .. 4095), 0 otherwise
__device__ __forceinline__ unsigned oz_ekey(double x) {
  const unsigned long long mag = (unsigned long long)__double_as_longlong(x) & kMagMask;
  return (mag != 0ULL && mag < kInfBits) ? (unsigned)(oz_scale_exp(mag) + OZ_EBIAS) : 0u;
}
// exponent held by a balancing word of this epoch, OZ_NOEXP if none
__device__ __forceinline__ int oz_word_exp(unsigned long long w, unsigned long long epoch) {
  return (w >> 12) == epoch ? (int)(w & 4095ULL) - OZ_EBIAS : OZ_NOEXP;
}

// Balancing exponents of one pass, both operands in one launch. Blocks
// [0, nab): 32 rows of A (m x kb) each; warp w takes columns k = w, w+8, ...
// (one coalesced 256-byte load per column, all of them issued before the first
// is used: one by one, as a bound test before each load made them, the pass took
// 32 memory latencies, 35 us at any size), reduces the lanes' exponent keys with
// one __reduce_max_sync and keeps the column's maximum in shared memory: c_k. Blocks after that: 64 columns of B (kb x n) each; warp w takes columns
// w, w+8, ..., lane l rows l, l+32, ...: h_k. Each block publishes its
// maxima with atomicMax into the epoch-tagged words. Small blocks with many
// independent loads, so the pass over both operands runs near copy speed.
__global__ void __launch_bounds__(256)
oz_kscale_kernel(const double* __restrict__ A, long long lda, int m, const double* __restrict__ B,
                 long long ldb, int n, int kb, int nab, unsigned long long* kinfo,
                 unsigned long long epoch) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __shared__ unsigned red[8][OZ_KMAX];
  if ((int)blockIdx.x < nab) {
    const int i = (int)blockIdx.x * 32 + lane;
    const double* arow = A + (i < m ? i : m - 1);  // (a repeated row changes no maximum)
    double v[OZ_KMAX / 8];  // every load of the warp's columns in flight at once
#pragma unroll
    for (int q = 0; q < OZ_KMAX / 8; ++q) v[q] = arow[(long long)min(warp + 8 * q, kb - 1) * lda];
#pragma unroll
    for (int q = 0; q < OZ_KMAX / 8; ++q) {
      const unsigned r = __reduce_max_sync(0xffffffffu, oz_ekey(v[q]));
      if (lane == 0) red[0][warp + 8 * q] = r;
    }
    __syncthreads();
    const int k = threadIdx.x;
    if (k < kb && red[0][k]) oz_raise_key(kinfo + OZ_KI_C + k, (epoch << 12) | red[0][k]);
    return;
  }
  const int c0 = ((int)blockIdx.x - nab) * 64;
  unsigned km[OZ_KMAX / 32];
#pragma unroll
  for (int r = 0; r < OZ_KMAX / 32; ++r) km[r] = 0u;
#pragma unroll
  for (int q0 = 0; q0 < 8; q0 += 4) {
    double v[4][OZ_KMAX / 32];  // four columns' loads in flight
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const double* col = B + (long long)min(c0 + warp + 8 * (q0 + q), n - 1) * ldb;
#pragma unroll
      for (int r = 0; r < OZ_KMAX / 32; ++r) v[q][r] = col[min(lane + 32 * r, kb - 1)];
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int r = 0; r < OZ_KMAX / 32; ++r)
        if (lane + 32 * r < kb) km[r] = max(km[r], oz_ekey(v[q][r]));
  }
#pragma unroll
  for (int r = 0; r < OZ_KMAX / 32; ++r) red[warp][lane + 32 * r] = km[r];
  __syncthreads();
  const int k = threadIdx.x;
  if (k < kb) {
    unsigned v = 0u;
#pragma unroll
    for (int w = 0; w < 8; ++w) v = max(v, red[w][k]);
    if (v) oz_raise_key(kinfo + OZ_KI_H + k, (epoch << 12) | v);
  }
}

// Both operands in one launch, after oz_kscale_kernel. Blocks [0, m_pad/32):
// 32 rows of A (m x kb, column-major) each, staged through shared memory 64 k
// at a time so that the reads run along the columns; slices Sa[s][i][kk] cut
// against e_i + d_k, and on side A the row's error-budget test. Blocks after
// that: 8 columns of B (kb x n, column-major, a column contiguous in k) each,
// one warp per column; slices Sb[t][j][kk] cut against f_j - d_k, and on side
// B the column's test. Padding rows, columns and k are zero; so is every k
// whose column of A or row of B is zero (its products vanish). ul.L set: side B, and
// a flag sends the pass to the FP64 route.
__global__ void __launch_bounds__(256)
oz_split_kernel(const double* __restrict__ A, long long lda, int m, const double* __restrict__ B,
                long long ldb, int n, int kb, int kpad, int m_pad, int n_pad,
                __nv_bfloat16* Sa, __nv_bfloat16* Sb, double* rs, double* cs,
                unsigned long long* kinfo, unsigned long long epoch, OzUnitLower ul) {
  __shared__ int s_c[OZ_KMAX], s_h[OZ_KMAX], s_d[OZ_KMAX];
  const bool side_b = ul.L != nullptr;
  if (blockIdx.x == 0 && (int)threadIdx.x < ul.nflags && ul.flags[threadIdx.x]) atomicMax(kinfo + OZ_KI_FLAG, epoch);
  // A blocks: the CTA's 32 rows x kpad of A, as bits, sA[kk * 33 + row],
  // loaded once (before the balancing words, so both reads overlap) and read
  // by the budget test and the slicing
  extern __shared__ unsigned long long sA[];
  const int nrb = m_pad / 32;
  if ((int)blockIdx.x < nrb) {
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int i = (int)blockIdx.x * 32 + tx;
    unsigned long long v[OZ_KMAX / 8];
#pragma unroll
    for (int q = 0; q < OZ_KMAX / 8; ++q) {
      const int kk = ty + 8 * q;
      v[q] = (i < m && kk < kb) ? (unsigned long long)__double_as_longlong(A[i + (long long)kk * lda])
                                : 0ULL;
    }
#pragma unroll
    for (int q = 0; q < OZ_KMAX / 8; ++q) {
      const int kk = ty + 8 * q;
      if (kk < kpad) sA[kk * 33 + tx] = v[q];
    }
  }
  for (int k = threadIdx.x; k < OZ_KMAX; k += 256) {
    int h = OZ_NOEXP, c = OZ_NOEXP;
    if (k < kb) {
      h = oz_word_exp(kinfo[OZ_KI_H + k], epoch);
      c = oz_word_exp(kinfo[OZ_KI_C + k], epoch);
      if (h == OZ_NOEXP || c == OZ_NOEXP) h = c = OZ_NOEXP;  // k contributes nothing
    }
    s_h[k] = h;
    s_c[k] = c;
    s_d[k] = (c == OZ_NOEXP) ? OZ_NOEXP : (side_b ? -h : c);
  }
  __syncthreads();
  if ((int)blockIdx.x < nrb) {
    __shared__ int redE[8][33], redF[8][33];
    __shared__ int s_e[32];
    __shared__ int s_bad[32];
    __shared__ int s_G;
    const int i0 = blockIdx.x * 32;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int i = i0 + tx;
    if (ty == 0) {  // G = max_k (c_k + h_k)
      int g = OZ_NOEXP;
      for (int q = 0; q < OZ_KMAX / 32; ++q) {
        const int k = tx + 32 * q;
        if (s_c[k] != OZ_NOEXP) g = max(g, s_c[k] + s_h[k]);
      }
      g = oz_warp_imax(g);
      if (tx == 0) s_G = g;
    }
    int em = OZ_NOEXP, fm = OZ_NOEXP, bad = 0;
    if (i < m)
      for (int kk = ty; kk < kb; kk += 8) {
        const unsigned long long mag = sA[kk * 33 + tx] & kMagMask;
        if (mag >= kInfBits) {
          bad = 1;
        } else if (mag != 0ULL && s_d[kk] != OZ_NOEXP) {
          const int ex = oz_scale_exp(mag);
          em = max(em, ex - s_d[kk]);
          fm = max(fm, ex + s_h[kk]);
        }
      }
    redE[ty][tx] = bad ? INT_MAX : em;
    redF[ty][tx] = fm;
    __syncthreads();
    if (ty == 0) {
      int r = OZ_NOEXP, F = OZ_NOEXP;
      bool anybad = false;
      for (int q = 0; q < 8; ++q) {
        anybad |= redE[q][tx] == INT_MAX;
        r = max(r, redE[q][tx] == INT_MAX ? OZ_NOEXP : redE[q][tx]);
        F = max(F, redF[q][tx]);
      }
      s_bad[tx] = anybad ? 1 : 0;
      s_e[tx] = r;
      // side A: row i's bound 2^(e_i + G) against its largest |A||B| term 2^F
      if (!anybad && r != OZ_NOEXP &&
          (!oz_scale_in_range(r) || (!side_b && r + s_G - F > OZ_BUDGET)))
        atomicMax(kinfo + OZ_KI_FLAG, epoch);
      if (i < m_pad) rs[i] = (i < m) ? oz_scale_value(r, anybad) : 0.0;
    }
    __syncthreads();
    const int r = threadIdx.x >> 3, g = threadIdx.x & 7;  // row r, k group g (8 values)
    const int row = i0 + r;
    const int e = s_e[r];
    const bool zero = s_bad[r] != 0 || e == OZ_NOEXP;
    for (int k0 = 0; k0 < kpad; k0 += 64) {
      unsigned long long W[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int kk = k0 + g * 8 + q;
        const unsigned long long bits = sA[kk * 33 + r];
        const int d = s_d[kk];
        W[q] = (zero || d == OZ_NOEXP) ? kDigitBias : oz_digits(bits, e + d);
      }
      if (row < m_pad) {
#pragma unroll
        for (int sl = 0; sl < OZ_S; ++sl) {
          uint4 h;
          h.x = oz_slice2(W[0], W[1], sl);
          h.y = oz_slice2(W[2], W[3], sl);
          h.z = oz_slice2(W[4], W[5], sl);
          h.w = oz_slice2(W[6], W[7], sl);
          *reinterpret_cast<uint4*>(Sa + ((size_t)sl * m_pad + row) * kpad + k0 + g * 8) = h;
        }
      }
    }
    return;
  }
  // columns of B: one warp per column, lane l holds k = l, l+32, ...
  const int j = ((int)blockIdx.x - nrb) * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (j >= n_pad) return;
  unsigned long long bits[OZ_KMAX / 32];
  int f = OZ_NOEXP, F = OZ_NOEXP, gg = OZ_NOEXP, bad = 0;
#pragma unroll
  for (int q = 0; q < OZ_KMAX / 32; ++q) {
    const int kk = lane + 32 * q;
    bits[q] = (j < n && kk < kb) ? (unsigned long long)__double_as_longlong(B[kk + (long long)j * ldb]) : 0ULL;
    const unsigned long long mag = bits[q] & kMagMask;
    if (s_d[kk] != OZ_NOEXP) gg = max(gg, s_c[kk] + s_h[kk]);
    if (mag >= kInfBits) {
      bad = 1;
    } else if (mag != 0ULL && s_d[kk] != OZ_NOEXP) {
      const int ex = oz_scale_exp(mag);
      f = max(f, ex + s_d[kk]);
      F = max(F, s_c[kk] + ex);
    }
  }
  f = oz_warp_imax(f);
  F = oz_warp_imax(F);
  gg = oz_warp_imax(gg);
  bad = __any_sync(0xffffffffu, bad) ? 1 : 0;
  if (lane == 0) {
    cs[j] = (j < n) ? oz_scale_value(f, bad != 0) : 0.0;
    // side B: column j's bound 2^(f_j + G) against its largest |A||B| term 2^F
    if (j < n && !bad && f != OZ_NOEXP &&
        (!oz_scale_in_range(f) || (side_b && f + gg - F > OZ_BUDGET)))
      atomicMax(kinfo + OZ_KI_FLAG, epoch);
  }
#pragma unroll
  for (int q = 0; q < OZ_KMAX / 32; ++q) {
    const int kk = lane + 32 * q;
    if (kk >= kpad) break;
    const int d = s_d[kk];
    const unsigned long long W =
        (bad || f == OZ_NOEXP || d == OZ_NOEXP) ? kDigitBias : oz_digits(bits[q], f - d);
#pragma unroll
    for (int sl = 0; sl < OZ_S; ++sl)
      Sb[((size_t)sl * n_pad + j) * kpad + kk] =
          __ushort_as_bfloat16((unsigned short)(oz_slice2(W, W, sl) & 0xffffu));
  }
}

// One tile of C (128 x 64) per CTA for K <= 64, balancing side A, keys already
// published: the CTA slices its own 128 x KP of A and KP x 64 of B into shared
// memory (where the tensor maps' swizzle puts them) instead of reading slices that
// oz_split_kernel left in memory. The same scales, digits and products as there;
// a row of A is sliced once per column tile, so this is for narrow C. A tile with a
// row outside the error budget (or a scale out of range) is computed in FP64
// arithmetic by itself.
//
// For the products inside a panel, one per 32 columns and on its critical path:
// what they take is latency (two launches, two trips through memory). Every LU
// factor is bit for bit the one of oz_split_kernel and ozgemm_kernel. Measured: a
// step of an LU of N = 4096 (128 of them) 6 us shorter.
template <int KP>
__global__ void __launch_bounds__(OZ_THREADS, 1)
oz_tile_kernel(const double* A, long long lda, int m, const double* B, long long ldb, int n, int kb,
               double alpha, double* C, long long ldc, int* status, unsigned long long* kinfo,
               unsigned long long epoch) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* base = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  unsigned char* sA = base;                        // 7 x 16 KB: rows of 128 bytes (64 k)
  unsigned char* sB = base + OZ_S * A_SLICE_BYTES; // 7 x 8 KB
  constexpr int VA = KP / 4, VB = KP / 8;          // values of A and of B per worker thread
  __shared__ uint64_t s_full;
  __shared__ uint32_t s_tmem;
  __shared__ int s_d[KP], s_h[KP];
  __shared__ int s_E[4][OBM], s_F[4][OBM];
  __shared__ double s_rs[OBM], s_cs[OBN];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  wait_for_previous();
  launch_dependents();
  const int failed = *(volatile int*)status != 0;  // an earlier wait gave up
  const int tiles_m = (m + OBM - 1) / OBM, tiles_n = (n + OBN - 1) / OBN;
  int m0, n0;
  oz_tile(blockIdx.x, tiles_m, tiles_n, m0, n0);
  // worker threads: 16 warps; thread t has row t % 128 and k range t / 128 of A,
  // column t / 8 and k range t % 8 of B
  const int t = (int)threadIdx.x - 64;
  const int ar = t & (OBM - 1), ak = (t >> 7) * VA, bc = t >> 3, bk = (t & 7) * VB;
  double av[VA], bv[VB];
  if (warp >= 2) {
    const double* arow = A + min(m0 + ar, m - 1);
    const double* bcol = B + (long long)min(n0 + bc, n - 1) * ldb;
#pragma unroll
    for (int q = 0; q < VA; ++q) av[q] = arow[(long long)min(ak + q, kb - 1) * lda];
#pragma unroll
    for (int q = 0; q < VB; ++q) bv[q] = bcol[min(bk + q, kb - 1)];
    if (t < KP) {
      int h = OZ_NOEXP, c = OZ_NOEXP;
      if (t < kb) {
        h = oz_word_exp(kinfo[OZ_KI_H + t], epoch);
        c = oz_word_exp(kinfo[OZ_KI_C + t], epoch);
        if (h == OZ_NOEXP || c == OZ_NOEXP) h = c = OZ_NOEXP;  // k contributes nothing
      }
      s_h[t] = h;
      s_d[t] = c;
    }
  } else if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)),
                 "r"(OZ_TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  } else if (lane == 0) {
    mbar_init(&s_full, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  const int skip = __syncthreads_or(failed);  // (threads may have read different words)
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = s_tmem;
  if (skip) {
    if (warp == 0)
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(OZ_TMEM_COLS));
    return;
  }

  // scales: e_i over the row's four k ranges, f_j over the column's eight
  int f = OZ_NOEXP, G = OZ_NOEXP;
  if (warp >= 2) {
    int em = OZ_NOEXP, fm = OZ_NOEXP;
    bool bad = false;
#pragma unroll
    for (int q = 0; q < VA; ++q) {
      if (m0 + ar >= m || ak + q >= kb) av[q] = 0.0;
      const unsigned long long mag = (unsigned long long)__double_as_longlong(av[q]) & kMagMask;
      const int d = s_d[ak + q];
      if (mag >= kInfBits) {
        bad = true;
      } else if (mag != 0ULL && d != OZ_NOEXP) {
        const int ex = oz_scale_exp(mag);
        em = max(em, ex - d);
        fm = max(fm, ex + s_h[ak + q]);
      }
    }
    s_E[t >> 7][ar] = bad ? INT_MAX : em;
    s_F[t >> 7][ar] = fm;
#pragma unroll
    for (int q = 0; q < VB; ++q) {
      if (n0 + bc >= n || bk + q >= kb) bv[q] = 0.0;
      const unsigned long long mag = (unsigned long long)__double_as_longlong(bv[q]) & kMagMask;
      const int d = s_d[bk + q];
      if (mag >= kInfBits) f = INT_MAX;
      else if (mag != 0ULL && d != OZ_NOEXP) f = max(f, oz_scale_exp(mag) + d);
    }
#pragma unroll
    for (int off = 4; off > 0; off >>= 1) f = max(f, __shfl_xor_sync(0xffffffffu, f, off));
#pragma unroll
    for (int k = lane; k < KP; k += 32)
      if (s_d[k] != OZ_NOEXP) G = max(G, s_d[k] + s_h[k]);
    G = oz_warp_imax(G);
  }
  __syncthreads();
  int e = OZ_NOEXP;
  bool out = false;
  if (warp >= 2) {
    e = max(max(s_E[0][ar], s_E[1][ar]), max(s_E[2][ar], s_E[3][ar]));
    const int F = max(max(s_F[0][ar], s_F[1][ar]), max(s_F[2][ar], s_F[3][ar]));
    // (as in oz_split_kernel: row i's bound 2^(e_i + G) against its largest term)
    if (e != INT_MAX && e != OZ_NOEXP) out = !oz_scale_in_range(e) || e + G - F > OZ_BUDGET;
    if (f != INT_MAX && f != OZ_NOEXP) out = out || !oz_scale_in_range(f);
    if (ak == 0) s_rs[ar] = oz_scale_value(e, e == INT_MAX);
    if (bk == 0) s_cs[bc] = oz_scale_value(f, f == INT_MAX);
  }
  if (__syncthreads_or(out)) {
    if (threadIdx.x == 0 && atomicMax(kinfo + OZ_KI_FLAG, epoch) < epoch) atomicAdd(&g_oz_fp64_routes, 1ULL);
    oz_fp64_tiles(base, m, n, kb, A, lda, B, ldb, alpha, C, ldc, blockIdx.x, 1, tiles_m, tiles_n, 0);
  } else {
    if (warp >= 2) {
      // slices; 8 values are one 16-byte piece of a row, piece p of row r at p ^ (r % 8)
#pragma unroll
      for (int q0 = 0; q0 < VA; q0 += 8) {
        unsigned long long W[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const int d = s_d[ak + q0 + q];
          W[q] = (e == INT_MAX || e == OZ_NOEXP || d == OZ_NOEXP)
                     ? kDigitBias
                     : oz_digits((unsigned long long)__double_as_longlong(av[q0 + q]), e + d);
        }
        unsigned char* dst = sA + ar * 128 + ((((ak + q0) >> 3) ^ (ar & 7)) << 4);
#pragma unroll
        for (int sl = 0; sl < OZ_S; ++sl)
          *reinterpret_cast<uint4*>(dst + sl * A_SLICE_BYTES) =
              make_uint4(oz_slice2(W[0], W[1], sl), oz_slice2(W[2], W[3], sl), oz_slice2(W[4], W[5], sl),
                         oz_slice2(W[6], W[7], sl));
      }
      unsigned long long W[VB];
#pragma unroll
      for (int q = 0; q < VB; ++q) {
        const int d = s_d[bk + q];
        W[q] = (f == INT_MAX || f == OZ_NOEXP || d == OZ_NOEXP)
                   ? kDigitBias
                   : oz_digits((unsigned long long)__double_as_longlong(bv[q]), f - d);
      }
      unsigned char* dst = sB + bc * 128 + (((bk >> 3) ^ (bc & 7)) << 4) + (bk & 7) * 2;
#pragma unroll
      for (int sl = 0; sl < OZ_S; ++sl)
#pragma unroll
        for (int q = 0; q < VB; q += 4)
          *reinterpret_cast<uint2*>(dst + sl * B_SLICE_BYTES + q * 2) =
              make_uint2(oz_slice2(W[q], W[q + 1], sl), oz_slice2(W[q + 2], W[q + 3], sl));
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // (the tensor core reads them)
    }
    __syncthreads();
    if (warp == 1) {
      if (lane == 0) {
        const uint64_t adesc = smem_desc_sw128(sA), bdesc = smem_desc_sw128(sB);
#pragma unroll
        for (int sl = 0; sl < OZ_S; ++sl)
#pragma unroll
          for (int kk = 0; kk < KP / 16; ++kk)
#pragma unroll
            for (int t0 = 0; t0 + sl < OZ_S; t0 += 4) {
              const int cnt = OZ_S - sl - t0 < 4 ? OZ_S - sl - t0 : 4;
              umma_f16(tmem + (uint32_t)((sl + t0) * OBN), adesc + (uint64_t)((sl * A_SLICE_BYTES + kk * 32) >> 4),
                       bdesc + (uint64_t)((t0 * B_SLICE_BYTES + kk * 32) >> 4), oz_idesc(cnt * OBN),
                       sl > 0 || kk > 0 ? 1u : 0u);
            }
        umma_commit(&s_full);
      }
    } else if (warp >= 2) {
      const int quad = warp & 3, cg = (warp - 2) >> 2;
      const int lr = quad * 32 + lane, nb0 = n0 + cg * OZ_EC;
      const int ncol = m0 + lr < m ? min(OZ_EC, n - nb0) : 0;
      double* crow = C + (long long)(m0 + lr) + (long long)nb0 * ldc;
      double cv[OZ_EC], sc[OZ_EC];
#pragma unroll
      for (int j = 0; j < OZ_EC; ++j) cv[j] = j < ncol ? crow[(long long)j * ldc] : 0.0;
      if (mbar_wait(&s_full, 0)) {
        asm volatile("tcgen05.fence::after_thread_sync;");
        long long I[OZ_EC];
        oz_read_sums(tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(cg * OZ_EC), I, [] {});
#pragma unroll
        for (int j = 0; j < OZ_EC; ++j) sc[j] = s_cs[cg * OZ_EC + j];
        oz_update_c(I, cv, crow, ldc, ncol, alpha, s_rs[lr], sc);
      } else if (lane == 0) {
        atomicExch(status, (int)kFlagTimeout);
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(OZ_TMEM_COLS));
}
constexpr int kTileSmem = 1024 + OZ_S * (A_SLICE_BYTES + B_SLICE_BYTES);

// 2D map over the slices: rows = S * rows_pad (slice-major), kpad columns of
// BF16, box {64, box_rows}, 128-byte swizzle.
bool make_slice_map(CUtensorMap* map, const void* ptr, int rows_total, int kpad, int box_rows) {
  auto enc = get_encode();
  if (!enc) return false;
  cuuint64_t dims[2] = {(cuuint64_t)kpad, (cuuint64_t)rows_total};
  cuuint64_t strides[1] = {(cuuint64_t)kpad * 2};
  cuuint32_t box[2] = {(cuuint32_t)OBK, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims,
                   strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

// dynamic shared memory of oz_split_kernel: the A rows of one CTA
inline size_t oz_split_smem(int kpad) { return (size_t)kpad * 33 * sizeof(unsigned long long); }

cudaError_t oz_smem_once() {
  static const cudaError_t e = cudaFuncSetAttribute(
      ozgemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)oz_smem_bytes());
  static const cudaError_t e2 = cudaFuncSetAttribute(
      oz_split_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)oz_split_smem(OZ_KMAX));
  static const cudaError_t e3 =
      cudaFuncSetAttribute(oz_tile_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTileSmem);
  static const cudaError_t e4 =
      cudaFuncSetAttribute(oz_tile_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTileSmem);
  for (cudaError_t x : {e, e2, e3, e4})
    if (x != cudaSuccess) return x;
  return cudaSuccess;
}

inline int round_up(int x, int q) { return (x + q - 1) / q * q; }

int g_oz_tiles_per_cta = 4;

// A product of k <= 64 in one launch (oz_tile_kernel): up to two tiles per SM, each
// tile slicing its operands itself. In us for a whole LU, with and without: N = 600
// 1699 / 1794, 4096 14020 / 14750; without the limit N = 16384 takes 117.2 ms instead
// of 115.8 (116.7 without), its products of 512 tiles then being the slower way.
inline bool oz_one_launch(int m, int n) {
  return (m + OBM - 1) / OBM * ((n + OBN - 1) / OBN) <= 2 * num_sms();
}

}  // namespace

void oz_set_tiles_per_cta(int t) { g_oz_tiles_per_cta = t < 1 ? 1 : (t > 4096 ? 4096 : t); }

size_t oz_scratch_bytes(int m, int n, int k) {
  const size_t kp = (size_t)round_up(k < OZ_KMAX ? k : OZ_KMAX, OBK);
  const size_t mp = (size_t)round_up(m, OBM), np = (size_t)round_up(n, OBN);
  return OZ_KINFO_BYTES + OZ_S * (mp + np) * kp * 2 + (mp + np) * sizeof(double) + 1024;
}

bool oz_fits(const OzScratch& sc, int m, int n, int k) {
  return sc.ptr && oz_scratch_bytes(m, n, k) <= sc.bytes;
}

// Passes that took the FP64 route on the current device since the library
// loaded (the count lives in device memory).
long long oz_fp64_routes() {
  unsigned long long v = 0;
  if (cudaMemcpyFromSymbol(&v, g_oz_fp64_routes, sizeof(v)) != cudaSuccess) return -1;
  return (long long)v;
}

// Epochs only grow (process-wide, 52 bits: no wrap in practice).
static std::atomic<unsigned long long> g_oz_epochs{0};

unsigned long long oz_new_epoch() {
  return (g_oz_epochs.fetch_add(1) + 1) & ((1ULL << 52) - 1);
}
unsigned long long* oz_ckeys(const OzScratch& sc) {
  return sc.ptr ? reinterpret_cast<unsigned long long*>(sc.ptr) + OZ_KI_C : nullptr;
}
unsigned long long* oz_hkeys(const OzScratch& sc) {
  return sc.ptr ? reinterpret_cast<unsigned long long*>(sc.ptr) + OZ_KI_H : nullptr;
}

// C (m x n) += alpha * A (m x k) * B (k x n), all FP64 column-major, through
// the sliced BF16 product; K is taken in passes of at most 256, each with its
// own balancing, budget test and (when the test trips) FP64 route.
static cudaError_t oz_dgemm_impl(const OzUnitLower& ul, unsigned long long keyed_epoch, const OzScratch& sc,
                                 int m, int n, int k, double alpha, const double* A, long long lda,
                                 const double* B, long long ldb, double* C, long long ldc,
                                 int* status, cudaStream_t s, int max_ctas = 0) {
  if (m <= 0 || n <= 0 || k <= 0) return cudaSuccess;
  if (!oz_fits(sc, m, n, k)) return cudaErrorMemoryAllocation;
  if (keyed_epoch && k > OZ_KMAX) return cudaErrorInvalidValue;
  SL_TRY(oz_smem_once());
  const int m_pad = round_up(m, OBM), n_pad = round_up(n, OBN);
  if (keyed_epoch && !ul.L && k <= 64 && oz_one_launch(m, n)) {
    unsigned long long* kinfo = reinterpret_cast<unsigned long long*>(sc.ptr);
    auto kern = k <= 32 ? oz_tile_kernel<32> : oz_tile_kernel<64>;
    count_launches(1);
    return launch_after(kern, dim3(m_pad / OBM * (n_pad / OBN)), OZ_THREADS, kTileSmem, s, A, lda, m, B, ldb, n, k,
                        alpha, C, ldc, status, kinfo, keyed_epoch);
  }
  for (int k0 = 0; k0 < k; k0 += OZ_KMAX) {
    const int kb = (k - k0) < OZ_KMAX ? (k - k0) : OZ_KMAX;
    const int kpad = round_up(kb, OBK);
    const unsigned long long epoch = keyed_epoch ? keyed_epoch : oz_new_epoch();
    unsigned char* p = reinterpret_cast<unsigned char*>(sc.ptr);
    unsigned long long* kinfo = reinterpret_cast<unsigned long long*>(p);
    __nv_bfloat16* sa = reinterpret_cast<__nv_bfloat16*>(p + OZ_KINFO_BYTES);
    __nv_bfloat16* sb = sa + (size_t)OZ_S * m_pad * kpad;
    double* rs = reinterpret_cast<double*>(sb + (size_t)OZ_S * n_pad * kpad);
    double* cs = rs + m_pad;
    const double* Ak = A + (long long)k0 * lda;
    const double* Bk = B + k0;
    const int nab = (m + 31) / 32, nbb = (n + 63) / 64;
    if (!keyed_epoch) {
      oz_kscale_kernel<<<nab + nbb, 256, 0, s>>>(Ak, lda, m, Bk, ldb, n, kb, nab, kinfo, epoch);
      count_launches(1);
    }
    oz_split_kernel<<<m_pad / 32 + n_pad / 8, 256, oz_split_smem(kpad), s>>>(Ak, lda, m, Bk, ldb, n, kb, kpad, m_pad,
                                                          n_pad, sa, sb, rs, cs, kinfo, epoch,
                                                          ul);
    CUtensorMap ta, tb;
    if (!make_slice_map(&ta, sa, OZ_S * m_pad, kpad, OBM) ||
        !make_slice_map(&tb, sb, OZ_S * n_pad, kpad, OBN))
      return cudaErrorInvalidResourceHandle;
    const int tiles = (m_pad / OBM) * (n_pad / OBN);
    // a few tiles per CTA: enough to overlap one tile's epilogue with the
    // next one's products, few enough that every SM gets work and SMs free
    // up often
    int tpc = std::max(1, std::min(g_oz_tiles_per_cta, tiles / num_sms()));
    if (max_ctas > 0 && (tiles + tpc - 1) / tpc > max_ctas) tpc = (tiles + max_ctas - 1) / max_ctas;
    const int grid = (tiles + tpc - 1) / tpc;
    ozgemm_kernel<<<grid, OZ_THREADS, oz_smem_bytes(), s>>>(ta, tb, m, n, kpad, m_pad, n_pad, rs,
                                                            cs, alpha, C, ldc, tpc, status, Ak,
                                                            lda, Bk, ldb, kb, kinfo, epoch, ul);
    count_launches(2);
    SL_TRY(cudaGetLastError());
  }
  return cudaSuccess;
}

cudaError_t oz_dgemm(const OzScratch& sc, int m, int n, int k, double alpha, const double* A,
                     long long lda, const double* B, long long ldb, double* C, long long ldc,
                     int* status, cudaStream_t s, int max_ctas) {
  return oz_dgemm_impl(OzUnitLower(), 0ULL, sc, m, n, k, alpha, A, lda, B, ldb, C, ldc, status, s, max_ctas);
}

cudaError_t oz_dgemm_keyed(const OzScratch& sc, unsigned long long epoch, int m, int n, int k,
                           double alpha, const double* A, long long lda, const double* B,
                           long long ldb, double* C, long long ldc, int* status, cudaStream_t s,
                           int max_ctas) {
  return oz_dgemm_impl(OzUnitLower(), epoch, sc, m, n, k, alpha, A, lda, B, ldb, C, ldc, status, s, max_ctas);
}

cudaError_t oz_unit_lower_solve(const OzScratch& sc, int m, int n, const double* N, long long ldn,
                                const double* L, long long ldl, const int* flags, int nflags, double* B,
                                long long ldb, int* status, cudaStream_t s, int max_ctas) {
  if (m > OZ_KMAX || nflags > OZ_KMAX) return cudaErrorInvalidValue;
  OzUnitLower ul;
  ul.L = L;
  ul.ldl = ldl;
  ul.flags = flags;
  ul.nflags = nflags;
  return oz_dgemm_impl(ul, 0ULL, sc, m, n, m, 1.0, N, ldn, B, ldb, B, ldb, status, s, max_ctas);
}

}  // namespace sl
