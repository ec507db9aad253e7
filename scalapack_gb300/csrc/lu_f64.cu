// FP64 LU factorization and solve on one GB300 (the plain FP64 drop-in path).
//
// Structure follows PDGETRF on a 1x1 grid (SRC/pdgetrf.f:219-295):
//   for each NB-wide block column j:
//     panel      PDGETF2 (SRC/pdgetf2.f:206-237)  -> panel_cluster_kernel / panel_kernel
//                                                    <double>, blocked by 32
//     swaps      PDLASWP (SRC/pdlaswp.f:163-172)  -> laswp_apply_kernel (composite plan of
//                                                    the panel's interchanges, both sides)
//     U12        PDTRSM  (SRC/pdgetrf.f:280-282)  -> inverse of L11 and a sliced product
//                                                    (trsm_strip_kernel in the DMMA mode)
//     update     PDGEMM  (SRC/pdgetrf.f:288-290)  -> oz_dgemm (FP64 from exact BF16 slice
//                                                    products, ozgemm_f64.cu; dgemm DMMA,
//                                                    dgemm_f64.cu, in the DMMA mode)
// with the next panel factored on a second stream (look-ahead), and PDGETRS
// (SRC/pdgetrs.f:250-284): pivots on B (PDLAPIV) as one composed permutation,
// then unit-lower and non-unit-upper solves: chained over 64-row blocks for few
// right-hand sides (trsv_f64.cu), else by 128-row blocks (diagonal-block inverses
// and sliced products for NOTRAN, substitution strips otherwise).
//
// The NB-wide panel is factored as 32-column sub-panels; each is one kernel whose
// CTAs hold disjoint row slices of the sub-panel in shared memory and exchange
// each column's pivot candidates, within a cluster through distributed shared
// memory or between more CTAs through tagged words in L2 (bounded polls, no grid
// barrier). The remaining columns of the panel are brought up to date by
// inpanel_step_kernel and a sliced product, so the final factors, pivots and INFO
// are those of the reference's column-by-column PDGETF2 in exact arithmetic.
#include <algorithm>
#include <climits>

#include <cmath>
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"
#include "lu_kernels.cuh"
#include "sl_internal.h"

namespace sl {

size_t panel_cand_doubles() { return kPanelCandDoubles; }
static_assert(kPanelCandDoubles == (size_t)PX_WORDS, "exchange area layout");

// Rows per CTA are capped by 200 KB of shared memory (rpc * 33 doubles),
// rounded down to a multiple of 8: 768 rows; one CTA per SM.
int panel_max_rows() { return num_sms() * 768; }
// Global rows of a tall panel: every CTA's slice (rows rounded up to 8), and
// their labels.
size_t panel_tile_doubles(int m) {
  const size_t rows = (size_t)m + (size_t)8 * PMAXG;
  return rows * PW + (rows + 1) / 2;
}

static long long g_spin_limit = kSpinLimit;
long long spin_limit() { return g_spin_limit; }
void set_spin_limit(long long polls) { g_spin_limit = polls < 0 ? kSpinLimit : polls; }

static int g_panel_min_rows = 0;  // 0: automatic (FP32 256, FP64 128)
int panel_min_rows() { return g_panel_min_rows; }
static int g_panel_ctas = 64;  // CTAs a panel's rows are spread over (before the minimum rows)
// Sub-panels per in-panel block (factor_panel); 0: one up to 12000 rows, where a
// block's second step costs a launch more than its deeper products save, two above,
// where the products are what takes the time. PDGETRF, ms, one / two: N = 4096 13.2 /
// 14.0, 6001 x 3007 11.1 / 11.7, N = 8192 31.7 / 32.7, N = 12000 61.6 / 62.6; 20000 x
// 4000 28.2 / 27.4, 30000 x 1000 8.2 / 7.6.
// One rounds C once per 32 columns inside a panel, two once per 64: where the diagonal is
// heavy and the updates small beside it the factors' error is up to 8 % larger (6001 x
// 3007 2.94e-16 / 2.72e-16 of their norm, N = 8192 3.86 / 3.76, N = 600 4.43 / 4.40); on
// uniform matrices it is the same to 1 % (N = 4096 3.95e-13 / 3.93e-13) or smaller (N = 600
// 1.91e-14 / 2.03e-14).
constexpr int kDeepPanelRows = 12000;
static int g_panel_ib = 0;
void set_panel_ib(int ib) { g_panel_ib = ib < 1 ? 0 : (ib > 8 ? 8 : ib); }
int panel_ctas() { return g_panel_ctas; }
int panel_cluster_rows() { return 128; }
void set_panel_ctas(int g) { g_panel_ctas = g < 8 ? 8 : (g > 224 ? 224 : g); }
void set_panel_min_rows(int rows) { g_panel_min_rows = rows <= 0 ? 0 : (rows < 8 ? 8 : (rows > 768 ? 768 : rows)); }

SplitKScratch& splitk_scratch() {
  static SplitKScratch sc;
  return sc;
}

// dst[i] = src[i] + delta (pivot base conversion at the C ABI).
__global__ void ipiv_shift_kernel(const int* __restrict__ src, int* dst, int n, int delta) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[i] = src[i] + delta;
}

cudaError_t ipiv_shift(const int* src, int* dst, int n, int delta, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  ipiv_shift_kernel<<<(n + 255) / 256, 256, 0, s>>>(src, dst, n, delta);
  count_launches(1);
  return cudaGetLastError();
}

// Composed row permutation of the n sequential interchanges j <-> ipiv[j]:
// perm[i] = original row that ends in row i. The interchanges are cut into at
// most kPermSegs segments; per segment, thread i walks its interchanges backwards
// from the last, following the row whose content ends in row i (interchange j
// moves it from ipiv[j] to j or from j to ipiv[j]), and rows then pass through
// the segments' maps from the last to the first (follow_perm). One walk of all n
// interchanges per row is a chain of two compares and selects each, 150 us at n =
// 8192; in 16 segments, on all SMs, the launch that also inverts the diagonal
// blocks takes 62. The pivots are
// compared, never used as addresses: a row label outside the matrix (from an
// invalid IPIV) is followed by walking the segment itself. A block does 256 rows
// of one segment, from shared memory (sp, kPermSmem ints) when it fits.
constexpr int kPermSmem = 8192;
__device__ __forceinline__ int walk_pivots(const int* pv, int lo, int hi, int q) {
#pragma unroll 4
  for (int j = hi - 1; j >= lo; --j) {
    const int p = pv[j - lo];
    q = (q == j) ? p : ((q == p) ? j : q);
  }
  return q;
}
__device__ __forceinline__ void perm_segment(int block, const int* __restrict__ ipiv, int n, int* maps,
                                             int* sp) {
  const int len = perm_seg_len(n), nrb = (n + 255) / 256;
  const int sgm = block / nrb, i = (block % nrb) * 256 + threadIdx.x;
  const int lo = sgm * len, hi = min(n, lo + len);
  const int* pv = ipiv + lo;
  if (len <= kPermSmem) {
    for (int j = threadIdx.x; j < hi - lo; j += 256) sp[j] = pv[j];
    __syncthreads();
    pv = sp;
  }
  const int q = walk_pivots(pv, lo, hi, i);
  if (i < n) maps[(size_t)sgm * n + i] = q;
}
__global__ void __launch_bounds__(256) perm_segments_kernel(const int* __restrict__ ipiv, int n, int* maps) {
  __shared__ int sp[kPermSmem];
  perm_segment(blockIdx.x, ipiv, n, maps, sp);
}
__global__ void __launch_bounds__(256)
perm_finish_kernel(const int* __restrict__ ipiv, int n, const int* __restrict__ maps, int* perm) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i < n) perm[i] = follow_perm(i, ipiv, n, maps);
}

cudaError_t perm_compose(const int* dipiv, int n, int* perm, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  const int nrb = (n + 255) / 256;
  perm_segments_kernel<<<nrb * perm_segs(n), 256, 0, s>>>(dipiv, n, perm + n);
  perm_finish_kernel<<<nrb, 256, 0, s>>>(dipiv, n, perm + n, perm);
  count_launches(2);
  return cudaGetLastError();
}

static int g_f64_update = 1;

void f64_update_set(int mode) { g_f64_update = (mode == 0) ? 0 : 1; }
int f64_update_get() { return g_f64_update; }

// C (m x n) -= A (m x k) * B (k x n) inside the factorization: the sliced
// tensor-core product when selected and its scratch fits, else FP64 DMMA.
// With look-ahead, the update of the columns right of the next panel runs
// beside that panel's kernels (on the auxiliary stream). The panel's
// cooperative kernel makes progress only once all its CTAs are resident, so
// the update keeps at least g_res_min SMs free for it; beyond that it takes
// the SMs it needs to finish within about one panel period (an SM's share of
// the sliced product being g_upd_flops_per_sm in that time) and leaves up to
// g_res_max to the panel chain. (0, 0): the update takes every SM.
static int g_res_min = 24, g_res_max = 88;
// Grid caps in the split step (bit mask): 1 the in-panel products and 2 the
// next panel's update keep to the SMs the trailing update leaves; 4 the
// caller's stream's U12 solve and interchanges keep to the update's SMs.
static int g_cap_mask = 7;
void set_inpanel_cap(int mask) { g_cap_mask = mask & 7; }
static double g_upd_flops_per_sm = 3.2e8;
void set_update_reserve(int min_sms, int max_sms) {
  g_res_min = std::max(0, std::min(min_sms, 120));
  g_res_max = std::max(g_res_min, std::min(max_sms, 120));
}
void set_update_share(double flops_per_sm) {
  g_upd_flops_per_sm = flops_per_sm > 1e6 ? flops_per_sm : 3.2e8;
}
static int update_ctas(double flops) {
  if (g_res_max <= 0) return 0;
  const int S = num_sms();
  const int want = (int)std::ceil(flops / g_upd_flops_per_sm);
  return std::max(1, std::max(S - g_res_max, std::min(S - g_res_min, want)));
}

static cudaError_t lu_update(const OzScratch& sc, int m, int n, int k, double alpha,
                             const double* A, long long lda, const double* B, long long ldb,
                             double* C, long long ldc, const LuWork& ws, cudaStream_t s,
                             int max_ctas = 0) {
  if (g_f64_update == 1 && oz_fits(sc, m, n, k))
    return oz_dgemm(sc, m, n, k, alpha, A, lda, B, ldb, C, ldc, ws.status, s, max_ctas);
  return dgemm(false, m, n, k, alpha, A, lda, B, ldb, 1.0, C, ldc, s);
}

// Largest NB whose inv(L11) - I is formed at the end of the panel (the U12 solve is
// then one product): the widest that factor_nb gives when blocks follow.
constexpr int kFullInvMax = 256;
static_assert(kDinv64Doubles >= (size_t)kFullInvMax * kFullInvMax, "inverse of L11");

// X = inv(L) - I for a unit-lower jb x jb L (jb <= 256): forward substitution of
// x = e_c per column c, in the order of a strip solve. A CTA takes the columns p
// and jb-1-p (a long one and a short one); its warp b owns rows 32b .. 32b+31, a
// lane per row. Block step s: warp s solves its 32 rows (x_q passed by a shuffle)
// and leaves them in shared memory, then the warps below subtract their 32 columns,
// L's next columns on their way meanwhile. Bound: the chain of 256 dependent FP64
// instructions and the FP64 unit's 20 cycles for each of a column's 1152: one warp
// per column (64 cycles for each of them) took 71 us, this 30. With a plan to make
// (plan != null), one extra block computes the panel's interchange plan
// (laswp_plan_block) in the same launch: both only read the finished panel.
//
// U12 = inv(L) A12 has an error of eps |inv(L)| |A12| where a substitution has eps |L|
// |U12|. flags[pair] = 1 where a column of the inverse has an entry of 64 or more, or one
// that is not finite: the U12 solve then substitutes (oz_unit_lower_solve). The largest
// entry in 256-wide blocks of random matrices, N = 256 .. 4096, is 4.2; scaled
// residual of U12 over random triangles, entries of the inverse up to 16: 0.1, up to
// 2^10: 0.5 (substitution 0.04), 2^12: 11, 2^40: 2e8.
__host__ __device__ inline int inv_cols_blocks(int jb) { return (jb + 1) / 2; }
__global__ void __launch_bounds__(256)
unit_lower_inv_cols_kernel(int jb, const double* L, long long ldl, double* X,
                           int ldx, int* flags, int k1, int k2, const int* ipiv, int* plan) {
  wait_for_previous();
  if (plan != nullptr && (int)blockIdx.x == inv_cols_blocks(jb)) {
    laswp_plan_block(k1, k2, ipiv, plan);
    return;
  }
  __shared__ double xs[2][2][32];  // [step parity][column][row]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, row = 32 * warp + lane;
  const int c0 = blockIdx.x, c1 = jb - 1 - c0;  // c0 <= c1; the same column when jb is odd
  const double* lrow = L + min(row, jb - 1);
  double x0 = row == c0 ? 1.0 : 0.0, x1 = row == c1 ? 1.0 : 0.0;
  const int nsteps = (jb + 31) / 32, sb = c0 / 32;
  // L(row, 32 s + q); outside the strict triangle's blocks the values are not used
  double lv[32], ln[32];
  auto load = [&](int s, double* v) {
    if (s <= warp && s < nsteps) {
#pragma unroll
      for (int q = 0; q < 32; ++q) v[q] = lrow[(long long)min(32 * s + q, jb - 1) * ldl];
    }
  };
  load(sb, lv);
  for (int s = sb; s < nsteps; ++s) {
    load(s + 1, ln);
    // column c begins at its own row: earlier columns of L do not enter
    const int f0 = c0 - 32 * s, f1 = c1 - 32 * s;
    const bool two = f1 <= 31;
    if (warp == s) {
#pragma unroll
      for (int q = 0; q < 32; ++q) {
        const double u0 = __shfl_sync(0xffffffffu, x0, q);
        if (lane > q && q >= f0) x0 = fma(-lv[q], u0, x0);
        if (two) {
          const double u1 = __shfl_sync(0xffffffffu, x1, q);
          if (lane > q && q >= f1) x1 = fma(-lv[q], u1, x1);
        }
      }
      xs[s & 1][0][lane] = x0;
      xs[s & 1][1][lane] = x1;
    }
    __syncthreads();
    if (warp > s && warp < nsteps) {
#pragma unroll
      for (int q = 0; q < 32; ++q)
        if (q >= f0) x0 = fma(-lv[q], xs[s & 1][0][q], x0);
      if (two) {
#pragma unroll
        for (int q = 0; q < 32; ++q)
          if (q >= f1) x1 = fma(-lv[q], xs[s & 1][1][q], x1);
      }
    }
#pragma unroll
    for (int q = 0; q < 32; ++q) lv[q] = ln[q];
  }
  if (row < jb) {
    X[row + (long long)c0 * ldx] = row > c0 ? x0 : 0.0;
    X[row + (long long)c1 * ldx] = row > c1 ? x1 : 0.0;
  }
  auto big = [](double x) { return ((__double2hiint(x) >> 20) & 0x7ff) >= 1023 + 6; };
  const int any = __syncthreads_or(row < jb && (big(x0) || big(x1)));
  if (threadIdx.x == 0) flags[blockIdx.x] = any;
}

// U12 = L11^-1 A12 (jb x nr, in place): with the sliced product and the inverse of L11
// at hand (formed at the end of its panel), A12 + (inv(L11) - I) A12 as one product,
// balanced by the rows of A12, which carry the pivots' scales. Otherwise the FP64
// strip solve.
static int* dinv_flags(double* dinv) { return reinterpret_cast<int*>(dinv + kDinvFlagsAt); }
static cudaError_t solve_u12(int jb, int nr, const double* L11, long long ldl, double* A12,
                             long long lda, const LuWork& ws, cudaStream_t s, int max_ctas = 0) {
  if (g_f64_update == 1 && ws.dinv64 && jb <= kFullInvMax && oz_fits(ws.oz, jb, nr, jb))
    return oz_unit_lower_solve(ws.oz, jb, nr, ws.dinv64, jb, L11, ldl, dinv_flags(ws.dinv64), inv_cols_blocks(jb),
                               A12, lda, ws.status, s, max_ctas);
  return trsm_strip<double, false, false, true>(jb, nr, L11, ldl, A12, lda, s);
}

// PDGETF2 on columns [j, j+jb), rows [j, m): 32-wide cooperative sub-panels,
// each followed by its row interchanges on the rest of the panel, the U solve
// and the GEMM update of the panel's remaining columns.
static cudaError_t factor_panel(int m, int n, double* dA, long long ldda, int* dipiv, int j, int jb,
                                const LuWork& ws, cudaStream_t s, int left = -1) {
  const int cb = left < 0 ? j : left;  // first column whose rows are interchanged
  auto Ap = [&](long long i, long long c) { return dA + i + c * ldda; };
  const OzScratch& sc = (ws.aux && s == ws.aux) ? ws.oz_aux : ws.oz;
  phase_begin(kPhPanel, s);
  double pflops = 0.0;
  // Sub-panels are grouped in blocks of ib: inside a block only the
  // next sub-panel's columns are brought up to date after each sub-panel
  // (left-looking, with every pivot row of the block so far), and the
  // columns beyond the block once at its end, with the block's rows -- fewer,
  // deeper in-panel products than one per sub-panel over all the remaining
  // columns.
  const int ib = g_panel_ib > 0 ? g_panel_ib : (m - j <= kDeepPanelRows ? 1 : 2);
  int blk_r0 = j;  // first row (= column) of the current block
  for (int c = 0, q = 0; c < jb; c += PW, ++q) {
    const int w = (jb - c) < PW ? (jb - c) : PW;
    const int r0 = j + c;
    const int kw = (m - r0) < w ? (m - r0) : w;
    double kflops = 0.0;
    for (int k = 0; k < kw; ++k) kflops += 2.0 * (double)(m - r0 - k - 1) * (w - k - 1) + (m - r0 - k - 1);
    pflops += kflops;
    phase_begin(kPhPanelKernel, s);
    SL_TRY(launch_panel<double>(dA, ldda, m, r0, r0, w, dipiv, ws, s, c > 0));
    phase_end(kPhPanelKernel, s, kflops, 16.0 * (double)(m - r0) * w);
    phase_begin(kPhPanelUpdate, s);
    if (c + w >= jb) {
      SL_TRY(inpanel_step<double>(dA, ldda, r0, r0 + kw, dipiv, cb, r0, r0 + w, j + jb, 0, kw, s));
    } else {
      const bool block_end = (q + 1) % ib == 0 || kw < w;
      // columns brought up to date now: the next sub-panel's, or at the end
      // of a block every remaining one; rows: the block's pivot rows (U, by
      // the strip solve) and every row below them (the product)
      const int ncols = block_end ? jb - c - w : ((jb - c - w) < PW ? (jb - c - w) : PW);
      const int kb = r0 + kw - blk_r0;
      const int rl = r0 + kw;  // first row below the block's pivot rows
      const bool fused = kb <= 64 && (kb - kw) % 32 == 0;  // (two sub-panels per block at most)
      if (!fused) SL_TRY(laswp<double>(dA, ldda, r0, r0 + kw, dipiv, cb, r0, r0 + w, j + jb, s));
      // (the block's earlier columns are read by the fused step: theirs first)
      else if (blk_r0 < r0) SL_TRY(laswp<double>(dA, ldda, r0, r0 + kw, dipiv, blk_r0, r0, r0, r0, s));
      // The solve also publishes the balancing keys of the product that
      // follows it: the row maxima of its own output (U) and, in extra blocks
      // of the same launch, the column maxima of the block's L.
      const bool keyed = rl < m && g_f64_update == 1 && oz_fits(sc, m - rl, ncols, kb);
      OzKeyJob kj;
      if (keyed) {
        kj.epoch = oz_new_epoch();
        kj.ckeys = oz_ckeys(sc);
        kj.hkeys = oz_hkeys(sc);
        kj.L = Ap(rl, blk_r0);
        kj.ldl = ldda;
        kj.lrows = m - rl;
        kj.lcols = kb;
      }
      if (fused)
        SL_TRY(inpanel_step<double>(dA, ldda, r0, r0 + kw, dipiv, cb, blk_r0, r0 + w, j + jb, ncols, kb, s, kj));
      else
        SL_TRY((trsm_strip<double, false, false, true>(kb, ncols, Ap(blk_r0, blk_r0), ldda,
                                                        Ap(blk_r0, r0 + w), ldda, s, kj)));
      pflops += (double)kb * kb * ncols;
      if (keyed) {
        SL_TRY(oz_dgemm_keyed(sc, kj.epoch, m - rl, ncols, kb, -1.0, Ap(rl, blk_r0), ldda,
                              Ap(blk_r0, r0 + w), ldda, Ap(rl, r0 + w), ldda, ws.status, s,
                              ws.aux && s == ws.aux ? ws.inpanel_ctas : 0));
        pflops += 2.0 * (double)(m - rl) * ncols * kb;
      } else if (rl < m) {
        SL_TRY(lu_update(sc, m - rl, ncols, kb, -1.0, Ap(rl, blk_r0), ldda, Ap(blk_r0, r0 + w), ldda,
                         Ap(rl, r0 + w), ldda, ws, s));
        pflops += 2.0 * (double)(m - rl) * ncols * kb;
      }
      if (block_end) blk_r0 = r0 + w;
    }
    phase_end(kPhPanelUpdate, s, 0.0, 0.0);
  }
  phase_begin(kPhPanelInverse, s);
  // the panel's interchanges in composite form, for the row interchanges of
  // the other columns (computed here, on the panel's stream)
  const int npiv = (m - j) < jb ? (m - j) : jb;
  const bool more = j + jb < n;  // columns to the right: they want both of what follows
  const bool want_plan = ws.swap_plan && npiv <= LSW_MAXP && (more || j > 0);
  // inverses of L11's diagonal blocks for the U12 solve of this step
  if (more && g_f64_update == 1 && ws.dinv64 && npiv == jb && jb <= kFullInvMax) {
    // inv(L11) - I whole (jb x jb, leading dimension jb), and the interchange
    // plan in the same launch
    if (want_plan && npiv <= 0) SL_TRY(cudaMemsetAsync(ws.swap_plan, 0, sizeof(int), s));
    const bool fused = want_plan && npiv > 0;
    SL_TRY(launch_after(unit_lower_inv_cols_kernel, dim3(inv_cols_blocks(jb) + (fused ? 1 : 0)), 256, 0, s, jb, Ap(j, j),
                        ldda, ws.dinv64, jb, dinv_flags(ws.dinv64), j, j + npiv, dipiv, fused ? ws.swap_plan : nullptr));
    count_launches(1);
  } else if (want_plan) {
    SL_TRY(laswp_plan(j, j + npiv, dipiv, ws.swap_plan, s));
  }
  phase_end(kPhPanelInverse, s, (double)jb * jb * jb / 3.0, 16.0 * (double)jb * jb);
  phase_end(kPhPanel, s, pflops, 16.0 * (double)(m - j) * jb);
  return cudaSuccess;
}

// Step 0 of the right-looking loop while the columns arrive in chunks (see
// dgetrf_device; m, n > 2 nb, panel 0 factored): the next panel's columns
// first, then the look-ahead panel on ws.aux, then the remaining columns of
// each chunk once it has landed.
template <typename WaitCols>
static cudaError_t step0_by_chunks(int m, int n, double* dA, long long ldda, int* dipiv, int nb,
                                   const LuWork& ws, cudaStream_t s, WaitCols& wait_cols) {
  auto Ap = [&](long long i, long long c) { return dA + i + c * ldda; };
  const int mn = m < n ? m : n;
  const int jb = nb, jn = nb;
  const int jb2 = (mn - jn) < nb ? (mn - jn) : nb;
  // step 0 on columns [c0, c1): interchanges, U12 solve, trailing update
  auto step_cols = [&](int c0, int c1, bool planned, const LuWork& w) -> cudaError_t {
    if (c1 <= c0) return cudaSuccess;
    const int nc = c1 - c0;
    phase_begin(kPhLaswp, s);
    if (planned) SL_TRY(laswp_planned<double>(dA, ldda, 0, jb, dipiv, w.swap_plan, 0, 0, c0, c1, s));
    else SL_TRY(laswp<double>(dA, ldda, 0, jb, dipiv, 0, 0, c0, c1, s));
    phase_end(kPhLaswp, s, 0.0, 32.0 * jb * (double)nc);
    phase_begin(kPhTrsm, s);
    SL_TRY(solve_u12(jb, nc, Ap(0, 0), ldda, Ap(0, c0), ldda, w, s));
    phase_end(kPhTrsm, s, (double)jb * jb * nc, 8.0 * (0.5 * jb * jb + 2.0 * jb * nc));
    if (jn < m) {
      const double mr = (double)(m - jn);
      phase_begin(kPhGemm, s);
      SL_TRY(lu_update(w.oz, m - jn, nc, jb, -1.0, Ap(jn, 0), ldda, Ap(0, c0), ldda, Ap(jn, c0),
                       ldda, w, s));
      phase_end(kPhGemm, s, 2.0 * mr * nc * jb, 8.0 * (mr * jb + (double)jb * nc + 2.0 * mr * nc));
    }
    return cudaSuccess;
  };
  SL_TRY(wait_cols(jn + jb2));
  SL_TRY(step_cols(jn, jn + jb2, true, ws));
  // the look-ahead panel rewrites the interchange plan and ws.dinv64: the
  // rest of step 0 reads dipiv and a copy of panel 0's inverses instead
  LuWork w0 = ws;
  w0.swap_plan = nullptr;
  if (g_f64_update == 1 && ws.dinv64) {
    SL_TRY(cudaMemcpyAsync(ws.dinv64_step0, ws.dinv64, kDinv64Doubles * sizeof(double), cudaMemcpyDeviceToDevice, s));
    w0.dinv64 = ws.dinv64_step0;
  }
  SL_TRY(cudaEventRecord(ws.ev_next, s));
  SL_TRY(cudaStreamWaitEvent(ws.aux, ws.ev_next, 0));
  SL_TRY(factor_panel(m, n, dA, ldda, dipiv, jn, jb2, ws, ws.aux));
  SL_TRY(cudaEventRecord(ws.ev_panel, ws.aux));
  const int nck = ws.ncol_chunks < kMaxColChunks ? ws.ncol_chunks : kMaxColChunks;
  for (int c = 0; c < nck; ++c) {
    const int lo = c ? ws.col_end[c - 1] : 0, hi = ws.col_end[c];
    const int a = lo > jn + jb2 ? lo : jn + jb2, b = hi < n ? hi : n;
    if (b <= a) continue;
    SL_TRY(wait_cols(b));
    SL_TRY(step_cols(a, b, false, w0));
  }
  return wait_cols(INT_MAX);
}

// The last columns of a factorization as one panel, as small matrices are (the
// launches of a block beside its panel cost more than the wider products), their
// interchanges applied to the `left` columns before them by the in-panel steps. In us,
// without / with: N = 1600 4519 / 4229, N = 2000 5746 / 5454 (up to 1536 columns: 5510),
// N = 3000 9198 / 8923, N = 4096 13210 / 13148, N = 8192 no difference. Its columns'
// updates are rounded once per 32 columns instead of once per 256: error of the factors
// with a heavy diagonal 2 % larger (N = 2000 5.00e-16 / 4.91e-16), of uniform ones 1 to 6 %
// smaller (1.56e-13 / 1.65e-13).
static bool one_panel_tail(int m, int n, int left) {
  return n <= 1024 && left <= 4096 && ((m + 127LL) / 128) * ((n + 63) / 64) <= 2LL * num_sms();
}

// Right-looking blocked LU. With look-ahead resources in `ws`, the panel of
// step j+1 is factored on ws.aux while the trailing update of step j runs on
// s: the columns of the next panel are updated first (event ev_next), the
// next panel starts as soon as they are ready, and step j+1 waits for it
// (event ev_panel). Panel and update touch disjoint columns, and each element
// is accumulated in the same order either way, so the factors are the same.
//
// With columns still arriving (ws.ncol_chunks > 0), s waits for each column
// chunk just before the first operation on it: panel 0 starts when its
// columns are in place, and step 0's interchanges, U12 solve and update run
// chunk by chunk as the rest lands. The interchanges and the update are
// independent per column; the U12 solve's first product balances its slices
// by the row maxima of the columns it is given, so those rows agree with the
// whole-width step to rounding (same pivots). After the look-ahead panel is
// launched the step-0 operations must not
// read the per-panel scratch that panel overwrites (the interchange plan and
// L11's block inverses): they take the interchanges from dipiv and a copy of
// the inverses (ws.dinv64_step0).
cudaError_t dgetrf_device(int m, int n, double* dA, long long ldda, int* dipiv, int nb,
                          const LuWork& ws, cudaStream_t s) {
  SL_TRY(cudaMemsetAsync(ws.status, 0, sizeof(int), s));
  SL_TRY(cudaMemsetAsync(ws.info_col, 0x7f, sizeof(int), s));
  const int mn = m < n ? m : n;
  if (nb > 1024 && !(nb == n && n <= m && n <= kOnePanelMax && g_f64_update == 1)) nb = 1024;
  auto Ap = [&](long long i, long long j) { return dA + i + j * ldda; };
  const bool lookahead = ws.aux && ws.ev_next && ws.ev_panel && mn > 2 * nb;
  // column chunks: s waits for every chunk that starts below column `upto`
  const int nck = (ws.ncol_chunks > 0 && ws.col_end && ws.ev_cols)
                      ? (ws.ncol_chunks < kMaxColChunks ? ws.ncol_chunks : kMaxColChunks) : 0;
  int next_chunk = 0;
  auto wait_cols = [&](int upto) -> cudaError_t {
    while (next_chunk < nck && (next_chunk ? ws.col_end[next_chunk - 1] : 0) < upto) {
      SL_TRY(cudaStreamWaitEvent(s, ws.ev_cols[next_chunk], 0));
      ++next_chunk;
    }
    return cudaSuccess;
  };
  const bool stream_step0 = nck > 0 && lookahead && ws.dinv64_step0 && ws.col_end[nck - 1] >= n;
  SL_TRY(wait_cols(stream_step0 ? nb : INT_MAX));
  if (mn > 0) SL_TRY(factor_panel(m, n, dA, ldda, dipiv, 0, (mn < nb ? mn : nb), ws, s));
  bool panel_on_aux = false;
  if (stream_step0) {
    SL_TRY(step0_by_chunks(m, n, dA, ldda, dipiv, nb, ws, s, wait_cols));
    panel_on_aux = true;
  }
  // Split look-ahead step (both buffer sets present, the panel stream's
  // scratch holding an m x nb x nb product): once panel j is factored, the
  // panel stream brings the next panel's columns up to date itself (their
  // interchanges, U12 solve and update) and factors that panel, while the
  // caller's stream handles every other column -- so only the next panel's
  // share of the step lies between two panels. cur holds the inverse and
  // interchange plan of the panel just factored, nxt receives the next one's;
  // the caller's stream is done with cur's before the panel stream rewrites
  // them two panels later (it waits for ev_next, recorded after that work).
  LuWork cur = ws, nxt = ws;
  const bool split = lookahead && ws.dinv64_alt && ws.swap_plan_alt && g_f64_update == 1 &&
                     oz_fits(ws.oz_aux, m, nb, nb);
  if (split) {
    nxt.dinv64 = ws.dinv64_alt;
    nxt.swap_plan = ws.swap_plan_alt;
  }
  for (int j = stream_step0 ? nb : 0; j < mn; j += nb) {
    const int jb = (mn - j) < nb ? (mn - j) : nb;
    if (panel_on_aux) SL_TRY(cudaStreamWaitEvent(s, ws.ev_panel, 0));
    panel_on_aux = false;
    const int jn = j + jb;                                   // next panel's first column
    const int jb2 = jn < mn ? ((mn - jn) < nb ? (mn - jn) : nb) : 0;
    const bool tail = nb < n && n <= m && jn < n && n - jn > jb2 && g_f64_update == 1 &&
                      one_panel_tail(m - jn, n - jn, jn) && oz_fits(ws.oz, m - jn, n - jn, nb);
    if (split && jb2 > 0 && !tail) {
      const double mr = (double)(m - jn);
      // panel j, and every update of the caller's stream before it
      SL_TRY(cudaEventRecord(ws.ev_next, s));
      SL_TRY(cudaStreamWaitEvent(ws.aux, ws.ev_next, 0));
      LuWork aw = cur;
      aw.oz = ws.oz_aux;
      phase_begin(kPhLaswp, ws.aux);
      SL_TRY(laswp_planned<double>(dA, ldda, j, jn, dipiv, cur.swap_plan, jn, jn + jb2, jn + jb2, jn + jb2, ws.aux));
      phase_end(kPhLaswp, ws.aux, 0.0, 32.0 * jb * (double)jb2);
      phase_begin(kPhTrsm, ws.aux);
      SL_TRY(solve_u12(jb, jb2, Ap(j, j), ldda, Ap(j, jn), ldda, aw, ws.aux));
      phase_end(kPhTrsm, ws.aux, (double)jb * jb * jb2, 8.0 * (0.5 * jb * jb + 2.0 * jb * jb2));
      // the next panel's update and in-panel products run on the SMs the
      // update of the other columns (beside them) leaves
      const int rest_cols = n - jn - jb2;
      const int upd = rest_cols > 0 ? update_ctas(2.0 * mr * rest_cols * jb) : 0;
      const int free_sms = upd > 0 ? num_sms() - upd : 0;
      phase_begin(kPhGemm, ws.aux);
      SL_TRY(lu_update(ws.oz_aux, m - jn, jb2, jb, -1.0, Ap(jn, j), ldda, Ap(j, jn), ldda, Ap(jn, jn),
                       ldda, ws, ws.aux, (g_cap_mask & 2) ? free_sms : 0));
      phase_end(kPhGemm, ws.aux, 2.0 * mr * jb2 * jb, 8.0 * (mr * jb + (double)jb * jb2 + 2.0 * mr * jb2));
      nxt.inpanel_ctas = (g_cap_mask & 1) ? free_sms : 0;
      SL_TRY(factor_panel(m, n, dA, ldda, dipiv, jn, jb2, nxt, ws.aux));
      SL_TRY(cudaEventRecord(ws.ev_panel, ws.aux));
      panel_on_aux = true;
      // the other columns on the caller's stream
      const int c2 = jn + jb2, rest = n - c2;
      const int main_cap = (g_cap_mask & 4) ? upd : 0;
      phase_begin(kPhLaswp, s);
      SL_TRY(laswp_planned<double>(dA, ldda, j, jn, dipiv, cur.swap_plan, 0, j, c2, n, s, main_cap));
      phase_end(kPhLaswp, s, 0.0, 32.0 * jb * (double)(n - jb - jb2));
      if (rest > 0) {
        phase_begin(kPhTrsm, s);
        SL_TRY(solve_u12(jb, rest, Ap(j, j), ldda, Ap(j, c2), ldda, cur, s, main_cap));
        phase_end(kPhTrsm, s, (double)jb * jb * rest, 8.0 * (0.5 * jb * jb + 2.0 * jb * rest));
        phase_begin(kPhGemm, s);
        SL_TRY(lu_update(ws.oz, m - jn, rest, jb, -1.0, Ap(jn, j), ldda, Ap(j, c2), ldda, Ap(jn, c2),
                         ldda, ws, s, update_ctas(2.0 * mr * rest * jb)));
        phase_end(kPhGemm, s, 2.0 * mr * rest * jb, 8.0 * (mr * jb + (double)jb * rest + 2.0 * mr * rest));
      }
      std::swap(cur, nxt);
      continue;
    }
    // ---- PDLASWP on the left and right column blocks ----
    phase_begin(kPhLaswp, s);
    SL_TRY(laswp_planned<double>(dA, ldda, j, j + jb, dipiv, cur.swap_plan, 0, j, j + jb, n, s));
    phase_end(kPhLaswp, s, 0.0, 32.0 * jb * (double)(n - jb));
    if (jn < n) {
      // ---- PDTRSM: U12 = L11^{-1} A12 ----
      const double nr = (double)(n - jn);
      phase_begin(kPhTrsm, s);
      SL_TRY(solve_u12(jb, n - jn, Ap(j, j), ldda, Ap(j, jn), ldda, cur, s));
      phase_end(kPhTrsm, s, (double)jb * jb * nr, 8.0 * (0.5 * jb * jb + 2.0 * jb * nr));
      // ---- PDGEMM: A22 -= L21 * U12 ----
      if (jn < m) {
        const double mr = (double)(m - jn);
        if (lookahead && jb2 > 0 && !tail) {
          // next panel's columns first, then the panel on the look-ahead stream
          phase_begin(kPhGemm, s);
          SL_TRY(lu_update(ws.oz, m - jn, jb2, jb, -1.0, Ap(jn, j), ldda, Ap(j, jn), ldda,
                           Ap(jn, jn), ldda, ws, s));
          phase_end(kPhGemm, s, 2.0 * mr * jb2 * jb, 8.0 * (mr * jb + (double)jb * jb2 + 2.0 * mr * jb2));
          SL_TRY(cudaEventRecord(ws.ev_next, s));
          SL_TRY(cudaStreamWaitEvent(ws.aux, ws.ev_next, 0));
          SL_TRY(factor_panel(m, n, dA, ldda, dipiv, jn, jb2, ws, ws.aux));
          SL_TRY(cudaEventRecord(ws.ev_panel, ws.aux));
          panel_on_aux = true;
          const int rest = n - jn - jb2;
          if (rest > 0) {
            phase_begin(kPhGemm, s);
            SL_TRY(lu_update(ws.oz, m - jn, rest, jb, -1.0, Ap(jn, j), ldda, Ap(j, jn + jb2), ldda,
                             Ap(jn, jn + jb2), ldda, ws, s,
                             update_ctas(2.0 * mr * rest * jb)));
            phase_end(kPhGemm, s, 2.0 * mr * rest * jb, 8.0 * (mr * jb + (double)jb * rest + 2.0 * mr * rest));
          }
        } else {
          phase_begin(kPhGemm, s);
          SL_TRY(lu_update(ws.oz, m - jn, n - jn, jb, -1.0, Ap(jn, j), ldda, Ap(j, jn), ldda,
                           Ap(jn, jn), ldda, ws, s));
          phase_end(kPhGemm, s, 2.0 * mr * nr * jb, 8.0 * (mr * jb + jb * nr + 2.0 * mr * nr));
        }
      }
    }
    if (tail) {
      SL_TRY(factor_panel(m, n, dA, ldda, dipiv, jn, n - jn, ws, s, 0));
      break;
    }
    if (jb2 > 0 && !panel_on_aux) SL_TRY(factor_panel(m, n, dA, ldda, dipiv, jn, jb2, ws, s));
  }
  if (panel_on_aux) SL_TRY(cudaStreamWaitEvent(s, ws.ev_panel, 0));
  return cudaGetLastError();
}

// Off-diagonal update of the blocked solves: C += alpha op(A) B.
template <>
cudaError_t gemm_update<double>(bool transa, int m, int n, int k, double alpha, const double* A,
                                long long lda, const double* B, long long ldb, double* C,
                                long long ldc, cudaStream_t s) {
  if (n <= 16) return gemm_skinny<double>(transa, m, n, k, alpha, A, lda, B, ldb, C, ldc, s);
  return dgemm(transa, m, n, k, alpha, A, lda, B, ldb, 1.0, C, ldc, s);
}

// Columns part, part + 4, ... of the inverse of a 64x64 diagonal block of the
// unit-lower L (LOWER) or the non-unit upper U of an n x n LU factor, for the
// blocked solves: block b at D + b*4096, column-major with leading dimension 64
// (D[c*64 + r] = inv(T_bb)(r, c)); a partial last block is padded with the
// identity. A warp per column: lane l owns rows l and l + 32, x_q is passed by a
// shuffle, in the order of a substitution. U's rows are divided by their
// diagonal beforehand, so that both triangles are unit ones. The four parts of a
// block are four CTAs: the FP64 unit of an SM takes 20 cycles per warp
// instruction whatever lanes are active, and a column of the inverse costs 32
// to 96 of them (one CTA per block and a barrier per row: 54 us for one block, 11
// with four).
//
// x = inv(T_bb) v has an error of eps |inv(T_bb)| |v|, a substitution one of eps |T_bb|
// |x|: what the inverse costs grows with its size against that of T_bb with its rows over
// their diagonal (the sizes of the rows do not matter). flag[part] = 1 where an entry of
// inv(T_bb) times its column's diagonal is 16 or more (8 may be taken for it), or is not finite, or
// a diagonal entry's reciprocal is not a normal number: such a block is solved by
// substitution. Largest over the 64-row blocks of the factors of random matrices, N = 256 ..
// 4096: 4.1 (uniform and normal entries; 1.0 with a heavy diagonal). Scaled residual of
// a 64-row solve, worst of 1500 triangles per size: entries up to 8: 0.7 (substitution
// 0.4), up to 64: 1.8, up to 2^11: 12, up to 2^16: 270; with 8 rows 1.5, 12 and 62 (bound
// of the tester: 16). Exponents are compared, off the FP64 unit.
constexpr int kInvSmem = (64 * 64 + 64 + 32) * (int)sizeof(double);
constexpr int kInvParts = 4;
template <bool LOWER>
__device__ __forceinline__ void tri_inv64_of(int b, int part, int n, const double* __restrict__ A,
                                             long long lda, double* D, int* flag, double* inv_smem) {
  double* Ts = inv_smem;  // Ts[q*64 + i] = T(i, q), zero outside the strict triangle
  double* rd = inv_smem + 64 * 64;
  int* de = reinterpret_cast<int*>(rd + 64);  // biased exponents of the diagonal
  auto exp_of = [](double x) { return (__double2hiint(x) >> 20) & 0x7ff; };
  bool bad = false;
  const int r0 = b * 64, rb = min(64, n - r0);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (!LOWER) {
    if (tid < 64) {
      const double d = tid < rb ? A[(r0 + tid) + (long long)(r0 + tid) * lda] : 1.0;
      rd[tid] = 1.0 / d;
      de[tid] = exp_of(d);
      bad = de[tid] == 0 || de[tid] > 2044;
    }
    __syncthreads();
  }
#pragma unroll 8
  for (int idx = tid; idx < 64 * 64; idx += 256) {
    const int i = idx & 63, q = idx >> 6;
    double v = 0.0;
    if (i < rb && q < rb && (LOWER ? q < i : q > i)) {
      v = A[(r0 + i) + (long long)(r0 + q) * lda];
      if (!LOWER) v *= rd[i];
    }
    Ts[idx] = v;
  }
  __syncthreads();
  double* Db = D + (size_t)b * 4096;
  for (int h = 0; h < 2; ++h) {
    const int c = part + kInvParts * (h ? 15 - warp : warp);  // a long column and a short one
    const double d = LOWER ? 1.0 : rd[c];
    double x0 = lane == c ? d : 0.0, x1 = lane + 32 == c ? d : 0.0;
    if (LOWER) {
      for (int q = c; q < 32; ++q) {
        const double xq = __shfl_sync(0xffffffffu, x0, q);
        if (lane > q) x0 = fma(-Ts[q * 64 + lane], xq, x0);
        x1 = fma(-Ts[q * 64 + lane + 32], xq, x1);
      }
      for (int q = c > 32 ? c : 32; q < 63; ++q) {
        const double xq = __shfl_sync(0xffffffffu, x1, q - 32);
        if (lane + 32 > q) x1 = fma(-Ts[q * 64 + lane + 32], xq, x1);
      }
    } else {
      for (int q = c; q >= 32; --q) {
        const double xq = __shfl_sync(0xffffffffu, x1, q - 32);
        if (lane + 32 < q) x1 = fma(-Ts[q * 64 + lane + 32], xq, x1);
        x0 = fma(-Ts[q * 64 + lane], xq, x0);
      }
      for (int q = c < 31 ? c : 31; q > 0; --q) {
        const double xq = __shfl_sync(0xffffffffu, x0, q);
        if (lane < q) x0 = fma(-Ts[q * 64 + lane], xq, x0);
      }
    }
    Db[c * 64 + lane] = x0;
    Db[c * 64 + lane + 32] = x1;
    const int e = max(exp_of(x0), exp_of(x1));
    bad = bad || e == 0x7ff || e + (LOWER ? 1023 : de[c]) > 2 * 1023 + 2;
  }
  const int any = __syncthreads_or(bad);
  if (tid == 0) flag[b * kInvParts + part] = any;
}

// Everything a solve needs before its first step, in one launch: the first
// blocks make the segment maps of the pivots' row permutation (perm_segment), the
// next kInvParts * nb64 invert L's diagonal blocks into D (flags: which of them not to
// use), as many more U's behind them; the tickets of the chained solve are reset.
__global__ void __launch_bounds__(256)
solve_prep_kernel(int n, const double* __restrict__ A, long long lda, double* D, int* flags,
                  const int* __restrict__ ipiv, int* maps, int* tickets) {
  extern __shared__ double inv_smem[];
  static_assert(kPermSmem * sizeof(int) <= (size_t)kInvSmem, "pivots of a segment");
  const int nb64 = (n + 63) / 64, nperm = (n + 255) / 256 * perm_segs(n);
  const int b = (int)blockIdx.x - nperm, part = b % kInvParts, blk = b / kInvParts;
  if (blockIdx.x == 0 && threadIdx.x == 0 && tickets) tickets[0] = tickets[1] = 0;
  launch_dependents();
  if (b < 0)
    perm_segment(blockIdx.x, ipiv, n, maps, reinterpret_cast<int*>(inv_smem));
  else if (blk < nb64) tri_inv64_of<true>(blk, part, n, A, lda, D, flags, inv_smem);
  else
    tri_inv64_of<false>(blk - nb64, part, n, A, lda, D + (size_t)nb64 * 4096, flags + nb64 * kInvParts, inv_smem);
}

// Balancing keys of the blocked NOTRAN solve's sliced products, once per
// solve: for column k of the factor, with b = k / 128, ck[k] is the largest
// exponent key of the unit-lower L's entries in rows [(b+1)*128, n) and
// ck[npad + k] that of U's entries in rows [0, b*128) -- the rows of the A
// operand of the product that follows block b's solve (the low 12 bits of
// oz_key_word; 0: no finite nonzero entry). One warp per column.
__global__ void __launch_bounds__(256)
solve_ckeys_kernel(int n, const double* __restrict__ A, long long lda, unsigned* ck, int npad) {
  const int k = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (k >= n) return;
  const double* col = A + (long long)k * lda;
  const int lo = (k / 128) * 128, hi = lo + 128;
  unsigned kl = 0u, ku = 0u;
  for (int i = hi + lane; i < n; i += 32) kl = max(kl, (unsigned)oz_key_word(col[i], 0ULL));
  for (int i = lane; i < lo; i += 32) ku = max(ku, (unsigned)oz_key_word(col[i], 0ULL));
  kl = __reduce_max_sync(0xffffffffu, kl);
  ku = __reduce_max_sync(0xffffffffu, ku);
  if (lane == 0) {
    ck[k] = kl;
    ck[npad + k] = ku;
  }
}

// One block step of the blocked NOTRAN solve: X(k0:k0+kb, c) =
// inv(T_bb) X(k0:k0+kb, c) for the 128-row block at k0 of the unit-lower L
// (LOWER, forward) or the upper U (backward), from the inverses of its two
// 64x64 diagonal blocks and its off-diagonal 64x64 block, staged in shared
// memory; a 64-row block whose four words of flags are not all zero is solved by
// substitution with its own triangle. CTA c < nrhs takes right-hand side c (threads 0..127 one row each);
// with ckeys set, the CTAs also publish the balancing keys of the sliced
// product that follows (A: the factor's columns k0..k0+kb outside the block,
// B: the solved rows): the h keys from each column's solved values and, in
// the extra CTA nrhs, the c keys from ck.
constexpr int kBlkSmem = 3 * 64 * 64 * (int)sizeof(double);
__device__ __forceinline__ bool block_flagged(const int* flags, int b) {
  static_assert(kInvParts == 4, "one int4 per block");
  const int4 f = reinterpret_cast<const int4*>(flags)[b];
  return (f.x | f.y | f.z | f.w) != 0;
}
// Ts[i*64 + r] = T(r, i) of the w x w triangle at T
__device__ __noinline__ void stage_triangle(int w, const double* __restrict__ T, long long lda, double* Ts) {
  for (int idx = threadIdx.x; idx < 4096; idx += 256) {
    const int r = idx & 63, i = idx >> 6;
    Ts[idx] = r < w && i < w ? T[r + (long long)i * lda] : 0.0;
  }
}
// y = inv(T) x by the calling warp, T from stage_triangle
template <bool LOWER>
__device__ __noinline__ void warp_solve_triangle(int w, const double* Ts, const double* x, double* y) {
  const int lane = threadIdx.x & 31;
  double x0 = x[lane], x1 = x[lane + 32];
  warp_substitute64(LOWER, LOWER, w, [&](int i, int k) { return Ts[k * 64 + i]; }, x0, x1);
  y[lane] = x0;
  y[lane + 32] = x1;
}
template <bool LOWER>
__global__ void __launch_bounds__(256)
solve_block128_kernel(int kb, const double* __restrict__ A, long long lda, int k0,
                      const double* __restrict__ D, const int* __restrict__ flags, double* X, long long ldx,
                      int nrhs, const unsigned* __restrict__ ck, unsigned long long* ckeys,
                      unsigned long long* hkeys, unsigned long long epoch) {
  extern __shared__ double blk_smem[];  // D0, D1 and the off-diagonal block O, each [c*64 + r]
  __shared__ double xs[128], ys[128];
  const int c = blockIdx.x, t = threadIdx.x;
  if (c == nrhs) {  // the c keys of the following product
    if (t < kb && ck[k0 + t]) atomicMax(ckeys + t, (epoch << 12) | ck[k0 + t]);
    return;
  }
  double* x = X + k0 + (long long)c * ldx;
  const int b0 = k0 / 64;  // first 64-block
  const int w0 = kb < 64 ? kb : 64, w1 = kb - w0;
  double* D0s = blk_smem;
  double* D1s = blk_smem + 4096;
  double* Os = blk_smem + 2 * 4096;
  {
    // every load of the staging is issued before the first store (one
    // memory round trip): D0 and D1 (D1 follows D0 in memory; only when the
    // block has a second half), O = L10 (rows 64.., columns 0..) or U01
    // (rows 0.., columns 64..), [i*64 + r], and this column's right-hand side
    const double2* Dg = reinterpret_cast<const double2*>(D + (size_t)b0 * 4096);
    const int nd = (w1 > 0 ? 2 : 1) * 2048;
    const double xv = (t < kb) ? x[t] : 0.0;
    double2 rd[16];
    double ro[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      const int idx = t + 256 * q;
      rd[q] = idx < nd ? Dg[idx] : make_double2(0.0, 0.0);
    }
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      const int idx = t + 256 * q;
      const int r = idx & 63, i = idx >> 6;
      const bool in = LOWER ? (r < w1 && i < w0) : (r < w0 && i < w1);
      const long long off = LOWER ? (k0 + 64 + r) + (long long)(k0 + i) * lda
                                  : (k0 + r) + (long long)(k0 + 64 + i) * lda;
      ro[q] = in ? A[off] : 0.0;
    }
    double2* d = reinterpret_cast<double2*>(blk_smem);
#pragma unroll
    for (int q = 0; q < 16; ++q) d[t + 256 * q] = rd[q];
#pragma unroll
    for (int q = 0; q < 16; ++q) Os[t + 256 * q] = ro[q];
    if (t < 128) xs[t] = xv;
  }
  const bool sub0 = block_flagged(flags, b0), sub1 = w1 > 0 && block_flagged(flags, b0 + 1);
  __syncthreads();
  if (sub0 || sub1) {
    if (sub0) stage_triangle(w0, A + k0 + (long long)k0 * lda, lda, D0s);
    if (sub1) stage_triangle(w1, A + (k0 + 64) + (long long)(k0 + 64) * lda, lda, D1s);
    __syncthreads();
  }
  if (LOWER) {
    // y0 = inv(L00) x0; x1 -= L10 y0; y1 = inv(L11) x1
    if (sub0) {
      if (t < 32) warp_solve_triangle<LOWER>(w0, D0s, xs, ys);
    } else if (t < 64) {
      double acc = 0.0;
      for (int i = 0; i < 64; ++i) acc = fma(D0s[i * 64 + t], xs[i], acc);
      ys[t] = acc;
    }
    __syncthreads();
    if (t >= 64 && t < 128 && t - 64 < w1) {
      double acc = xs[t];
      for (int i = 0; i < w0; ++i) acc = fma(-Os[i * 64 + (t - 64)], ys[i], acc);
      xs[t] = acc;
    }
    __syncthreads();
    if (sub1) {
      if (t < 32) warp_solve_triangle<LOWER>(w1, D1s, xs + 64, ys + 64);
    } else if (t >= 64 && t < 128 && w1 > 0) {  // (no second 64-block when kb <= 64)
      const int r = t - 64;
      double acc = 0.0;
      for (int i = 0; i < 64; ++i) acc = fma(D1s[i * 64 + r], xs[64 + i], acc);
      ys[t] = acc;
    }
  } else {
    // y1 = inv(U11) x1; x0 -= U01 y1; y0 = inv(U00) x0
    if (sub1) {
      if (t < 32) warp_solve_triangle<LOWER>(w1, D1s, xs + 64, ys + 64);
    } else if (t >= 64 && t < 128 && w1 > 0) {
      const int r = t - 64;
      double acc = 0.0;
      for (int i = 0; i < 64; ++i) acc = fma(D1s[i * 64 + r], xs[64 + i], acc);
      ys[t] = acc;
    } else if (t >= 64 && t < 128) {
      ys[t] = 0.0;
    }
    __syncthreads();
    if (t < 64 && w1 > 0) {
      double acc = xs[t];
      for (int i = 0; i < w1; ++i) acc = fma(-Os[i * 64 + t], ys[64 + i], acc);
      xs[t] = acc;
    }
    __syncthreads();
    if (sub0) {
      if (t < 32) warp_solve_triangle<LOWER>(w0, D0s, xs, ys);
    } else if (t < 64) {
      double acc = 0.0;
      for (int i = 0; i < 64; ++i) acc = fma(D0s[i * 64 + t], xs[i], acc);
      ys[t] = acc;
    }
  }
  __syncthreads();
  if (t < kb) {
    x[t] = ys[t];
    if (hkeys) {
      const unsigned long long w = oz_key_word(ys[t], epoch);
      if (w) oz_raise_key(hkeys + t, w);
    }
  }
}

// The same block step for many right-hand sides: a CTA stages the two inverses and
// the coupling block once and takes eight right-hand sides at a time, two columns
// per thread, so that all its warps feed the FP64 unit (the kernel above reloads 96
// KB per right-hand side and leaves six of eight warps idle in each product); the
// sums run in the same order. The triangles' zero quarters are skipped. Bound: the
// FP64 pipe, 10240 FMAs per right-hand side and block. n = 3000, 3000 right-hand
// sides: the whole solve 9.7 -> 7.4 ms.
constexpr int kWideCols = 8;
constexpr int kWideSmem = (3 * 64 * 64 + 2 * 128 * kWideCols) * (int)sizeof(double) + 128 * (int)sizeof(unsigned);
template <bool LOWER>
__global__ void __launch_bounds__(256)
solve_block128_wide_kernel(int kb, const double* __restrict__ A, long long lda, int k0,
                           const double* __restrict__ D, const int* __restrict__ flags, double* X,
                           long long ldx, int nrhs, const unsigned* __restrict__ ck, unsigned long long* ckeys,
                           unsigned long long* hkeys, unsigned long long epoch) {
  extern __shared__ double blk_smem[];  // D0, D1 and the coupling block O, each [i*64 + r]
  double* D0s = blk_smem;
  double* D1s = blk_smem + 4096;
  double* Os = blk_smem + 2 * 4096;
  double* xs = blk_smem + 3 * 4096;           // [col][128]
  double* ys = xs + 128 * kWideCols;
  unsigned* s_h = reinterpret_cast<unsigned*>(ys + 128 * kWideCols);
  const int t = threadIdx.x, r = t & 63, c = t >> 6;  // row, columns c and c + 4
  const int w0 = kb < 64 ? kb : 64, w1 = kb - w0;
  if (blockIdx.x == 0 && hkeys && t < kb && ck[k0 + t]) atomicMax(ckeys + t, (epoch << 12) | ck[k0 + t]);
  const double* Dg = D + (size_t)(k0 / 64) * 4096;
#pragma unroll 8
  for (int idx = t; idx < 4096; idx += 256) {
    const int rr = idx & 63, i = idx >> 6;
    const bool in = LOWER ? (rr < w1 && i < w0) : (rr < w0 && i < w1);
    const long long off = LOWER ? (k0 + 64 + rr) + (long long)(k0 + i) * lda
                                : (k0 + rr) + (long long)(k0 + 64 + i) * lda;
    D0s[idx] = Dg[idx];
    D1s[idx] = w1 > 0 ? Dg[4096 + idx] : 0.0;
    Os[idx] = in ? A[off] : 0.0;
  }
  if (t < 128) s_h[t] = 0u;
  const bool sub0 = block_flagged(flags, k0 / 64), sub1 = w1 > 0 && block_flagged(flags, k0 / 64 + 1);
  if (sub0 || sub1) {
    __syncthreads();
    if (sub0) stage_triangle(w0, A + k0 + (long long)k0 * lda, lda, D0s);
    if (sub1) stage_triangle(w1, A + (k0 + 64) + (long long)(k0 + 64) * lda, lda, D1s);
  }
  // y = M v for 64 rows: v, y at offset h of a column; i runs over the warp's part
  // of the triangle (i0 .. i1)
  // (sub: M is the triangle itself, a warp per column)
  auto tri = [&](const double* M, int h, int i0, int i1, bool sub) {
    if (sub) {
      warp_solve_triangle<LOWER>(h ? w1 : w0, M, xs + (t >> 5) * 128 + h, ys + (t >> 5) * 128 + h);
      return;
    }
    double a0 = 0.0, a1 = 0.0;
    for (int i = i0; i < i1; ++i) {
      const double m = M[i * 64 + r];
      a0 = fma(m, xs[c * 128 + h + i], a0);
      a1 = fma(m, xs[(c + 4) * 128 + h + i], a1);
    }
    ys[c * 128 + h + r] = a0;
    ys[(c + 4) * 128 + h + r] = a1;
  };
  // x -= O y, x at offset hx, y at offset hy, w columns of O
  auto couple = [&](int hx, int hy, int w) {
    double a0 = xs[c * 128 + hx + r], a1 = xs[(c + 4) * 128 + hx + r];
    for (int i = 0; i < w; ++i) {
      const double m = Os[i * 64 + r];
      a0 = fma(-m, ys[c * 128 + hy + i], a0);
      a1 = fma(-m, ys[(c + 4) * 128 + hy + i], a1);
    }
    xs[c * 128 + hx + r] = a0;
    xs[(c + 4) * 128 + hx + r] = a1;
  };
  const int lo_i0 = LOWER ? 0 : (r & 32), lo_i1 = LOWER ? (r & 32) + 32 : 64;
  for (int g = blockIdx.x * kWideCols; g < nrhs; g += gridDim.x * kWideCols) {
    __syncthreads();  // the staging, or the previous group's last reads
#pragma unroll
    for (int q = 0; q < kWideCols / 2; ++q) {
      const int row = t & 127, col = (t >> 7) + 2 * q;
      xs[col * 128 + row] = (row < kb && g + col < nrhs) ? X[k0 + row + (long long)(g + col) * ldx] : 0.0;
    }
    __syncthreads();
    if (LOWER) {  // y0 = inv(L00) x0; x1 -= L10 y0; y1 = inv(L11) x1
      tri(D0s, 0, lo_i0, lo_i1, sub0);
      __syncthreads();
      couple(64, 0, w0);
      __syncthreads();
      tri(D1s, 64, lo_i0, lo_i1, sub1);
    } else {      // y1 = inv(U11) x1; x0 -= U01 y1; y0 = inv(U00) x0
      tri(D1s, 64, lo_i0, lo_i1, sub1);
      __syncthreads();
      couple(0, 64, max(w1, 0));
      __syncthreads();
      tri(D0s, 0, lo_i0, lo_i1, sub0);
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kWideCols / 2; ++q) {
      const int row = t & 127, col = (t >> 7) + 2 * q;
      if (row < kb && g + col < nrhs) {
        const double y = ys[col * 128 + row];
        X[k0 + row + (long long)(g + col) * ldx] = y;
        if (hkeys) atomicMax(&s_h[row], (unsigned)(oz_key_word(y, 0ULL) & 4095ULL));
      }
    }
  }
  __syncthreads();
  if (hkeys && t < kb && s_h[t]) oz_raise_key(hkeys + t, (epoch << 12) | s_h[t]);
}

// Blocked NOTRAN solve with the diagonal-block inverses (ws.dinv_solve: L
// blocks, then U blocks, then the column keys) and the off-diagonal updates
// as sliced products on the tensor cores: 128-row blocks, each applied by
// inverse and then subtracted from the rest. The products take their
// balancing keys from the block step (no key pass over the factor per step).
// With triangular set (LOWER), X is lower triangular on entry (an identity) and
// stays so: a block step concerns only the columns up to its own.
static cudaError_t tri_solve_inv(bool lower, int n, int ncols, const double* A, long long lda,
                                 double* X, long long ldx, const LuWork& ws, cudaStream_t s,
                                 bool triangular = false) {
  constexpr int KB = 128;
  const int nblk = (n + KB - 1) / KB;
  const int nb64 = (n + 63) / 64;
  const double* D = ws.dinv_solve + (lower ? 0 : (size_t)nb64 * 4096);
  const int* flags = solve_inv_flags(ws.dinv_solve, n) + (lower ? 0 : nb64 * kInvParts);
  const unsigned* ck = reinterpret_cast<const unsigned*>(ws.dinv_solve + (size_t)2 * nb64 * 4096) +
                       (lower ? 0 : nb64 * 64);
  unsigned long long* ckeys = oz_ckeys(ws.oz);
  unsigned long long* hkeys = oz_hkeys(ws.oz);
  for (int bi = 0; bi < nblk; ++bi) {
    const int b = lower ? bi : nblk - 1 - bi;
    const int k0 = b * KB, kb = (n - k0) < KB ? (n - k0) : KB;
    const int rest = lower ? n - k0 - kb : k0;
    const int nrhs = triangular ? std::min(ncols, k0 + kb) : ncols;
    const unsigned long long ep = rest > 0 ? oz_new_epoch() : 0ULL;
    if (nrhs >= kWideRhs) {
      const int grid = std::min(2 * num_sms(), (nrhs + kWideCols - 1) / kWideCols);
      if (lower)
        solve_block128_wide_kernel<true><<<grid, 256, kWideSmem, s>>>(
            kb, A, lda, k0, D, flags, X, ldx, nrhs, ck, ckeys, rest > 0 ? hkeys : nullptr, ep);
      else
        solve_block128_wide_kernel<false><<<grid, 256, kWideSmem, s>>>(
            kb, A, lda, k0, D, flags, X, ldx, nrhs, ck, ckeys, rest > 0 ? hkeys : nullptr, ep);
    } else if (lower)
      solve_block128_kernel<true><<<nrhs + (rest > 0 ? 1 : 0), 256, kBlkSmem, s>>>(
          kb, A, lda, k0, D, flags, X, ldx, nrhs, ck, ckeys, rest > 0 ? hkeys : nullptr, ep);
    else
      solve_block128_kernel<false><<<nrhs + (rest > 0 ? 1 : 0), 256, kBlkSmem, s>>>(
          kb, A, lda, k0, D, flags, X, ldx, nrhs, ck, ckeys, rest > 0 ? hkeys : nullptr, ep);
    count_launches(1);
    SL_TRY(cudaGetLastError());
    if (rest > 0 && lower)
      SL_TRY(oz_dgemm_keyed(ws.oz, ep, rest, nrhs, kb, -1.0, A + (k0 + kb) + (long long)k0 * lda, lda,
                            X + k0, ldx, X + k0 + kb, ldx, ws.status, s));
    else if (rest > 0)
      SL_TRY(oz_dgemm_keyed(ws.oz, ep, k0, nrhs, kb, -1.0, A + (long long)k0 * lda, lda, X + k0, ldx,
                            X, ldx, ws.status, s));
  }
  return cudaSuccess;
}

// Shared-memory opt-in of the blocked solve's kernels, once.
static cudaError_t blocked_solve_attrs() {
  static const cudaError_t a[] = {
      cudaFuncSetAttribute(solve_prep_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kInvSmem),
      cudaFuncSetAttribute(solve_block128_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kBlkSmem),
      cudaFuncSetAttribute(solve_block128_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kBlkSmem),
      cudaFuncSetAttribute(solve_block128_wide_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kWideSmem),
      cudaFuncSetAttribute(solve_block128_wide_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kWideSmem)};
  for (cudaError_t e : a) SL_TRY(e);
  return cudaSuccess;
}

// Diagonal-block inverses, the pivots' permutation (ws.perm) and, for the blocked
// solve, the column keys.
static cudaError_t prepare_solve(int n, const double* dA, long long ldda, const int* dipiv, const LuWork& ws,
                                 int* tickets, bool blocked, cudaStream_t s) {
  SL_TRY(blocked_solve_attrs());
  const int nrb = (n + 255) / 256, nb64 = (n + 63) / 64;
  solve_prep_kernel<<<2 * kInvParts * nb64 + nrb * perm_segs(n), 256, kInvSmem, s>>>(
      n, dA, ldda, ws.dinv_solve, solve_inv_flags(ws.dinv_solve, n), dipiv, ws.perm + n, tickets);
  count_launches(1);
  if (blocked) {
    perm_finish_kernel<<<nrb, 256, 0, s>>>(dipiv, n, ws.perm + n, ws.perm);
    solve_ckeys_kernel<<<(n + 7) / 8, 256, 0, s>>>(
        n, dA, ldda, reinterpret_cast<unsigned*>(ws.dinv_solve + (size_t)2 * nb64 * 4096), nb64 * 64);
    count_launches(2);
  }
  return cudaGetLastError();
}

// dst(:, perm[i]) = X(:, i), n x n.
__global__ void scatter_columns_kernel(int n, const double* __restrict__ X, double* dst, long long ldd,
                                       const int* __restrict__ perm) {
  const int c = blockIdx.y, p = perm[c];
  const int r = blockIdx.x * 256 + threadIdx.x;
  if (r < n && (unsigned)p < (unsigned)n) dst[r + (long long)p * ldd] = X[r + (long long)c * n];
}

// inv(A) = inv(U) inv(L) P: L's inverse is formed as a lower triangle (a third of
// a full solve's work), U's solve runs over all columns, and the interchanges are
// a permutation of the result's columns. n = 3000: 5.75 ms, 7.5 with the identity
// permuted first and both solves full.
bool inverse_fits(int n, const LuWork& ws) {
  return n >= kWideRhs && n <= 65535 && g_f64_update == 1 && ws.dinv_solve &&
         ws.dinv_solve_len >= kSolveInvDoubles(n) && oz_fits(ws.oz, n, n, 128);
}
cudaError_t inverse_from_factors(int n, double* dA, long long ldda, const int* dipiv, double* X,
                                 const LuWork& ws, cudaStream_t s) {
  phase_begin(kPhSolve, s);
  SL_TRY(prepare_solve(n, dA, ldda, dipiv, ws, nullptr, true, s));
  SL_TRY(tri_solve_inv(true, n, n, dA, ldda, X, n, ws, s, true));
  SL_TRY(tri_solve_inv(false, n, n, dA, ldda, X, n, ws, s));
  scatter_columns_kernel<<<dim3((n + 255) / 256, n), 256, 0, s>>>(n, X, dA, ldda, ws.perm);
  count_launches(1);
  phase_end(kPhSolve, s, 4.0 * (double)n * n * n / 3.0, 24.0 * (double)n * n);
  return cudaGetLastError();
}

cudaError_t dgetrs_device(char trans, int n, int nrhs, const double* dA, long long ldda,
                          const int* dipiv, double* dB, long long lddb, const LuWork& ws,
                          cudaStream_t s) {
  if (n <= 0 || nrhs <= 0) return cudaSuccess;
  const bool notran = (trans == 'N' || trans == 'n');
  phase_begin(kPhSolve, s);
  double* X = ws.bswap;  // n x nrhs, ld = n
  // any NRHS whose products fit the scratch (PDGETRI solves with NRHS = N)
  const bool inv_path = g_f64_update == 1 && ws.dinv_solve && ws.dinv_solve_len >= kSolveInvDoubles(n) &&
                        oz_fits(ws.oz, n, nrhs, 128);
  // Few right-hand sides go through the chained solves, whose FP64 work grows with n^2
  // nrhs: NOTRAN while n nrhs <= 2^18, beyond which the blocked solve, its products on
  // the tensor cores, takes less. In ms, chained / blocked: n = 2048, 128 columns
  // 1.24 / 1.39; n = 4096, 64: 2.36 / 2.99, 96: 3.41 / 2.99; n = 8192, 32: 4.54 /
  // 5.81, 48: 6.57 / 6.03; n = 16384, 16: 9.08 / 12.33, 24: 13.14 / 12.36.
  // Transposed always (n = 8192, 64 columns: 8.6 / 31 ms: the blocked form there
  // substitutes and multiplies on the FP64 pipe).
  const bool few = nrhs <= kChainRhs && (!notran || (long long)n * nrhs <= 1LL << 18);
  const bool chain_path = g_f64_update == 1 && few && ws.dinv_solve &&
                          ws.dinv_solve_len >= kSolveInvDoubles(n) && ws.chain && ws.chain_epoch &&
                          ws.chain_values >= (size_t)n * nrhs;
  unsigned long long* words = chain_path ? reinterpret_cast<unsigned long long*>(ws.chain + 16) : nullptr;
  if (chain_path && (*ws.chain_epoch == 0 || *ws.chain_epoch > UINT_MAX - 2)) {
    // (before the preparation: the chained launches follow a kernel, launch_after)
    SL_TRY(cudaMemsetAsync(words, 0, ws.chain_values * 16, s));
    *ws.chain_epoch = 0;
  }
  if (notran ? (inv_path || chain_path) : chain_path) {
    SL_TRY(prepare_solve(n, dA, ldda, dipiv, ws, chain_path ? ws.chain : nullptr, !chain_path, s));
  } else {
    SL_TRY(perm_compose(dipiv, n, ws.perm, s));
  }
  if (chain_path) {
    // L then U (N), or U^T then L^T (T): the pivots' permutation is applied as
    // the first triangle reads B, or as the second one writes it
    const size_t ub = (size_t)((n + 63) / 64) * 4096, uf = (size_t)((n + 63) / 64) * kInvParts;
    const int* flags = solve_inv_flags(ws.dinv_solve, n);
    const unsigned e1 = ++*ws.chain_epoch, e2 = ++*ws.chain_epoch;
    SL_TRY(trsv64_chain(notran, !notran, dA, ldda, n, ws.dinv_solve + (notran ? 0 : ub), flags + (notran ? 0 : uf), dB, lddb,
                        notran ? dipiv : nullptr, X, n, nullptr, ws.perm + n, nrhs, ws.chain, words, e1, ws.status, s));
    SL_TRY(trsv64_chain(!notran, !notran, dA, ldda, n, ws.dinv_solve + (notran ? ub : 0), flags + (notran ? uf : 0), X, n, nullptr, dB,
                        lddb, notran ? nullptr : dipiv, ws.perm + n, nrhs, ws.chain + 1, words, e2, ws.status, s));
    phase_end(kPhSolve, s, 2.0 * (double)n * n * nrhs, 8.0 * ((double)n * n + 4.0 * (double)n * nrhs));
    return cudaSuccess;
  }
  if (notran && inv_path) {
    SL_TRY((permute_rows<double, double>(dB, lddb, X, n, ws.perm, n, nrhs, 0, s)));
    SL_TRY(tri_solve_inv(true, n, nrhs, dA, ldda, X, n, ws, s));
    SL_TRY(tri_solve_inv(false, n, nrhs, dA, ldda, X, n, ws, s));
    SL_TRY(cudaMemcpy2DAsync(dB, lddb * sizeof(double), X, n * sizeof(double),
                             n * sizeof(double), nrhs, cudaMemcpyDeviceToDevice, s));
  } else if (notran) {
    SL_TRY((permute_rows<double, double>(dB, lddb, X, n, ws.perm, n, nrhs, 0, s)));
    SL_TRY(tri_solve<double>(true, false, true, n, nrhs, dA, ldda, X, n, s));
    SL_TRY(tri_solve<double>(false, false, false, n, nrhs, dA, ldda, X, n, s));
    SL_TRY(cudaMemcpy2DAsync(dB, lddb * sizeof(double), X, n * sizeof(double),
                             n * sizeof(double), nrhs, cudaMemcpyDeviceToDevice, s));
  } else {
    SL_TRY(cudaMemcpy2DAsync(X, n * sizeof(double), dB, lddb * sizeof(double),
                             n * sizeof(double), nrhs, cudaMemcpyDeviceToDevice, s));
    SL_TRY(tri_solve<double>(false, true, false, n, nrhs, dA, ldda, X, n, s));
    SL_TRY(tri_solve<double>(true, true, true, n, nrhs, dA, ldda, X, n, s));
    SL_TRY((permute_rows<double, double>(X, n, dB, lddb, ws.perm, n, nrhs, 1, s)));
  }
  phase_end(kPhSolve, s, 2.0 * (double)n * n * nrhs, 8.0 * ((double)n * n + 4.0 * (double)n * nrhs));
  return cudaSuccess;
}

}  // namespace sl
