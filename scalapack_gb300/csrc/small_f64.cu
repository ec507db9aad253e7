// PDGESV of one small system (n <= 32, at most 16 right-hand sides) in one launch
// (SRC/pdgesv.f:229,236): the ordinary path is a chain of eight launches, each
// of them mostly latency, where the whole computation fits four warps'
// registers.
//
// Lane l holds row l of the matrix and of the right-hand sides; warp v the columns
// v, v + 4, .. of both. Column k's warp finds the pivot (IDAMAX: first maximal |x|
// by label, a leading NaN stays), scales by its reciprocal and passes the
// multipliers through shared memory; after one barrier every warp updates its own
// columns, the pivot row's value coming by a shuffle. Rows keep their lanes and
// change labels instead of being interchanged. The right-hand sides are updated
// among the columns, so only the backward substitution is left: a warp per
// right-hand side. Every element of the factors takes the updates of columns 0,
// 1, ... in order, one fma each, as in the panel kernels (the same factors bit for
// bit). Bound: about 900 dependent cycles per column, a third of them the division.
// Measured, n = 17 with the caller's copies and the host call: 60 us (136 as eight
// launches; n = 32: 86 of 161).
#include <climits>
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"
#include "lu_kernels.cuh"
#include "sl_internal.h"

namespace sl {
namespace {

template <int CPW>  // columns per warp: n + nrhs <= 4 * CPW
__global__ void __launch_bounds__(128)
small_gesv_kernel(int n, int nrhs, double* A, long long lda, double* B, long long ldb, int* ipiv,
                  int* status, int* info_col) {
  __shared__ double s_l[2][32];
  __shared__ int s_win[2], s_piv[2];
  __shared__ double s_U[32 * 33];            // factors by label, column-major
  __shared__ double s_Y[kSmallGesvRhs * 33];
  __shared__ int s_info;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nc = n + nrhs;
  double a[CPW];
#pragma unroll
  for (int q = 0; q < CPW; ++q) {
    const int c = 4 * q + warp;
    a[q] = 0.0;
    if (lane < n && c < n) a[q] = A[lane + (long long)c * lda];
    else if (lane < n && c < nc) a[q] = B[lane + (long long)(c - n) * ldb];
  }
  if (threadIdx.x == 0) s_info = INT_MAX;
  int lab = lane < n ? lane : -1;  // where this row's content stands; ~k once it is pivot row k
  int zero_col = INT_MAX;
#pragma unroll
  for (int q = 0; q < CPW; ++q) {
    for (int w = 0; w < 4; ++w) {
      const int k = 4 * q + w, buf = k & 1;
      if (k >= n) break;
      if (warp == w) {
        const double v = a[q];
        long long key = -2;
        if (lab >= 0) {
          key = amax_ikey(v);
          if (key < 0 && lab == k) key = LLONG_MAX;
        }
        const int win = warp_best(key, lab >= 0 ? lab : INT_MAX);
        const double g = __shfl_sync(0xffffffffu, v, win);
        const bool zero = ((unsigned long long)__double_as_longlong(g) << 1) == 0;
        const double rinv = zero ? 1.0 : 1.0 / g;  // ONE/GMAX (pdgetf2.f:224)
        const double l = v * rinv;
        if (lab >= 0 && lane != win) a[q] = l;
        s_l[buf][lane] = l;
        const int piv = __shfl_sync(0xffffffffu, lab, win);
        if (lane == 0) {
          s_win[buf] = win;
          s_piv[buf] = piv;
          ipiv[k] = piv + 1;
          if (zero) zero_col = min(zero_col, k);
        }
      }
      __syncthreads();
      const int win = s_win[buf], piv = s_piv[buf];
      const double l = s_l[buf][lane];
      if (lane == win) lab = ~k;
      else if (lab == k) lab = piv;  // the diagonal row goes where the pivot row stood
#pragma unroll
      for (int p = 0; p < CPW; ++p) {
        if (p < q) continue;
        const int c = 4 * p + warp;
        const double u = __shfl_sync(0xffffffffu, a[p], win);
        if (c > k && c < nc && lab >= 0) a[p] = fma(-l, u, a[p]);
      }
    }
  }
  if (lane == 0 && zero_col != INT_MAX) atomicMin(&s_info, zero_col);
  const int row = lab < 0 ? ~lab : lab;
#pragma unroll
  for (int q = 0; q < CPW; ++q) {
    const int c = 4 * q + warp;
    if (lane < n && c < n) {
      A[row + (long long)c * lda] = a[q];
      s_U[c * 33 + row] = a[q];
    } else if (lane < n && c < nc) {
      s_Y[(c - n) * 33 + row] = a[q];
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    *status = 0;
    *info_col = s_info;
  }
  if (s_info != INT_MAX) return;  // exactly singular: B stays (pdgesv.f:231)
  const double d = lane < n ? s_U[lane * 33 + lane] : 1.0, rd = 1.0 / d;
  for (int r = warp; r < nrhs; r += 4) {
    double x = lane < n ? s_Y[r * 33 + lane] : 0.0;
    for (int k = n - 1; k >= 0; --k) {
      if (lane == k) x = div_by(x, d, rd);
      const double xk = __shfl_sync(0xffffffffu, x, k);
      if (lane < k) x = fma(-s_U[k * 33 + lane], xk, x);
    }
    if (lane < n) B[lane + (long long)r * ldb] = x;
  }
}

}  // namespace

cudaError_t small_gesv(int n, int nrhs, double* A, long long lda, double* B, long long ldb, int* ipiv,
                       int* status, int* info_col, cudaStream_t s) {
  if (n < 1 || n > kSmallGesvMax || nrhs < 1 || nrhs > kSmallGesvRhs) return cudaErrorInvalidValue;
  if (n + nrhs <= 32) small_gesv_kernel<8><<<1, 128, 0, s>>>(n, nrhs, A, lda, B, ldb, ipiv, status, info_col);
  else small_gesv_kernel<12><<<1, 128, 0, s>>>(n, nrhs, A, lda, B, ldb, ipiv, status, info_col);
  count_launches(1);
  return cudaGetLastError();
}

}  // namespace sl
