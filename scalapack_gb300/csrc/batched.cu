// Batched solver: thousands of independent dense systems A_i X_i = B_i of
// uneven order (N_i <= 512) in one persistent launch. Each system is the same
// computation as PDGESV on a 1x1 grid (SRC/pdgesv.f: PDGETRF then PDGETRS),
// with LAPACK/ScaLAPACK pivoting semantics (first maximal |x|, scale by the
// reciprocal, INFO = first exactly-zero pivot).
//
// Layout: every system keeps its own column-major A_i (lda_i), B_i and X_i
// (ldb_i, ldx_i) in device memory; A_i and B_i are not modified. The plan
// holds a per-system workspace (a copy of A_i in the factorization precision)
// where the factors live, and the per-system outputs: pivots, INFO, refinement
// steps and the scaled residual ||b - A x||_inf / (||A||_inf ||x||_inf N eps).
//
// Scheduling: systems are sorted by decreasing N on the host (largest first,
// so the tail of the launch is made of small systems); CTAs of one persistent
// grid take the next system from an atomic ticket until the queue is empty.
//
// Per system, one CTA (two share an SM):
//   factor   blocked right-looking LU with 16-column panels held in shared
//            memory (factor_system), the right-hand sides among the columns it
//            updates, so that their forward solve is part of it; the trailing
//            update as a register-tiled GEMM (each thread owns rows)
//   solve    32-row blocked backward (refinement steps: forward too)
//            substitution, one warp per right-hand side for the diagonal blocks,
//            all threads for the off-diagonal update
//   refine   (mode 1) FP32 factors, FP64 residual and update, at most kMaxIr
//            steps; a system that does not reach the tolerance is queued for
//            the FP64 pass, which is a second persistent launch in the same
//            CUDA graph.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <numeric>
#include <vector>

#include "common.cuh"
#include "lu_kernels.cuh"
#include "sl_internal.h"

namespace sl {

constexpr int kBMaxN = 512;   // largest system order
constexpr int kBMaxRhs = 8;   // largest number of right-hand sides
constexpr int kBPB = 16;      // panel width
constexpr int kMaxIr = 10;    // refinement steps in mode 1

struct BatchArgs {
  int batch;
  const int* n;
  const int* nrhs;
  const double* const* A;
  const int* lda;
  const double* const* B;
  const int* ldb;
  double* const* X;
  const int* ldx;
  int* const* ipiv;
  void* const* W;        // per-system factor workspace (n x n in the factor type)
  void* const* W64;      // per-system FP64 workspace of the FP64 pass (== W in mode 0)
  const int* order;      // processing order (sorted by decreasing n)
  int* queue;            // [0] ticket of the main pass, [1] ticket of the fallback pass,
                         // [2] number of systems queued for the fallback pass
  int* fallback_list;    // systems queued for the FP64 pass
  int* info;
  int* iters;            // refinement steps; -1 = solved by the FP64 pass after refinement stalled
  double* sresid;
  double tol;
  int nmax, rmax;        // largest order and number of right-hand sides in the batch
};

// ------------------------------------------------------------ factorization
constexpr int kPL = kBPB + 1;  // shared row stride of the panel: conflict-free row and column walks

// Columns of a trailing update's chunk.
template <typename T>
__host__ __device__ constexpr int chunk_cols() { return 16; }

// The next column's offset: an addition the compiler keeps where it stands (as
// products c * n it hoists a dozen of them out of every loop, and spills).
__device__ __forceinline__ int next_col(int off, int ld) {
  off += ld;
  asm volatile("" : "+r"(off));
  return off;
}

// Shared memory of one system of order <= nmax: while it is factored the panel
// P [nmax][kPL], the rows' labels, and two chunks of U; afterwards, over the same
// bytes, the right-hand sides (Xs, and Cx for FP32 factors), the residual, X in
// FP64 and a diagonal block. The row order (org) lasts through both.
template <typename T>
struct BatchSmem {
  T *P, *Us;
  int* lab;
  int* org;
  T *Xs, *Ds;
  double *Xsh, *Rs;
  static size_t factor_bytes(int nmax) {
    return sizeof(T) * ((size_t)nmax * kPL + 2 * kBPB * chunk_cols<T>()) + sizeof(int) * (size_t)nmax;
  }
  static size_t solve_bytes(int nmax, int rmax) {
    // Xs and X in FP64 share their bytes; Rs (FP32 factors only) stands alone
    return sizeof(double) * (size_t)nmax * rmax * (sizeof(T) == 8 ? 1 : 2) + sizeof(T) * 32 * 33;
  }
  static size_t bytes(int nmax, int rmax) {
    const size_t f = factor_bytes(nmax), v = solve_bytes(nmax, rmax);
    return sizeof(int) * (size_t)nmax + (f > v ? f : v) + 16;
  }
  __device__ BatchSmem(unsigned char* p, int nmax, int rmax) {
    org = reinterpret_cast<int*>(p);
    unsigned char* q = p + (sizeof(int) * (size_t)nmax + 15) / 16 * 16;
    P = reinterpret_cast<T*>(q);
    Us = P + (size_t)nmax * kPL;
    lab = reinterpret_cast<int*>(Us + 2 * kBPB * chunk_cols<T>());
    Xsh = reinterpret_cast<double*>(q);
    Xs = reinterpret_cast<T*>(q);
    Rs = Xsh + (size_t)nmax * rmax;
    Ds = sizeof(T) == 8 ? reinterpret_cast<T*>(Xsh + (size_t)nmax * rmax)
                        : reinterpret_cast<T*>(Rs + (size_t)nmax * rmax);
  }
};

// Factor the leading n columns of the n x ncols matrix W (column-major, ld n)
// in place and apply the interchanges and inv(L) to the columns beyond (the
// right-hand sides: their forward solve). ipiv receives 0-based rows, org[i] the
// original row that ends in row i; *info the first zero pivot (1-based) or 0.
//
// A panel's rows keep their place in shared memory and carry a label, the row
// where their content stands after the interchanges so far (~k once it is pivot
// row k), so a column takes one barrier: every warp reduces the warps' IDAMAX
// candidates (integer keys, warp_best), each thread then scales and updates its
// rows from the pivot row where it stands and forms their keys for the next
// column. The labels are the panel's interchanges in composite form: one thread
// per other column gathers its pivot rows, sends the displaced rows where they
// go and solves with L11 in registers. Bound: the FP64 unit (FP64 factors) in the
// trailing update; two systems share an SM so that the panels of one run beside
// the updates of another (a third one's 80 registers a thread cost more in spills
// than it gave). Measured, 4096 systems of order 16 .. 512:
// FP64 119 ms (the unit's floor is 103; 188 with 32-column panels of four
// barriers and FP64 compares per column and one system per SM), FP32 factors
// with refinement 31.5 ms (87), a third of it FP64 residuals.
template <typename T, int NT>
__device__ __forceinline__ void factor_system(T* W, int n, int ncols, int* ipiv, int* info, const BatchSmem<T>& sm) {
  constexpr int CH = chunk_cols<T>();
  constexpr int NW = NT / 32;
  T* P = sm.P;
  int* lab = sm.lab;
  __shared__ long long s_wk[2][NW];
  __shared__ int s_wr[2][NW], s_wl[2][NW];
  __shared__ int s_rowof[kBPB], s_dsp[kBPB];
  __shared__ T s_L[kBPB][kPL];  // L11 by label
  __shared__ int s_info;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) s_info = 0;
  for (int r = tid; r < n; r += NT) sm.org[r] = r;
  auto row_key = [&](T v, int label, int k) -> long long {
    const long long key = amax_ikey(v);
    return (key < 0 && label == k) ? LLONG_MAX : key;  // IDAMAX keeps a leading NaN
  };
  auto put_candidate = [&](int buf, long long key, int label, int lrow) {
    if (lane == warp_best(key, label)) {
      s_wk[buf][warp] = key;
      s_wr[buf][warp] = label;
      s_wl[buf][warp] = lrow;
    }
  };
  for (int j = 0; j < n; j += kBPB) {
    const int jb = min(kBPB, n - j), m = n - j;
    {
      long long key = -2;
      int label = INT_MAX, lrow = 0;
      for (int r = tid; r < m; r += NT) {
        const T* src = W + (j + r) + (long long)j * n;
        T v[kBPB];
#pragma unroll
        for (int c = 0, o = 0; c < kBPB; ++c, o = next_col(o, n)) v[c] = c < jb ? src[o] : (T)0;
#pragma unroll
        for (int c = 0; c < kBPB; ++c) P[r * kPL + c] = v[c];
        lab[r] = r;
        const long long k2 = row_key(v[0], r, 0);
        if (k2 > key) { key = k2; label = r; lrow = r; }
      }
      put_candidate(0, key, label, lrow);
    }
    for (int k = 0; k < jb; ++k) {
      const int buf = k & 1;
      __syncthreads();
      long long key = lane < NW ? s_wk[buf][lane] : -3;
      int label = lane < NW ? s_wr[buf][lane] : INT_MAX;
      const int cw = warp_best(key, label);
      const int lr = s_wl[buf][cw];
      key = s_wk[buf][cw];
      label = s_wr[buf][cw];
      const T* U = P + lr * kPL;
      const T g = U[k];
      T rinv;  // ONE/GMAX, 1 for a zero pivot (its column is not scaled)
      bool zero;
      if constexpr (sizeof(T) == 8) {
        const unsigned long long kb = (unsigned long long)key, gb = (unsigned long long)__double_as_longlong(g);
        zero = (gb << 1) == 0;
        if (kb - 1ULL < 0x7FEFFFFFFFFFFFFFULL)
          rinv = __longlong_as_double(__double_as_longlong(recip_bits(kb)) | (long long)(gb & (1ULL << 63)));
        else
          rinv = zero ? 1.0 : 1.0 / g;
      } else {
        zero = g == (T)0;
        rinv = zero ? (T)1 : (T)1 / g;
      }
      if (tid == 0) {
        ipiv[j + k] = j + label;
        if (zero && s_info == 0) s_info = j + k + 1;
      }
      long long nkey = -2;
      int nlab = INT_MAX, nrow = 0;
      const int kn = k + 1;
      for (int r = tid; r < m; r += NT) {
        int lb = lab[r];
        if (r == lr) lab[r] = ~k;
        if (lb < 0 || r == lr) continue;
        if (lb == k) lab[r] = lb = label;
        T* row = P + r * kPL;
        const T l = row[k] * rinv;
        row[k] = l;
        if (kn < jb) {
          const T v = fma(-l, U[kn], row[kn]);
          row[kn] = v;
          const long long k2 = row_key(v, lb, kn);
          if (k2 > nkey || (k2 == nkey && lb < nlab)) { nkey = k2; nlab = lb; nrow = r; }
#pragma unroll 4
          for (int c = kn + 1; c < jb; ++c) row[c] = fma(-l, U[c], row[c]);
        }
      }
      if (kn < jb) put_candidate(buf ^ 1, nkey, nlab, nrow);
    }
    __syncthreads();
    // rows to where their content stands; the interchanges for the other columns
    int mv[kBMaxN / NT > 0 ? kBMaxN / NT : 1];
    {
      int q = 0;
      for (int r = tid; r < m; r += NT, ++q) {
        const int lb = lab[r], L = lb < 0 ? ~lb : lb;
        mv[q] = sm.org[j + r];
        T* dst = W + (j + L) + (long long)j * n;
#pragma unroll
        for (int c = 0, o = 0; c < kBPB; ++c, o = next_col(o, n))
          if (c < jb) dst[o] = P[r * kPL + c];
        if (L < jb) {
          s_rowof[L] = r;
#pragma unroll
          for (int c = 0; c < kBPB; ++c) s_L[L][c] = P[r * kPL + c];
        }
        if (r < jb) s_dsp[r] = L >= jb ? L : -1;
      }
    }
    __syncthreads();
    {
      int q = 0;
      for (int r = tid; r < m; r += NT, ++q) {
        const int lb = lab[r], L = lb < 0 ? ~lb : lb;
        if (L != r) sm.org[j + L] = mv[q];
      }
    }
    // one thread per other column: PDLASWP, and on the right U12 = inv(L11) A12
    for (int ci = tid; ci < ncols - jb; ci += NT) {
      const int c = ci < j ? ci : ci + jb;
      T* col = W + (long long)c * n + j;
      T x[kBPB], y[kBPB];
#pragma unroll
      for (int k = 0; k < kBPB; ++k) {
        x[k] = k < jb ? col[s_rowof[k]] : (T)0;
        y[k] = (k < jb && s_dsp[k] >= 0) ? col[k] : (T)0;
      }
#pragma unroll
      for (int k = 0; k < kBPB; ++k)
        if (k < jb && s_dsp[k] >= 0) col[s_dsp[k]] = y[k];
      if (c >= j + jb) {
#pragma unroll
        for (int k = 0; k < kBPB; ++k)
#pragma unroll
          for (int r = k + 1; r < kBPB; ++r)
            if (r < jb) x[r] = fma(-s_L[r][k], x[k], x[r]);
      }
#pragma unroll
      for (int k = 0; k < kBPB; ++k)
        if (k < jb) col[k] = x[k];
    }
    __syncthreads();
    if (m <= jb) break;
    // A22 -= L21 U12 (jb = kBPB here): a chunk of U12 in shared memory, each
    // thread owns rows and CH accumulators, C on its way meanwhile
    for (int c0 = j + jb, it = 0; c0 < ncols; c0 += CH, ++it) {
      T* Us = sm.Us + (it & 1) * kBPB * CH;
      const int cw = min(CH, ncols - c0);
      for (int idx = tid; idx < kBPB * CH; idx += NT) {
        const int k = idx % kBPB, c = idx / kBPB;
        Us[k * CH + c] = c < cw ? W[(j + k) + (long long)(c0 + c) * n] : (T)0;
      }
      __syncthreads();
      for (int r = tid; r < m; r += NT) {
        const int L = lab[r];
        if (L < 0) continue;
        T* crow = W + (j + L) + (long long)c0 * n;
        T cv[CH], acc[CH];
#pragma unroll
        for (int c = 0, o = 0; c < CH; ++c, o = next_col(o, n)) cv[c] = c < cw ? crow[o] : (T)0;
        const T* lrow = P + r * kPL;
#pragma unroll
        for (int k = 0; k < kBPB; ++k) {
          const T a = lrow[k];
#pragma unroll
          for (int c = 0; c < CH; ++c) acc[c] = k == 0 ? a * Us[c] : fma(a, Us[k * CH + c], acc[c]);
        }
#pragma unroll
        for (int c = 0, o = 0; c < CH; ++c, o = next_col(o, n))
          if (c < cw) crow[o] = cv[c] - acc[c];
      }
    }
    __syncthreads();
  }
  __syncthreads();
  if (tid == 0) *info = s_info;
  __syncthreads();
}

__device__ __forceinline__ float div_by(float x, float d, float) { return x / d; }

// Triangular solve with the unit-lower L (LOWER) or the upper U of the factors
// in W on Xs (n x nrhs, shared), 32-row blocks: the diagonal block in shared
// memory, a warp per right-hand side, then all threads subtract its columns
// from the remaining rows, 16 loads in flight.
template <typename T, int NT, bool LOWER>
__device__ __forceinline__ void solve_tri(const T* W, int n, T* Xs, int nrhs, T* Ds) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nblk = (n + 31) / 32;
  for (int bi = 0; bi < nblk; ++bi) {
    const int k0 = (LOWER ? bi : nblk - 1 - bi) * 32, kb = min(32, n - k0);
    for (int idx = tid; idx < 32 * 32; idx += NT) {
      const int i = idx & 31, k = idx >> 5;
      Ds[k * 33 + i] = (i < kb && k < kb) ? W[(k0 + i) + (long long)(k0 + k) * n] : (T)0;
    }
    __syncthreads();
    for (int c = warp; c < nrhs; c += NT / 32) {
      T x = lane < kb ? Xs[k0 + lane + c * n] : (T)0;
      if (LOWER) {
        for (int i = 0; i < kb; ++i) {
          const T xi = __shfl_sync(0xffffffffu, x, i);
          if (lane > i) x = fma(-Ds[i * 33 + lane], xi, x);
        }
      } else {
        const T d = lane < kb ? Ds[lane * 33 + lane] : (T)1;
        const T rd = (T)1 / d;
        for (int i = kb - 1; i >= 0; --i) {
          const T q = div_by(x, d, rd);
          if (lane == i) x = q;
          const T xi = __shfl_sync(0xffffffffu, x, i);
          if (lane < i) x = fma(-Ds[i * 33 + lane], xi, x);
        }
      }
      if (lane < kb) Xs[k0 + lane + c * n] = x;
    }
    __syncthreads();
    const int lo = LOWER ? k0 + kb : 0, hi = LOWER ? n : k0;
    for (int r = lo + tid; r < hi; r += NT) {
      T acc[kBMaxRhs];
#pragma unroll
      for (int c = 0; c < kBMaxRhs; ++c) acc[c] = (T)0;
      for (int i0 = 0; i0 < kb; i0 += 16) {
        T l[16];
        const T* wr = W + r + (long long)(k0 + i0) * n;
#pragma unroll
        for (int i = 0, o = 0; i < 16; ++i, o = next_col(o, n)) l[i] = i0 + i < kb ? wr[o] : (T)0;
#pragma unroll
        for (int i = 0; i < 16; ++i)
          if (i0 + i < kb) {
#pragma unroll
            for (int c = 0; c < kBMaxRhs; ++c)
              if (c < nrhs) acc[c] = fma(l[i], Xs[k0 + i0 + i + c * n], acc[c]);
          }
      }
#pragma unroll
      for (int c = 0; c < kBMaxRhs; ++c)
        if (c < nrhs) Xs[r + c * n] -= acc[c];
    }
    __syncthreads();
  }
}

// |v| as an integer: larger for larger magnitudes, largest for NaN, so that a
// maximum keeps a NaN once seen (the tester's norm semantics) without FP64
// compares.
__device__ __forceinline__ unsigned long long mag_key(double v) {
  return (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffULL;
}
__device__ __forceinline__ unsigned long long warp_max64(unsigned long long v) {
  const unsigned h = (unsigned)(v >> 32), hm = __reduce_max_sync(0xffffffffu, h);
  const unsigned l = __reduce_max_sync(0xffffffffu, h == hm ? (unsigned)v : 0u);
  return ((unsigned long long)hm << 32) | l;
}

// Scaled residual max_c ||b_c - A x_c|| / (||A|| ||x_c|| n eps) (tester
// semantics, LIN/pdlaschk.f) of Xsh (n x nrhs, shared); with Rs set, the
// residuals go there. rmax[c] receives the magnitude of ||r_c||_inf. The pass
// over A is the only global stream, 8 loads in flight per thread.
template <int NT>
__device__ __forceinline__ double residual_system(const double* A, int lda, int n, const double* B, int ldb,
                                  const double* Xsh, int nrhs, double* Rs, double anorm, double* rmax) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  __shared__ unsigned long long s_rm[kBMaxRhs], s_xm[kBMaxRhs];
  __shared__ double s_worst;
  if (tid < kBMaxRhs) s_rm[tid] = s_xm[tid] = 0ULL;
  __syncthreads();
  for (int r0 = 0; r0 < n; r0 += NT) {
    const int r = r0 + tid;
    const bool in = r < n;
    double acc[kBMaxRhs];
#pragma unroll
    for (int c = 0; c < kBMaxRhs; ++c) acc[c] = (in && c < nrhs) ? B[r + (long long)c * ldb] : 0.0;
    if (__any_sync(0xffffffffu, in)) {
      const double* ar = A + (in ? r : n - 1);
      for (int k0 = 0; k0 < n; k0 += 8) {
        double a[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) a[k] = ar[(long long)min(k0 + k, n - 1) * lda];
#pragma unroll
        for (int k = 0; k < 8; ++k)
          if (k0 + k < n) {
#pragma unroll
            for (int c = 0; c < kBMaxRhs; ++c)
              if (c < nrhs) acc[c] = fma(-a[k], Xsh[k0 + k + c * n], acc[c]);
          }
      }
#pragma unroll
      for (int c = 0; c < kBMaxRhs; ++c)
        if (c < nrhs) {
          if (in && Rs) Rs[r + c * n] = acc[c];
          const unsigned long long r1 = warp_max64(in ? mag_key(acc[c]) : 0ULL);
          const unsigned long long x1 = warp_max64(in ? mag_key(Xsh[r + c * n]) : 0ULL);
          if (lane == 0) {
            atomicMax(&s_rm[c], r1);
            atomicMax(&s_xm[c], x1);
          }
        }
    }
  }
  __syncthreads();
  if (warp == 0) {
    double v = 0.0;
    if (lane < nrhs) {
      const double rn = __longlong_as_double((long long)s_rm[lane]);
      rmax[lane] = rn;
      // (a zero right-hand side and its zero solution are exact, not 0 / 0)
      v = rn == 0.0 ? 0.0 : rn / (__longlong_as_double((long long)s_xm[lane]) * anorm * ldexp(1.0, -53) * n);
    }
    const unsigned long long w = warp_max64(mag_key(v));
    if (lane == 0) s_worst = __longlong_as_double((long long)w);
  }
  __syncthreads();
  return s_worst;
}

template <typename TF, int NT>
__device__ __forceinline__ void run_system(const BatchArgs& a, int sys, bool fp64_pass, unsigned char* smem) {
  const int n = a.n[sys], nrhs = a.nrhs[sys];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const double* A = a.A[sys];
  const int lda = a.lda[sys];
  TF* W = reinterpret_cast<TF*>(fp64_pass ? a.W64[sys] : a.W[sys]);  // n x (n + nrhs)
  int* ipiv = a.ipiv[sys];
  double* X = a.X[sys];
  const int ldx = a.ldx[sys];
  const double* B = a.B[sys];
  const int ldb = a.ldb[sys];
  const BatchSmem<TF> sm(smem, a.nmax, a.rmax);
  __shared__ unsigned long long s_red[NT / 32];
  __shared__ double s_rmax[kBMaxRhs];
  __shared__ int s_exp[kBMaxRhs];
  __shared__ double s_anorm;
  __shared__ int s_info;
  // Working copy in the factorization precision; one thread per row, so the
  // same pass gives ||A||_inf (row sums of |a|). The right-hand sides follow
  // as columns n .. n+nrhs-1 (FP32 factors: each scaled by a power of two), so
  // that the factorization does their forward solve.
  {
    unsigned long long rs_max = 0ULL;
    for (int r = tid; r < n; r += NT) {
      double rs = 0.0;
      const double* ar = A + r;
      for (int c0 = 0; c0 < n; c0 += 8) {
        double v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = ar[(long long)min(c0 + q, n - 1) * lda];
#pragma unroll
        for (int q = 0; q < 8; ++q)
          if (c0 + q < n) {
            rs += fabs(v[q]);
            W[r + (long long)(c0 + q) * n] = (TF)v[q];
          }
      }
      rs_max = max(rs_max, mag_key(rs));
    }
    rs_max = warp_max64(rs_max);
    if (lane == 0) s_red[warp] = rs_max;
    if constexpr (sizeof(TF) == 4) {
      for (int c = warp; c < nrhs; c += NT / 32) {
        unsigned long long bm = 0ULL;
        for (int i = lane; i < n; i += 32) bm = max(bm, mag_key(B[i + (long long)c * ldb]));
        bm = warp_max64(bm);
        if (lane == 0) s_rmax[c] = __longlong_as_double((long long)bm);
      }
    }
    __syncthreads();
    if (tid == 0) {
      unsigned long long an = 0ULL;
      for (int w = 0; w < NT / 32; ++w) an = max(an, s_red[w]);
      s_anorm = __longlong_as_double((long long)an);
    }
    if (tid < nrhs) {
      int e = 0;
      if constexpr (sizeof(TF) == 4) {
        const double mx = s_rmax[tid];
        if (mx > 0.0 && isfinite(mx)) frexp(mx, &e);
      }
      s_exp[tid] = e;
    }
    __syncthreads();
    for (int c = 0; c < nrhs; ++c)
      for (int i = tid; i < n; i += NT) {
        const double b = B[i + (long long)c * ldb];
        W[i + (long long)(n + c) * n] = sizeof(TF) == 4 ? (TF)ldexp(b, -s_exp[c]) : (TF)b;
      }
    __syncthreads();
  }
  factor_system<TF, NT>(W, n, n + nrhs, ipiv, &s_info, sm);
  const int info = s_info;
  if (info != 0) {
    // Exactly singular in the factorization precision: in mode 1 hand the
    // system to the FP64 pass, else report INFO and leave X untouched.
    if (!fp64_pass && sizeof(TF) == 4) {
      if (tid == 0) {
        int slot = atomicAdd(&a.queue[2], 1);
        a.fallback_list[slot] = sys;
      }
    } else if (tid == 0) {
      a.info[sys] = info;
      a.iters[sys] = 0;
      a.sresid[sys] = -1.0;
    }
    __syncthreads();
    return;
  }
  TF* Xs = sm.Xs;
  for (int c = 0; c < nrhs; ++c)
    for (int i = tid; i < n; i += NT) Xs[i + c * n] = W[i + (long long)(n + c) * n];
  __syncthreads();
  solve_tri<TF, NT, false>(W, n, Xs, nrhs, sm.Ds);
  if constexpr (sizeof(TF) == 8) {
    for (int c = 0; c < nrhs; ++c)
      for (int i = tid; i < n; i += NT) X[i + (long long)c * ldx] = Xs[i + c * n];
    const double sr = residual_system<NT>(A, lda, n, B, ldb, sm.Xsh, nrhs, nullptr, s_anorm, s_rmax);
    if (tid == 0) {
      a.info[sys] = 0;
      a.iters[sys] = fp64_pass ? -1 : 0;
      a.sresid[sys] = sr;
    }
    __syncthreads();
    return;
  } else {
    // FP32 factors + FP64 refinement: the first correction (from x = 0) stands
    // in Xs; X accumulates in global memory, Xsh holds it during the residual
    int steps = 1;
    double sr = 0.0;
    bool ok = false;
    for (;;) {
      for (int c = 0; c < nrhs; ++c)
        for (int i = tid; i < n; i += NT) {
          const double d = ldexp((double)Xs[i + c * n], s_exp[c]);
          double* xp = X + i + (long long)c * ldx;
          *xp = steps == 1 ? d : *xp + d;
        }
      __syncthreads();
      for (int c = 0; c < nrhs; ++c)
        for (int i = tid; i < n; i += NT) sm.Xsh[i + c * n] = X[i + (long long)c * ldx];
      __syncthreads();
      sr = residual_system<NT>(A, lda, n, B, ldb, sm.Xsh, nrhs, sm.Rs, s_anorm, s_rmax);
      if (sr <= a.tol) { ok = true; break; }
      if (steps == kMaxIr) break;
      // correction: scale each residual column by a power of two into FP32, solve
      if (tid < nrhs) {
        const double mx = s_rmax[tid];
        int e = 0;
        if (mx > 0.0 && isfinite(mx)) frexp(mx, &e);
        s_exp[tid] = e;
      }
      __syncthreads();
      for (int c = 0; c < nrhs; ++c)
        for (int i = tid; i < n; i += NT) Xs[i + c * n] = (TF)ldexp(sm.Rs[sm.org[i] + c * n], -s_exp[c]);
      __syncthreads();
      solve_tri<TF, NT, true>(W, n, Xs, nrhs, sm.Ds);
      solve_tri<TF, NT, false>(W, n, Xs, nrhs, sm.Ds);
      ++steps;
    }
    if (tid == 0) {
      if (ok) {
        a.info[sys] = 0;
        a.iters[sys] = steps;
        a.sresid[sys] = sr;
      } else {
        int slot = atomicAdd(&a.queue[2], 1);
        a.fallback_list[slot] = sys;
      }
    }
    __syncthreads();
  }
}

template <typename TF, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) batched_kernel(BatchArgs a, int fp64_pass) {
  extern __shared__ __align__(16) unsigned char bsmem[];
  __shared__ int s_item;
  const int ticket = fp64_pass ? 1 : 0;
  const int count = fp64_pass ? a.queue[2] : a.batch;
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) s_item = atomicAdd(&a.queue[ticket], 1);
    __syncthreads();
    const int item = s_item;
    if (item >= count) break;
    const int sys = fp64_pass ? a.fallback_list[item] : a.order[item];
    run_system<TF, NT>(a, sys, fp64_pass != 0, bsmem);
  }
}

template <typename TF, int NT, int MINB>
cudaError_t launch_batched(const BatchArgs& a, int fp64_pass, int ctas_per_sm, cudaStream_t s) {
  const size_t smem = BatchSmem<TF>::bytes(a.nmax, a.rmax);
  auto kern = batched_kernel<TF, NT, MINB>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  int occ = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, NT, smem);
  if (e != cudaSuccess) return e;
  if (occ < 1) return cudaErrorInvalidConfiguration;
  const int per_sm = std::min(occ, std::max(1, ctas_per_sm));
  kern<<<num_sms() * per_sm, NT, smem, s>>>(a, fp64_pass);
  count_launches(1);
  return cudaGetLastError();
}

// threads in {128, 256, 512}; as many CTAs per SM as fit, up to ctas
template <typename TF>
cudaError_t launch_batched(const BatchArgs& a, int fp64_pass, int threads, int ctas, cudaStream_t s) {
  if (threads == 128) return launch_batched<TF, 128, 4>(a, fp64_pass, ctas, s);
  if (threads == 512) return launch_batched<TF, 512, 1>(a, fp64_pass, ctas, s);
  return launch_batched<TF, 256, 2>(a, fp64_pass, ctas, s);
}

// ------------------------------------------------------------ plan
struct BatchPlan {
  int batch = 0, mode = 0;
  double tol = 1.0;
  // device arrays
  int *d_n = nullptr, *d_nrhs = nullptr, *d_lda = nullptr, *d_ldb = nullptr, *d_ldx = nullptr;
  const double** d_A = nullptr;
  const double** d_B = nullptr;
  double** d_X = nullptr;
  int** d_ipiv = nullptr;
  void** d_W = nullptr;
  int *d_order = nullptr, *d_queue = nullptr, *d_fb = nullptr;
  int *d_info = nullptr, *d_iters = nullptr;
  double* d_sresid = nullptr;
  void* work = nullptr;        // factor workspaces (one block)
  void* work64 = nullptr;      // FP64 workspaces of the FP64 pass (mode 1)
  void** d_W64 = nullptr;
  int* ipiv_pool = nullptr;    // pivots (one block)
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  int threads = 256, chunk = 16, ctas_per_sm = 1;
  int nmax = 1, rmax = 1;
  double flops = 0.0;
};

static BatchArgs plan_args(const BatchPlan& p) {
  BatchArgs a;
  a.batch = p.batch; a.n = p.d_n; a.nrhs = p.d_nrhs; a.A = p.d_A; a.lda = p.d_lda;
  a.B = p.d_B; a.ldb = p.d_ldb; a.X = p.d_X; a.ldx = p.d_ldx; a.ipiv = p.d_ipiv; a.W = p.d_W;
  a.W64 = p.mode == 0 ? p.d_W : p.d_W64;
  a.order = p.d_order; a.queue = p.d_queue; a.fallback_list = p.d_fb; a.info = p.d_info;
  a.iters = p.d_iters; a.sresid = p.d_sresid; a.tol = p.tol; a.nmax = p.nmax; a.rmax = p.rmax;
  return a;
}

static cudaError_t record_plan(const BatchPlan& p, int threads, int ctas, cudaStream_t s) {
  BatchArgs a = plan_args(p);
  SL_TRY(cudaMemsetAsync(p.d_queue, 0, 4 * sizeof(int), s));
  if (p.mode == 0) return launch_batched<double>(a, 0, threads, ctas, s);
  SL_TRY(launch_batched<float>(a, 0, threads, ctas, s));
  // FP64 pass over the systems the refinement could not finish (may be empty)
  return launch_batched<double>(a, 1, 256, 2, s);
}

cudaError_t batch_plan_create(BatchPlan** out, int batch, const int* n, const int* nrhs,
                              const double* const* A, const int* lda, const double* const* B,
                              const int* ldb, double* const* X, const int* ldx, int mode,
                              double tol, int autotune, cudaStream_t s) {
  *out = nullptr;
  BatchPlan* p = new BatchPlan();
  p->batch = batch;
  p->mode = mode;
  p->tol = tol > 0 ? tol : 1.0;
  std::vector<int> order(batch);
  std::iota(order.begin(), order.end(), 0);
  std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return n[x] > n[y]; });
  const size_t esz = mode == 0 ? sizeof(double) : sizeof(float);
  std::vector<size_t> woff(batch), poff(batch);
  size_t wtot = 0, ptot = 0;
  for (int i = 0; i < batch; ++i) {
    woff[i] = wtot;
    wtot += ((size_t)n[i] * (n[i] + nrhs[i]) * esz + 255) / 256 * 256;
    p->nmax = std::max(p->nmax, n[i]);
    p->rmax = std::max(p->rmax, nrhs[i]);
    poff[i] = ptot;
    ptot += (size_t)n[i];
    p->flops += 2.0 * n[i] * (double)n[i] * n[i] / 3.0;
  }
  cudaError_t e = cudaSuccess;
  auto alloc = [&](auto** ptr, size_t bytes) {
    if (e == cudaSuccess) e = cudaMalloc((void**)ptr, bytes < 4 ? 4 : bytes);
  };
  alloc(&p->d_n, sizeof(int) * batch);
  alloc(&p->d_nrhs, sizeof(int) * batch);
  alloc(&p->d_lda, sizeof(int) * batch);
  alloc(&p->d_ldb, sizeof(int) * batch);
  alloc(&p->d_ldx, sizeof(int) * batch);
  alloc(&p->d_A, sizeof(double*) * batch);
  alloc(&p->d_B, sizeof(double*) * batch);
  alloc(&p->d_X, sizeof(double*) * batch);
  alloc(&p->d_ipiv, sizeof(int*) * batch);
  alloc(&p->d_W, sizeof(void*) * batch);
  alloc(&p->d_order, sizeof(int) * batch);
  alloc(&p->d_queue, sizeof(int) * 4);
  alloc(&p->d_fb, sizeof(int) * batch);
  alloc(&p->d_info, sizeof(int) * batch);
  alloc(&p->d_iters, sizeof(int) * batch);
  alloc(&p->d_sresid, sizeof(double) * batch);
  alloc(&p->work, wtot);
  alloc(&p->ipiv_pool, sizeof(int) * ptot);
  std::vector<size_t> w64off(batch);
  size_t w64 = 0;
  if (mode == 1) {
    for (int i = 0; i < batch; ++i) {
      w64off[i] = w64;
      w64 += ((size_t)n[i] * (n[i] + nrhs[i]) * sizeof(double) + 255) / 256 * 256;
    }
    alloc(&p->work64, w64);
    alloc(&p->d_W64, sizeof(void*) * batch);
  }
  if (e != cudaSuccess) { batch_plan_destroy(p); return e; }
  std::vector<void*> W(batch), W64(batch);
  std::vector<int*> piv(batch);
  for (int i = 0; i < batch; ++i) {
    W[i] = (unsigned char*)p->work + woff[i];
    if (mode == 1) W64[i] = (unsigned char*)p->work64 + w64off[i];
    piv[i] = p->ipiv_pool + poff[i];
  }
  auto up = [&](void* dst, const void* src, size_t bytes) {
    if (e == cudaSuccess) e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s);
  };
  up(p->d_n, n, sizeof(int) * batch);
  up(p->d_nrhs, nrhs, sizeof(int) * batch);
  up(p->d_lda, lda, sizeof(int) * batch);
  up(p->d_ldb, ldb, sizeof(int) * batch);
  up(p->d_ldx, ldx, sizeof(int) * batch);
  up(p->d_A, A, sizeof(double*) * batch);
  up(p->d_B, B, sizeof(double*) * batch);
  up(p->d_X, X, sizeof(double*) * batch);
  up(p->d_ipiv, piv.data(), sizeof(int*) * batch);
  up(p->d_W, W.data(), sizeof(void*) * batch);
  if (mode == 1) up(p->d_W64, W64.data(), sizeof(void*) * batch);
  up(p->d_order, order.data(), sizeof(int) * batch);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) { batch_plan_destroy(p); return e; }
  // autotune: time the candidate shapes on this batch and keep the fastest
  struct Cand { int threads, ctas; };
  std::vector<Cand> cands = {{256, 8}, {512, 8}, {128, 16}};
  Cand best = p->nmax <= 128 ? cands[2] : cands[0];
  if (autotune) {
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    float best_ms = 1e30f;
    for (const Cand& c : cands) {
      cudaEventRecord(e0, s);
      cudaError_t r = record_plan(*p, c.threads, c.ctas, s);
      cudaEventRecord(e1, s);
      if (r != cudaSuccess) { cudaGetLastError(); continue; }
      if (cudaEventSynchronize(e1) != cudaSuccess) break;
      float ms = 0.f;
      cudaEventElapsedTime(&ms, e0, e1);
      if (ms < best_ms) { best_ms = ms; best = c; }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
  }
  p->threads = best.threads;
  p->chunk = mode == 0 ? chunk_cols<double>() : chunk_cols<float>();
  p->ctas_per_sm = best.ctas;
  // capture the execution in a CUDA graph
  cudaStream_t cs;
  e = cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal);
  if (e == cudaSuccess) {
    cudaError_t r = record_plan(*p, p->threads, p->ctas_per_sm, cs);
    cudaGraph_t g = nullptr;
    e = cudaStreamEndCapture(cs, &g);
    if (r != cudaSuccess) e = r;
    if (e == cudaSuccess) {
      p->graph = g;
      e = cudaGraphInstantiate(&p->exec, g, 0);
    }
  }
  cudaStreamDestroy(cs);
  if (e != cudaSuccess) { batch_plan_destroy(p); return e; }
  *out = p;
  return cudaSuccess;
}

cudaError_t batch_plan_execute(BatchPlan* p, cudaStream_t s) {
  phase_begin(kPhBatched, s);
  cudaError_t e = cudaGraphLaunch(p->exec, s);
  count_launches(p->mode == 0 ? 1 : 2);
  phase_end(kPhBatched, s, p->flops, 0.0);
  return e;
}

cudaError_t batch_plan_results(BatchPlan* p, int* info, int* iters, double* sresid,
                               cudaStream_t s) {
  cudaError_t e = cudaSuccess;
  if (info) e = cudaMemcpyAsync(info, p->d_info, sizeof(int) * p->batch, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess && iters)
    e = cudaMemcpyAsync(iters, p->d_iters, sizeof(int) * p->batch, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess && sresid)
    e = cudaMemcpyAsync(sresid, p->d_sresid, sizeof(double) * p->batch, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  return e;
}

void batch_plan_shape(const BatchPlan* p, int* threads, int* chunk, int* ctas) {
  *threads = p->threads;
  *chunk = p->chunk;
  *ctas = p->ctas_per_sm;
}

void batch_plan_destroy(BatchPlan* p) {
  if (!p) return;
  if (p->exec) cudaGraphExecDestroy(p->exec);
  if (p->graph) cudaGraphDestroy(p->graph);
  cudaFree(p->d_n); cudaFree(p->d_nrhs); cudaFree(p->d_lda); cudaFree(p->d_ldb); cudaFree(p->d_ldx);
  cudaFree(p->d_A); cudaFree(p->d_B); cudaFree(p->d_X); cudaFree(p->d_ipiv); cudaFree(p->d_W);
  cudaFree(p->d_order); cudaFree(p->d_queue); cudaFree(p->d_fb); cudaFree(p->d_info);
  cudaFree(p->d_iters); cudaFree(p->d_sresid); cudaFree(p->work); cudaFree(p->ipiv_pool);
  cudaFree(p->work64); cudaFree(p->d_W64);
  delete p;
}

}  // namespace sl
