// Chained FP64 triangular solves for few right-hand sides (PDGETRS,
// SRC/pdgetrs.f:250-284, both TRANS): two launches, one per triangle, instead
// of two or three launches per 128 rows.
//
// Work is cut into 64-row blocks of op(T) times groups of NR right-hand sides;
// each CTA takes the next (block, group) in solve order from an atomic ticket,
// so every block it depends on belongs to a CTA that has already started and
// the waits always end (no residency assumption). A CTA streams its 64x64
// blocks of the factor through a ring in shared memory with cp.async, ahead of
// the solutions it needs; solved values are published as single-copy atomic
// 16-byte words {x, epoch}, so a consumer polls the data itself (one L2 round
// trip, no flag, no fence). With all of them applied, x_b = inv(T_bb) v_b from
// the precomputed inverse of the diagonal block (the last tile of the ring).
//
// Bound: n^2 nrhs FMAs on the FP64 pipe (a 64x64 block times one vector takes
// 2560 cycles of an SM) when there are many right-hand sides; with one, the
// chain of n/64 steps (one poll, one block product, one inverse product: about
// 4 us each). One right-hand side per CTA keeps that chain short; two halve the
// factor's reads through L2 once the pipe is the bound. Measured, GB300: n = 8192
// with one right-hand side, 0.97 ms for the whole PDGETRS (two chains of 0.39,
// the rest before them; 6.27 with three launches per 128 rows); n = 8192, TRANS
// = 'T', 16 right-hand sides, 3.07 ms (16.96 by substitution and DMMA
// products), of which the FP64 pipe needs 2.0.
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"
#include "sl_internal.h"

namespace sl {
namespace {

constexpr int TB = 64;             // rows of a block
constexpr int TSLOT = TB * 65;     // doubles of a ring slot (stride 65 when transposed)
constexpr int TRING = 3;

__device__ __forceinline__ void cp_async8(double* dst, const double* src, bool in) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(in ? 8 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// {x, epoch} in one 16-byte word
__device__ __forceinline__ void put_x(unsigned long long* p, double x, uint32_t epoch) {
  asm volatile("{ .reg .b128 t;\n mov.b128 t, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], t; }" ::"l"(p),
               "l"((unsigned long long)__double_as_longlong(x)), "l"((unsigned long long)epoch)
               : "memory");
}
__device__ __forceinline__ bool get_x(const unsigned long long* p, uint32_t epoch, double& x) {
  unsigned long long a, b;
  asm volatile("{ .reg .b128 t;\n ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t; }"
               : "=l"(a), "=l"(b)
               : "l"(p)
               : "memory");
  x = __longlong_as_double((long long)a);
  return (uint32_t)b == epoch;
}

// op(T) X = S for one triangle of the LU factors A; TRANS: op(T) = T^T.
// forward: block rows from the top (lower, or upper transposed). Row i of S is
// row i of src, of X row i of dst, or in either place the row that the pivots
// `gather` / `scatter` permute there (null: i; maps: their segments' maps,
// follow_perm). D: inverses of T's diagonal blocks,
// 4096 doubles each, column-major.
template <int NR, bool TRANS>
__global__ void __launch_bounds__(256)
trsv64_chain_kernel(const double* __restrict__ A, long long lda, int n, int forward,
                    const double* __restrict__ D, const double* __restrict__ src, long long lds,
                    const int* __restrict__ gather, double* dst, long long ldd,
                    const int* __restrict__ scatter, const int* __restrict__ maps, int nrhs,
                    int ngroups, int* ticket,
                    unsigned long long* words, uint32_t epoch, int* status) {
  extern __shared__ double trsv_ring[];     // TRING tiles
  __shared__ double xs[2][TB * NR];         // solutions of the block being applied
  __shared__ double part[4][TB * NR];
  __shared__ double vs[TB * NR];
  __shared__ int s_t, s_fail;
  const int tid = threadIdx.x;
  if (tid == 0) {
    s_t = atomicAdd(ticket, 1);
    s_fail = *(volatile int*)status != 0;  // an earlier wait gave up: nothing more comes
  }
  __syncthreads();
  const int nblk = (n + TB - 1) / TB;
  const int sidx = s_t / ngroups, c0 = (s_t % ngroups) * NR;
  if (sidx >= nblk || s_fail) return;
  const int b = forward ? sidx : nblk - 1 - sidx;
  const int r0 = b * TB, rb = min(TB, n - r0);
  const int r = tid & (TB - 1), q = tid >> 6;

  // tile t of the ring: block (b, k(t)) of op(T) for t < sidx, inv(T_bb) for
  // t = sidx; columns of the stored block at stride 64, or 65 when transposed
  // (both ways the threads of a warp then read one column of op(T) without
  // bank conflicts)
  constexpr int CS = TRANS ? TB + 1 : TB;
  auto fetch = [&](int t) {
    if (t <= sidx) {
      double* slot = trsv_ring + (t % TRING) * TSLOT;
      const int k0 = (forward ? t : nblk - 1 - t) * TB;
      const double* g = t == sidx ? D + (size_t)b * (TB * TB)
                                  : (TRANS ? A + k0 + (long long)r0 * lda : A + r0 + (long long)k0 * lda);
      const long long ld = t == sidx ? TB : lda;
      const int kb = t == sidx ? TB : min(TB, n - k0);
      const int rows = t == sidx ? TB : (TRANS ? kb : rb), cols = t == sidx ? TB : (TRANS ? rb : kb);
#pragma unroll 4
      for (int idx = tid; idx < TB * TB; idx += 256) {
        const int i = idx & (TB - 1), j = idx >> 6;
        const bool in = i < rows && j < cols;
        cp_async8(slot + j * CS + i, in ? g + i + (long long)j * ld : g, in);
      }
    }
    cp_commit();
  };
#pragma unroll
  for (int t = 0; t < TRING - 1; ++t) fetch(t);

  // thread (pi, pc) of the first TB*NR carries value pi of right-hand side pc
  const int pi = tid & (TB - 1), pc = tid >> 6;
  const bool mine = pc < NR && pi < rb && c0 + pc < nrhs;
  double bv = 0.0;
  int drow = r0 + pi;
  if (mine) {
    const int srow = gather ? follow_perm(drow, gather, n, maps) : drow;
    if ((unsigned)srow < (unsigned)n) bv = src[srow + (long long)(c0 + pc) * lds];
    if (scatter) drow = follow_perm(drow, scatter, n, maps);
  }

  double acc[NR];
#pragma unroll
  for (int c = 0; c < NR; ++c) acc[c] = 0.0;
  for (int t = 0; t < sidx; ++t) {
    const int k0 = (forward ? t : nblk - 1 - t) * TB;
    if (pc < NR) {
      double v = 0.0;
      if (k0 + pi < n && c0 + pc < nrhs) {
        const unsigned long long* p = words + ((size_t)(c0 + pc) * n + k0 + pi) * 2;
        for (long long spins = 0; !get_x(p, epoch, v);) {
          if (++spins > kSpinLimit) { s_fail = 1; break; }
          // far from its turn a CTA leaves the L2 to the ones that are next
          if (sidx - t > 2) __nanosleep(200);
        }
      }
      xs[t & 1][pi * NR + pc] = v;
    }
    cp_wait<TRING - 2>();
    __syncthreads();
    if (s_fail) {
      if (tid == 0) atomicExch(status, (int)kFlagTimeout);
      cp_wait<0>();
      return;
    }
    fetch(t + TRING - 1);  // into the slot that step t-1 has finished with
    // a tile's 16 terms are summed before they join the row's running sum, so
    // that a row of any length meets one rounding per tile at the sum's size
    const double* T = trsv_ring + (t % TRING) * TSLOT;
    const double* x = xs[t & 1];
    double p[NR];
#pragma unroll
    for (int kk = 0; kk < 16; ++kk) {
      const int k = q * 16 + kk;
      const double a = TRANS ? T[r * CS + k] : T[k * CS + r];
#pragma unroll
      for (int c = 0; c < NR; ++c) p[c] = kk == 0 ? a * x[k * NR + c] : fma(a, x[k * NR + c], p[c]);
    }
#pragma unroll
    for (int c = 0; c < NR; ++c) acc[c] += p[c];
  }
#pragma unroll
  for (int c = 0; c < NR; ++c) part[q][r * NR + c] = acc[c];
  cp_wait<0>();
  __syncthreads();
  if (pc < NR) {
    const int e = pi * NR + pc;
    vs[e] = bv - ((part[0][e] + part[1][e]) + (part[2][e] + part[3][e]));
  }
  __syncthreads();
  {
    // x = inv(T_bb) v over the triangle only, so that an Inf or NaN in v
    // reaches no row that does not depend on it
    const double* T = trsv_ring + (sidx % TRING) * TSLOT;
#pragma unroll
    for (int c = 0; c < NR; ++c) acc[c] = 0.0;
#pragma unroll
    for (int kk = 0; kk < 16; ++kk) {
      const int k = q * 16 + kk;
      const double a = TRANS ? T[r * CS + k] : T[k * CS + r];
      if (forward ? k <= r : k >= r) {
#pragma unroll
        for (int c = 0; c < NR; ++c) acc[c] = fma(a, vs[k * NR + c], acc[c]);
      }
    }
#pragma unroll
    for (int c = 0; c < NR; ++c) part[q][r * NR + c] = acc[c];
  }
  __syncthreads();
  if (mine) {
    const int e = pi * NR + pc;
    const double x = (part[0][e] + part[1][e]) + (part[2][e] + part[3][e]);
    put_x(words + ((size_t)(c0 + pc) * n + r0 + pi) * 2, x, epoch);
    if ((unsigned)drow < (unsigned)n) dst[drow + (long long)(c0 + pc) * ldd] = x;  // (an invalid IPIV writes nothing)
  }
}

template <int NR, bool TRANS>
cudaError_t launch_chain(const double* A, long long lda, int n, bool forward, const double* D,
                         const double* src, long long lds, const int* gather, double* dst,
                         long long ldd, const int* scatter, const int* maps, int nrhs, int* ticket,
                         unsigned long long* words, uint32_t epoch, int* status, cudaStream_t s) {
  constexpr int smem = TRING * TSLOT * (int)sizeof(double);
  auto kern = trsv64_chain_kernel<NR, TRANS>;
  static const cudaError_t attr = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  SL_TRY(attr);
  const int ngroups = (nrhs + NR - 1) / NR;
  kern<<<(n + TB - 1) / TB * ngroups, 256, smem, s>>>(A, lda, n, forward ? 1 : 0, D, src, lds, gather, dst,
                                                      ldd, scatter, maps, nrhs, ngroups, ticket, words, epoch, status);
  count_launches(1);
  return cudaGetLastError();
}

}  // namespace

cudaError_t trsv64_chain(bool lower, bool trans, const double* A, long long lda, int n, const double* D,
                         const double* src, long long lds, const int* gather, double* dst,
                         long long ldd, const int* scatter, const int* maps, int nrhs, int* ticket,
                         unsigned long long* words, uint32_t epoch, int* status, cudaStream_t s) {
  const bool forward = lower != trans;
  // two right-hand sides a CTA once one each would queue several CTAs per SM
  const bool two = nrhs > 1 && (long long)((n + TB - 1) / TB) * nrhs > 2LL * num_sms();
#define SL_CH(NR, TR)                                                                                 \
  return launch_chain<NR, TR>(A, lda, n, forward, D, src, lds, gather, dst, ldd, scatter, maps, nrhs, ticket, \
                              words, epoch, status, s)
  if (two) {
    if (trans) SL_CH(2, true);
    SL_CH(2, false);
  }
  if (trans) SL_CH(1, true);
  SL_CH(1, false);
#undef SL_CH
}

}  // namespace sl
