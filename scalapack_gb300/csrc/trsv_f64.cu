// Chained FP64 triangular solves for few right-hand sides (PDGETRS,
// SRC/pdgetrs.f:250-284, both TRANS): two launches, one per triangle, instead
// of two or three launches per 128 rows.
//
// Work is cut into 64-row blocks of op(T) times right-hand sides; each CTA takes
// the next (block, right-hand side) in solve order from an atomic ticket,
// so every block it depends on belongs to a CTA that has already started and
// the waits always end (no residency assumption); each is bounded all the same
// (spin_limit polls), and a CTA that gives up sets the status word, at which the
// CTAs after it leave at once. A CTA streams its 64x64
// blocks of the factor through a ring in shared memory with cp.async, ahead of
// the solutions it needs; solved values are published as single-copy atomic
// 16-byte words {x, epoch}, so a consumer polls the data itself (one L2 round
// trip, no flag, no fence). With all of them applied, x_b = inv(T_bb) v_b from
// the precomputed inverse of the diagonal block (the last tile of the ring); a block
// whose inverse is large (tri_inv64_of) is solved by substitution instead, its own
// triangle then being the last tile.
//
// Bound: n^2 nrhs FMAs on the FP64 pipe (a 64x64 block times one vector takes
// 2560 cycles of an SM) when there are many right-hand sides; with one, the
// chain of n/64 steps (one poll, one block product, one inverse product: about
// 3.5 us each). Two right-hand sides per CTA would halve the factor's reads
// through L2, which are not the bound, and lengthen a block's turn in the chain,
// which is: n = 4096, 8 right-hand sides 0.93 ms (one per CTA: 0.59), n = 8192, 16
// of them 2.98 (2.56), n = 16384 9.70 (9.12). Measured, GB300: n = 8192 with one
// right-hand side, 0.91 ms for the whole PDGETRS (two chains of 0.39, the rest
// before them; 6.27 with three launches per 128 rows); n = 8192, TRANS = 'T', 16
// right-hand sides, 2.55 ms (16.96 by substitution and DMMA products), of which
// the FP64 pipe needs 2.0. The three launches of a PDGETRS overlap (launch_after):
// n = 64 56 -> 46 us, n = 1000 with 16 columns 173 -> 167.
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

// x = op(T) \ v over the tile T by the first warp, out: four partial sums of x (the
// first is x). Not inlined: a CTA comes to the end of the kernel once, and what stands
// between the loop and the product there is fetched on every step of the chain (n = 8192
// with one right-hand side: 0.90 ms without this way, 0.91 with it, 1.00 inlined).
template <bool TRANS>
__device__ __noinline__ void substitute_tile(int forward, int w, const double* T, const double* v, double* out) {
  constexpr int CS = TRANS ? TB + 1 : TB;
  const int tid = threadIdx.x;
  if (tid < 32) {
    double x0 = v[tid], x1 = v[tid + 32];
    // (the unit triangle is L: forward without TRANS, backward with it)
    warp_substitute64(forward, (forward != 0) != TRANS, w,
                      [&](int i, int k) { return TRANS ? T[i * CS + k] : T[k * CS + i]; }, x0, x1);
    out[tid] = x0;
    out[tid + 32] = x1;
  }
  if (tid >= TB) out[tid] = 0.0;
}

// op(T) X = S for one triangle of the LU factors A; TRANS: op(T) = T^T.
// forward: block rows from the top (lower, or upper transposed). Row i of S is
// row i of src, of X row i of dst, or in either place the row that the pivots
// `gather` / `scatter` permute there (null: i; maps: their segments' maps,
// follow_perm). D: inverses of T's diagonal blocks, 4096 doubles each, column-major;
// flags: four words per block, nonzero where it is solved by substitution.
template <bool TRANS>
__global__ void __launch_bounds__(256)
trsv64_chain_kernel(const double* __restrict__ A, long long lda, int n, int forward,
                    const double* __restrict__ D, const int* __restrict__ flags, const double* __restrict__ src,
                    long long lds, const int* __restrict__ gather, double* dst, long long ldd,
                    const int* __restrict__ scatter, const int* __restrict__ maps, int nrhs,
                    int* ticket, unsigned long long* words, uint32_t epoch, int* status, long long spin_limit) {
  extern __shared__ double trsv_ring[];  // TRING tiles
  __shared__ double xs[2][TB];           // solution of the block being applied
  __shared__ double part[4][TB];
  __shared__ double vs[TB];
  __shared__ int s_t, s_fail;
  const int tid = threadIdx.x;
  wait_for_previous();
  if (tid == 0) {
    s_t = atomicAdd(ticket, 1);
    s_fail = *(volatile int*)status != 0;  // an earlier wait gave up: nothing more comes
  }
  __syncthreads();
  const int nblk = (n + TB - 1) / TB;
  const int sidx = s_t / nrhs, col = s_t % nrhs;
  if (sidx >= nblk || s_fail) return;
  const int b = forward ? sidx : nblk - 1 - sidx;
  const int r0 = b * TB, rb = min(TB, n - r0);
  const int r = tid & (TB - 1), q = tid >> 6;
  const int4 fl = reinterpret_cast<const int4*>(flags)[b];
  const bool subst = (fl.x | fl.y | fl.z | fl.w) != 0;

  // tile t of the ring: block (b, k(t)) of op(T) for t < sidx, inv(T_bb) (or T_bb) for
  // t = sidx; columns of the stored block at stride 64, or 65 when transposed
  // (both ways the threads of a warp then read one column of op(T) without
  // bank conflicts)
  constexpr int CS = TRANS ? TB + 1 : TB;
  auto fetch = [&](int t) {
    if (t <= sidx) {
      double* slot = trsv_ring + (t % TRING) * TSLOT;
      const int k0 = (forward ? t : nblk - 1 - t) * TB;
      const bool inv = t == sidx && !subst;
      const double* g = inv ? D + (size_t)b * (TB * TB)
                            : (TRANS ? A + k0 + (long long)r0 * lda : A + r0 + (long long)k0 * lda);
      const long long ld = inv ? TB : lda;
      const int kb = inv ? TB : min(TB, n - k0);
      const int rows = inv ? TB : (TRANS ? kb : rb), cols = inv ? TB : (TRANS ? rb : kb);
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

  // thread r of the first TB carries value r of the block
  const bool mine = tid < rb;
  double bv = 0.0;
  int drow = r0 + r;
  if (mine) {
    const int srow = gather ? follow_perm(drow, gather, n, maps) : drow;
    if ((unsigned)srow < (unsigned)n) bv = src[srow + (long long)col * lds];
    if (scatter) drow = follow_perm(drow, scatter, n, maps);
  }

  double acc = 0.0;
  for (int t = 0; t < sidx; ++t) {
    const int k0 = (forward ? t : nblk - 1 - t) * TB;
    int fail = 0;
    if (tid < TB) {
      double v = 0.0;
      if (k0 + r < n) {
        const unsigned long long* p = words + ((size_t)col * n + k0 + r) * 2;
        for (long long spins = 0;; ++spins) {
          if (spins >= spin_limit) { fail = 1; break; }
          if (get_x(p, epoch, v)) break;
          // far from its turn a CTA leaves the L2 to the ones that are next
          if (sidx - t > 2) __nanosleep(200);
        }
      }
      xs[t & 1][r] = v;
    }
    cp_wait<TRING - 2>();
    if (__syncthreads_or(fail)) {  // (the CTA gives up as a whole)
      if (tid == 0) atomicExch(status, (int)kFlagTimeout);
      cp_wait<0>();
      return;
    }
    fetch(t + TRING - 1);  // into the slot that step t-1 has finished with
    // a tile's 16 terms are summed before they join the row's running sum, so
    // that a row of any length meets one rounding per tile at the sum's size
    const double* T = trsv_ring + (t % TRING) * TSLOT;
    const double* x = xs[t & 1];
    double p = 0.0;
#pragma unroll
    for (int kk = 0; kk < 16; ++kk) {
      const int k = q * 16 + kk;
      const double a = TRANS ? T[r * CS + k] : T[k * CS + r];
      p = kk == 0 ? a * x[k] : fma(a, x[k], p);
    }
    acc += p;
  }
  launch_dependents();  // the other triangle's CTAs come up when the last block is this far
  part[q][r] = acc;
  cp_wait<0>();
  __syncthreads();
  if (tid < TB) vs[r] = bv - ((part[0][r] + part[1][r]) + (part[2][r] + part[3][r]));
  __syncthreads();
  const double* T = trsv_ring + (sidx % TRING) * TSLOT;
  if (__builtin_expect(subst, false)) {
    substitute_tile<TRANS>(forward, rb, T, vs, part[0]);
  } else {
    // x = inv(T_bb) v over the triangle only, so that an Inf or NaN in v
    // reaches no row that does not depend on it
    acc = 0.0;
#pragma unroll
    for (int kk = 0; kk < 16; ++kk) {
      const int k = q * 16 + kk;
      const double a = TRANS ? T[r * CS + k] : T[k * CS + r];
      if (forward ? k <= r : k >= r) acc = fma(a, vs[k], acc);
    }
    part[q][r] = acc;
  }
  __syncthreads();
  if (mine) {
    const double x = (part[0][r] + part[1][r]) + (part[2][r] + part[3][r]);
    put_x(words + ((size_t)col * n + r0 + r) * 2, x, epoch);
    if ((unsigned)drow < (unsigned)n) dst[drow + (long long)col * ldd] = x;  // (an invalid IPIV writes nothing)
  }
}

template <bool TRANS>
cudaError_t launch_chain(const double* A, long long lda, int n, bool forward, const double* D,
                         const int* flags, const double* src, long long lds, const int* gather, double* dst,
                         long long ldd, const int* scatter, const int* maps, int nrhs, int* ticket,
                         unsigned long long* words, uint32_t epoch, int* status, cudaStream_t s) {
  constexpr int smem = TRING * TSLOT * (int)sizeof(double);
  auto kern = trsv64_chain_kernel<TRANS>;
  static const cudaError_t attr = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  SL_TRY(attr);
  count_launches(1);
  return launch_after(kern, dim3((n + TB - 1) / TB * nrhs), 256, smem, s, A, lda, n, forward ? 1 : 0, D, flags, src, lds, gather,
                      dst, ldd, scatter, maps, nrhs, ticket, words, epoch, status, spin_limit());
}

}  // namespace

cudaError_t trsv64_chain(bool lower, bool trans, const double* A, long long lda, int n, const double* D,
                         const int* flags, const double* src, long long lds, const int* gather, double* dst,
                         long long ldd, const int* scatter, const int* maps, int nrhs, int* ticket,
                         unsigned long long* words, uint32_t epoch, int* status, cudaStream_t s) {
  const bool forward = lower != trans;
  auto launch = trans ? launch_chain<true> : launch_chain<false>;
  return launch(A, lda, n, forward, D, flags, src, lds, gather, dst, ldd, scatter, maps, nrhs, ticket, words, epoch, status, s);
}

}  // namespace sl
