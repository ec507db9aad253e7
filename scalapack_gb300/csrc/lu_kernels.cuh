// Type-generic LU kernels (T = double for the plain FP64 path, float for the
// FP32 panel of the mixed-precision path) and their launch helpers.
//
//   panel_kernel<T>      PDGETF2 (SRC/pdgetf2.f:206-237) on a <=32-column sub-panel
//   laswp_kernel<T>      PDLASWP (SRC/pdlaswp.f:163-172)
//   trsm_strip_kernel<T> PDTRSM diagonal-block solves (PB_CptrsmAB.c)
//   permute_rows_kernel<T>, gemm_skinny_kernel<T>  PDLAPIV and the narrow
//                        off-diagonal updates of PDGETRS
#pragma once
#include <algorithm>
#include <climits>
#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>

#include "common.cuh"
#include "sl_internal.h"

namespace sl {

namespace {
// Dynamic shared-memory opt-in, once per kernel and translation unit. Kernels
// are registered per translation unit, so the record of which kernels were
// raised must not be shared between units: it lives in an unnamed namespace.
inline cudaError_t smem_attr_once(const void* kern, int bytes) {
  static std::mutex mu;
  static const void* done_k[64];
  static int done_b[64];
  static int ndone = 0;
  std::lock_guard<std::mutex> lk(mu);
  for (int i = 0; i < ndone; ++i)
    if (done_k[i] == kern && done_b[i] >= bytes) return cudaSuccess;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess && ndone < 64) {
    done_k[ndone] = kern;
    done_b[ndone] = bytes;
    ++ndone;
  }
  return e;
}
}  // namespace

constexpr int PW = 32;       // sub-panel width held in shared memory (<= 64)
constexpr int PMAXG = 160;   // max CTAs of the panel kernel
// Exchange area of the panel kernel, in 8-byte words: the candidate keys
// [2 parities][PMAXG readers][PMAXG writers], each {key, label | tag << 32} in
// one 16-byte word, so that a CTA polls lines that no other CTA reads, and the
// candidate rows [PMAXG][2 parities][2*PW] in tagged 8-byte words.
constexpr int PX_KEYS = 0;
constexpr int PX_VALS = PX_KEYS + 2 * PMAXG * PMAXG * 2;
constexpr int PX_WORDS = PX_VALS + PMAXG * 2 * 2 * PW;
constexpr int PTR = 256;     // row threads per panel CTA
constexpr int PT = PTR + 32; // and the exchange warp
constexpr int PKP = 2;        // key polls a lane keeps in flight (64 CTAs)
constexpr int PCH = 16;       // columns a row thread copies at a time
constexpr int PLD = PW + 1;  // shared row stride: conflict-free row and column walks

// Factor rows [r0, m) x columns [c0, c0+w) (w <= 32) of A in place (the
// panel kernel below): writes ipiv[c0+k] = r0 + pivot (0-based rows of A) for
// k < min(w, m-r0) and the first exactly-zero pivot column into *info_col.
//
// Tagged 8-byte words {32-bit payload, 32-bit tag} carry the per-column
// exchange between the panel's CTAs: a word is valid once its tag equals the
// column's tag, so readers poll the data itself and no separate grid barrier
// or fence is needed (each aligned 8-byte access is single-copy atomic).
__device__ __forceinline__ void st_tagged(unsigned long long* p, uint32_t v, uint32_t tag) {
  const unsigned long long wd = ((unsigned long long)tag << 32) | v;
  asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(wd) : "memory");
}
__device__ __forceinline__ unsigned long long ld_tagged(const unsigned long long* p) {
  unsigned long long wd;
  asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(wd) : "l"(p) : "memory");
  return wd;
}
__device__ __forceinline__ void ld_tagged2(const unsigned long long* p, unsigned long long& a,
                                           unsigned long long& b) {
  asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}
__device__ __forceinline__ bool tag_ok(unsigned long long wd, uint32_t tag) {
  return (uint32_t)(wd >> 32) == tag;
}
__device__ __forceinline__ uint32_t payload(unsigned long long wd) { return (uint32_t)wd; }
__device__ __forceinline__ unsigned long long join(unsigned long long lo, unsigned long long hi) {
  return ((unsigned long long)payload(hi) << 32) | payload(lo);
}

// A candidate key with its label and tag, one single-copy atomic 16-byte word.
__device__ __forceinline__ void st_key(unsigned long long* p, long long key, int label, uint32_t tag) {
  const unsigned long long hi = ((unsigned long long)tag << 32) | (uint32_t)label;
  asm volatile("{ .reg .b128 t;\n mov.b128 t, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], t; }" ::"l"(p),
               "l"((unsigned long long)key), "l"(hi)
               : "memory");
}
__device__ __forceinline__ void ld_key(const unsigned long long* p, unsigned long long& key, unsigned long long& hi) {
  asm volatile("{ .reg .b128 t;\n ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t; }"
               : "=l"(key), "=l"(hi)
               : "l"(p)
               : "memory");
}

// Value v of a row as tagged words (FP32: one word, FP64: two).
template <typename T>
__device__ __forceinline__ void st_value(unsigned long long* p, int j, T v, uint32_t tag) {
  if constexpr (sizeof(T) == 4) {
    st_tagged(p + j, __float_as_uint(v), tag);
  } else {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    const unsigned long long t = (unsigned long long)tag << 32;
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p + 2 * j), "l"(t | (uint32_t)b),
                 "l"(t | (b >> 32)) : "memory");
  }
}

// Polls value j of a published row until its tag matches, at most `limit`
// times; false on timeout.
template <typename T>
__device__ __forceinline__ bool ld_value(const unsigned long long* p, int j, uint32_t tag, T& v,
                                         long long limit) {
  for (long long spins = 0; spins < limit; ++spins) {
    if constexpr (sizeof(T) == 4) {
      const unsigned long long a = ld_tagged(p + j);
      if (tag_ok(a, tag)) { v = __uint_as_float(payload(a)); return true; }
    } else {
      unsigned long long a0, a1;
      ld_tagged2(p + 2 * j, a0, a1);
      if (tag_ok(a0, tag) && tag_ok(a1, tag)) { v = __longlong_as_double((long long)join(a0, a1)); return true; }
    }
  }
  return false;
}

// IDAMAX key of a value: the bit pattern of |x| as an integer (monotonic in
// |x| for IEEE formats, +0 and -0 equal; an FP32 pattern in the high half), -1
// for NaN so that NaN never wins. Integer keys keep the pivot search off the
// FP64 pipe.
__device__ __forceinline__ long long amax_ikey(double v) {
  const long long b = __double_as_longlong(v) & 0x7FFFFFFFFFFFFFFFLL;
  return b > 0x7FF0000000000000LL ? -1LL : b;
}
__device__ __forceinline__ long long amax_ikey(float v) {
  const int b = __float_as_int(v) & 0x7FFFFFFF;
  return b > 0x7F800000 ? -1LL : (long long)b << 32;
}
// The lane that holds the warp's best (key, row): largest key, lowest row among
// ties. One integer warp reduction (28 cycles) over the keys' high halves decides
// unless two lanes tie there (two more then, over the low halves and the rows),
// instead of five rounds of three dependent shuffles (42 cycles each), three
// times on every panel column's critical path.
__device__ __forceinline__ int warp_best(long long key, int row) {
  const int h = (int)(key >> 32);
  const int hm = __reduce_max_sync(0xffffffffu, h);
  unsigned hit = __ballot_sync(0xffffffffu, h == hm);
  if (hit & (hit - 1)) {  // (the same on every lane: all take part in what follows)
    const bool t0 = (hit >> (threadIdx.x & 31)) & 1u;
    const unsigned l = t0 ? (unsigned)key : 0u;
    const unsigned lm = __reduce_max_sync(0xffffffffu, l);
    const bool t1 = t0 && l == lm;
    const unsigned r = t1 ? (unsigned)row : 0xffffffffu;
    const unsigned rm = __reduce_min_sync(0xffffffffu, r);
    hit = __ballot_sync(0xffffffffu, t1 && r == rm);
  }
  return __ffs(hit) - 1;
}

// 1/x for a positive finite x, rounded to nearest, from its bit pattern. The
// FP64 pipe of this GPU takes 64 cycles per warp instruction, so a division
// there (a chain of them, beside the other warps' updates) would cost more
// than the L2 round trip it can hide behind; this one runs on the integer
// pipe: Newton's iteration for the reciprocal of the 53-bit significand in
// 64-bit fixed point from a 23-bit seed, then one exact comparison that picks
// the nearest of two neighbours. Subnormal operands or results divide.
__device__ __forceinline__ double recip_bits(unsigned long long bits) {
  const int bexp = (int)(bits >> 52);
  if (bexp == 0 || bexp >= 2045) return 1.0 / __longlong_as_double((long long)bits);
  const unsigned long long frac = bits & 0xfffffffffffffULL;
  if (frac == 0) return __longlong_as_double((long long)((unsigned long long)(2046 - bexp) << 52));
  const unsigned long long m = frac | (1ULL << 52);
  const unsigned long long d = m << 11;                       // D = d / 2^64 in (1/2, 1)
  const float rf = __frcp_rn((float)(unsigned)(d >> 40));     // in (2^-24, 2^-23]
  const float sf = rf * 36028797018963968.0f;                 // 2^55: Y = 1/D in units of 2^-31
  const unsigned y0 = sf >= 4294967040.0f ? 4294967040u : (unsigned)sf;
  // Y <- Y (2 - D Y), twice; e = 2^63 (1 - D Y)
  unsigned long long y = (unsigned long long)y0 << 32;
  long long e = (long long)((1ULL << 63) - __umul64hi(d, y));
  y += (unsigned long long)(((long long)y0 * (e >> 12)) >> 19);
  e = (long long)((1ULL << 63) - __umul64hi(d, y));
  y += (unsigned long long)(((long long)(y >> 32) * e) >> 31);
  // y is within a few units of 2^64 / (2 D): 16 units below the rounding
  // boundary the lower neighbour is q, and q + 1 is nearer exactly when
  // m (2q + 1) < 2^106
  unsigned long long q = (y + 1024 - 16) >> 11;
  if (__umul64hi(m, 2 * q + 1) < (1ULL << 42)) ++q;
  return __longlong_as_double((long long)(((unsigned long long)(2045 - bexp) << 52) + (q - (1ULL << 52))));
}

// Cooperative unblocked LU of a sub-panel (PDGETF2, SRC/pdgetf2.f:206-237)
// over rows r0..m-1 and columns c0..c0+w-1 of A, w <= PW. CTA b owns rows
// r0 + b*rpc .. +rpc-1 in shared memory; rows are never moved: each has a
// label, the row of the sub-panel where its content stands after the
// interchanges so far (negative, ~k, once it is pivot row k), and goes back to
// that row of A at the end. PTR row threads update the rows: tpr of them, lanes
// of one warp, share a row (4, 2 or 1, so that a CTA's rows keep four warps
// busy: the FP64 unit is one per SM, takes a warp instruction every 20 cycles
// whatever lanes are active, and has one of a warp's in flight at a time, for 64
// cycles), the first of them owns it. One more warp runs the exchange. Per
// column k:
//   1. barrier; every warp reduces the row warps' IDAMAX candidates (first max
//      by label, NaN never wins unless it stands in the diagonal row --
//      PBLAS/SRC/pdamax_.c:414-486 through idamax_). The exchange warp
//      publishes the CTA's key and label as tagged words; the row warp that
//      holds the candidate publishes that row with column k-1's update applied
//      (a lane per column), and then all row warps apply that update to their
//      rows while the exchange is under way;
//   2. the exchange warp polls all CTAs' keys (lane q reads CTAs q, q+32, ..,
//      PKP in flight) until the tags match, reduces them to the winner
//      (largest |x|, lowest label on ties), reads the winner's row -- U(k, :),
//      the diagonal row's swap being a change of label -- and forms 1/|pivot|
//      from the key while that row is on its way;
//   3. barrier; the row threads scale column k by the reciprocal of the pivot
//      and update column k+1 (PDSWAP/PDSCAL/PDGER, pdgetf2.f:218-233), which
//      gives the next column's IDAMAX keys.
// Every element receives the updates of columns 0, 1, ... in order, as one
// fma each.
//
// Bound: the L2 round trips of a column's exchange (publish and poll the keys,
// about 950 cycles between two CTAs, 1900 over 64 CTAs on both dies; read the
// winner's row, 600), two barriers, and a chain of dependent FP64 and warp
// reductions (about 1200); the rest of the rank-1 update hides behind them up to
// about 256 rows per SM. Keys are pushed to each reader's own lines: 64 CTAs
// polling the same 64 sectors cost 1200 cycles more. Measured, per column: 2.4
// us over 32 CTAs (R = 4096), 2.6 over 64 (R = 8192), 2.2 with two; 3.74 with
// shuffle reductions, rows swapped in place, the diagonal row published too and
// the reciprocal divided on the FP64 pipe. PDGESV N = 4096 28.0 -> 22.3 ms.
//
// Column k's words carry tag tag0 + k, where tag0 differs from launch to
// launch, so nothing is cleared between launches. A word of parity k&1 is
// rewritten only at column k+2, after every CTA has read column k+1 -- which
// it can only do after finishing column k -- so two parities suffice. Every
// poll is bounded (at most spin_limit polls); a CTA that gives up records
// kFlagTimeout and returns, and block 0 then writes the identity for the
// pivots it has not chosen, so the interchanges launched after it stay inside
// the matrix.
//
// GTILE: for panels taller than the CTAs' shared memory holds (more than 768
// FP64 rows per CTA on every SM), each CTA's rows live in a global buffer
// instead (gtile, column-major per CTA: rpc rows x PW columns, so a warp's
// row walk is one coalesced access; the labels follow all rows); the algorithm
// is unchanged.
//
// ONE: a row thread has at most one row (rpc * tpr <= PTR), whose label stays in a
// register (its loops cost 400 cycles of a column's 4600).
template <typename T, bool GTILE = false, bool ONE = false>
__global__ void __launch_bounds__(PT, GTILE ? 1 : 3)
panel_kernel(T* A, long long lda, int m, int r0, int c0, int w, int rpc, int* ipiv,
             int* info_col, double* cand, int* status, long long spin_limit, T* gtile,
             uint32_t tag0, int tpr) {
  extern __shared__ __align__(16) unsigned char panel_smem[];
  // element (r, c) of this CTA's rows: [rpc][PLD] in shared memory, or
  // column-major rpc x PW in the global buffer
  T* tile = GTILE ? gtile + (size_t)blockIdx.x * (size_t)rpc * PW : reinterpret_cast<T*>(panel_smem);
  int* lab = GTILE ? reinterpret_cast<int*>(gtile + (size_t)gridDim.x * (size_t)rpc * PW) + (size_t)blockIdx.x * rpc
                   : reinterpret_cast<int*>(reinterpret_cast<T*>(panel_smem) + (size_t)rpc * PLD);
  auto tix = [&](int r, int c) -> size_t {
    return GTILE ? (size_t)c * (size_t)rpc + (size_t)r : (size_t)r * PLD + (size_t)c;
  };
  constexpr int NW = PTR / 32;  // row warps
  __shared__ T s_U[2][PW];      // U(k, :) by column parity
  __shared__ long long s_wk[NW];  // row warps' candidates: key, label, local row
  __shared__ int s_wr[NW], s_wl[NW];
  __shared__ int s_piv, s_own, s_fail;
  __shared__ T s_rinv;

  const int G = gridDim.x, b = blockIdx.x, tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  const bool exch = warp == NW;
  const int R = m - r0;
  const int kw = min(w, R);
  const int lo = b * rpc;                   // first local row (relative to r0)
  const int nr = max(0, min(rpc, R - lo));  // rows owned
  unsigned long long* words = reinterpret_cast<unsigned long long*>(cand);
  unsigned long long* keyw = words + PX_KEYS;
  unsigned long long* valw = words + PX_VALS;
  // block 0 on a timeout at column k: pivots k.. become the diagonal rows
  auto give_up = [&](int k) {
    if (b == 0)
      for (int q = k + tid; q < kw; q += PT) ipiv[c0 + q] = r0 + q;
  };
  // a row's IDAMAX key for column k: a NaN in the diagonal row stays (IDAMAX
  // keeps the first element when it is NaN), elsewhere it never wins
  auto row_key = [&](T v, int label, int k) -> long long {
    const long long key = amax_ikey(v);
    return (key < 0 && label == k) ? LLONG_MAX : key;
  };
  auto put_candidate = [&](long long key, int label, int lrow) {
    if (lane == warp_best(key, label)) {
      s_wk[warp] = key;
      s_wr[warp] = label;
      s_wl[warp] = lrow;
    }
  };
  // row thread tid: part `part` of rows row0, row0 + rstep, ...
  const int part = tid & (tpr - 1), row0 = exch ? nr : tid / tpr, rstep = PTR / tpr;
  int mylab = row0 < nr ? lo + row0 : -1;  // ONE: the label of row row0

  if (!exch) {
    // Sub-panel rows into shared memory, PCH columns' loads in flight at
    // once, and the row warps' IDAMAX candidates of column 0; those of column
    // k+1 come out of column k's rank-1 update.
    long long key = -2;
    int label = INT_MAX, lrow = 0;
    for (int r = tid; r < nr; r += PTR) {
      const T* src = A + (long long)(r0 + lo + r) + (long long)c0 * lda;
#pragma unroll
      for (int cb = 0; cb < PW; cb += PCH) {
        T v[PCH];
#pragma unroll
        for (int c = 0; c < PCH; ++c) v[c] = (cb + c < w) ? src[(long long)(cb + c) * lda] : (T)0;
#pragma unroll
        for (int c = 0; c < PCH; ++c)
          if (cb + c < w) tile[tix(r, cb + c)] = v[c];
      }
      lab[r] = lo + r;
    }
    asm volatile("bar.sync 1, %0;" ::"n"(PTR) : "memory");  // the rows' owners differ from their loaders
    if (part == 0)
      for (int r = row0; r < nr; r += rstep) {
        const long long k2 = row_key(tile[tix(r, 0)], lo + r, 0);
        if (k2 > key) { key = k2; label = lo + r; lrow = r; }
      }
    put_candidate(key, label, lrow);
  }
  if (tid == 0) s_fail = 0;

  // columns kp+2 .. w-1 of the active rows, column by column in turn among a
  // row's threads; the next column's operands are read while one is updated
  auto finish_update = [&](int kp) {
    const T* U = s_U[kp & 1];
    for (int r = row0; r < nr; r += ONE ? nr : rstep) {
      if ((ONE ? mylab : lab[r]) < 0) continue;
      const T l = tile[tix(r, kp)];
      int j = kp + 2 + part;
      if (j >= w) continue;
      T v = tile[tix(r, j)], u = U[j];
#pragma unroll 2
      for (; j + tpr < w; j += tpr) {
        const T vn = tile[tix(r, j + tpr)], un = U[j + tpr];
        tile[tix(r, j)] = fma(-l, u, v);
        v = vn;
        u = un;
      }
      tile[tix(r, j)] = fma(-l, u, v);
    }
  };

  for (int k = 0; k < kw; ++k) {
    const int par = k & 1;
    const uint32_t tag = tag0 + (uint32_t)k;
    __syncthreads();
    // --- this CTA's candidate ---
    long long key = lane < NW ? s_wk[lane] : -3;
    int label = lane < NW ? s_wr[lane] : INT_MAX;
    const int cw = warp_best(key, label);  // row warp that holds it
    const int lrow = s_wl[cw];
    if (!exch) {
      if (warp == cw && s_wr[cw] != INT_MAX) {
        // the candidate row, its columns beyond k with column k-1's update
        const T l = k > 0 ? tile[tix(lrow, k - 1)] : (T)0;
        for (int c = lane; c < w; c += 32) {
          T v = tile[tix(lrow, c)];
          if (k > 0 && c > k) v = fma(-l, s_U[par ^ 1][c], v);
          st_value<T>(valw + ((size_t)b * 2 + par) * 2 * PW, c, v, tag);
        }
        __syncwarp();
      }
      if (k > 0) finish_update(k - 1);
    } else {
      key = __shfl_sync(0xffffffffu, key, cw);
      label = __shfl_sync(0xffffffffu, label, cw);
      for (int q = lane; q < G; q += 32)
        st_key(keyw + (((size_t)par * PMAXG + q) * PMAXG + b) * 2, key, label, tag);
      // --- poll every CTA's key; the polls spin without sleeping (a sleep
      //     costs more than it saves here), bounded by spin_limit ---
      bool fail = false;
      key = -3;
      label = INT_MAX;
      int own = 0;  // CTA of this lane's best key
      const unsigned long long* kq = keyw + ((size_t)par * PMAXG + b) * PMAXG * 2;
      for (int q0 = lane; q0 < G; q0 += 32 * PKP) {
        for (long long spins = 0;; ++spins) {
          unsigned long long kk[PKP], hi[PKP];
          bool all = true;
#pragma unroll
          for (int i = 0; i < PKP; ++i)
            if (q0 + 32 * i < G) ld_key(kq + 2 * (q0 + 32 * i), kk[i], hi[i]);
#pragma unroll
          for (int i = 0; i < PKP; ++i)
            if (q0 + 32 * i < G) all = all && tag_ok(hi[i], tag);
          if (spins >= spin_limit) { fail = true; break; }
          if (!all) continue;
#pragma unroll
          for (int i = 0; i < PKP; ++i)
            if (q0 + 32 * i < G) {
              const long long k2 = (long long)kk[i];
              const int l2 = (int)payload(hi[i]);
              if (k2 > key || (k2 == key && l2 < label)) { key = k2; label = l2; own = q0 + 32 * i; }
            }
          break;
        }
        if (fail) break;
      }
      fail = __any_sync(0xffffffffu, fail);
      const int wl = warp_best(key, label);
      key = __shfl_sync(0xffffffffu, key, wl);
      label = __shfl_sync(0xffffffffu, label, wl);
      own = __shfl_sync(0xffffffffu, own, wl);
      // --- the winner's row: U(k, :), and 1/|pivot| meanwhile ---
      T v = (T)0, ra = (T)0;
      if (!fail) {
        const unsigned long long* vq = valw + ((size_t)own * 2 + par) * 2 * PW;
        if constexpr (sizeof(T) == 8) {
          // first look at the row, the reciprocal while it is in flight
          unsigned long long a0 = 0, a1 = 0;
          if (lane < w) ld_tagged2(vq + 2 * lane, a0, a1);
          const unsigned long long kb = (unsigned long long)key;
          if (kb - 1ULL < 0x7FEFFFFFFFFFFFFFULL) ra = recip_bits(kb);
          asm volatile("" ::"d"(ra));  // (here, not after the row's arrival)
          if (tag_ok(a0, tag) && tag_ok(a1, tag)) v = __longlong_as_double((long long)join(a0, a1));
          else if (lane < w && !ld_value<T>(vq, lane, tag, v, spin_limit)) fail = true;
        } else {
          if (lane < w && !ld_value<T>(vq, lane, tag, v, spin_limit)) fail = true;
        }
      }
      fail = __any_sync(0xffffffffu, fail);
      if (fail) {
        if (lane == 0) {
          atomicExch(status, (int)kFlagTimeout);
          s_fail = 1;
        }
      } else {
        if (lane < w) s_U[par][lane] = v;
        if (lane == k) {  // ONE/GMAX (pdgetf2.f:224)
          // (its zero test and sign on the integer pipe, see recip_bits)
          T rinv;
          bool zero;
          if constexpr (sizeof(T) == 8) {
            const unsigned long long kb = (unsigned long long)key, vb = (unsigned long long)__double_as_longlong(v);
            zero = (vb << 1) == 0;
            if (kb - 1ULL < 0x7FEFFFFFFFFFFFFFULL)
              rinv = __longlong_as_double(__double_as_longlong(ra) | (long long)(vb & (1ULL << 63)));
            else
              rinv = zero ? (T)1 : (T)1 / v;
          } else {
            zero = v == (T)0;
            rinv = zero ? (T)1 : (T)1 / v;
          }
          s_rinv = rinv;
          s_piv = label;
          s_own = own;
          if (b == 0) {
            ipiv[c0 + k] = r0 + label;
            if (zero) atomicMin(info_col, c0 + k);
          }
        }
      }
    }
    __syncthreads();
    if (s_fail) { give_up(k); return; }
    // --- labels (PDSWAP), scale (PDSCAL) and the first column of the rank-1
    //     update (PDGER); the row's next-column entry gives its IDAMAX key for
    //     column k+1 ---
    if (!exch) {
      const T rinv = s_rinv;  // 1 for a zero pivot: its column is not scaled
      const int piv = s_piv, mine = s_own == b ? lrow : -1;
      const int kn = k + 1;
      const T un = s_U[par][kn < w ? kn : k];
      if constexpr (ONE) {
        const int r = min(row0, rpc - 1);
        T l = tile[tix(r, k)];
        const T a = tile[tix(r, kn < w ? kn : k)];
        l *= rinv;
        const T v = fma(-l, un, a);
        const bool act = mylab >= 0 && row0 != mine && part == 0;
        if (mylab == k) mylab = piv;   // the diagonal row goes where the pivot row stood
        if (row0 == mine) mylab = ~k;  // pivot row k
        if (act) {
          tile[tix(r, k)] = l;
          if (kn < w) tile[tix(r, kn)] = v;
        }
        if (kn < kw)
          put_candidate(act ? row_key(v, mylab, kn) : -2LL, act ? mylab : INT_MAX, row0);
        continue;
      }
      long long nkey = -2;
      int nlab = INT_MAX, nrow = 0;
      for (int r = part == 0 ? row0 : nr; r < nr; r += rstep) {
        // straight-line: all of a row's operands at once, stores where it counts
        const int lb = lab[r];
        T l = tile[tix(r, k)];
        const T a = tile[tix(r, kn < w ? kn : k)];
        l *= rinv;
        const T v = fma(-l, un, a);
        const bool act = lb >= 0 && r != mine;
        const int ln = lb == k ? piv : lb;  // the diagonal row goes where the pivot row stood
        if (act) tile[tix(r, k)] = l;
        if (act && kn < w) tile[tix(r, kn)] = v;
        if (r == mine) lab[r] = ~k;  // pivot row k
        else if (lb == k) lab[r] = ln;
        const long long k2 = act ? row_key(v, ln, kn) : -2LL;
        if (k2 > nkey || (k2 == nkey && act && ln < nlab)) { nkey = k2; nlab = ln; nrow = r; }
      }
      if (kn < kw) put_candidate(nkey, nlab, nrow);
    }
  }
  // the last column's remaining update (columns beyond kw when the panel has
  // fewer rows than columns), then every row to where its content stands
  launch_dependents();
  if (exch) return;
  if (kw > 0) finish_update(kw - 1);
  if (ONE && part == 0 && row0 < nr) lab[row0] = mylab;
  asm volatile("bar.sync 1, %0;" ::"n"(PTR) : "memory");
  for (int r = tid; r < nr; r += PTR) {
    const int lb = lab[r];
    T* dst = A + (long long)(r0 + (lb < 0 ? ~lb : lb)) + (long long)c0 * lda;
#pragma unroll
    for (int cb = 0; cb < PW; cb += PCH) {
      T v[PCH];
#pragma unroll
      for (int c = 0; c < PCH; ++c) v[c] = (cb + c < w) ? tile[tix(r, cb + c)] : (T)0;
#pragma unroll
      for (int c = 0; c < PCH; ++c)
        if (cb + c < w) dst[(long long)(cb + c) * lda] = v[c];
    }
  }
}

// The same factorization by one thread-block cluster of up to CMAXG CTAs, for
// panels short enough that the cluster's FP64 units keep up (launch_panel): a
// CTA's candidate row, key and label go straight into every CTA's shared memory
// (st.async, counted by an mbarrier there), so that a column costs one
// shared-memory hop between SMs instead of two round trips through L2, and every
// warp then picks the winner by itself: one block barrier per column. Measured,
// per column, FP64: 1.4 us at R = 600 (2.3 through L2), 1.8 at R = 2048 (2.4; with
// 256 rows per CTA the FP64 units take as long, so launch_panel stops at 128);
// FP32, R = 4096: 1.4 (2.1). Three
// inboxes: column k's pivot row is read until column k+1 has been sent for, so a
// CTA may be sent column k+2's while it still reads column k's, but not k+3's.
// Waits are bounded (spin_limit polls). A warp that gives up at column k raises the
// column parity's flag, which is read only after the barrier of column k+1, when no
// warp can still write it: all of a CTA's warps stop at the same column. The CTAs
// may stop one column apart; each tells the others how many columns it has sent, and
// after the cluster barrier the ones behind send the missing column (its content is
// not used), so that every message has its count of bytes and can be waited for
// before shared memory goes.
constexpr int CMAXG = 16;
template <typename T>
struct PanelInbox {
  long long key;
  long long label;
  double rmag;  // 1/|pivot| (FP64)
  double pad;
  T row[PW];
};
template <typename T>
__host__ __device__ constexpr size_t panel_inbox_bytes() {
  return 3 * CMAXG * sizeof(PanelInbox<T>);
}
__device__ __forceinline__ uint32_t cluster_addr(uint32_t local, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// What all CTAs send one of them per column.
template <typename T>
__host__ __device__ constexpr uint32_t panel_column_bytes(int CS) {
  return (uint32_t)(CS * (16 + (sizeof(T) == 8 ? 8 : 0) + PW * sizeof(T)));
}

// After a give-up, by all threads of CTA b (sent: what panel_cluster_kernel keeps in
// s_sent, the same on every CTA): its first warp sends the column that others have
// begun and it has not, and the CTA waits for all that it was sent.
template <typename T>
__device__ __noinline__ void panel_cluster_finish(const int* sent, int CS, int b, uint32_t bar0, uint32_t in0) {
  const int lane = threadIdx.x & 31;
  int most = 0;
  for (int q = 0; q < CS; ++q) most = max(most, sent[q]);
  if (threadIdx.x < 32)
    for (int c = sent[b]; c < most; ++c) {
      const uint32_t bar = bar0 + 8 * (c % 3);
      const uint32_t slot = in0 + (uint32_t)((c % 3 * CMAXG + b) * sizeof(PanelInbox<T>));
      if (lane == 0)
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(panel_column_bytes<T>(CS))
                     : "memory");
      // (zeros, in pieces of 8 bytes: key and label, reciprocal, row)
      for (int q = 0; q < CS; ++q) {
        constexpr int kHead = sizeof(T) == 8 ? 3 : 2;
        for (int i = lane; i < kHead + (int)(PW * sizeof(T) / 8); i += 32)
          asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(
                           cluster_addr(slot + 8 * (i < kHead ? i : i - kHead + 4), q)),
                       "l"(0LL), "r"(cluster_addr(bar, q))
                       : "memory");
      }
    }
  __syncthreads();
  for (int c = max(0, most - 3); c < most; ++c)
    for (long long spins = 0; spins < kSpinLimit; ++spins) {
      uint32_t done;
      asm volatile(
          "{\n .reg .pred p;\n mbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
          " selp.u32 %0, 1, 0, p;\n}\n"
          : "=r"(done)
          : "r"(bar0 + 8 * (c % 3)), "r"((uint32_t)((c / 3) & 1))
          : "memory");
      if (done) break;
    }
}

// NTR row threads and the reciprocal's warp; a row thread has at most one row (rpc *
// tpr <= NTR), whose label stays in a register.
template <typename T, int NTR>
__global__ void __launch_bounds__(NTR + 32, 512 / NTR)
panel_cluster_kernel(T* A, long long lda, int m, int r0, int c0, int w, int rpc, int* ipiv, int* info_col,
                     int* status, long long spin_limit, int tpr) {
  extern __shared__ __align__(16) unsigned char panel_smem[];
  PanelInbox<T>* inbox = reinterpret_cast<PanelInbox<T>*>(panel_smem);  // [3][CMAXG]
  T* tile = reinterpret_cast<T*>(panel_smem + panel_inbox_bytes<T>());
  int* lab = reinterpret_cast<int*>(tile + (size_t)rpc * PLD);
  constexpr int NW = NTR / 32;
  __shared__ __align__(8) unsigned long long s_bar[3];
  __shared__ long long s_wk[2][NW];
  __shared__ int s_wr[2][NW], s_wl[2][NW];
  __shared__ int s_fail[2];       // a wait gave up, by column parity
  __shared__ int s_sent[CMAXG];   // columns each CTA has sent
  __shared__ int s_any;           // some CTA gave up

  const int CS = gridDim.x, b = blockIdx.x, tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  const bool exch = warp == NW;  // the warp that forms the reciprocal
  const int R = m - r0;
  const int kw = min(w, R);
  const int lo = b * rpc;
  const int nr = max(0, min(rpc, R - lo));
  const uint32_t bar0 = (uint32_t)__cvta_generic_to_shared(s_bar);
  const uint32_t in0 = (uint32_t)__cvta_generic_to_shared(inbox);
  if (tid < CMAXG) s_sent[tid] = kw;
  if (tid == 0) {
    s_fail[0] = s_fail[1] = s_any = 0;
    for (int i = 0; i < 3; ++i) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar0 + 8 * i));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  auto row_key = [&](T v, int label, int k) -> long long {
    const long long key = amax_ikey(v);
    return (key < 0 && label == k) ? LLONG_MAX : key;
  };
  auto put_candidate = [&](int buf, long long key, int label, int lrow) {
    if (lane == warp_best(key, label)) {
      s_wk[buf][warp] = key;
      s_wr[buf][warp] = label;
      s_wl[buf][warp] = lrow;
    }
  };
  const int part = tid & (tpr - 1), row0 = exch ? nr : tid / tpr;
  int mylab = row0 < nr ? lo + row0 : -1;  // the label of row row0
  wait_for_previous();
  if (!exch) {
    long long key = -2;
    int label = INT_MAX, lrow = 0;
    for (int r = tid; r < nr; r += NTR) {
      const T* src = A + (long long)(r0 + lo + r) + (long long)c0 * lda;
#pragma unroll
      for (int cb = 0; cb < PW; cb += PCH) {
        T v[PCH];
#pragma unroll
        for (int c = 0; c < PCH; ++c) v[c] = (cb + c < w) ? src[(long long)(cb + c) * lda] : (T)0;
#pragma unroll
        for (int c = 0; c < PCH; ++c) tile[r * PLD + cb + c] = v[c];
      }
    }
    asm volatile("bar.sync 1, %0;" ::"n"(NTR) : "memory");
    if (part == 0 && row0 < nr) {
      key = row_key(tile[row0 * PLD], lo + row0, 0);
      label = lo + row0;
      lrow = row0;
    }
    put_candidate(0, key, label, lrow);
  }
  cluster_sync();  // every CTA's barriers are there

  // columns kp+2 .. w-1 of the active rows, U = the pivot row of column kp
  auto finish_update = [&](int kp, const T* U) {
    if (row0 >= nr || mylab < 0) return;
    T* row = tile + row0 * PLD;
    const T l = row[kp];
    int j = kp + 2 + part;
    if (j >= w) return;
    T v = row[j], u = U[j];
#pragma unroll 2
    for (; j + tpr < w; j += tpr) {
      const T vn = row[j + tpr], un = U[j + tpr];
      row[j] = fma(-l, u, v);
      v = vn;
      u = un;
    }
    row[j] = fma(-l, u, v);
  };

  const T* Uprev = nullptr;  // pivot row of column k-1
  int k = 0;                 // columns sent
  for (; k < kw; ++k) {
    const int buf = k % 3, par = k & 1;
    __syncthreads();
    if (s_fail[par ^ 1]) break;
    // --- this CTA's candidate, into every CTA's inbox ---
    long long key = lane < NW ? s_wk[par][lane] : -3;
    int label = lane < NW ? s_wr[par][lane] : INT_MAX;
    const int cw = warp_best(key, label);
    const int lrow = s_wl[par][cw];
    if (tid == 0)
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar0 + 8 * buf),
                   "r"(panel_column_bytes<T>(CS))
                   : "memory");
    if (warp == cw) {
      // the candidate row with column k-1's update of its columns beyond k
      T v = (T)0;
      if (nr > 0 && lane < w) {
        v = tile[lrow * PLD + lane];
        if (k > 0 && lane > k) v = fma(-tile[lrow * PLD + k - 1], Uprev[lane], v);
      }
      const uint32_t slot = in0 + (uint32_t)((buf * CMAXG + b) * sizeof(PanelInbox<T>));
      const long long ck = s_wk[par][cw];
      const long long cl = s_wr[par][cw];
      if (lane < CS)
        asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(
                         cluster_addr(slot, lane)),
                     "l"(ck), "l"(cl), "r"(cluster_addr(bar0 + 8 * buf, lane))
                     : "memory");
      const uint32_t mine = slot + 32 + (uint32_t)(lane * sizeof(T));
      for (int q = 0; q < CS; ++q) {
        const uint32_t dst = cluster_addr(mine, q), bar = cluster_addr(bar0 + 8 * buf, q);
        if constexpr (sizeof(T) == 8)
          asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(dst),
                       "l"(__double_as_longlong(v)), "r"(bar)
                       : "memory");
        else
          asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(dst),
                       "r"(__float_as_uint(v)), "r"(bar)
                       : "memory");
      }
      __syncwarp();  // (the row is read before its owner goes on)
    }
    if (exch) {
      if constexpr (sizeof(T) == 8) {
        // 1/|candidate| on the integer pipe while the rows are updated: 450
        // cycles that every thread would otherwise wait for after the exchange
        const unsigned long long kb = (unsigned long long)s_wk[par][cw];
        const double ra = kb - 1ULL < 0x7FEFFFFFFFFFFFFFULL ? recip_bits(kb) : 0.0;
        const uint32_t slot = in0 + (uint32_t)((buf * CMAXG + b) * sizeof(PanelInbox<T>));
        if (lane < CS)
          asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(
                           cluster_addr(slot + 16, lane)),
                       "l"(__double_as_longlong(ra)), "r"(cluster_addr(bar0 + 8 * buf, lane))
                       : "memory");
      }
    } else if (k > 0) {
      finish_update(k - 1, Uprev);
    }
    // --- every CTA's candidate is here: the winner, U(k, :) and 1/pivot ---
    bool ok = false;
    for (long long spins = 0; spins < 8 * spin_limit; ++spins) {  // (a poll here takes an eighth of one in L2)
      uint32_t done;
      asm volatile(
          "{\n .reg .pred p;\n mbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
          " selp.u32 %0, 1, 0, p;\n}\n"
          : "=r"(done)
          : "r"(bar0 + 8 * buf), "r"((uint32_t)((k / 3) & 1))
          : "memory");
      if (done) { ok = true; break; }
    }
    ok = __all_sync(0xffffffffu, ok);
    if (!ok) {
      if (lane == 0) {
        atomicExch(status, (int)kFlagTimeout);
        s_fail[par] = 1;
      }
      continue;
    }
    const PanelInbox<T>* in = inbox + buf * CMAXG;
    key = lane < CS ? in[lane].key : -3;
    label = lane < CS ? (int)in[lane].label : INT_MAX;
    const int own = warp_best(key, label);
    key = in[own].key;
    label = (int)in[own].label;
    const T* U = in[own].row;
    const T g = U[k];
    T rinv;  // ONE/GMAX (pdgetf2.f:224), 1 for a zero pivot: its column is not scaled
    bool zero;
    if constexpr (sizeof(T) == 8) {
      const unsigned long long kb = (unsigned long long)key, gb = (unsigned long long)__double_as_longlong(g);
      zero = (gb << 1) == 0;
      if (kb - 1ULL < 0x7FEFFFFFFFFFFFFFULL)
        rinv = __longlong_as_double(__double_as_longlong(in[own].rmag) | (long long)(gb & (1ULL << 63)));
      else
        rinv = zero ? (T)1 : (T)1 / g;
    } else {
      zero = g == (T)0;
      rinv = zero ? (T)1 : (T)1 / g;
    }
    if (b == 0 && tid == 0) {
      ipiv[c0 + k] = r0 + label;
      if (zero) atomicMin(info_col, c0 + k);
    }
    const int piv = label, mine = own == b ? lrow : -1;
    const int kn = k + 1;
    const T un = U[kn < w ? kn : k];
    {
      T* row = tile + min(row0, rpc - 1) * PLD;
      T l = row[k];
      const T a = row[kn < w ? kn : k];
      l *= rinv;
      const T v = fma(-l, un, a);
      const bool act = mylab >= 0 && row0 != mine && part == 0;
      if (mylab == k) mylab = piv;   // the diagonal row goes where the pivot row stood
      if (row0 == mine) mylab = ~k;  // pivot row k
      if (act) {
        row[k] = l;
        if (kn < w) row[kn] = v;
      }
      if (kn < kw && !exch)
        put_candidate(par ^ 1, act ? row_key(v, mylab, kn) : -2LL, act ? mylab : INT_MAX, row0);
    }
    Uprev = U;
  }
  launch_dependents();
  __syncthreads();
  if (s_fail[0] | s_fail[1]) {
    // pivots from the first one that was not chosen become the diagonal rows
    if (b == 0)
      for (int q = max(k - 1, 0) + tid; q < kw; q += NTR + 32) ipiv[c0 + q] = r0 + q;
    if (tid < CS) {
      asm volatile("st.relaxed.cluster.shared::cluster.b32 [%0], %1;" ::"r"(
                       cluster_addr((uint32_t)__cvta_generic_to_shared(s_sent) + 4 * b, tid)),
                   "r"(k)
                   : "memory");
      asm volatile("st.relaxed.cluster.shared::cluster.b32 [%0], %1;" ::"r"(
                       cluster_addr((uint32_t)__cvta_generic_to_shared(&s_any), tid)),
                   "r"(1)
                   : "memory");
    }
  } else {
    if (kw > 0) finish_update(kw - 1, Uprev);
    if (part == 0 && row0 < nr) lab[row0] = mylab;
    __syncthreads();
    for (int r = exch ? nr : tid; r < nr; r += NTR) {
      const int lb = lab[r];
      T* dst = A + (long long)(r0 + (lb < 0 ? ~lb : lb)) + (long long)c0 * lda;
#pragma unroll
      for (int cb = 0; cb < PW; cb += PCH) {
        T v[PCH];
#pragma unroll
        for (int c = 0; c < PCH; ++c) v[c] = (cb + c < w) ? tile[r * PLD + cb + c] : (T)0;
#pragma unroll
        for (int c = 0; c < PCH; ++c)
          if (cb + c < w) dst[(long long)(cb + c) * lda] = v[c];
      }
    }
  }
  cluster_sync();
  if (!*(volatile int*)&s_any) return;  // every CTA has received all columns
  panel_cluster_finish<T>(s_sent, CS, b, bar0, in0);
  cluster_sync();
}

// Sequential row interchanges k1..k2-1 (rows i <-> ipiv[i]) on the columns
// [cb1,ce1) and [cb2,ce2); one thread per column (PDLASWP 'Forward','Rows').
// Used when the interchanges outnumber the composite form's table.
template <typename T>
__global__ void __launch_bounds__(256)
laswp_seq_kernel(T* A, long long lda, int k1, int k2, const int* __restrict__ ipiv, int cb1,
                 int ce1, int cb2, int ce2) {
  const int npiv = k2 - k1;
  const long long n1 = ce1 - cb1, n2 = ce2 - cb2;
  long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= n1 + n2) return;
  long long col = idx < n1 ? cb1 + idx : cb2 + (idx - n1);
  T* a = A + col * lda;
  for (int i = 0; i < npiv; ++i) {
    int p = ipiv[k1 + i];
    int r = k1 + i;
    if (p != r) {
      T t = a[r];
      a[r] = a[p];
      a[p] = t;
    }
  }
}

// The same interchanges applied as one composite permutation (PDLASWP
// 'Forward','Rows', SRC/pdlaswp.f:163-172): warp 0 of each CTA replays the
// swaps on row labels in shared memory -- entries for rows k1..k2-1 plus the
// pivot rows below them -- giving, for every touched row, the row whose
// original content ends up there. Then one warp per column loads all moved
// values at once and stores them, so a column costs one round trip instead of
// k2-k1 dependent ones. The result is bitwise that of the sequential swaps.
constexpr int LSW_MAXP = 256;
template <typename T>
__global__ void __launch_bounds__(256)
laswp_kernel(T* A, long long lda, int k1, int k2, const int* __restrict__ ipiv, int cb1, int ce1,
             int cb2, int ce2) {
  __shared__ int s_piv[LSW_MAXP];
  __shared__ int s_row[2 * LSW_MAXP];  // touched row of entry e
  __shared__ int s_src[2 * LSW_MAXP];  // row whose original content lands in s_row[e]
  __shared__ int s_cnt;
  const int npiv = k2 - k1;  // <= LSW_MAXP (checked by the launcher)
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < npiv; i += blockDim.x) {
    s_piv[i] = ipiv[k1 + i];
    s_row[i] = k1 + i;
    s_src[i] = k1 + i;
  }
  __syncthreads();
  if (warp == 0) {
    int cnt = npiv;
    for (int i = 0; i < npiv; ++i) {
      const int p = s_piv[i];
      if (p == k1 + i) continue;
      int e;
      if (p >= k1 && p < k2) {
        e = p - k1;
      } else {
        e = -1;
        for (int base = npiv; base < cnt && e < 0; base += 32) {
          const int q = base + lane;
          const unsigned hit = __ballot_sync(0xffffffffu, q < cnt && s_row[q] == p);
          if (hit) e = base + __ffs(hit) - 1;
        }
        if (e < 0) {
          e = cnt++;
          if (lane == 0) { s_row[e] = p; s_src[e] = p; }
        }
      }
      __syncwarp();
      if (lane == 0) {
        const int t = s_src[i];
        s_src[i] = s_src[e];
        s_src[e] = t;
      }
      __syncwarp();
    }
    if (lane == 0) s_cnt = cnt;
  }
  __syncthreads();
  const int cnt = s_cnt;
  const long long n1 = ce1 - cb1, ncols = n1 + (ce2 - cb2);
  constexpr int PER = 2 * LSW_MAXP / 32;
  for (long long ci = (long long)blockIdx.x * 8 + warp; ci < ncols; ci += (long long)gridDim.x * 8) {
    const long long col = ci < n1 ? cb1 + ci : cb2 + (ci - n1);
    T* a = A + col * lda;
    T v[PER];
#pragma unroll
    for (int q = 0; q < PER; ++q) {
      const int e = lane + 32 * q;
      v[q] = (e < cnt && s_src[e] != s_row[e]) ? a[s_src[e]] : (T)0;
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < PER; ++q) {
      const int e = lane + 32 * q;
      if (e < cnt && s_src[e] != s_row[e]) a[s_row[e]] = v[q];
    }
  }
}

// Plan of the interchanges k1..k2-1 (k2-k1 <= LSW_MAXP) in composite form:
// plan[0] = number of pairs, then (row, src) pairs for every touched row whose
// content changes (row receives the original content of src). The touched
// rows are k1..k2-1, then each row outside them in the order the interchanges
// first reach it; every thread walks the interchanges backwards for its rows
// (interchange i moves the content followed from ipiv[k1+i] to k1+i or the
// other way), so the cost is npiv shared-memory reads per row, in parallel.
// The pairs come out in the order of a sequential replay. Computed once per
// panel, on the panel's stream; laswp_apply_kernel then only moves data.
static __device__ __noinline__ void laswp_plan_block(int k1, int k2, const int* ipiv, int* plan) {
  __shared__ int s_piv[LSW_MAXP], s_row[2 * LSW_MAXP];
  const int npiv = k2 - k1, tid = threadIdx.x, nt = blockDim.x;
  for (int i = tid; i < npiv; i += nt) s_piv[i] = ipiv[k1 + i];
  // exclusive rank of this thread's flag among the block's (in thread order), and
  // the total: ballots and the warps' counts
  __shared__ int s_wc[32];
  auto rank = [&](bool f, int& total) {
    const unsigned m = __ballot_sync(0xffffffffu, f);
    __syncthreads();
    if ((tid & 31) == 0) s_wc[tid >> 5] = __popc(m);
    __syncthreads();
    int before = 0;
    total = 0;
    for (int w = 0; w < nt / 32; ++w) {
      if (w < tid / 32) before += s_wc[w];
      total += s_wc[w];
    }
    return before + __popc(m & ((1u << (tid & 31)) - 1u));
  };
  __syncthreads();
  // each outside row where an interchange reaches it for the first time
  int cnt = npiv, tot = 0;
  for (int i0 = 0; i0 < npiv; i0 += nt) {
    const int i = i0 + tid, p = i < npiv ? s_piv[i] : k1;
    bool first = p < k1 || p >= k2;
    for (int i2 = 0; i2 < min(i, npiv); ++i2)
      if (s_piv[i2] == p) first = false;
    const int q = rank(first, tot);
    if (i < npiv) s_row[i] = k1 + i;
    if (first) s_row[cnt + q] = p;
    cnt += tot;
  }
  __syncthreads();
  int np = 0;
  for (int e0 = 0; e0 < cnt; e0 += nt) {
    const int e = e0 + tid, row = e < cnt ? s_row[e] : -1;
    int q = row;
    if (e < cnt)
      for (int i = npiv - 1; i >= 0; --i) {
        const int p = s_piv[i];
        q = (q == k1 + i) ? p : ((q == p) ? k1 + i : q);
      }
    const bool moved = e < cnt && q != row;
    const int at = np + rank(moved, tot);
    if (moved) {
      plan[1 + 2 * at] = row;
      plan[2 + 2 * at] = q;
    }
    np += tot;
  }
  if (tid == 0) plan[0] = np;
}

static __global__ void laswp_plan_kernel(int k1, int k2, const int* __restrict__ ipiv, int* plan) {
  laswp_plan_block(k1, k2, ipiv, plan);
}

// Applies a plan of laswp_plan_kernel to the columns [cb1,ce1) and
// [cb2,ce2): one warp per column loads every moved value, then stores them.
template <typename T>
__global__ void __launch_bounds__(256)
laswp_apply_kernel(T* A, long long lda, const int* __restrict__ plan, int cb1, int ce1, int cb2,
                   int ce2) {
  __shared__ int s_row[2 * LSW_MAXP], s_src[2 * LSW_MAXP];
  const int np = plan[0];
  for (int e = threadIdx.x; e < np; e += blockDim.x) {
    s_row[e] = plan[1 + 2 * e];
    s_src[e] = plan[2 + 2 * e];
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long n1 = ce1 - cb1, ncols = n1 + (ce2 - cb2);
  constexpr int PER = 2 * LSW_MAXP / 32;
  for (long long ci = (long long)blockIdx.x * 8 + warp; ci < ncols; ci += (long long)gridDim.x * 8) {
    const long long col = ci < n1 ? cb1 + ci : cb2 + (ci - n1);
    T* a = A + col * lda;
    T v[PER];
#pragma unroll
    for (int q = 0; q < PER; ++q) {
      const int e = lane + 32 * q;
      v[q] = (e < np) ? a[s_src[e]] : (T)0;
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < PER; ++q) {
      const int e = lane + 32 * q;
      if (e < np) a[s_row[e]] = v[q];
    }
  }
}

// A sub-panel's in-panel step in one launch: its interchanges k1..k2-1 (at most
// 32) on the panel's other columns [cb1, ce1) and [cb2, ce2), then, on the first
// `nsolve` columns from cb2, the solve with the unit-lower kb x kb triangle T (kb
// = k2 - k1, or 32 more: the rows of the sub-panel before it in the same block
// come first, and the interchanges of T's and kj.L's columns are done beforehand) of
// rows k2-kb .. k2-1, and the balancing keys of the product that
// follows (kj: row maxima of the solution, and in extra CTAs column maxima of
// kj.L). A warp per column: the composed interchanges bring the pivot rows into
// the lane that solves for them (lane l owns rows l and l + 32 of the triangle),
// and x_q is passed by a shuffle. The interchanges are composed by walking them
// backwards for every touched row at once. Bound: the dependent steps (a shuffle
// and an FP64 instruction each, about 110 cycles); four columns per CTA, since
// four warps are what an SM's FP64 unit serves without queueing. One launch of
// about 11 us instead of two of 12 and 13.
constexpr int IPC = 4;  // columns (warps) per CTA
template <typename T>
__global__ void __launch_bounds__(32 * IPC)
inpanel_step_kernel(T* A, long long lda, int k1, int k2, const int* ipiv, int cb1, int ce1,
                    int cb2, int ce2, int nsolve, int kb, OzKeyJob kj) {
  __shared__ T Ls[64 * 64];  // T(i, q) at q*64 + i, rows below the diagonal
  __shared__ int s_piv[32], s_row[64], s_src[64];
  __shared__ unsigned s_h[64];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n1 = ce1 - cb1, ncols = n1 + (ce2 - cb2), ncta = (ncols + IPC - 1) / IPC;
  wait_for_previous();
  launch_dependents();
  if ((int)blockIdx.x >= ncta) {
    if constexpr (sizeof(T) == 8) {
      // column maxima of kj.L, 32 rows per CTA
      const double* row = kj.L + min(((int)blockIdx.x - ncta) * 32 + lane, kj.lrows - 1);
      double v[64 / IPC];
#pragma unroll
      for (int q = 0; q < 64 / IPC; ++q) v[q] = row[(long long)min(warp + IPC * q, kj.lcols - 1) * kj.ldl];
#pragma unroll
      for (int q = 0; q < 64 / IPC; ++q) {
        const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(oz_key_word(v[q], 0ULL) & 4095ULL));
        if (lane == 0 && hi && warp + IPC * q < kj.lcols)
          oz_raise_key(kj.ckeys + warp + IPC * q, (kj.epoch << 12) | hi);
      }
    }
    return;
  }
  const int npiv = k2 - k1, base = k2 - kb;  // base: first row of the triangle
  const int ci = blockIdx.x * IPC + warp;
  const bool in = ci < ncols;
  const int col = ci < n1 ? cb1 + ci : cb2 + (ci - n1);
  const bool solve = in && ci >= n1 && ci - n1 < nsolve;
  T* a = A + (long long)(in ? col : cb2) * lda;
  T x0 = (T)0, x1 = (T)0;
  if (solve && kb > npiv && lane < kb - npiv) x0 = a[base + lane];
  if (blockIdx.x * IPC + IPC > n1 && nsolve > 0) {  // some column of the CTA is solved
    const T* Tm = A + base + (long long)base * lda;
#pragma unroll 8
    for (int idx = tid; idx < kb * 64; idx += 32 * IPC) {
      const int i = idx & 63, q = idx >> 6;
      Ls[idx] = (i > q && i < kb) ? Tm[i + (long long)q * lda] : (T)0;
    }
  }
  if (tid < npiv) s_piv[tid] = ipiv[k1 + tid];
  if (tid < 64) s_h[tid] = 0u;
  __syncthreads();
  if (tid < 64) {
    // touched rows: k1.., then each pivot row outside them, once
    int row = -1;
    if (tid < 32) {
      if (tid < npiv) row = k1 + tid;
    } else if (tid - 32 < npiv) {
      const int p = s_piv[tid - 32];
      bool first = p < k1 || p >= k2;
      for (int i = 0; i < tid - 32; ++i) first = first && s_piv[i] != p;
      if (first) row = p;
    }
    int q = row;
    for (int i = npiv - 1; i >= 0; --i) {
      const int p = s_piv[i];
      q = (q == k1 + i) ? p : ((q == p) ? k1 + i : q);
    }
    s_row[tid] = row;
    s_src[tid] = q;
  }
  __syncthreads();
  if (in) {
    const int ra = s_row[lane], rb = s_row[lane + 32];
    const T va = ra >= 0 ? a[s_src[lane]] : (T)0, vb = rb >= 0 ? a[s_src[lane + 32]] : (T)0;
    __syncwarp();
    if (rb >= 0) a[rb] = vb;
    if (!solve) {
      if (ra >= 0) a[ra] = va;
    } else {
      if (kb > npiv) x1 = va;
      else x0 = va;
      for (int q = 0; q < min(kb, 32); ++q) {
        const T xq = __shfl_sync(0xffffffffu, x0, q);
        if (lane > q) x0 = fma(-Ls[q * 64 + lane], xq, x0);
        if (kb > 32) x1 = fma(-Ls[q * 64 + lane + 32], xq, x1);
      }
      for (int q = 32; q < kb; ++q) {
        const T xq = __shfl_sync(0xffffffffu, x1, q - 32);
        if (lane + 32 > q) x1 = fma(-Ls[q * 64 + lane + 32], xq, x1);
      }
      if (lane < kb) a[base + lane] = x0;
      if (lane + 32 < kb) a[base + lane + 32] = x1;
      if constexpr (sizeof(T) == 8) {
        if (kj.hkeys) {
          const unsigned h0 = (unsigned)(oz_key_word(x0, 0ULL) & 4095ULL), h1 = (unsigned)(oz_key_word(x1, 0ULL) & 4095ULL);
          if (lane < kb && h0) atomicMax(&s_h[lane], h0);
          if (lane + 32 < kb && h1) atomicMax(&s_h[lane + 32], h1);
        }
      }
    }
  }
  if (kj.hkeys) {
    __syncthreads();
    if (tid < kb && s_h[tid]) oz_raise_key(kj.hkeys + tid, (kj.epoch << 12) | s_h[tid]);
  }
}

// op(T) X = B for a w x w triangle (w <= 256) and a strip of NC columns of B
// per CTA, held in shared memory. FORWARD solves top-down (lower, or upper^T),
// otherwise bottom-up. The triangle is staged in shared memory eb (<= 32)
// columns at a time (all loads of a block in flight together), so the w
// dependent steps read only shared memory. Non-unit diagonals divide
// (reference DTRSM semantics).
constexpr int TRSM_EB = 32;
template <typename T, bool UPPER, bool TRANS, bool UNIT, int NC>
__global__ void __launch_bounds__(256)
trsm_strip_kernel(int w, int ncols, int eb, const T* __restrict__ Tm, long long ldt, T* B,
                  long long ldb, OzKeyJob kj) {
  constexpr bool FORWARD = (UPPER == TRANS);
  const int nsolve = (ncols + NC - 1) / NC;
  if ((int)blockIdx.x >= nsolve) {
    // extra blocks: column maxima of kj.L, 32 rows each (warp w: columns w,
    // w+8, ...; one coalesced load per column)
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const int i = ((int)blockIdx.x - nsolve) * 32 + lane;
    const double* row = kj.L + min(i, kj.lrows - 1);  // (a repeated row changes no maximum)
    for (int c0 = wp; c0 < kj.lcols; c0 += 64) {
      double v[8];  // eight columns' loads in flight
#pragma unroll
      for (int q = 0; q < 8; ++q) v[q] = row[(long long)min(c0 + 8 * q, kj.lcols - 1) * kj.ldl];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(oz_key_word(v[q], 0ULL) & 4095ULL));
        if (lane == 0 && hi && c0 + 8 * q < kj.lcols) oz_raise_key(kj.ckeys + c0 + 8 * q, (kj.epoch << 12) | hi);
      }
    }
    return;
  }
  constexpr int RG = 256 / NC;  // row groups
  extern __shared__ __align__(16) unsigned char strip_smem[];
  T* Bs = reinterpret_cast<T*>(strip_smem);  // [w][NC+1]
  const int LD = NC + 1;
  T* Es = Bs + (size_t)w * LD;                // [eb][w+1]: Es[ii*(w+1) + r] = op(T)(r, i(ii))
  const int LE = w + 1;
  const int tid = threadIdx.x;
  const int c = tid % NC, rg = tid / NC;
  const long long col0 = (long long)blockIdx.x * NC;
  const int nc = (int)min((long long)NC, ncols - col0);
  for (int i = tid; i < w * NC; i += 256) {
    int r = i % w, cc = i / w;
    Bs[r * LD + cc] = cc < nc ? B[r + (col0 + cc) * ldb] : (T)0;
  }
  for (int s0 = 0; s0 < w; s0 += eb) {
    const int nb = min(eb, w - s0);
    __syncthreads();  // the previous block's steps are done with Es
    for (int idx = tid; idx < nb * w; idx += 256) {
      int ii, r;
      if (!TRANS) { r = idx % w; ii = idx / w; }    // coalesced along r
      else { ii = idx % nb; r = idx / nb; }         // coalesced along i
      const int i = FORWARD ? s0 + ii : w - 1 - (s0 + ii);
      Es[ii * LE + r] = TRANS ? Tm[i + (long long)r * ldt] : Tm[r + (long long)i * ldt];
    }
    __syncthreads();
    for (int ii = 0; ii < nb; ++ii) {
      const int i = FORWARD ? s0 + ii : w - 1 - (s0 + ii);
      const T* Ei = Es + ii * LE;
      if (!UNIT) {
        if (tid < NC) Bs[i * LD + tid] = Bs[i * LD + tid] / Ei[i];
        __syncthreads();
      }
      const T xi = Bs[i * LD + c];
      if (FORWARD) {
        for (int r = i + 1 + rg; r < w; r += RG) Bs[r * LD + c] = fma(-Ei[r], xi, Bs[r * LD + c]);
      } else {
        for (int r = rg; r < i; r += RG) Bs[r * LD + c] = fma(-Ei[r], xi, Bs[r * LD + c]);
      }
      __syncthreads();
    }
  }
  for (int i = tid; i < w * NC; i += 256) {
    int r = i % w, cc = i / w;
    if (cc < nc) B[r + (col0 + cc) * ldb] = Bs[r * LD + cc];
  }
  // row maxima of this strip of the solution: the balancing keys of the
  // product that takes it as its right operand
  if constexpr (sizeof(T) == 8) {
    if (kj.hkeys != nullptr)
      for (int r = tid; r < w; r += 256) {
        unsigned long long km = 0ULL;
        for (int cc = 0; cc < nc; ++cc) {
          const unsigned long long v = oz_key_word(Bs[r * LD + cc], kj.epoch);
          km = v > km ? v : km;
        }
        if (km) oz_raise_key(kj.hkeys + r, km);
      }
  }
}

// L X = B in place for a unit-lower w x w triangle (w <= 256) and many columns: a
// warp takes TCC columns, lane l owning rows l, l + 32, .. of each in registers, and
// x_q passes by a shuffle; the triangle comes through shared memory 32 columns at a
// time, with a barrier per 32 steps instead of one per step. Elements take their
// updates in the order of the substitution, one fma each. Bound: the triangle's
// reads from shared memory. FP32, w = 256, 8192 columns: 30 us (trsm_strip_kernel,
// 145).
constexpr int TCC = 2;
template <typename T>
__global__ void __launch_bounds__(256)
trsm_cols_kernel(int w, int ncols, const T* __restrict__ L, long long ldl, T* B, long long ldb) {
  __shared__ T Es[32 * 256];  // L(r, s0 + i) at i*256 + r
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int col0 = ((int)blockIdx.x * 8 + warp) * TCC;
  T x[TCC][8];
#pragma unroll
  for (int c = 0; c < TCC; ++c)
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      const int r = lane + 32 * t;
      x[c][t] = (r < w && col0 + c < ncols) ? B[r + (long long)(col0 + c) * ldb] : (T)0;
    }
  // thread tid stages row tid: the next 32 columns are on their way (addresses
  // clamped into the triangle's square, no test before a load) while these are used
  const T* lrow = L + min(tid, w - 1);
  T e[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) e[i] = lrow[(long long)min(i, w - 1) * ldl];
#pragma unroll
  for (int tq = 0; tq < 8; ++tq) {
    const int s0 = 32 * tq;
    if (s0 >= w) break;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 32; ++i) Es[i * 256 + tid] = (tid < w && s0 + i < tid) ? e[i] : (T)0;
    __syncthreads();
    if (s0 + 32 < w) {
#pragma unroll
      for (int i = 0; i < 32; ++i) e[i] = lrow[(long long)min(s0 + 32 + i, w - 1) * ldl];
    }
#pragma unroll 4
    for (int i = 0; i < 32; ++i) {
      T xq[TCC];
#pragma unroll
      for (int c = 0; c < TCC; ++c) xq[c] = __shfl_sync(0xffffffffu, x[c][tq], i);
#pragma unroll
      for (int t = tq; t < 8; ++t) {
        const T l = Es[i * 256 + lane + 32 * t];
#pragma unroll
        for (int c = 0; c < TCC; ++c)
          if (t > tq || lane > i) x[c][t] = fma(-l, xq[c], x[c][t]);
      }
    }
  }
#pragma unroll
  for (int c = 0; c < TCC; ++c)
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      const int r = lane + 32 * t;
      if (r < w && col0 + c < ncols) B[r + (long long)(col0 + c) * ldb] = x[c][t];
    }
}

// op(T) x = b for a w x w diagonal block (w <= 128) and few right-hand sides:
// one CTA per right-hand side stages the block's triangle in shared memory
// (row stride w+1, conflict-free) with all its warps, then warp 0 solves the
// column with its 4 rows per lane held in registers;
// x_i is broadcast with a shuffle, so no block-wide barrier sits on the
// dependency chain. Non-unit diagonals divide (reference DTRSM semantics).
template <typename T, bool UPPER, bool TRANS, bool UNIT>
__global__ void __launch_bounds__(256)
trsv_warp_kernel(int w, int ncols, const T* __restrict__ Tm, long long ldt, T* B, long long ldb) {
  extern __shared__ __align__(16) unsigned char trsv_smem[];
  T* Ts = reinterpret_cast<T*>(trsv_smem);  // Ts[r*(w+1) + i] = op(T)(r, i)
  const int W1 = w + 1;
  constexpr bool FORWARD = (UPPER == TRANS);
  // stage only the triangle the solve reads (the diagonal too when non-unit),
  // many loads in flight per thread
#pragma unroll 8
  for (int idx = threadIdx.x; idx < w * w; idx += blockDim.x) {
    int r, i;
    if (!TRANS) { r = idx % w; i = idx / w; }  // coalesced along r
    else { i = idx % w; r = idx / w; }         // coalesced along i
    const bool need = FORWARD ? (r > i || (!UNIT && r == i)) : (r < i || (!UNIT && r == i));
    if (need) Ts[r * W1 + i] = TRANS ? Tm[i + (long long)r * ldt] : Tm[r + (long long)i * ldt];
  }
  __syncthreads();
  // one right-hand side per CTA, solved by warp 0: GB300's FP64 pipe is narrow
  // per SM, so the columns' solves are spread over as many SMs as there are
  // columns; the other warps only help staging
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long col = blockIdx.x;
  if (warp != 0 || col >= ncols) return;
  T x[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    int r = lane + 32 * q;
    x[q] = r < w ? B[r + col * ldb] : (T)0;
  }
  for (int s = 0; s < w; ++s) {
    const int i = FORWARD ? s : w - 1 - s;
    const int qi = i >> 5, li = i & 31;
    if (!UNIT && lane == li) {
      const T dinv = Ts[i * W1 + i];
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (q == qi) x[q] = x[q] / dinv;
    }
    T own = x[0];
#pragma unroll
    for (int q = 1; q < 4; ++q)
      if (q == qi) own = x[q];
    const T xi = __shfl_sync(0xffffffffu, own, li);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int r = lane + 32 * q;
      if (r < w && (FORWARD ? r > i : r < i)) x[q] = fma(-Ts[r * W1 + i], xi, x[q]);
    }
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    int r = lane + 32 * q;
    if (r < w) B[r + col * ldb] = x[q];
  }
}

// Single-launch blocked triangular solve for few right-hand sides (nrhs <=
// NRM), FP32: FORWARD solves with the unit-lower L, otherwise with the
// non-unit upper U, of an n x n LU factor, X (n x nrhs) overwritten in place.
//
// Each CTA takes the next 64-row block (in solve order) from an atomic
// ticket, so every block it depends on belongs to a CTA that has already
// started: the waits below always end (no residency assumption). Solved
// blocks are published as tagged words {x bits, epoch} in xt, so a consumer
// polls the values themselves (one round trip, no flag and no fence). A CTA
// stages the inverse of its diagonal block (precomputed once per factorization,
// diag_inv) and M_b = inv(T_bb) T_bp for its immediate predecessor p in
// shared memory, consumes the earlier solved blocks in chunks as they appear
// (4 thread groups of 64 rows x 16 columns apply the 64x64 blocks of the
// factor), forms y_b = inv(T_bb) v_b before the predecessor is solved, and
// when x_p arrives one 64x64 product from shared memory remains on the chain,
// x_b = y_b - M_b x_p (no serial substitution). Waits are bounded
// (kSpinLimit); on timeout the CTA records kFlagTimeout in *status and stops.
// TM: storage of the factor and of the diagonal-block inverses (FP32). TV:
// the arithmetic and the vectors: FP32, or FP64 for a preconditioner applied
// in the working precision (the FP32 factors and inverses then define the
// operator exactly and only FP64 rounding enters). An FP64 value travels as
// two tagged words (low and high halves).
template <typename TM, typename TV, bool FORWARD, int NRM>
__global__ void __launch_bounds__(256)
trsv_chain_kernel(const TM* __restrict__ A, long long lda, int n, TV* X, long long ldx, int nrhs,
                  const TM* __restrict__ Dinv, const TM* __restrict__ Mp, int* ticket,
                  unsigned long long* xt, int epoch, int* status) {
  static_assert(sizeof(TM) == 4, "FP32 factors");
  constexpr int VW = sizeof(TV) / 4;  // tagged words per value
  constexpr int KB = 64;
  constexpr int kChunk = NRM > 4 ? 1 : (NRM > 1 ? 4 : 8);  // static shared memory under 48 KB
  __shared__ TM Ds[KB][KB + 1];         // inverse of the diagonal block, Ds[r][i]
  __shared__ TM Ms[KB][KB + 1];         // M_b = inv(T_bb) T_bp, Ms[r][i]
  __shared__ TV xs[kChunk * KB][NRM];   // x of the blocks being applied
  __shared__ TV part[4][KB][NRM];       // partial sums of the 4 column groups
  __shared__ int s_b, s_fail, s_bad[kChunk];
  const uint32_t tag = (uint32_t)epoch;
  auto word = [&](int c, long long row) { return xt + ((size_t)c * n + row) * VW; };
  // reads one published value; false while its tag(s) are not the current one
  auto read_val = [&](const unsigned long long* p, TV& v) -> bool {
    if constexpr (VW == 1) {
      unsigned long long wd;
      asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(wd) : "l"(p) : "memory");
      v = __uint_as_float((uint32_t)wd);
      return (uint32_t)(wd >> 32) == tag;
    } else {
      unsigned long long lo, hi;
      asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(lo), "=l"(hi) : "l"(p) : "memory");
      v = __longlong_as_double((long long)(((unsigned long long)(uint32_t)hi << 32) | (uint32_t)lo));
      return (uint32_t)(lo >> 32) == tag && (uint32_t)(hi >> 32) == tag;
    }
  };
  auto publish = [&](unsigned long long* p, TV v) {
    if constexpr (VW == 1) {
      const unsigned long long wd = ((unsigned long long)tag << 32) | __float_as_uint(v);
      asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(wd) : "memory");
    } else {
      const unsigned long long bits = (unsigned long long)__double_as_longlong(v);
      const unsigned long long lo = ((unsigned long long)tag << 32) | (uint32_t)bits;
      const unsigned long long hi = ((unsigned long long)tag << 32) | (uint32_t)(bits >> 32);
      asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(lo), "l"(hi) : "memory");
    }
  };
  const int tid = threadIdx.x;
  const int nblk = (n + KB - 1) / KB;
  if (tid == 0) { s_b = atomicAdd(ticket, 1); s_fail = 0; }
  __syncthreads();
  const int sidx = s_b;
  if (sidx >= nblk) return;
  const int b = FORWARD ? sidx : nblk - 1 - sidx;
  const int r0 = b * KB, rb = min(KB, n - r0);
  const int kp = FORWARD ? b - 1 : b + 1;  // predecessor in solve order
  const int wp = (sidx > 0) ? min(KB, n - kp * KB) : 0;
  const TM* Db = Dinv + (size_t)b * KB * KB;  // row-major [KB][KB]
  const TM* Mb = Mp + (size_t)b * KB * KB;
  for (int idx = tid; idx < KB * KB; idx += 256) {
    Ds[idx / KB][idx % KB] = Db[idx];
    Ms[idx / KB][idx % KB] = (sidx > 0) ? Mb[idx] : (TM)0;
  }
  const int r = tid & (KB - 1), q = tid >> 6;
  const int warp = tid >> 5, lane = tid & 31;
  // the block's right-hand side, read now rather than on the chain (warp c
  // owns column c; only this CTA writes these rows)
  TV bx0 = (TV)0, bx1 = (TV)0;
  if (warp < nrhs) {
    if (lane < rb) bx0 = X[(r0 + lane) + (long long)warp * ldx];
    if (lane + 32 < rb) bx1 = X[(r0 + lane + 32) + (long long)warp * ldx];
  }
  TV acc[NRM];
#pragma unroll
  for (int c = 0; c < NRM; ++c) acc[c] = (TV)0;
  // Blocks 0 .. sidx-2 in solve order: chunks of the consecutive solved blocks
  // that are already published (at least the first one, waited for).
  int t = 0;
  long long spins = 0;
  while (t < sidx - 1) {
    const int want = min(kChunk, sidx - 1 - t);
    const int kfirst = FORWARD ? t : nblk - 1 - (t + want - 1);  // lowest block of the chunk
    const int k0 = kfirst * KB;
    const int kn = min(want * KB, n - k0);
    if (tid == 0) {
      // one thread watches the chunk's first block (its last value) before the
      // whole chunk is read, so waiting CTAs do not stream through L2
      const int kb0 = FORWARD ? t : nblk - 1 - t;
      const unsigned long long* p = word(0, kb0 * KB + min(KB, n - kb0 * KB) - 1);
      for (long long sp = 0;; ++sp) {
        TV v;
        if (read_val(p, v)) break;
        if (sp > kSpinLimit) { s_fail = 1; break; }
      }
    }
    if (tid < kChunk) s_bad[tid] = 0;
    __syncthreads();
    if (s_fail) {
      if (tid == 0) atomicExch(status, (int)kFlagTimeout);
      return;
    }
    for (int idx = tid; idx < kn * nrhs; idx += 256) {
      const int i = idx % kn, c = idx / kn;
      TV v;
      if (!read_val(word(c, k0 + i), v)) {
        const int blk = i / KB;                                  // chunk block, matrix order
        s_bad[FORWARD ? blk : want - 1 - blk] = 1;               // solve order
      }
      xs[i][c] = v;
    }
    __syncthreads();
    int av = 0;
    while (av < want && s_bad[av] == 0) ++av;
    if (av == 0) {  // the watched value arrived before the rest of its block
      if (++spins > kSpinLimit) {
        if (tid == 0) atomicExch(status, (int)kFlagTimeout);
        return;
      }
      __syncthreads();  // everyone has read s_bad before it is reset
      continue;
    }
    // columns of the av complete blocks, in matrix order
    const int c0 = FORWARD ? 0 : (want - av) * KB;
    const int c1 = FORWARD ? min(av * KB, kn) : kn;
    if (r < rb) {
      for (int g0 = c0 + q * 16; g0 < c1; g0 += 64) {
        const int g1 = min(g0 + 16, c1);
        for (int kk = g0; kk < g1; ++kk) {
          const TV a = (TV)A[(r0 + r) + (long long)(k0 + kk) * lda];
#pragma unroll
          for (int c = 0; c < NRM; ++c)
            if (c < nrhs) acc[c] = fma(a, xs[kk][c], acc[c]);
        }
      }
    }
    __syncthreads();
    t += av;
  }
#pragma unroll
  for (int c = 0; c < NRM; ++c) part[q][r][c] = acc[c];
  __syncthreads();
  // v = b - sum of the partials (warp c owns column c, lanes rows lane and
  // lane+32), then y = inv(T_bb) v by all four thread groups
  __shared__ TV vs[NRM][KB];
  if (warp < nrhs) {
    const int c = warp;
    TV v0 = (TV)0, v1 = (TV)0;
    if (lane < rb) v0 = bx0 - (part[0][lane][c] + part[1][lane][c] + part[2][lane][c] + part[3][lane][c]);
    if (lane + 32 < rb)
      v1 = bx1 - (part[0][lane + 32][c] + part[1][lane + 32][c] + part[2][lane + 32][c] + part[3][lane + 32][c]);
    vs[c][lane] = v0;
    vs[c][lane + 32] = v1;
  }
  __syncthreads();
  {
#pragma unroll
    for (int c = 0; c < NRM; ++c) acc[c] = (TV)0;
#pragma unroll
    for (int i = q * 16; i < q * 16 + 16; ++i) {
      const TV d = (TV)Ds[r][i];
#pragma unroll
      for (int c = 0; c < NRM; ++c)
        if (c < nrhs) acc[c] = fma(d, vs[c][i], acc[c]);
    }
#pragma unroll
    for (int c = 0; c < NRM; ++c) part[q][r][c] = acc[c];
  }
  __syncthreads();
  TV x0 = (TV)0, x1 = (TV)0;
  if (warp < nrhs) {
    const int c = warp;
    x0 = part[0][lane][c] + part[1][lane][c] + part[2][lane][c] + part[3][lane][c];
    x1 = part[0][lane + 32][c] + part[1][lane + 32][c] + part[2][lane + 32][c] + part[3][lane + 32][c];
  }
  // The predecessor: poll its x (the chain's one round trip), x -= M_b x_p.
  if (sidx > 0) {
    for (int idx = tid; idx < wp * nrhs; idx += 256) {
      const int i = idx % wp, c = idx / wp;
      const unsigned long long* p = word(c, kp * KB + i);
      TV v = (TV)0;
      for (long long sp = 0;; ++sp) {
        if (read_val(p, v)) break;
        if (sp > kSpinLimit) { s_fail = 1; break; }
      }
      xs[i][c] = v;
    }
    __syncthreads();  // also orders the reads of part above before the writes below
    if (s_fail) {
      if (tid == 0) atomicExch(status, (int)kFlagTimeout);
      return;
    }
#pragma unroll
    for (int c = 0; c < NRM; ++c) acc[c] = (TV)0;
#pragma unroll 4
    for (int kk = q * 16; kk < q * 16 + 16; ++kk) {
      if (kk < wp) {
        const TV m = (TV)Ms[r][kk];
#pragma unroll
        for (int c = 0; c < NRM; ++c)
          if (c < nrhs) acc[c] = fma(m, xs[kk][c], acc[c]);
      }
    }
#pragma unroll
    for (int c = 0; c < NRM; ++c) part[q][r][c] = acc[c];
    __syncthreads();
    if (warp < nrhs) {
      const int c = warp;
      x0 -= part[0][lane][c] + part[1][lane][c] + part[2][lane][c] + part[3][lane][c];
      x1 -= part[0][lane + 32][c] + part[1][lane + 32][c] + part[2][lane + 32][c] + part[3][lane + 32][c];
    }
  }
  // publish: tagged words for the consumers, plain values for the result
  if (warp < nrhs) {
    const int c = warp;
    if (lane < rb) {
      publish(word(c, r0 + lane), x0);
      X[(r0 + lane) + (long long)c * ldx] = x0;
    }
    if (lane + 32 < rb) {
      publish(word(c, r0 + lane + 32), x1);
      X[(r0 + lane + 32) + (long long)c * ldx] = x1;
    }
  }
}

// Launch the chained solve; `sync` holds 1 ticket int (64 bytes reserved)
// followed by the tagged words: n x nrhs values of 1 (FP32) or 2 (FP64) words
// (zeroed once; epoch must differ from every earlier one).
template <typename TM, typename TV, bool FORWARD>
inline cudaError_t trsv_chain(const TM* A, long long lda, int n, TV* X, long long ldx, int nrhs,
                              const TM* Dinv, const TM* Mp, int* sync, int epoch, int* status,
                              cudaStream_t s) {
  if (n <= 0 || nrhs <= 0) return cudaSuccess;
  const int nblk = (n + 63) / 64;
  SL_TRY(cudaMemsetAsync(sync, 0, sizeof(int), s));
  unsigned long long* xt = reinterpret_cast<unsigned long long*>(sync + 16);
  if (nrhs <= 1)
    trsv_chain_kernel<TM, TV, FORWARD, 1><<<nblk, 256, 0, s>>>(A, lda, n, X, ldx, nrhs, Dinv, Mp, sync, xt, epoch, status);
  else if constexpr (sizeof(TV) == 8)
    return cudaErrorInvalidValue;  // FP64 vectors: one right-hand side (GMRES)
  else if (nrhs <= 4)
    trsv_chain_kernel<TM, TV, FORWARD, 4><<<nblk, 256, 0, s>>>(A, lda, n, X, ldx, nrhs, Dinv, Mp, sync, xt, epoch, status);
  else
    trsv_chain_kernel<TM, TV, FORWARD, 8><<<nblk, 256, 0, s>>>(A, lda, n, X, ldx, nrhs, Dinv, Mp, sync, xt, epoch, status);
  count_launches(1);
  return cudaGetLastError();
}

// dst(i, c) = src(perm[i], c) (forward) or dst(perm[i], c) = src(i, c) (inverse).
template <typename TS, typename TD>
__global__ void permute_rows_kernel(const TS* __restrict__ src, long long lds, TD* dst,
                                    long long ldd, const int* __restrict__ perm, int n, int nrhs,
                                    int inverse) {
  long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)n * nrhs) return;
  int i = (int)(idx % n), c = (int)(idx / n);
  int p = perm[i];
  if (!inverse) dst[i + c * ldd] = (TD)src[p + c * lds];
  else dst[p + c * ldd] = (TD)src[i + c * lds];
}

// C (m x n) += alpha * op(A) (m x k) * B (k x n) for n <= NC <= 16 and any k:
// one thread per row of C, B staged in 64-row chunks through shared memory.
// Used for the narrow off-diagonal updates of the triangular solves and for
// residuals b - A x with a few right-hand sides.
template <typename T, bool TRANSA, int NC>
__global__ void __launch_bounds__(256)
gemm_skinny_kernel(int m, int n, int k, T alpha, const T* __restrict__ A, long long lda,
                   const T* __restrict__ B, long long ldb, T* C, long long ldc) {
  __shared__ T Bs[64][NC];
  const long long row = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  T acc[NC];
#pragma unroll
  for (int j = 0; j < NC; ++j) acc[j] = (T)0;
  for (int k0 = 0; k0 < k; k0 += 64) {
    const int kc = min(64, k - k0);
    __syncthreads();
    for (int c = threadIdx.x; c < 64 * NC; c += blockDim.x) {
      int kk = c % 64, nn = c / 64;
      Bs[kk][nn] = (kk < kc && nn < n) ? B[(k0 + kk) + (long long)nn * ldb] : (T)0;
    }
    __syncthreads();
    if (row < m) {
#pragma unroll 16
      for (int kk = 0; kk < kc; ++kk) {
        T a = TRANSA ? A[(k0 + kk) + row * lda] : A[row + (long long)(k0 + kk) * lda];
#pragma unroll
        for (int j = 0; j < NC; ++j) acc[j] = fma(a, Bs[kk][j], acc[j]);
      }
    }
  }
  if (row < m) {
#pragma unroll
    for (int j = 0; j < NC; ++j)
      if (j < n) C[row + (long long)j * ldc] += alpha * acc[j];
  }
}

// ------------------------------------------------------------ launch helpers

// Threads of the widest one-cluster panel (FP64 rows per CTA never pass PTR), and its
// rows per CTA at most.
template <typename T>
constexpr int kClusterThreads = sizeof(T) == 4 ? 2 * PTR : PTR;
template <typename T>
inline int panel_cluster_rows_of() { return sizeof(T) == 4 ? 512 : panel_cluster_rows(); }
template <typename T>
inline size_t panel_cluster_smem(int rpc) {
  return panel_inbox_bytes<T>() + (sizeof(T) * PLD + sizeof(int)) * (size_t)rpc;
}

// Prepares the one-cluster panel's kernels, once; whether the device gives a cluster of
// CMAXG of them room (a part of a GPU may not: the other form runs there).
template <typename T>
inline bool panel_cluster_fits() {
  static const bool fits = [] {
    const void* kerns[] = {(const void*)panel_cluster_kernel<T, PTR>,
                           (const void*)panel_cluster_kernel<T, kClusterThreads<T>>};
    for (const void* f : kerns)
      if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024) != cudaSuccess ||
          cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
        cudaGetLastError();
        return false;
      }
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute la[1];
    la[0].id = cudaLaunchAttributeClusterDimension;
    la[0].val.clusterDim.x = CMAXG;
    la[0].val.clusterDim.y = la[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(CMAXG);
    cfg.blockDim = dim3(kClusterThreads<T> + 32);
    cfg.dynamicSmemBytes = panel_cluster_smem<T>(panel_cluster_rows_of<T>());
    cfg.attrs = la;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kerns[1], &cfg) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    return n > 0;
  }();
  return fits;
}

template <typename T>
inline cudaError_t launch_panel(T* A, long long lda, int m, int r0, int c0, int w, int* ipiv,
                                const LuWork& ws, cudaStream_t s, bool after_kernel = false) {
  const int R = m - r0;
  // One cluster (16 CTAs at most, of 32 rows at least) while its rows stay
  // within what its SMs' FP64 units do in a column's time. (The tuning knobs of
  // the row slices and CTAs ask for the other form.)
  if (panel_min_rows() == 0 && panel_ctas() == 64 && R <= CMAXG * panel_cluster_rows_of<T>() && w > 0 &&
      panel_cluster_fits<T>()) {
    int cs = 1;
    while (cs < CMAXG && R > 32 * cs) cs *= 2;
    int crpc = ((R + cs - 1) / cs + 7) & ~7;
    const size_t csmem = panel_cluster_smem<T>(crpc);
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute la[2];
    la[0].id = cudaLaunchAttributeClusterDimension;
    la[0].val.clusterDim.x = cs;
    la[0].val.clusterDim.y = la[0].val.clusterDim.z = 1;
    la[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // (see launch_after)
    la[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = dim3(cs);
    const int ntr = crpc > PTR ? kClusterThreads<T> : PTR;
    cfg.blockDim = dim3(ntr + 32);
    cfg.dynamicSmemBytes = csmem;
    cfg.stream = s;
    cfg.attrs = la;
    cfg.numAttrs = after_kernel ? 2 : 1;
    int ctpr = crpc > PTR / 4 ? 1 : (crpc > PTR / 8 ? 2 : 4);
    count_launches(1);
    auto kern = ntr == PTR ? panel_cluster_kernel<T, PTR> : panel_cluster_kernel<T, kClusterThreads<T>>;
    return cudaLaunchKernelEx(&cfg, kern, A, lda, m, r0, c0, w, crpc, ipiv, ws.info_col, ws.status,
                              spin_limit(), ctpr);
  }
  // Rows per CTA: about 64 CTAs per panel, and at least the type's minimum
  // (FP32 256, FP64 128, or the tuning knob). Fewer CTAs make the per-column
  // exchange cheaper (fewer keys to poll, less cross-die skew); more rows per
  // CTA make the rank-1 update longer -- on GB300's FP64 pipe sooner than on
  // the FP32 one.
  // Tall panels beyond 64 CTAs' shared memory spread over every SM instead;
  // beyond every SM's shared memory the rows go to the global buffer ws.ptile.
  const int rpc_max = (int)((200 * 1024) / (sizeof(T) * PLD)) & ~7;
  const int ctas = std::min(panel_ctas(), PMAXG);
  int rpc = (R + ctas - 1) / ctas;
  const int lo_rows = panel_min_rows() > 0 ? panel_min_rows() : (sizeof(T) == 4 ? 256 : 128);
  if (rpc < lo_rows) rpc = lo_rows;
  if (rpc > rpc_max) rpc = (R + num_sms() - 1) / num_sms();
  rpc = (rpc + 7) & ~7;
  int G = (R + rpc - 1) / rpc;
  size_t smem = sizeof(T) * (size_t)rpc * PLD;  // and the labels
  const bool global_tile = smem > 200 * 1024 || G > PMAXG;
  smem += sizeof(int) * (size_t)rpc;
  T* gtile = nullptr;
  if (global_tile) {
    if constexpr (sizeof(T) != 8) {
      return cudaErrorInvalidValue;  // M beyond the FP32 panel limit
    } else {
      G = std::min(PMAXG, num_sms());
      rpc = ((R + G - 1) / G + 7) & ~7;
      G = (R + rpc - 1) / rpc;
      if (!ws.ptile || ws.ptile_len < (size_t)G * rpc * PW + ((size_t)G * rpc + 1) / 2)
        return cudaErrorInvalidValue;
      gtile = ws.ptile;
      smem = 0;
    }
  }
  if (!global_tile) {
    SL_TRY(smem_attr_once((const void*)panel_kernel<T, false, false>, 212 * 1024));
    SL_TRY(smem_attr_once((const void*)panel_kernel<T, false, true>, 212 * 1024));
  }
  // Tags of this launch's words: 64 per launch, never used before in this
  // area since it was cleared (when new and when the launch count wraps).
  // Without a launch count the words are cleared for every launch.
  constexpr unsigned kLaunches = 1u << 26;
  unsigned id = 1;
  if (!ws.cand_launches || *ws.cand_launches == 0 || *ws.cand_launches + 1 >= kLaunches) {
    SL_TRY(cudaMemsetAsync(ws.cand, 0, sizeof(unsigned long long) * (size_t)PX_WORDS, s));
    if (ws.cand_launches) *ws.cand_launches = 0;
  }
  if (ws.cand_launches) id = ++*ws.cand_launches;
  uint32_t tag0 = id * 64u;
  int tpr = global_tile || rpc > PTR / 4 ? 1 : (rpc > PTR / 8 ? 2 : 4);  // threads per row
  long long limit = spin_limit();
  void* args[] = {&A, &lda, &m, &r0, &c0, &w, (void*)&rpc, &ipiv, (void*)&ws.info_col,
                  (void*)&ws.cand, (void*)&ws.status, (void*)&limit, (void*)&gtile, (void*)&tag0, (void*)&tpr};
  count_launches(1);
  if (global_tile)
    return cudaLaunchCooperativeKernel((void*)panel_kernel<T, true>, dim3(G), dim3(PT), args, 0, s);
  void* kern = rpc * tpr <= PTR ? (void*)panel_kernel<T, false, true> : (void*)panel_kernel<T, false, false>;
  return cudaLaunchCooperativeKernel(kern, dim3(G), dim3(PT), args, smem, s);
}

template <typename T>
inline cudaError_t laswp(T* A, long long lda, int k1, int k2, const int* ipiv, int cb1, int ce1,
                         int cb2, int ce2, cudaStream_t s) {
  const long long ncols = (long long)(ce1 - cb1) + (ce2 - cb2);
  if (ncols <= 0 || k2 <= k1) return cudaSuccess;
  if (k2 - k1 > LSW_MAXP) {
    dim3 grid((unsigned)((ncols + 255) / 256));
    laswp_seq_kernel<T><<<grid, 256, 0, s>>>(A, lda, k1, k2, ipiv, cb1, ce1, cb2, ce2);
  } else {
    // one warp per column, at most 4 CTAs per SM's worth of CTAs
    const long long want = (ncols + 7) / 8;
    const long long cap = 4LL * num_sms();
    laswp_kernel<T><<<(unsigned)(want < cap ? want : cap), 256, 0, s>>>(A, lda, k1, k2, ipiv, cb1,
                                                                         ce1, cb2, ce2);
  }
  count_launches(1);
  return cudaGetLastError();
}

// The in-panel step of a sub-panel (kb <= 64, a multiple of 32 above k2 - k1), see
// inpanel_step_kernel.
template <typename T>
inline cudaError_t inpanel_step(T* A, long long lda, int k1, int k2, const int* ipiv, int cb1, int ce1,
                                int cb2, int ce2, int nsolve, int kb, cudaStream_t s,
                                const OzKeyJob& kj = OzKeyJob()) {
  const int ncols = (ce1 - cb1) + (ce2 - cb2);
  if (ncols <= 0 || k2 <= k1) return cudaSuccess;
  const int grid = (ncols + IPC - 1) / IPC + (kj.ckeys ? (kj.lrows + 31) / 32 : 0);
  count_launches(1);
  return launch_after(inpanel_step_kernel<T>, dim3(grid), 32 * IPC, 0, s, A, lda, k1, k2, ipiv, cb1, ce1, cb2, ce2,
                      nsolve, kb, kj);
}

// Plan of a panel's interchanges (k2 - k1 <= LSW_MAXP), see laswp_plan_kernel.
inline cudaError_t laswp_plan(int k1, int k2, const int* ipiv, int* plan, cudaStream_t s) {
  if (k2 - k1 > LSW_MAXP) return cudaErrorInvalidValue;
  if (k2 <= k1) return cudaMemsetAsync(plan, 0, sizeof(int), s);
  laswp_plan_kernel<<<1, 256, 0, s>>>(k1, k2, ipiv, plan);
  count_launches(1);
  return cudaGetLastError();
}

// Row interchanges from a plan when one is available, else as laswp().
template <typename T>
inline cudaError_t laswp_planned(T* A, long long lda, int k1, int k2, const int* ipiv,
                                 const int* plan, int cb1, int ce1, int cb2, int ce2,
                                 cudaStream_t s, int max_ctas = 0) {
  const long long ncols = (long long)(ce1 - cb1) + (ce2 - cb2);
  if (ncols <= 0 || k2 <= k1) return cudaSuccess;
  if (!plan || k2 - k1 > LSW_MAXP) return laswp<T>(A, lda, k1, k2, ipiv, cb1, ce1, cb2, ce2, s);
  const long long want = (ncols + 7) / 8;
  const long long cap = max_ctas > 0 ? (long long)max_ctas : 4LL * num_sms();
  laswp_apply_kernel<T><<<(unsigned)(want < cap ? want : cap), 256, 0, s>>>(A, lda, plan, cb1, ce1,
                                                                            cb2, ce2);
  count_launches(1);
  return cudaGetLastError();
}

// Unit-lower solve of many columns: trsm_cols_kernel up to 256 rows, else strips.
template <typename T, bool UPPER, bool TRANS, bool UNIT, int NC = 8>
inline cudaError_t trsm_strip(int w, int ncols, const T* Tm, long long ldt, T* B, long long ldb,
                              cudaStream_t s, const OzKeyJob& kj = OzKeyJob());
template <typename T>
inline cudaError_t trsm_cols(int w, int ncols, const T* L, long long ldl, T* B, long long ldb, cudaStream_t s) {
  if (w <= 0 || ncols <= 0) return cudaSuccess;
  if (w > 256) return trsm_strip<T, false, false, true>(w, ncols, L, ldl, B, ldb, s);
  trsm_cols_kernel<T><<<(ncols + 8 * TCC - 1) / (8 * TCC), 256, 0, s>>>(w, ncols, L, ldl, B, ldb);
  count_launches(1);
  return cudaGetLastError();
}

template <typename T, bool UPPER, bool TRANS, bool UNIT, int NC>
inline cudaError_t trsm_strip(int w, int ncols, const T* Tm, long long ldt, T* B, long long ldb,
                              cudaStream_t s, const OzKeyJob& kj) {
  if (w <= 0 || ncols <= 0) return cudaSuccess;
  // staged triangle columns per block: up to 32, within 200 KB of shared memory
  constexpr size_t kBudget = 200 * 1024;
  const size_t bbytes = sizeof(T) * (size_t)w * (NC + 1);
  const size_t ecol = sizeof(T) * (size_t)(w + 1);
  if (bbytes + ecol > kBudget) return cudaErrorInvalidValue;
  const int eb = (int)std::min<size_t>(TRSM_EB, (kBudget - bbytes) / ecol);
  const size_t smem = bbytes + (size_t)eb * ecol;
  auto kern = trsm_strip_kernel<T, UPPER, TRANS, UNIT, NC>;
  SL_TRY(smem_attr_once((const void*)kern, (int)kBudget));
  dim3 grid((ncols + NC - 1) / NC + (kj.ckeys ? (kj.lrows + 31) / 32 : 0));
  kern<<<grid, 256, smem, s>>>(w, ncols, eb, Tm, ldt, B, ldb, kj);
  count_launches(1);
  return cudaGetLastError();
}

// The same product with each row tile split across NC/4 column groups of 4
// (64 rows per CTA for NC = 16, 128 for NC = 8): 4x more CTAs than
// gemm_skinny_kernel, so that a product with few rows still fills every SM
// (the off-diagonal updates of a blocked triangular solve with 8-16 right-hand
// sides).
template <typename T, bool TRANSA, int NC>
__global__ void __launch_bounds__(256)
gemm_skinny_rt_kernel(int m, int n, int k, T alpha, const T* __restrict__ A, long long lda,
                      const T* __restrict__ B, long long ldb, T* C, long long ldc) {
  static_assert(NC % 4 == 0 && NC >= 8, "column groups of 4");
  constexpr int G = NC / 4;    // column groups
  constexpr int RT = 256 / G;  // rows per CTA
  __shared__ T Bs[64][NC];
  const int g = threadIdx.x / RT, rl = threadIdx.x % RT;
  const long long row = (long long)blockIdx.x * RT + rl;
  T acc[4] = {(T)0, (T)0, (T)0, (T)0};
  for (int k0 = 0; k0 < k; k0 += 64) {
    const int kc = min(64, k - k0);
    __syncthreads();
    for (int c = threadIdx.x; c < 64 * NC; c += blockDim.x) {
      int kk = c % 64, nn = c / 64;
      Bs[kk][nn] = (kk < kc && nn < n) ? B[(k0 + kk) + (long long)nn * ldb] : (T)0;
    }
    __syncthreads();
    if (row < m) {
#pragma unroll 16
      for (int kk = 0; kk < kc; ++kk) {
        const T a = TRANSA ? A[(k0 + kk) + row * lda] : A[row + (long long)(k0 + kk) * lda];
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[j] = fma(a, Bs[kk][g * 4 + j], acc[j]);
      }
    }
  }
  if (row < m) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = g * 4 + j;
      if (c < n) C[row + (long long)c * ldc] += alpha * acc[j];
    }
  }
}

template <typename T, bool TA, int NC>
inline cudaError_t launch_skinny(int m, int n, int k, T alpha, const T* A, long long lda,
                                 const T* B, long long ldb, T* C, long long ldc, cudaStream_t s) {
  dim3 grid((m + 255) / 256);
  gemm_skinny_kernel<T, TA, NC><<<grid, 256, 0, s>>>(m, n, k, alpha, A, lda, B, ldb, C, ldc);
  count_launches(1);
  return cudaGetLastError();
}

// Split-K form for long k (matrix-vector products of the refinement): CTA
// (bx, by) computes rows 256*bx.. of op(A)[:, kslice(by)] * B into its own
// partial slot; gemm_skinny_reduce adds the ksplit partials in a fixed order.
template <typename T, int NC>
__global__ void __launch_bounds__(256)
gemm_skinny_splitk_kernel(int m, int n, int k, int kslice, const T* __restrict__ A, long long lda,
                          const T* __restrict__ B, long long ldb, T* part) {
  __shared__ T Bs[64][NC];
  const long long row = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int kbeg = blockIdx.y * kslice, kend = min(k, kbeg + kslice);
  T acc[2][NC];
#pragma unroll
  for (int j = 0; j < NC; ++j) { acc[0][j] = (T)0; acc[1][j] = (T)0; }
  for (int k0 = kbeg; k0 < kend; k0 += 64) {
    const int kc = min(64, kend - k0);
    __syncthreads();
    for (int c = threadIdx.x; c < 64 * NC; c += blockDim.x) {
      int kk = c % 64, nn = c / 64;
      Bs[kk][nn] = (kk < kc && nn < n) ? B[(k0 + kk) + (long long)nn * ldb] : (T)0;
    }
    __syncthreads();
    if (row < m) {
      int kk = 0;
      for (; kk + 1 < kc; kk += 2) {  // two independent accumulator chains
        const T a0 = A[row + (long long)(k0 + kk) * lda];
        const T a1 = A[row + (long long)(k0 + kk + 1) * lda];
#pragma unroll
        for (int j = 0; j < NC; ++j) {
          acc[0][j] = fma(a0, Bs[kk][j], acc[0][j]);
          acc[1][j] = fma(a1, Bs[kk + 1][j], acc[1][j]);
        }
      }
      if (kk < kc) {
        const T a0 = A[row + (long long)(k0 + kk) * lda];
#pragma unroll
        for (int j = 0; j < NC; ++j) acc[0][j] = fma(a0, Bs[kk][j], acc[0][j]);
      }
    }
  }
  if (row < m) {
#pragma unroll
    for (int j = 0; j < NC; ++j)
      if (j < n) part[((long long)blockIdx.y * n + j) * m + row] = acc[0][j] + acc[1][j];
  }
}

template <typename T>
__global__ void gemm_skinny_reduce_kernel(int m, int n, int ksplit, T alpha, const T* part, T* C,
                                          long long ldc) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)m * n) return;
  const int row = (int)(idx % m), j = (int)(idx / m);
  T s = (T)0;
  for (int q = 0; q < ksplit; ++q) s += part[((long long)q * n + j) * m + row];
  C[row + (long long)j * ldc] += alpha * s;
}

// C += alpha * op(A) * B for n <= 16 columns.
template <typename T>
inline cudaError_t gemm_skinny(bool transa, int m, int n, int k, T alpha, const T* A,
                               long long lda, const T* B, long long ldb, T* C, long long ldc,
                               cudaStream_t s) {
  if (m <= 0 || n <= 0 || k <= 0) return cudaSuccess;
  if (!transa && n <= 4 && k >= 4096) {
    // long products: spread k over ksplit CTA columns so every SM works
    const int rb = (m + 255) / 256;
    int ksplit = (4 * num_sms() + rb - 1) / rb;
    if (ksplit > 32) ksplit = 32;
    if (ksplit > 1) {
      SplitKScratch& sc = splitk_scratch();
      const size_t need = sizeof(T) * (size_t)ksplit * n * m;
      if (sc.ptr && sc.bytes >= need) {
        const int kslice = ((k + ksplit - 1) / ksplit + 63) / 64 * 64;
        ksplit = (k + kslice - 1) / kslice;
        dim3 grid(rb, ksplit);
        T* part = reinterpret_cast<T*>(sc.ptr);
        if (n == 1) gemm_skinny_splitk_kernel<T, 1><<<grid, 256, 0, s>>>(m, n, k, kslice, A, lda, B, ldb, part);
        else gemm_skinny_splitk_kernel<T, 4><<<grid, 256, 0, s>>>(m, n, k, kslice, A, lda, B, ldb, part);
        const long long tot = (long long)m * n;
        gemm_skinny_reduce_kernel<T><<<(unsigned)((tot + 255) / 256), 256, 0, s>>>(m, n, ksplit, alpha, part, C, ldc);
        count_launches(2);
        return cudaGetLastError();
      }
    }
  }
  if (n > 4 && (m + 255) / 256 < 2 * num_sms()) {
    // few rows: split each row tile over column groups so that every SM works
    const int nc = n <= 8 ? 8 : 16;
    const int rt = 256 / (nc / 4);
    dim3 grid((unsigned)((m + rt - 1) / rt));
    if (nc == 8) {
      if (transa) gemm_skinny_rt_kernel<T, true, 8><<<grid, 256, 0, s>>>(m, n, k, alpha, A, lda, B, ldb, C, ldc);
      else gemm_skinny_rt_kernel<T, false, 8><<<grid, 256, 0, s>>>(m, n, k, alpha, A, lda, B, ldb, C, ldc);
    } else {
      if (transa) gemm_skinny_rt_kernel<T, true, 16><<<grid, 256, 0, s>>>(m, n, k, alpha, A, lda, B, ldb, C, ldc);
      else gemm_skinny_rt_kernel<T, false, 16><<<grid, 256, 0, s>>>(m, n, k, alpha, A, lda, B, ldb, C, ldc);
    }
    count_launches(1);
    return cudaGetLastError();
  }
#define SL_SK(NC)                                                                              \
  return transa ? launch_skinny<T, true, NC>(m, n, k, alpha, A, lda, B, ldb, C, ldc, s)        \
                : launch_skinny<T, false, NC>(m, n, k, alpha, A, lda, B, ldb, C, ldc, s)
  if (n == 1) { SL_SK(1); }
  if (n <= 2) { SL_SK(2); }
  if (n <= 4) { SL_SK(4); }
  if (n <= 8) { SL_SK(8); }
  SL_SK(16);
#undef SL_SK
}

template <typename TS, typename TD>
inline cudaError_t permute_rows(const TS* src, long long lds, TD* dst, long long ldd,
                                const int* perm, int n, int nrhs, int inverse, cudaStream_t s) {
  const long long total = (long long)n * nrhs;
  if (total <= 0) return cudaSuccess;
  permute_rows_kernel<TS, TD><<<(unsigned)((total + 255) / 256), 256, 0, s>>>(
      src, lds, dst, ldd, perm, n, nrhs, inverse);
  count_launches(1);
  return cudaGetLastError();
}

// C += alpha op(A) B for the off-diagonal blocks of the solves (defined per
// type: FP64 in lu_f64.cu with DMMA for wide B, FP32 in mixed.cu).
template <typename T>
cudaError_t gemm_update(bool transa, int m, int n, int k, T alpha, const T* A, long long lda,
                        const T* B, long long ldb, T* C, long long ldc, cudaStream_t s);
template <>
cudaError_t gemm_update<double>(bool, int, int, int, double, const double*, long long,
                                const double*, long long, double*, long long, cudaStream_t);
template <>
cudaError_t gemm_update<float>(bool, int, int, int, float, const float*, long long, const float*,
                               long long, float*, long long, cudaStream_t);

template <typename T, bool UPPER, bool TRANS, bool UNIT>
inline cudaError_t diag_solve(int kb, int nrhs, const T* Td, long long lda, T* X, long long ldx,
                              cudaStream_t s) {
  if (kb <= 128 && nrhs <= 16) {
    // Few right-hand sides: one warp per column, the block in shared memory.
    auto kern = trsv_warp_kernel<T, UPPER, TRANS, UNIT>;
    SL_TRY(smem_attr_once((const void*)kern, 140 * 1024));
    const size_t smem = sizeof(T) * (size_t)kb * (kb + 1);
    kern<<<nrhs, 256, smem, s>>>(kb, nrhs, Td, lda, X, ldx);
    count_launches(1);
    return cudaGetLastError();
  }
  return trsm_strip<T, UPPER, TRANS, UNIT, 8>(kb, nrhs, Td, lda, X, ldx, s);
}

// Blocked triangular solve op(T) X = X with the n x n LU factors in A:
// lower = unit-lower L, otherwise non-unit upper U; trans solves with T^T.
// Diagonal blocks (256 wide for large n, 64 otherwise) are solved in shared
// memory; off-diagonal blocks are applied with gemm_update.
template <typename T>
inline cudaError_t tri_solve(bool lower, bool trans, bool unit, int n, int nrhs, const T* A,
                             long long lda, T* X, long long ldx, cudaStream_t s) {
  const int KB = nrhs <= 16 ? 128 : (n >= 2048 ? 256 : 64);
  const bool forward = (lower != trans);
  const int nblk = (n + KB - 1) / KB;
  for (int bi = 0; bi < nblk; ++bi) {
    const int b = forward ? bi : nblk - 1 - bi;
    const int k0 = b * KB;
    const int kb = (n - k0) < KB ? (n - k0) : KB;
    const T* Td = A + k0 + (long long)k0 * lda;
    if (lower && !trans) SL_TRY((diag_solve<T, false, false, true>(kb, nrhs, Td, lda, X + k0, ldx, s)));
    else if (!lower && !trans) {
      if (unit) SL_TRY((diag_solve<T, true, false, true>(kb, nrhs, Td, lda, X + k0, ldx, s)));
      else SL_TRY((diag_solve<T, true, false, false>(kb, nrhs, Td, lda, X + k0, ldx, s)));
    } else if (!lower && trans) SL_TRY((diag_solve<T, true, true, false>(kb, nrhs, Td, lda, X + k0, ldx, s)));
    else SL_TRY((diag_solve<T, false, true, true>(kb, nrhs, Td, lda, X + k0, ldx, s)));
    if (forward) {
      const int rest = n - k0 - kb;
      if (rest > 0) {
        // X[k0+kb:] -= op(T)[k0+kb:, k0:k0+kb] * X[k0:k0+kb]
        const T* Aoff = trans ? A + k0 + (long long)(k0 + kb) * lda : A + (k0 + kb) + (long long)k0 * lda;
        SL_TRY(gemm_update<T>(trans, rest, nrhs, kb, (T)-1, Aoff, lda, X + k0, ldx, X + k0 + kb, ldx, s));
      }
    } else if (k0 > 0) {
      // X[0:k0] -= op(T)[0:k0, k0:k0+kb] * X[k0:k0+kb]
      const T* Aoff = trans ? A + k0 : A + (long long)k0 * lda;
      SL_TRY(gemm_update<T>(trans, k0, nrhs, kb, (T)-1, Aoff, lda, X + k0, ldx, X, ldx, s));
    }
  }
  return cudaSuccess;
}

}  // namespace sl
