// 32x32 tile operations of the dense root's LDL' (no pivoting), one tile at a time: the diagonal
// tile's factorisation, the off-diagonal tiles and the trailing products, in FP64, FP32 or
// double-float. Used by the one-CTA factor (denseLdlt) and the whole-GPU one (gridLdlt*).
//
// Two properties of GB300 shape them. An FP64 instruction holds its SM sub-partition's FP64 unit
// for 64 cycles whatever the number of active lanes (measured: 64.8 cycles per dependent FMA of
// one warp with 1 or 32 lanes, one to four independent chains; two warps of one sub-partition
// take twice as long), so FP64 work is counted in warp instructions per sub-partition; and one
// warp's dependent FP32 operation takes about 5 cycles, so double-float work is bound by chains
// of such operations unless it is spread over warps. Every entry keeps one order of operations
// however the work is spread, so results do not depend on the number of warps.
#pragma once

#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "cxg_df64.cuh"
#include "cxg_kernels.h"
#include "cxg_layout.h"

namespace cxg {

// Pivot statistics written by the factoring warps (shared memory, read after a barrier).
struct PivotStats {
  int nreg, zero, wrong;
  int next;  // queue of trailing tile products of the current tile column (denseLdlt)
  double minAbs;
};

template <typename T>
__device__ __forceinline__ T shflT(T v, int src) { return __shfl_sync(0xffffffffu, v, src); }
__device__ __forceinline__ df64 shflT(df64 v, int src) {
  return df64(__shfl_sync(0xffffffffu, v.hi, src), __shfl_sync(0xffffffffu, v.lo, src));
}
// c - a b in the tile arithmetic (one FMA for float/double, the fused double-float form)
template <typename T>
__device__ __forceinline__ T msubT(T c, T a, T b) { return c - a * b; }
__device__ __forceinline__ df64 msubT(df64 c, df64 a, df64 b) { return dfMad(c, -a, b); }
// Accumulation inside tile products: accT (no renormalisation for double-float), then accEnd.
template <typename T>
__device__ __forceinline__ T accT(T c, T a, T b) { return c + a * b; }
__device__ __forceinline__ df64 accT(df64 c, df64 a, df64 b) { return dfMadLoose(c, a, b); }
template <typename T>
__device__ __forceinline__ T accEnd(T c) { return c; }
__device__ __forceinline__ df64 accEnd(df64 c) { return dfNorm(c); }

// A row of 32 values held in registers (indices are compile-time after unrolling).
template <typename T>
struct Row32 {
  T v[32];
  __device__ __forceinline__ T get(int k) const { return v[k]; }
  __device__ __forceinline__ void set(int k, T x) { v[k] = x; }
};

// 1/d for a pivot. FP32: the IEEE reciprocal intrinsic. FP64 and double-float: Newton-Raphson
// iteration r <- r + r (1 - d r) from the FP32 reciprocal of the leading part (each step doubles
// the correct bits: 23 -> 46 -> full; two steps for FP64, one for double-float), falling back to
// a division when d is outside the float range or not finite.
__device__ __forceinline__ float recipT(float d) { return __frcp_rn(d); }
__device__ __forceinline__ double recipT(double d) {
  const float f = __double2float_rn(d);
  const float af = fabsf(f);
  if (!(af >= 1e-37f && af <= 1e37f)) return 1.0 / d;
  double r = (double)__frcp_rn(f);
  double e = fma(-d, r, 1.0);
  r = fma(r, e, r);
  e = fma(-d, r, 1.0);
  return fma(r, e, r);
}
static __device__ __noinline__ float2 dfRecipFar(float hi, float lo) {
  const df64 q = df64(1.0f, 0.0f) / df64(hi, lo);
  return make_float2(q.hi, q.lo);
}
__device__ __forceinline__ df64 recipT(df64 d) {
  const float af = fabsf(d.hi);
  if (!(af >= 1e-37f && af <= 1e37f)) {
    const float2 q = dfRecipFar(d.hi, d.lo);
    return df64(q.x, q.y);
  }
  // one step from the 23-bit seed gives ~46 bits, the double-float rounding level
  const df64 r(__frcp_rn(d.hi), 0.0f);
  const df64 one(1.0f, 0.0f);
  return r + r * (one - d * r);
}

// Barrier over the first `threads` threads of the block (a multiple of 32), on named barrier 1.
__device__ __forceinline__ void groupSync(int threads) {
  if (threads == 32) __syncwarp();
  else asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory");
}

// Pivot statistics of diagonal tile J's rows (one warp): exact zeros, wrong signs, smallest |D|.
// The tests read the sign, exponent and order of each |D| from its bits, since FP64 compares
// would each hold the FP64 unit for 64 cycles.
template <typename T>
__device__ __forceinline__ void tilePivotStats(const T* A, int J, int nr, int nx, bool regularized, PivotStats* ps) {
  const int r = threadIdx.x & 31, g = J * 32 + r;
  const bool real = g < nr;
  const long long bits = __double_as_longlong((double)A[r * kTileLd + r]);
  const long long mag = bits & 0x7fffffffffffffffll;
  const bool finite = (mag >> 52) != 0x7ff, nan = mag > 0x7ff0000000000000ll;
  const bool positive = mag != 0 && !nan && ((bits >= 0) == (g < nx));
  const unsigned zeroMask = __ballot_sync(0xffffffffu, real && mag == 0);
  const unsigned wrongMask = __ballot_sync(0xffffffffu, real && !positive);
  const unsigned badMask = __ballot_sync(0xffffffffu, real && !finite);
  long long m = real ? mag : 0x7ff0000000000000ll;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const long long o = __shfl_xor_sync(0xffffffffu, m, off);
    m = o < m ? o : m;
  }
  if (r == 0) {
    if (!regularized && zeroMask) ps->zero = 1;
    if (wrongMask) ps->wrong = 1;
    const long long old = __double_as_longlong(ps->minAbs);  // >= 0, or NaN (above every number)
    if (old > 0x7ff0000000000000ll || badMask) ps->minAbs = NAN;
    else if (m < old) ps->minAbs = __longlong_as_double(m);
  }
}

// Factors diagonal tile J in place (one warp), FP32 form. Global row of tile row r is J*32 + r.
// Lane r keeps row r of the tile in registers (entries right of the diagonal mirrored from the
// lower triangle) and the 32 elimination steps broadcast pivot column j by shuffles. The same
// steps applied to the identity (Gauss-Jordan) give row r of the inverse of the unit-lower
// factor, which is stored transposed in the upper half: Linv(r, c) at r*ld + c. Only the
// per-pivot regularisation test runs inside the loop, in the tile's own arithmetic.
template <typename T>
__device__ __noinline__ void tileFactorDiagRegs(T* A, int J, int nr, int nx, const DevSettings& st, PivotStats* ps, T* invD) {
  const int r = threadIdx.x & 31;
  const bool regularized = st.linear_solver == 2;
  const T epsT = (T)st.dynamic_reg_eps, deltaT = (T)st.dynamic_reg_delta;
  Row32<T> a, e;
#pragma unroll
  for (int col = 0; col < 32; ++col) {
    a.set(col, (col <= r) ? A[col * kTileLd + r] : A[r * kTileLd + col]);
    e.set(col, (col == r) ? (T)1 : (T)0);
  }
  int nreg = 0;
#pragma unroll
  for (int j = 0; j < 32; ++j) {
    T dj = shflT(a.get(j), j);
    if (regularized) {
      const int g = J * 32 + j;
      if (g < nr) {
        const T sg = (g < nx) ? (T)1 : (T)-1;
        if (dj * sg < epsT) {
          dj = dj + sg * deltaT;
          if (dj * sg < epsT) dj = sg * deltaT;
          ++nreg;
        }
      }
    }
    const T inv = recipT(dj);
    const T lj = a.get(j) * inv;
#pragma unroll
    for (int k = j + 1; k < 32; ++k) {
      const T akj = shflT(a.get(j), k);
      a.set(k, msubT(a.get(k), lj, akj));
    }
    // Gauss-Jordan on the identity: row j of the inverse is final at step j
#pragma unroll
    for (int c = 0; c <= j; ++c) {
      const T ejc = shflT(e.get(c), j);
      if (r > j) e.set(c, msubT(e.get(c), lj, ejc));
    }
    if (r > j) a.set(j, lj);
    if (r == j) {
      a.set(j, dj);
      invD[r] = inv;
    }
  }
  __syncwarp();
#pragma unroll
  for (int col = 0; col < 32; ++col) {
    if (col <= r) A[col * kTileLd + r] = a.get(col);
    if (col < r) A[r * kTileLd + col] = e.get(col);
  }
  __syncwarp();
  if (r == 0) ps->nreg += nreg;
  tilePivotStats(A, J, nr, nx, regularized, ps);
  __syncwarp();
}

// ---- diagonal tile, 8-byte arithmetic (FP64, double-float) --------------------------------------
// Blocked right-looking LDL' in 8-column blocks (entry (i, k) at k*ld + i) by a group of warps:
//  (1) leaf (warp 0): the 8x8 diagonal block, rows in registers of its 8 lanes, pivots by shuffle;
//  (2) panel (warp 0): every row below finishes its 8 entries of the block by substitution with the
//      leaf, keeps them unscaled in the upper half of the tile for (3) and scales them by the
//      pivot reciprocals;
//  (3) trailing (all warps): the entries below subtract the block's rank-8 product.
// The inverse of the unit-lower factor, stored transposed in the upper half (Linv(R, C) at R*ld + C
// for C < R), follows one block behind: while warp 0 factors leaf b, the other warps finish block
// row b-1 of the inverse and form the products of block row b, so that only the last block row's
// is left after the last leaf. One warp alone did all of it in sequence before: 50k cycles per
// tile in double-float, 43% of them pivots (the chain that is left now).

// The pivot rule (regularized: a pivot below eps with the expected sign is corrected). A function of its
// own, as dfRecipFar is: eight copies of the two were half of the leaf's code.
template <typename T>
__device__ __noinline__ void pivotRule(T& dj, int g, int nr, int nx, T epsT, T deltaT, int& nreg) {
  if (g >= nr) return;
  const T sg = (g < nx) ? (T)1 : (T)-1;
  if (dj * sg < epsT) {
    dj = dj + sg * deltaT;
    if (dj * sg < epsT) dj = sg * deltaT;
    ++nreg;
  }
}

// Leaf block b and its panel; one warp. Returns the number of regularised pivots.
template <typename T>
__device__ __forceinline__ int tileLeafPanel(T* A, int b, int J, int nr, int nx, bool regularized, T epsT, T deltaT,
                                             T* invD) {
  const int r = threadIdx.x & 31, c0 = 8 * b, li = r - c0;
  const bool leaf = li >= 0 && li < 8;
  int nreg = 0;
  T invMine = (T)0;  // 1 / D(r), kept by lane r
  T a[8];
#pragma unroll
  for (int t = 0; t < 8; ++t) {
    const int ct = c0 + t;
    const T v = A[(t <= li) ? ct * kTileLd + r : r * kTileLd + ct];
    a[t] = leaf ? v : (T)0;
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    T dj = shflT(a[j], c0 + j);
    if (regularized) pivotRule(dj, J * 32 + c0 + j, nr, nx, epsT, deltaT, nreg);
    const T inv = recipT(dj);
    if (li == j) invMine = inv;
    const T lj = a[j] * inv;
#pragma unroll
    for (int k = j + 1; k < 8; ++k) {
      const T akj = shflT(a[j], c0 + k);
      a[k] = msubT(a[k], lj, akj);
    }
    if (li > j) a[j] = lj;
    if (li == j) a[j] = dj;
  }
  if (leaf) {
    invD[r] = invMine;
#pragma unroll
    for (int t = 0; t < 8; ++t)
      if (t <= li) A[(c0 + t) * kTileLd + r] = a[t];
  }
  __syncwarp();
  if (c0 + 8 < 32) {
    const bool below = r >= c0 + 8;
    // rows not below: the leaf's last one, without use (their own entries are those that the other warps
    // write meanwhile, tileInverseSum)
    const int ru = below ? r : c0 + 7;
    T u[8];
#pragma unroll
    for (int t = 0; t < 8; ++t) u[t] = A[(c0 + t) * kTileLd + ru];
#pragma unroll
    for (int t = 0; t < 8; ++t) {
#pragma unroll
      for (int s2 = t + 1; s2 < 8; ++s2) u[s2] = msubT(u[s2], u[t], A[(c0 + t) * kTileLd + c0 + s2]);
    }
    if (below) {
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        A[(c0 + t) * kTileLd + r] = u[t] * invD[c0 + t];
        A[r * kTileLd + c0 + t] = u[t];
      }
    }
  }
  return nreg;
}

#ifndef CXG_UNROLLED_LEAF
// The double-float form of the batched kernels: rolled loops over the pivots, the row shifted down by
// one entry a step (entry 0 is the pivot column's), seven updates a step for the first four and three
// for the others. Alone it takes 13% longer than the unrolled form (4870 cycles a leaf, 4300), which the
// whole-GPU kernels have; but that is 50 KB of code, and a batch whose SMs run different code then
// spends 20% more on the factor. Entries shifted in from beyond the block are never used.
template <int kUpd>
__device__ __forceinline__ void dfLeafSteps(df64 (&a)[8], df64* A, int c0, int j0, int g0, int nr, int nx,
                                            bool regularized, df64 epsT, df64 deltaT, int& nreg, df64& invMine) {
  const int r = threadIdx.x & 31, li = r - c0;
#pragma unroll 1
  for (int j = j0; j < j0 + 4; ++j) {
    const df64 aj = a[0];
    df64 dj = shflT(aj, c0 + j);
    if (regularized) pivotRule(dj, g0 + j, nr, nx, epsT, deltaT, nreg);
    const df64 inv = recipT(dj);
    if (li == j) invMine = inv;
    const df64 lj = aj * inv;
#pragma unroll
    for (int k = 1; k <= kUpd; ++k) a[k - 1] = msubT(a[k], lj, shflT(aj, (c0 + j + k) & 31));
    if (li >= j && li < 8) A[(c0 + j) * kTileLd + r] = (li > j) ? lj : dj;
  }
}
template <int kUpd>
__device__ __forceinline__ void dfPanelSteps(df64 (&u)[8], df64* A, int c0, int t0, const df64* invD) {
  const int r = threadIdx.x & 31;
#pragma unroll 1
  for (int t = t0; t < t0 + 4; ++t) {
    const df64* Ac = A + (c0 + t) * kTileLd + c0;
    const df64 ut = u[0];
#pragma unroll
    for (int k = 1; k <= kUpd; ++k) u[k - 1] = msubT(u[k], ut, Ac[min(t + k, 7)]);
    if (r >= c0 + 8) {
      A[(c0 + t) * kTileLd + r] = ut * invD[c0 + t];
      A[r * kTileLd + c0 + t] = ut;
    }
  }
}
__device__ __forceinline__ int tileLeafPanel(df64* A, int b, int J, int nr, int nx, bool regularized, df64 epsT,
                                             df64 deltaT, df64* invD) {
  const int r = threadIdx.x & 31, c0 = 8 * b, li = r - c0;
  const bool leaf = li >= 0 && li < 8;
  int nreg = 0;
  df64 invMine(0.0f, 0.0f), a[8];
#pragma unroll
  for (int t = 0; t < 8; ++t) {
    const int ct = c0 + t;
    const df64 v = A[(t <= li) ? ct * kTileLd + r : r * kTileLd + ct];
    a[t] = leaf ? v : df64(0.0f, 0.0f);
  }
  __syncwarp();
  dfLeafSteps<7>(a, A, c0, 0, J * 32 + c0, nr, nx, regularized, epsT, deltaT, nreg, invMine);
  dfLeafSteps<3>(a, A, c0, 4, J * 32 + c0, nr, nx, regularized, epsT, deltaT, nreg, invMine);
  if (leaf) invD[r] = invMine;
  __syncwarp();
  if (c0 + 8 < 32) {
    const int ru = r >= c0 + 8 ? r : c0 + 7;  // as above
    df64 u[8];
#pragma unroll
    for (int t = 0; t < 8; ++t) u[t] = A[(c0 + t) * kTileLd + ru];
    dfPanelSteps<7>(u, A, c0, 0, invD);
    dfPanelSteps<3>(u, A, c0, 4, invD);
  }
  return nreg;
}
#endif

// Trailing entries (r, k), c0 + 8 <= k <= r < end, of block b: thread t of nt.
template <typename T>
__device__ __forceinline__ void tileTrailing(T* A, int b, int end, int t, int nt) {
  const int c0 = 8 * b, o = c0 + 8, m = end - o;
#pragma unroll 1
  for (int e = t; e < m * (m + 1) / 2; e += nt) {
    // e = i (i + 1) / 2 + k
    int i = (int)((sqrtf(8.0f * (float)e + 1.0f) - 1.0f) * 0.5f);
    if (i * (i + 1) / 2 > e) --i;
    if ((i + 1) * (i + 2) / 2 <= e) ++i;
    const int r = o + i, k = o + e - i * (i + 1) / 2;
    T acc = A[k * kTileLd + r];
#pragma unroll
    for (int q = 0; q < 8; ++q) acc = accT(acc, -A[r * kTileLd + c0 + q], A[(c0 + q) * kTileLd + k]);
    A[k * kTileLd + r] = accEnd(acc);
  }
}

// Inverse of the 8x8 unit-lower leaf block b, lane c < 8 its column c; one warp.
template <typename T>
__device__ __forceinline__ void tileLeafInverse(T* A, int b) {
  const int o = 8 * b, c = threadIdx.x & 31;
  if (c >= 8) return;
  T y[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    T acc = (T)0;
#pragma unroll
    for (int k = 0; k < i; ++k) acc = accT(acc, A[(o + k) * kTileLd + o + i], y[k]);
    y[i] = (i < c) ? (T)0 : ((i == c) ? (T)1 : -accEnd(acc));
  }
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if (i > c) A[(o + i) * kTileLd + o + c] = y[i];
}

// Linv(I, Jb) = -Linv(I, I) S(I, Jb), S in place (tileInverseSum); one warp, two entries a lane.
template <typename T>
__device__ __forceinline__ void tileInverseFinish(T* A, int I, int Jb) {
  const int lane = threadIdx.x & 31, o = 8 * I, C = 8 * Jb + (lane & 7), i0 = lane >> 3;
  T v[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int i = i0 + 4 * h;
    T acc = A[(o + i) * kTileLd + C];
#pragma unroll
    for (int k = 0; k < 7; ++k) {
      if (k >= 3 + 4 * h) break;
      const T l = A[(o + i) * kTileLd + o + k];
      acc = accT(acc, k < i ? l : (T)0, A[(o + k) * kTileLd + C]);
    }
    v[h] = -accEnd(acc);
  }
  __syncwarp();
  A[(o + i0) * kTileLd + C] = v[0];
  A[(o + i0 + 4) * kTileLd + C] = v[1];
  __syncwarp();
}

// S(I, Jb) = sum over K = Jb .. I-1 of L(I, K) Linv(K, Jb), into the place of Linv(I, Jb); one
// warp, two entries a lane, even and odd terms in two sums.
template <typename T>
__device__ __forceinline__ void tileInverseSum(T* A, int I, int Jb) {
  const int lane = threadIdx.x & 31, C = 8 * Jb + (lane & 7), R = 8 * I + (lane >> 3);
  T a0 = (T)0, a1 = (T)0, b0 = (T)0, b1 = (T)0;
#pragma unroll 4
  for (int k = 8 * Jb; k < 8 * I; k += 2) {
    const T l0 = A[k * kTileLd + C], l1 = A[(k + 1) * kTileLd + C];
    const T lv0 = (k > C) ? l0 : ((k == C) ? (T)1 : (T)0), lv1 = (k + 1 > C) ? l1 : ((k + 1 == C) ? (T)1 : (T)0);
    a0 = accT(a0, A[k * kTileLd + R], lv0);
    a1 = accT(a1, A[(k + 1) * kTileLd + R], lv1);
    b0 = accT(b0, A[k * kTileLd + R + 4], lv0);
    b1 = accT(b1, A[(k + 1) * kTileLd + R + 4], lv1);
  }
  A[R * kTileLd + C] = accEnd(a0) + accEnd(a1);
  A[(R + 4) * kTileLd + C] = accEnd(b0) + accEnd(b1);
}

// Factors diagonal tile J in place with the calling warps 0 .. gw-1 (gw >= 1; named barrier 1 when
// gw > 1); its pivot reciprocals go to invD[32] (shared). Rows beyond nr are identity padding with
// zero off-diagonal entries: their 8-blocks are left as they are. Ends with a group barrier.
template <typename T>
__device__ __noinline__ void tileFactorDiagBlocked(T* A, int J, int nr, int nx, const DevSettings& st, PivotStats* ps,
                                                   T* invD, int gw) {
  const int warp = threadIdx.x >> 5, gt = 32 * gw;
  const bool regularized = st.linear_solver == 2;
  const T epsT = (T)st.dynamic_reg_eps, deltaT = (T)st.dynamic_reg_delta;
  const int real = min(32, nr - J * 32), nb = (real + 7) >> 3;
  const int helpers = max(gw - 1, 1), hw = (gw > 1) ? warp - 1 : 0;  // this warp among the helpers
  int nreg = 0;
  if (warp == 0 && (int)(threadIdx.x & 31) >= 8 * nb) invD[threadIdx.x & 31] = (T)1;
#pragma unroll 1
  for (int b = 0; b < nb; ++b) {
    if (warp == 0) nreg += tileLeafPanel(A, b, J, nr, nx, regularized, epsT, deltaT, invD);
    if (gw == 1) __syncwarp();
    // the inverse's block row b-1, and the sums of block row b
    if (b > 0 && (gw == 1 || warp > 0)) {
      if (hw == 0) tileLeafInverse(A, b - 1);
      if (helpers > 1) asm volatile("bar.sync 2, %0;" ::"r"(32 * helpers) : "memory");
      else __syncwarp();
#pragma unroll 1
      for (int Jb = hw; Jb < b; Jb += helpers) {
        if (Jb < b - 1) tileInverseFinish(A, b - 1, Jb);
        tileInverseSum(A, b, Jb);
      }
      if (gw == 1) __syncwarp();
    }
    groupSync(gt);
    if (b + 1 < nb) {
      tileTrailing(A, b, 8 * nb, (int)threadIdx.x, gt);
      groupSync(gt);
    }
  }
  if (warp == 0 && (threadIdx.x & 31) == 0) ps->nreg += nreg;
  if (warp == gw - 1) tilePivotStats(A, J, nr, nx, regularized, ps);
  // the last block row of the inverse
  if (gw == 1 || warp > 0) {
    if (hw == 0) tileLeafInverse(A, nb - 1);
    if (helpers > 1) asm volatile("bar.sync 2, %0;" ::"r"(32 * helpers) : "memory");
    else __syncwarp();
#pragma unroll 1
    for (int Jb = hw; Jb < nb - 1; Jb += helpers) tileInverseFinish(A, nb - 1, Jb);
  }
  groupSync(gt);
}

// Diagonal tile factorisation by warps 0 .. gw-1 (the register form for FP32, warp 0 alone; the
// blocked form for 8-byte types).
template <typename T>
__device__ __forceinline__ void tileFactorDiag(T* A, int J, int nr, int nx, const DevSettings& st, PivotStats* ps,
                                               T* invD, int gw) {
  if constexpr (sizeof(T) == 4) {
    if (threadIdx.x < 32) tileFactorDiagRegs<T>(A, J, nr, nx, st, ps, invD);
    groupSync(32 * gw);
  } else {
    tileFactorDiagBlocked<T>(A, J, nr, nx, st, ps, invD, gw);
  }
}

// ---- off-diagonal tile: L_IJ = A_IJ Linv_JJ^T D_J^-1 ----------------------------------------------
// Columns 8 g .. 8 g + 7 of the result, one warp, lane = row. Column c needs columns k <= c of A
// only (products with the zeros above are left out: 640 multiply-adds a lane for the whole tile
// instead of 1024); the result stays in registers since other warps may still read A.
template <typename T>
__device__ __forceinline__ void tileOffDiagGroup(const T* Aij, const T* Ajj, const T* invD, int g, T (&out)[8]) {
  const int lane = threadIdx.x & 31, c0 = 8 * g;
#pragma unroll
  for (int j = 0; j < 8; ++j) out[j] = (T)0;
#pragma unroll 2
  for (int k = 0; k < c0; ++k) {
    const T av = Aij[k * kTileLd + lane];
#pragma unroll
    for (int j = 0; j < 8; ++j) out[j] = accT(out[j], av, Ajj[(c0 + j) * kTileLd + k]);
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const T av = Aij[(c0 + k) * kTileLd + lane];
    out[k] = accT(out[k], av, (T)1);
#pragma unroll
    for (int j = k + 1; j < 8; ++j) out[j] = accT(out[j], av, Ajj[(c0 + j) * kTileLd + c0 + k]);
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) out[j] = accEnd(out[j]) * invD[c0 + j];
}

template <typename T>
__device__ __forceinline__ void tileOffDiagStore(T* Aij, int g, const T (&out)[8]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int j = 0; j < 8; ++j) Aij[(8 * g + j) * kTileLd + lane] = out[j];
}

// ---- trailing products: C -= A diag(d) B^T, d = diagonal of the factored tile Ajj -----------------
// Columns 16 h .. 16 h + 15, one warp: lane (lr, lc) takes rows 4 i + lr, i < 8, and columns
// 16 h + 2 lc, + 1 (two scalings by d for sixteen multiply-adds).
template <typename T>
__device__ __noinline__ void tileSyrkHalf(T* C, const T* A, const T* B, const T* Ajj, int h) {
  const int lane = threadIdx.x & 31, lr = lane & 3, c0 = 16 * h + 2 * (lane >> 2);
  T acc[8][2];
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i][0] = acc[i][1] = (T)0;
#pragma unroll 2
  for (int k = 0; k < 32; ++k) {
    const T dk = Ajj[k * kTileLd + k];
    const T b0 = B[k * kTileLd + c0] * dk, b1 = B[k * kTileLd + c0 + 1] * dk;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const T av = A[k * kTileLd + 4 * i + lr];
      acc[i][0] = accT(acc[i][0], av, b0);
      acc[i][1] = accT(acc[i][1], av, b1);
    }
  }
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int i = 0; i < 8; ++i) C[(c0 + j) * kTileLd + 4 * i + lr] -= accEnd(acc[i][j]);
}

// Unit u < 6 of the lower half of a diagonal tile's product (its upper half is never read): the
// 16x16 quadrants (0,0), (1,0), (1,1) in halves of eight columns, one warp, lane (lr, lc) rows
// 4 i + lr, i < 4, of one column. Each entry gets tileSyrkHalf's operations in its order.
template <typename T>
__device__ __noinline__ void tileSyrkDiagUnit(T* C, const T* A, const T* Ajj, int u) {
  const int lane = threadIdx.x & 31, q = u >> 1;
  const int r0 = (q == 0 ? 0 : 16) + (lane & 3), c0 = (q == 2 ? 16 : 0) + 8 * (u & 1) + (lane >> 2);
  T acc[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) acc[i] = (T)0;
#pragma unroll 4
  for (int k = 0; k < 32; ++k) {
    const T bv = A[k * kTileLd + c0] * Ajj[k * kTileLd + k];
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[i] = accT(acc[i], A[k * kTileLd + r0 + 4 * i], bv);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) C[c0 * kTileLd + r0 + 4 * i] -= accEnd(acc[i]);
}

}  // namespace cxg
