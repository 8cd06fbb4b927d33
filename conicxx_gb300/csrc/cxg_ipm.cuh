// The interior-point hot path on the GPU (device code, instantiated by cxg_ipm_f32.cu,
// cxg_ipm_f32s.cu, cxg_ipm_f64.cu, cxg_ipm_gridf.cu, cxg_ipm_gridd.cu and cxg_ipm_probe.cu, which
// compile in parallel). One CTA runs the complete homogeneous self-dual embedding IPM of ConicXX
// (SolverImpl::solve and its helpers, src/conicxx/solver_impl.cpp:102-466) for one instance:
//  - batched form (ipmKernel): persistent CTAs take instances from an atomic queue per size
//    bucket; iterates in shared memory when they fit, the problem data in HBM/L2;
//  - whole-GPU form (ipmGridKernel): one large instance, CTA 0 running the iteration on vectors in
//    its scratch while every SM joins the root assembly, LDL', triangular solves and the larger
//    products with P and A (gridSync).
//
// Precision: cone scaling, residuals, refinement residuals, step lengths and termination are
// FP64. The dense root LDL' (see cxg_layout.h) is FP32 (MIXED) or FP64. In MIXED mode a KKT
// solve whose FP64-refined relative residual stays above mixed_fallback_tol (or is not finite),
// or whose FP32 factor has a pivot of the wrong sign, switches that instance to the double-float
// factor (about 48 bits, on the FP32 pipe) for the rest of its solve ("sticky" fallback, counted
// in DevResult::fp64_fallbacks).
#pragma once

#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "cxg_cones.cuh"
#include "cxg_df64.cuh"
#include "cxg_kernels.h"
#include "cxg_layout.h"
#include "cxg_tc.cuh"
#include "cxg_tiles.cuh"

namespace cxg {

// Rolled loops in the batched kernels: most run once or twice, and the unrolled copies were a third of
// 1.6 MB of code, far more than an SM's instruction caches hold. SMs that run different code then slow
// each other down: in a batch of 4096 problems an iteration of a 165-row root took 860 us where it takes
// 630 us alone; with 0.5 MB less of code on its path 650 to 700 us. The whole-GPU kernels, one instance
// with vectors in global memory, unroll by four to have more loads in flight.
#ifndef CXG_VEC_UNROLL
#define CXG_VEC_UNROLL "unroll 1"
#endif
#define FOR_T(i, n) _Pragma(CXG_VEC_UNROLL) for (int i = (int)threadIdx.x; i < (n); i += (int)blockDim.x)
// The elements a thread sums: over the first `vb` threads of the block (Ctx::vb). A sum's order, and so its
// rounding, is that of a block of vb threads whatever the block's real size; a batch that leaves SMs
// free runs blocks wider than that (threads beyond vb add zeros to nothing).
#define FOR_V(i, n, vb) _Pragma(CXG_VEC_UNROLL) for (int i = (int)threadIdx.x < (vb) ? (int)threadIdx.x : (n); i < (n); i += (vb))

// A sparse matrix in the plan's slice order (sliceRows): rows sorted by length, 32 a slice.
struct Sliced {
  const double* val;
  const int *col, *ptr, *perm;  // per entry; slot ptr; slot -> row
  int rows;
  const int* src;               // kGather: the entries' places in val, or null (val is in slice order)
};

// Products of the 32 rows of slice `sl` with x, one row a lane (a whole warp calls it); row receives
// this lane's row, or -1. init (by row, negated when kNeg; may be null) + sum of val * x[col]. kFour:
// four interleaved sums over the whole groups of eight entries, the rest added to the first, then
// ((0 + 1) + (2 + 3)); else one sum in sequence, without the entries with col < cmin.
//
// The order puts a warp's k-th entries next to each other, sorted rows make a slice's lengths alike, and
// no load hangs on a branch (a lane without an entry reads its slice's first one and multiplies zeros),
// so the loads of eight entries are in flight together, during the eight before. With one row per
// thread in plain CSR order a 189-row P of 9 100 entries took 19 000 cycles, now 11 400; the same order
// with the loads under their conditions 29 000. One FP64 instruction (64 cycles) per entry of a slice's
// longest row is 7 000. Inlined: a function would save and restore its registers through L1.
// kGather: values through their source index, for working memory without A's copies in slice order
// (LaunchArgs::gatherA); a form of its own, since the second dependent load costs the other one time.
template <bool kGather>
__device__ __forceinline__ double sliceDot(const Sliced& A, bool kFour, int sl, const double* x, int& row,
                                           const double* init = nullptr, bool negInit = false, int cmin = 0) {
  const int lane = threadIdx.x & 31, slot = 32 * sl + lane, rows = A.rows;
  const int *ptr = A.ptr, *col = A.col, *src = kGather ? A.src : nullptr;
  const double* val = A.val;
  const bool real = slot < rows;
  const int b0 = ptr[min(slot, rows)], b1 = ptr[min(slot + 1, rows)], r0 = A.perm[min(slot, rows - 1)];
  row = real ? r0 : -1;
  const int len = b1 - b0;
  const int start = __shfl_sync(0xffffffffu, b0, 0), longest = __shfl_sync(0xffffffffu, len, 0);
  const int whole = kFour ? (len & ~7) : 0;
  double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
  if (init) {
    const double i0 = init[r0];
    a0 = negInit ? -i0 : i0;
  }
  if (longest == 0) return a0;
  int base = start + lane;
  double v[8];
  int ci[8];
  auto load = [&](int k) {
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const bool on = k + u < len;
      const int at = on ? base : start;
      v[u] = val[kGather && src ? src[at] : at];
      ci[u] = col[at];
      base += __popc(__ballot_sync(0xffffffffu, on));
    }
  };
  load(0);
  for (int k = 0; k < longest; k += 8) {
    double w[8], xv[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) xv[u] = x[ci[u]];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const bool on = k + u < len && ci[u] >= cmin;
      w[u] = on ? v[u] : 0.0;
      xv[u] = on ? xv[u] : 0.0;
    }
    if (k + 8 < longest) load(k + 8);
    const bool four = k < whole;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      if (u > 0 && k + u >= longest) break;
      if ((u & 3) == 0) {
        a0 = fma(w[u], xv[u], a0);
      } else {
        double& a = (u & 3) == 1 ? a1 : (u & 3) == 2 ? a2 : a3;
        const double t = fma(w[u], xv[u], four ? a : a0);
        a = four ? t : a;
        a0 = four ? a0 : t;
      }
    }
  }
  if (kFour && longest >= 8) return (a0 + a1) + (a2 + a3);
  return a0;
}

// The task of a warp in round `round` of a list that comes longest first: back and forth over the SM's
// four sub-partitions (warp w runs on sub-partition w % 4), so that they get alike shares.
__device__ __forceinline__ int snakeTask(int round) {
  const int nw = blockDim.x >> 5, q = round * nw + (threadIdx.x >> 5);
  if (nw & 3) return round * nw + ((round & 1) ? nw - 1 - (int)(threadIdx.x >> 5) : (int)(threadIdx.x >> 5));
  return ((q >> 2) & 1) ? (q ^ 3) : q;
}

// ------------------------------------------------------------------------------------------
// block reductions (deterministic: fixed summation order, identical result in every thread)
// ------------------------------------------------------------------------------------------
// An FP64 instruction holds its sub-partition's FP64 unit for 64 cycles whatever the number of
// active lanes, so the trees below pack the additions of several values (and of several warps'
// partials) into one instruction's lanes, and comparisons run on the integer pipe. Six sums over
// 256 threads take 14 FP64 instructions a warp where one tree per value took 72.

// Lane of warpSums' result k of K: the bit pattern of k, lowest bit in lane bit 4.
__device__ __forceinline__ int sumLane(int k) { return ((k & 1) << 4) | ((k & 2) << 2) | (k & 4); }

// Sums of K values (K <= 8) over the warp: v_k = ((v_k[0] + v_k[16]) + (v_k[8] + v_k[24])) + ..., the
// shuffle-down tree's order (additions commute), in lane sumLane(k) of the result.
template <int K>
__device__ __forceinline__ double warpSums(const double (&v)[K]) {
  const int lane = threadIdx.x & 31;
  double w[K];
#pragma unroll
  for (int k = 0; k < K; ++k) w[k] = v[k];
  int n = K;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < (K + 1) / 2; ++i) {
      if (2 * i + 1 < n) {  // two values: the lower half of the lanes goes on with the first
        const double keep = up ? w[2 * i + 1] : w[2 * i], give = up ? w[2 * i] : w[2 * i + 1];
        w[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
      } else if (2 * i < n) {
        w[i] = w[2 * i] + __shfl_xor_sync(0xffffffffu, w[2 * i], o);
      }
    }
    n = (n + 1) / 2;
  }
  return w[0];
}

// Totals of the warps' partials red[k * 16 + w], w < nw, pairwise over the warps, of the (up to
// 32 / nw) values from k0 on: value k0 + i's in the lanes i * nw .. of the calling warp. Block
// sizes of 1, 2, 4 or 8 warps.
__device__ __forceinline__ double warpTotals(const double* red, int k0, int nw) {
  const int lane = threadIdx.x & 31, sh = 31 - __clz(nw);
  double t = red[min(k0 + (lane >> sh), 7) * 16 + (lane & (nw - 1))];
#pragma unroll 1
  for (int o = 1; o < nw; o <<= 1) t = t + __shfl_xor_sync(0xffffffffu, t, o);
  return t;
}

template <int K>
__device__ __forceinline__ void blockPartials(const double (&v)[K], double* red, int nw) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const double p = warpSums<K>(v);
  const int k = ((lane >> 4) & 1) | ((lane >> 2) & 2) | (lane & 4);
  __syncthreads();  // the last reduction's readers are done with red
  if (w < nw && lane == sumLane(k) && k < K) red[k * 16 + w] = p;
  __syncthreads();
}

// A function of its own, called with K = 2, 4 and 6: inlined it was 25 KB of code at six sums.
template <int K>
__device__ __noinline__ void blockSum(double (&v)[K], double* red, int vb) {
  const int nw = vb >> 5, lane = threadIdx.x & 31;
  blockPartials<K>(v, red, nw);
  if (nw & (nw - 1)) {  // a number of warps that is no power of two: in sequence, value k in lane k
    double t = 0.0;
#pragma unroll 1
    for (int j = 0; j < nw; ++j) t += red[min(lane, 7) * 16 + j];
#pragma unroll
    for (int k = 0; k < K; ++k) v[k] = __shfl_sync(0xffffffffu, t, k);
    return;
  }
#pragma unroll
  for (int k0 = 0; k0 < K; k0 += 4) {
    const double t = warpTotals(red, k0, nw);
#pragma unroll
    for (int k = k0; k < min(k0 + 4, K); ++k) v[k] = __shfl_sync(0xffffffffu, t, (k - k0) * nw);
  }
}

// One of four values by the lowest two bits of k.
__device__ __forceinline__ double pick4(int k, double a, double b, double c, double d) {
  const double t = (k & 1) ? b : a, u = (k & 1) ? d : c;
  return (k & 2) ? u : t;
}

__device__ __forceinline__ double blockMin(double v, double* red) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = minBits(v, __shfl_xor_sync(0xffffffffu, v, o));
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  double t = red[0];
  for (int j = 1; j < nw; ++j) t = minBits(t, red[j]);
  return t;
}

__device__ __forceinline__ bool blockAny(int v) { return __syncthreads_or(v) != 0; }

__device__ __forceinline__ int blockMaxInt(int v, int* redi) {
  if (!__syncthreads_or(v > 0)) return 0;
  if (threadIdx.x == 0) redi[0] = 0;
  __syncthreads();
  if (v) atomicMax(redi, v);
  __syncthreads();
  return redi[0];
}

// ------------------------------------------------------------------------------------------
// per-instance context (pointers into shared memory, scratch and the pools)
// ------------------------------------------------------------------------------------------
struct GridCtl;

struct Ctx {
  int n, m, p, l, nsoc, nr, nUnits;
  int vb;  // threads of the block whose sums the instance has (FOR_V)
  bool gather;  // no copies of A in slice order: values through their source index (LaunchArgs::gatherA)
  const InstanceDesc* D;
  const int *pdiag, *plowSrc, *ap, *ai, *arSrc;
  const int *azSrc, *socOff, *socDim, *unitAd, *unitSup, *tgtBeg, *contrib, *scUnit, *scOff;
  Sliced sP, sAc, sAr;  // P, A by columns, A by rows
  const long long *plowIdx, *azIdx, *tgtIdx;  // 64-bit root element offsets (8-byte aligned in the pool)
  // FP64 scratch (scaled data)
  double *Pu, *Pv, *Av, *Avc, *Avr, *Ad, *T, *qs, *bs, *root64;
  // shared-memory (or scratch) vectors
  double *x, *s, *z, *rx, *rz, *x1, *z1, *Px1, *dx, *dz, *ds, *dcon, *lam, *tn, *tm, *tm2;
  double *rhs, *sol, *res, *cor, *rr, *cw, *cu, *ev;
  SocScale* sp;
  void* root;      // FactT root (shared or scratch)
  double* red;
  int* redi;
  double* sc;      // scalar broadcast area
  double* kry;     // whole-GPU form: GMRES Krylov area (krylovDoubles) in scratch
  unsigned char* slices;  // whole-GPU mixed form: double-float panel slices (dfSliceBytes) in scratch
  GridCtl* grid;   // whole-GPU launch: the root jobs run on every CTA (null: this CTA alone)
};

// scalar slots in Ctx::sc
enum {
  SC_TAU = 0, SC_KAPPA, SC_EXTRA_P, SC_EXTRA_A, SC_USE64, SC_NFB, SC_RSTEPS, SC_MAXREL,
  SC_ATTEMPTS, SC_FACTOK, SC_GMRES, SC_ITREL, SC_FAULTF, SC_FAULTS, SC_ESC, SC_SOCLVL, SC_HSFLOOR, SC_PXOK, SC_COUNT
};



// Phase cycle counters (record_timings), kept by thread 0 in the scalar area after PivotStats.
enum { TM_FACTOR = 0, TM_SOLVE = 1, TM_ASSEMBLE = 2, TM_LDLT = 3, TM_DSOLVE = 4, TM_RESID = 5, TM_COUNT = 6 };
__device__ __forceinline__ long long* timers(Ctx& c) { return reinterpret_cast<long long*>(c.sc + SC_COUNT + 4); }

// ------------------------------------------------------------------------------------------
// instance prologue: scaled copies of the data (equilibration.cpp:102-127)
// ------------------------------------------------------------------------------------------
static __device__ __noinline__ void loadInstance(Ctx& c, const LaunchArgs& a) {
  const InstanceDesc& D = *c.D;
  const double* dvec = a.dpool + D.dD;
  const double* evec = a.dpool + D.dE;
  const double cs = D.cscale;
  const double* Px = a.Px + D.vPx;
  const double* Ax = a.Ax + D.vAx;
  const double* q = a.q + D.vQ;
  const double* b = a.b + D.vB;
  const int* Pp = a.ipool + D.iPp;
  const int* Pi = a.ipool + D.iPi;
  const int* psSrc = a.ipool + D.iPsSrc;
  // scaleP / scaleA / scaleQ / scaleB with the reference's operation order
  FOR_T(j, c.n) {
    for (int k = Pp[j]; k < Pp[j + 1]; ++k) c.Pu[k] = Px[k] * (cs * dvec[Pi[k]] * dvec[j]);
    for (int k = c.ap[j]; k < c.ap[j + 1]; ++k) c.Av[k] = Ax[k] * (evec[c.ai[k]] * dvec[j]);
    c.qs[j] = q[j] * (cs * dvec[j]);
  }
  FOR_T(r, c.m) {
    c.bs[r] = b[r] * evec[r];
    c.ev[r] = (r < c.p) ? 0.0 : ((r < c.p + c.l) ? 1.0 : 0.0);
  }
  __syncthreads();
  FOR_T(b2, c.nsoc) c.ev[c.socOff[b2]] = 1.0;
  FOR_T(k, D.nnzPs) c.Pv[k] = c.Pu[psSrc[k]];
  const int* acSrc = a.ipool + D.iAcSrc;
  if (!c.gather)
    FOR_T(k, D.nnzA) {
      c.Avc[k] = c.Av[acSrc[k]];
      c.Avr[k] = c.Av[c.arSrc[k]];
    }
  const int* adSrc = a.ipool + D.iAdSrc;
  FOR_T(k, D.nAd) {
    const int src = adSrc[k];
    c.Ad[k] = (src >= 0) ? c.Av[src] : 0.0;
  }
  __syncthreads();
}

// ------------------------------------------------------------------------------------------
// cone-set operations over all units of the instance (cone_set.cpp)
// ------------------------------------------------------------------------------------------
// Also leaves in c.sc[SC_SOCLVL] the first attempt of the regularisation ladder at which every SOC
// block's dense pivots pass in the reference's arithmetic (socRefLadderLevel; 0 when the test is
// off): the earlier attempts of factorizeWithRetry fail as the reference's do. From the first
// iteration with such a failure on, the instance's blocks hold Hs at the dense form's resolution
// (kind 3, hsSmall; flag SC_HSFLOOR).
static __device__ __noinline__ void coneUpdateScaling(Ctx& c, const DevSettings& st, const double* s, const double* z) {
  int lvl = 0;
  // three lists of work, one after another over the threads: the SOC blocks' scaling, their pivot
  // tests and the NN rows; each list starts at a warp of its own (a warp with lanes of two lists
  // would run both, one after the other)
  constexpr int al = 31;
  const bool test = st.soc_ref_dense && st.linear_solver != 2;
  const int o1 = (c.nsoc + al) & ~al, o2 = o1 + (test ? ((c.nsoc + al) & ~al) : 0);
  FOR_T(t, o2 + c.l) {
    if (t < o1) {
      if (t < c.nsoc) {
        const int off = c.socOff[t], d = c.socDim[t];
        socUpdateScaling(s + off, z + off, d, c.sp[t], c.cu + off);
      }
    } else if (t < o2) {
      if (t - o1 < c.nsoc) {
        const int off = c.socOff[t - o1], d = c.socDim[t - o1];
        lvl = max(lvl, socRefLadderLevel(s + off, z + off, d, st.static_reg_A, st.dynamic_reg_eps,
                                         st.dynamic_reg_delta, lvl));
      }
    } else {
      const int r = c.p + (t - o2);
      c.cw[r] = sqrt(s[r] / z[r]);  // nonnegative_cone.cpp:24
    }
  }
  const int mx = blockMaxInt(lvl, c.redi);
  // once a block's dense form has lost its small eigenvalue (the reference's pivot test fails),
  // the instance's blocks take Hs at the dense form's resolution, from this iteration on (sticky)
  const bool floorHs = c.sc[SC_HSFLOOR] != 0.0 || mx > 0;
  if (floorHs) FOR_T(b, c.nsoc) if (socKind(c.cu + c.socOff[b]) == 2) setSocKind(c.cu + c.socOff[b], 3);
  __syncthreads();
  if (threadIdx.x == 0) {
    c.sc[SC_SOCLVL] = (double)mx;
    if (floorHs) c.sc[SC_HSFLOOR] = 1.0;
  }
  __syncthreads();
}

// out = f(W) x on every cone row (Zero rows: 0, or eps * x for kHsEps). `sync`: with a barrier at the end.
static __device__ __noinline__ void coneApply(Ctx& c, int f, double eps, const double* x, double* out,
                                               bool sync = true) {
  FOR_T(r, c.p) out[r] = (f == kHsEps) ? eps * x[r] : 0.0;
  FOR_T(t, c.l + c.nsoc) {  // the longer SOC units first, packed into as few warps as they fill
    if (t >= c.nsoc) {
      const int r = c.p + (t - c.nsoc);
      out[r] = wfun(f, c.cw[r], eps) * x[r];
    } else {
      const int b = t;
      const int off = c.socOff[b], d = c.socDim[b];
      socApply(c.sp[b], c.cu + off, d, f, eps, x + off, out + off);
    }
  }
  if (sync) __syncthreads();
}

// out = G x on the cone rows with the G eigenvalues prepared at factorisation (Zero rows: 0, or left as
// they are).
static __device__ __noinline__ void coneApplyG(Ctx& c, const double* x, double* out, bool zeroRows) {
  if (zeroRows) FOR_T(r, c.p) out[r] = 0.0;
  FOR_T(t, c.l + c.nsoc) {
    if (t >= c.nsoc) {
      const int r = c.p + (t - c.nsoc);
      out[r] = c.cu[r] * x[r];
    } else {
      const int b = t;
      const int off = c.socOff[b], d = c.socDim[b];
      socApplyG(c.sp[b], c.cu + off, d, x + off, out + off);
    }
  }
  __syncthreads();
}

// Jordan product / inverse product (Zero rows -> 0).
static __device__ __noinline__ void coneProduct(Ctx& c, bool inverse, const double* u, const double* v, double* out) {
  FOR_T(r, c.p) out[r] = 0.0;
  FOR_T(t, c.l + c.nsoc) {
    if (t >= c.nsoc) {
      const int r = c.p + (t - c.nsoc);
      out[r] = inverse ? v[r] / u[r] : u[r] * v[r];
    } else {
      const int b = t;
      const int off = c.socOff[b], d = c.socDim[b];
      if (inverse) socInverseProduct(u + off, v + off, d, out + off);
      else socProduct(u + off, v + off, d, out + off);
    }
  }
  __syncthreads();
}

// ConeSet::maxStep (cone_set.cpp:108-115) of (s, ds) and (z, dz) as one block-wide min of per-unit
// limits.
static __device__ __noinline__ double coneMaxStep2(Ctx& c, double amax) {
  double al = amax;
  const int nu = c.l + c.nsoc;
  FOR_T(t2, 2 * nu) {  // the SOC blocks of both, then the NN rows of both
    const bool soc = t2 < 2 * c.nsoc;
    const int t1 = soc ? t2 : t2 - 2 * c.nsoc, len = soc ? c.nsoc : c.l;
    const bool second = t1 >= len;
    const int t = second ? t1 - len : t1;
    const double* x = second ? c.s : c.z;
    const double* dx = second ? c.ds : c.dz;
    if (!soc) {
      const int r = c.p + t;
      if (negBits(dx[r])) al = minBits(al, -x[r] / dx[r]);
    } else {
      const int b = t;
      const int off = c.socOff[b], d = c.socDim[b];
      al = minBits(al, socMaxStep(x + off, dx + off, d, amax));
    }
  }
  return blockMin(al, c.red);
}

// ConeSet::margins (cone_set.cpp:77-90): the NN block contributes ONE margin (its minimum).
static __device__ __noinline__ void coneMargins(Ctx& c, const double* x, double& mn, double& pos) {
  double nnmin = INFINITY;
  FOR_T(t, c.l) nnmin = fmin(nnmin, x[c.p + t]);
  double smin = INFINITY, spos = 0.0;
  FOR_V(b, c.nsoc, c.vb) {
    const double mg = socMargin(x + c.socOff[b], c.socDim[b]);
    smin = fmin(smin, mg);
    spos += fmax(mg, 0.0);
  }
  nnmin = blockMin(nnmin, c.red);
  smin = blockMin(smin, c.red);
  double v[1] = {spos};
  blockSum<1>(v, c.red, c.vb);
  mn = fmin(nnmin, smin);
  pos = v[0] + ((c.l > 0) ? fmax(nnmin, 0.0) : 0.0);
  if (!isfinite(mn)) mn = 0.0;
}

static __device__ void coneShift(Ctx& c, double* x, double alpha) {
  FOR_T(t, c.l) x[c.p + t] += alpha;
  FOR_T(b, c.nsoc) x[c.socOff[b]] += alpha;
  __syncthreads();
}

// shiftToInteriorCold (solver_impl.cpp:104-116 in the reference numbering of SolverImpl)
static __device__ void shiftToInteriorCold(Ctx& c, double* v, int degree) {
  double mn, pos;
  coneMargins(c, v, mn, pos);
  const double deg = (double)max(degree, 1);
  const double target = fmax(1.0, 0.1 * pos / deg);
  if (mn <= 0.0) {
    coneShift(c, v, -mn);
    coneShift(c, v, target);
  } else if (mn < target) {
    coneShift(c, v, target - mn);
  }
}

static __device__ void ensureStrictlyInteriorWarm(Ctx& c, double* v) {
  double mn, pos;
  coneMargins(c, v, mn, pos);
  if (mn <= 1e-8) coneShift(c, v, -mn + 1e-6);
}

// ------------------------------------------------------------------------------------------
// SpMVs with the scaled data (FP64)
// ------------------------------------------------------------------------------------------
// Slices of 32 rows.
__device__ __forceinline__ int slices(int rows) { return (rows + 31) >> 5; }

// What sliceProducts forms, and how.
enum {
  kProdP = 1,         // px = P x
  kProdCols = 2,      // atz = A' z
  kProdRows = 4,      // ax = A x
  kProdColsFour = 8,  // A' z in four interleaved sums
  kProdInit = 16,     // A_C' z + init (without the Zero rows) and A_C x - init (on the cone rows)
  kProdColsF32 = 32, kProdColsDf = 64  // atz is an array of float / df64
};

// Products to form: `what`, the vectors and where the results go.
struct ProductJob {
  int what;
  const double *x, *z;
  double* px;
  void* atz;
  double* ax;
  const double* init;
};

__device__ __forceinline__ int productTasks(const Ctx& c, int what) {
  return ((what & kProdP) ? slices(c.n) : 0) + ((what & kProdCols) ? slices(c.n) : 0) +
         ((what & kProdRows) ? slices(c.m) : 0);
}

// The products asked for, the slices of all of them as one list of tasks, the long rows of P first: the
// CTA's warps take them all (`first` < 0), or warp `first`'s of `count` over the grid. One function for
// every product of the iteration: each inlined copy of sliceDot was 5 to 11 KB of code.
template <bool kGather>
static __device__ __noinline__ void sliceTasks(const Ctx& c, const ProductJob& p, int first, int count) {
  const int what = p.what, sn = slices(c.n), end = productTasks(c, what);
  const int eP = (what & kProdP) ? sn : 0, eC = eP + ((what & kProdCols) ? sn : 0);
  const bool add = what & kProdInit;
#pragma unroll 1
  for (int i = 0;; ++i) {
    const int base = i * (first < 0 ? (int)(blockDim.x >> 5) : count);
    if (base >= end) break;
    const int q = first < 0 ? snakeTask(i) : base + first;
    if (q >= end) continue;
    const int kind = (q >= eP) + (q >= eC);
    const Sliced& A = kind == 0 ? c.sP : kind == 1 ? c.sAc : c.sAr;
    int row;
    const double v = sliceDot<kGather>(A, kind == 0 || (kind == 1 && (what & kProdColsFour)), q - (kind == 0 ? 0 : kind == 1 ? eP : eC),
                                       kind == 1 ? p.z : p.x, row, add ? p.init : nullptr, kind == 2,
                                       add && kind == 1 ? c.p : 0);
    if (row < 0) continue;
    if (kind == 0) p.px[row] = v;
    else if (kind == 2) { if (!add || row >= c.p) p.ax[row] = v; }
    else if (what & kProdColsF32) reinterpret_cast<float*>(p.atz)[row] = (float)v;
    else if (what & kProdColsDf) reinterpret_cast<df64*>(p.atz)[row] = (df64)v;
    else reinterpret_cast<double*>(p.atz)[row] = v;
  }
}

#ifdef CXG_GRID_KERNELS
// Whole-GPU kernels: products of more than four tasks a warp go to the other CTAs (two grid barriers,
// about 5 us, against 15 us and more for CTA 0 alone), which leaves CTA 0 free until productsEnd.
static __device__ bool gridProductsPost(Ctx& c, const ProductJob& p);
static __device__ void gridProductsWait(Ctx& c);
__device__ __forceinline__ bool productsBegin(Ctx& c, const ProductJob& p) {
  if (!c.grid || productTasks(c, p.what) <= 4 * (int)(blockDim.x >> 5)) return false;
  gridProductsPost(c, p);
  return true;
}
#else
__device__ __forceinline__ bool productsBegin(Ctx&, const ProductJob&) { return false; }
#endif
// Ends with a barrier. `begun`: productsBegin's answer.
__device__ __forceinline__ void productsEnd(Ctx& c, const ProductJob& p, bool begun) {
#ifdef CXG_GRID_KERNELS
  if (begun) {
    gridProductsWait(c);
    return;
  }
  sliceTasks<false>(c, p, -1, 0);
#else
  (void)begun;
  if (c.gather) sliceTasks<true>(c, p, -1, 0);
  else sliceTasks<false>(c, p, -1, 0);
#endif
  __syncthreads();
}
__device__ __forceinline__ void sliceProducts(Ctx& c, int what, const double* x, const double* z, double* px, void* atz,
                                              double* ax, const double* init) {
  const ProductJob p{what, x, z, px, atz, ax, init};
  productsEnd(c, p, productsBegin(c, p));
}

// y = P_sym x (full symmetric P)
static __device__ __forceinline__ void pmul(Ctx& c, const double* x, double* y) {
  sliceProducts(c, kProdP, x, nullptr, y, nullptr, nullptr, nullptr);
}

// px = P x, atz = A'z (interleaved sums) and ax = A x
__device__ __forceinline__ ProductJob kktProducts(const double* x, const double* z, double* px, double* atz, double* ax) {
  return {kProdP | kProdCols | kProdRows | kProdColsFour, x, z, px, atz, ax, nullptr};
}

// res = rhs - K sol for the statically-regularised K (the matrix refinement targets,
// kkt_system.cpp:296-311): top = (P + epsP I) x + A'z, bottom = A x - (Hs + epsA I) z. Returns
// |res| / rhsNorm; rhsNorm is computed when `first` (the first residual for this rhs), and P x is
// left in c.tn.
static __device__ __noinline__ double kktResidualImpl(Ctx& c, const DevSettings& st, const double* rhs, const double* sol,
                                  double* res, double& rhsNorm, bool first) {
  const int n = c.n, m = c.m;
  const double* xs = sol;
  const double* zs = sol + n;
  double acc2[2] = {0.0, 0.0};
  // (Hs + epsA I) z, then the products, with one barrier for both: warps without cone units go ahead
  const ProductJob prod = kktProducts(xs, zs, c.tn, c.dx, res + n);  // dx: free during a solve
  const bool begun = productsBegin(c, prod);
  coneApply(c, kHsEps, st.static_reg_A, zs, c.tm2, false);
  productsEnd(c, prod, begun);
  // the residual and its norm in one pass, each thread the elements that it sums
  FOR_V(t, n + m, c.vb) {
    double r;
    if (t < n) {
      // the product with the small regularisation rounded first (not fused into the sum)
      r = rhs[t] - (__dadd_rn(__dmul_rn(st.static_reg_P, xs[t]), c.tn[t]) + c.dx[t]);
    } else {
      r = (rhs[t] - res[t]) + c.tm2[t - n];
    }
    res[t] = r;
    acc2[0] += r * r;
    if (first) acc2[1] += rhs[t] * rhs[t];
  }
  // both norms and the quotient by one warp: a square root and a division hold the FP64 unit for
  // some 600 cycles each
  if (c.vb & (c.vb - 1)) {
    blockSum<2>(acc2, c.red, c.vb);
    if (first) rhsNorm = fmax(sqrt(acc2[1]), 1e-30);
    return sqrt(acc2[0]) / rhsNorm;
  }
  const int nw = c.vb >> 5;
  blockPartials<2>(acc2, c.red, nw);
  if (threadIdx.x < 32) {
    const double norm = sqrt(warpTotals(c.red, 0, nw));
    const double rn = first ? fmax(__shfl_sync(0xffffffffu, norm, nw), 1e-30) : rhsNorm;
    const double rel = norm / rn;
    if (threadIdx.x == 0) {
      c.red[120] = rel;
      c.red[121] = rn;
    }
  }
  __syncthreads();
  rhsNorm = c.red[121];
  return c.red[120];
}

// y = K sol for the same statically regularised K (the operator of the GMRES refinement).
static __device__ __noinline__ void kktApply(Ctx& c, const DevSettings& st, const double* sol, double* y) {
  const int n = c.n, m = c.m;
  const double* xs = sol;
  const double* zs = sol + n;
  const ProductJob prod = kktProducts(xs, zs, c.tn, c.dx, y + n);
  const bool begun = productsBegin(c, prod);
  coneApply(c, kHsEps, st.static_reg_A, zs, c.tm2, false);
  productsEnd(c, prod, begun);
  FOR_T(t, n + m) {
    if (t < n) y[t] = __dadd_rn(__dmul_rn(st.static_reg_P, xs[t]), c.tn[t]) + c.dx[t];
    else y[t] -= c.tm2[t - n];
  }
  __syncthreads();
}

static __device__ double kktResidual(Ctx& c, const DevSettings& st, const double* rhs, const double* sol, double* res,
                              double& rhsNorm, bool first) {
  const long long t0 = (st.record_timings && threadIdx.x == 0) ? clock64() : 0;
  const double r = kktResidualImpl(c, st, rhs, sol, res, rhsNorm, first);
  if (st.record_timings && threadIdx.x == 0) timers(c)[TM_RESID] += clock64() - t0;
  return r;
}

// ------------------------------------------------------------------------------------------
// dense LDL' of the tiled root (no pivoting) and its solve
// ------------------------------------------------------------------------------------------
// Right-looking over 32-wide tile columns J (tile operations in cxg_tiles.cuh). Pivot rules: QDLDL
// (qdldl_ldlt.cpp:64-68) fails on an exact zero pivot; REGULARIZED (regularized_ldlt.cpp:132-139,
// 251-253) corrects a pivot below eps with the expected sign (+ on x rows, - on Zero-cone rows)
// and fails if > 5% were corrected.

// Warps that factor the diagonal tile together in a block of nw warps; with eight warps the other
// four start on the trailing products at once.
__device__ __forceinline__ int diagWarps(int nw) { return nw >= 8 ? 4 : min(nw, 2); }

// The root's LDL' by one CTA, right-looking by tile column J with a one-column lookahead:
//  (1) the off-diagonal tiles of column J by groups of eight columns;
//  (2) the next diagonal tile's product on up to six warps, then its factorisation by
//      diagWarps() warps while the others take the other products of column J from a queue
//      (half a tile each), joined by the factoring warps when they are done.
// The order in which warps take products does not change a result: each is one warp's own.
template <typename T>
__device__ __noinline__ void denseLdlt(Ctx& c, T* M, const DevSettings& st, int& fail, int& wrongSign, double& minAbsD) {
  const int nr = c.nr, nx = c.n, Tn = rootTiles(nr);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int gw = diagWarps(nw), lw = min(nw, 6);
  PivotStats* ps = reinterpret_cast<PivotStats*>(c.sc + SC_COUNT);
  T* invD = reinterpret_cast<T*>(c.red);  // pivot reciprocals of the current tile column
  if (threadIdx.x == 0) {
    ps->nreg = 0;
    ps->zero = 0;
    ps->wrong = 0;
    ps->minAbs = INFINITY;
  }
  __syncthreads();
  if (warp < gw) tileFactorDiag<T>(M, 0, nr, nx, st, ps, invD, gw);
  __syncthreads();
  for (int J = 0; J + 1 < Tn; ++J) {
    T* Ajj = M + tileBase(Tn, J, J);
    const int rem = Tn - J - 1;
    if (threadIdx.x == 0) ps->next = 0;
    // column groups (tileOffDiagGroup) of the column's tiles, one a warp and round, the last (longest)
    // groups first. A group reads its own and earlier columns of its tile: what a round stores, after
    // the barrier, is not read by that tile's groups still to come.
#pragma unroll 1
    for (int t = warp; t - warp < 4 * rem; t += nw) {
      T o[8];
      const int g = 3 - t / rem;
      T* Aij = M + tileBase(Tn, J + 1 + t % rem, J);
      if (t < 4 * rem) tileOffDiagGroup(Aij, Ajj, invD, g, o);
      __syncthreads();
      if (t < 4 * rem) tileOffDiagStore(Aij, g, o);
    }
    __syncthreads();
    const int ntask = rem * (rem + 1) - 2;  // halves of the pairs (I, K), J < K <= I, but the first
    T* Anext = M + tileBase(Tn, J + 1, J + 1);
    const T* Lnext = M + tileBase(Tn, J + 1, J);
    for (int u = warp; u < 6 && warp < lw; u += lw) tileSyrkDiagUnit<T>(Anext, Lnext, Ajj, u);
    if (nw <= 6) __syncthreads();
    else if (warp < lw) asm volatile("bar.sync 3, %0;" ::"r"(32 * lw) : "memory");
    if (warp < gw) tileFactorDiag<T>(Anext, J + 1, nr, nx, st, ps, invD, gw);
    for (;;) {
      int q = 0;
      if (lane == 0) q = atomicAdd(&ps->next, 1);
      q = __shfl_sync(0xffffffffu, q, 0);
      if (q >= ntask) break;
      // pairs column by column, (J + 1, J + 1) first
      int K = J + 1, t = 1 + (q >> 1), len = rem;
      while (t >= len) { t -= len; --len; ++K; }
      const int I = K + t;
      const T *Lik = M + tileBase(Tn, I, J), *Lkj = M + tileBase(Tn, K, J);
      T* C = M + tileBase(Tn, I, K);
      if (I == K && (q & 1)) {
        // the upper right quadrant of a diagonal tile is never read
        tileSyrkDiagUnit<T>(C, Lik, Ajj, 4);
        tileSyrkDiagUnit<T>(C, Lik, Ajj, 5);
      } else {
        tileSyrkHalf<T>(C, Lik, Lkj, Ajj, q & 1);
      }
    }
    __syncthreads();
  }
  const bool regularized = st.linear_solver == 2;
  fail = regularized ? (((double)ps->nreg > 0.05 * (double)nr) ? 1 : 0) : ps->zero;
  wrongSign = ps->wrong;
  minAbsD = ps->minAbs;
  __syncthreads();
}

template <typename T>
__device__ __forceinline__ T shflXorT(T v, int m) { return __shfl_xor_sync(0xffffffffu, v, m); }
__device__ __forceinline__ df64 shflXorT(df64 v, int m) {
  return df64(__shfl_xor_sync(0xffffffffu, v.hi, m), __shfl_xor_sync(0xffffffffu, v.lo, m));
}

// log2 of the largest split s in {1, 2, 4, 8} of a 32-term dot product such that rows * s threads fit in
// one pass of a block of vb threads (rows is a multiple of 32, so each warp holds whole groups of s lanes).
__device__ __forceinline__ int dotSplit(int rows, int vb) {
  int ls = 0;
  while (ls < 3 && (rows << (ls + 1)) <= vb) ++ls;
  return ls;
}

// Sum of a dot-product partial over the s consecutive lanes of a group (s a power of two <= 8).
template <typename T>
__device__ __forceinline__ T groupSum(T v, int s) {
  for (int m = 1; m < s; m <<= 1) v = v + shflXorT(v, m);
  return v;
}

// y <- M^-1 y for the factored tiled root; y has Tn*32 entries (padding entries are zero).
// Every block product (the diagonal tile's Linv and each off-diagonal tile) is a set of 32-term
// dot products, split over s lanes per row (dotSplit) and reduced by shuffles, so that the few
// rows of the late steps still occupy the whole block. A solved tile goes to a buffer in the
// reduction area first, so that a step takes two barriers. (Half of the warps on the chain of
// diagonal tiles and half on the rows beyond, with one barrier, was slower by a third: the chain
// is bound by the issue of its double-float operations, not by the barriers.)
// (Split and row index are powers of two and shifts: a division by the split cost as much as a product.)
template <typename T, bool kForward>
__device__ __forceinline__ void denseSolvePass(Ctx& c, const T* M, T* y) {
  const int Tn = rootTiles(c.nr), tid = threadIdx.x, nth = blockDim.x;
  const int lsd = dotSplit(32, c.vb), wd = 32 >> lsd;
  const int di = tid >> lsd, d0 = (tid & ((1 << lsd) - 1)) * wd;  // row and first column in a diagonal product
  T* x = reinterpret_cast<T*>(c.red);
#pragma unroll 1
  for (int q = 0; q < Tn; ++q) {
    const int J = kForward ? q : Tn - 1 - q;
    const T* Ajj = M + tileBase(Tn, J, J);
    T* yJ = y + J * 32;
    if (tid < (32 << lsd)) {
      // forward: Linv_JJ y_J, backward: Linv_JJ' y_J (Linv(r, k) at r * ld + k)
      const T* Ad = Ajj + (kForward ? di * kTileLd + d0 : d0 * kTileLd + di);
      T acc = (T)0;
#pragma unroll 1
      for (int k = 0; k < wd; k += 4) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const T l = Ad[kForward ? u : u * kTileLd];
          const int at = d0 + k + u;
          acc = accT(acc, (kForward ? at < di : at > di) ? l : (T)0, yJ[at]);
        }
        Ad += kForward ? 4 : 4 * kTileLd;
      }
      const T tot = groupSum(accEnd(acc), 1 << lsd);
      if (d0 == 0) x[di] = yJ[di] + tot;
    }
    __syncthreads();
    if (tid < 32) yJ[tid] = x[tid];
    const int rows = (kForward ? Tn - J - 1 : J) * 32;
    if (rows > 0) {
      const int ls = dotSplit(rows, c.vb), w = 32 >> ls;
#pragma unroll 1
      for (int t = tid; t < rows << ls; t += nth) {
        const int row = t >> ls, p = (t & ((1 << ls) - 1)) * w, rr = row & 31;
        const int I = (kForward ? J + 1 : 0) + (row >> 5);
        const T* L = kForward ? M + tileBase(Tn, I, J) + p * kTileLd + rr : M + tileBase(Tn, J, I) + rr * kTileLd + p;
        T acc = (T)0;
#pragma unroll 1
        for (int k = 0; k < w; k += 4) {
#pragma unroll
          for (int u = 0; u < 4; ++u) acc = accT(acc, L[kForward ? u * kTileLd : u], x[p + k + u]);
          L += kForward ? 4 * kTileLd : 4;
        }
        acc = groupSum(accEnd(acc), 1 << ls);
        if (p == 0) y[I * 32 + rr] -= acc;
      }
    }
    __syncthreads();
  }
}

template <typename T>
__device__ void denseSolve(Ctx& c, const T* M, T* y) {
  const int Tn = rootTiles(c.nr);
  denseSolvePass<T, true>(c, M, y);   // y_J = Linv_JJ y_J, then y_I -= L_IJ y_J for I > J
#pragma unroll 1
  for (int t = threadIdx.x; t < Tn * 32; t += blockDim.x) {
    const int J = t / 32, rr = t % 32;
    y[t] /= M[tileBase(Tn, J, J) + rr * kTileLd + rr];
  }
  __syncthreads();
  denseSolvePass<T, false>(c, M, y);  // x_J = Linv_JJ^T y_J, then y_K -= L_JK^T x_J for K < J
}

// ------------------------------------------------------------------------------------------
// whole-GPU root (single large instance)
// ------------------------------------------------------------------------------------------
// One instance whose root is too large for one SM runs as a cooperative launch with one CTA
// per SM: CTA 0 runs the interior-point iteration exactly as the batched kernel does, and at the
// two root-sized steps, assembly + LDL' and the triangular solves, it posts a job that every
// CTA runs with it. Jobs are the same tile operations in the same order per tile as the
// single-CTA root, spread over the warps of the grid, with a grid barrier between dependent
// steps of the factor (two per tile column); the triangular passes hand solved tiles over by flags.
enum { kGridOpFactor = 1, kGridOpSolve = 2, kGridOpExit = 3, kGridOpProducts = 4, kGridOpSave = 5 };

constexpr int kGridMaxTiles = 131072 / kTile;  // of the largest whole-GPU root

struct GridCtl {
  unsigned arrive;   // barrier: arrivals in the current round
  unsigned gen;      // barrier: completed rounds
  int error;         // a barrier wait ran out; every later barrier fails at once
  int op;            // job posted by CTA 0
  int arith;         // root arithmetic of the job: 0 FP64, 1 FP32, 2 double-float
  int epoch;         // number of the job (tile flags of the triangular solves)
  void* M;           // root of the job
  void* y;           // solve vector (root arithmetic), rootTiles(nr) * 32 entries; save: FP64 copy of the root
  double ep, ea;     // regularisation bumps of the assembly
  int64_t stageOff;  // byte offset of the tile staging area in dynamic shared memory
  unsigned long long waitNs;  // longest wait at a barrier or for a tile; 0 = kGridWaitNs
  int leaveJob;      // tests: CTA 1 leaves the launch at its job of this number, undone (0: none)
  ProductJob prod;   // products job
  Ctx ctx;           // CTA 0's instance context (pointers into global memory only)
  int flags[2 * kGridMaxTiles];  // job whose forward / backward pass has solved the tile
};

template <typename T> struct ArithOf;
template <> struct ArithOf<double> { static constexpr int v = 0; };
template <> struct ArithOf<float> { static constexpr int v = 1; };
template <> struct ArithOf<df64> { static constexpr int v = 2; };

__device__ __forceinline__ unsigned long long globalNs() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Longest wait at one grid barrier. CTA 0's own work between two root jobs (cone scaling,
// residuals, KKT residual products) takes milliseconds; a wait this long means a CTA is gone.
constexpr unsigned long long kGridWaitNs = 30ull * 1000ull * 1000ull * 1000ull;

// Grid-wide barrier of a cooperative launch (every CTA resident). Thread 0 of each CTA arrives
// after a fence (release); the last arrival resets the count and opens the next round; the
// others poll the round number and fence after it changes (acquire). Each wait is bounded by
// kGridWaitNs: a wait that runs out records an error, and from then on every barrier of every
// CTA returns false at once, so the launch always ends.
static __device__ __noinline__ bool gridSync(GridCtl* g) {
  __shared__ int sOk;
  __syncthreads();
  if (threadIdx.x == 0) {
    volatile GridCtl* vg = g;
    int ok = vg->error == 0;
    if (ok) {
      unsigned long long limit = vg->waitNs;
      if (limit == 0) limit = kGridWaitNs;
      const unsigned gen = vg->gen;
      __threadfence();
      const unsigned prev = atomicAdd(&g->arrive, 1u);
      if (prev == gridDim.x - 1) {
        atomicExch(&g->arrive, 0u);
        __threadfence();
        atomicAdd(&g->gen, 1u);
      } else {
        const unsigned long long t0 = globalNs();
        unsigned backoff = 32;  // ns, doubled up to 512 while the wait lasts
        while (vg->gen == gen) {
          if (vg->error) { ok = 0; break; }
          if (globalNs() - t0 > limit) {
            atomicExch(&g->error, 1);
            ok = 0;
            break;
          }
          __nanosleep(backoff);
          if (backoff < 512) backoff <<= 1;
        }
      }
      __threadfence();
    }
    sOk = ok;
  }
  __syncthreads();
  return sOk != 0;
}

// Whether a wait of this launch has run out (every barrier fails from then on); for a whole CTA.
static __device__ __forceinline__ bool gridFailed(GridCtl* g) {
  return __syncthreads_or(threadIdx.x == 0 && reinterpret_cast<volatile GridCtl*>(g)->error != 0) != 0;
}

#ifdef CXG_GRID_KERNELS
// The products job on CTAs 1 ..: the tasks go round the CTAs first, so that few of them share an SM. After
// a failed barrier the results are those of an earlier product: the next root job fails as well, and what
// was judged from them until then does not count (gridFailed).
static __device__ __forceinline__ void gridProductsShare(GridCtl* g) {
  if (blockIdx.x > 0) {
    const int ctas = (int)gridDim.x - 1, w = threadIdx.x >> 5;
    sliceTasks<false>(g->ctx, g->prod, (int)blockIdx.x - 1 + ctas * w, ctas * (int)(blockDim.x >> 5));
  }
}
static __device__ bool gridProductsPost(Ctx& c, const ProductJob& p) {
  if (threadIdx.x == 0) {
    c.grid->op = kGridOpProducts;
    c.grid->prod = p;
  }
  return gridSync(c.grid);
}
static __device__ void gridProductsWait(Ctx& c) { gridSync(c.grid); }

// The factored root as FP64, for the adjoint: the share of CTA `cta` of `ctas`. CTA 0 alone took 32 ms for
// the 147 MB of a 5940-row root, a tenth of the whole solve.
template <typename T>
__device__ __forceinline__ void gridSaveShare(GridCtl* g, int cta, int ctas) {
  const T* R = reinterpret_cast<const T*>(g->M);
  double* out = reinterpret_cast<double*>(g->y);
  const int64_t rs = rootSize(g->ctx.nr), step = (int64_t)ctas * blockDim.x;
#pragma unroll 4
  for (int64_t t = (int64_t)cta * blockDim.x + threadIdx.x; t < rs; t += step) out[t] = (double)R[t];
}
static __device__ __forceinline__ void gridSaveJob(GridCtl* g, int cta, int ctas) {
  const int arith = g->arith;
  if (arith == 0) gridSaveShare<double>(g, cta, ctas);
  else if (arith == 1) gridSaveShare<float>(g, cta, ctas);
  else gridSaveShare<df64>(g, cta, ctas);
}
// CTA 0. Where a barrier fails (nothing follows this job that would notice), all of it by this CTA: the
// others write the same values, if any.
static __device__ void gridSaveRoot(Ctx& c, int arith, void* M, double* out) {
  if (threadIdx.x == 0) {
    c.grid->op = kGridOpSave;
    c.grid->arith = arith;
    c.grid->M = M;
    c.grid->y = out;
  }
  if (gridSync(c.grid)) {
    gridSaveJob(c.grid, 0, (int)gridDim.x);
    if (gridSync(c.grid)) return;
  }
  gridSaveJob(c.grid, 0, 1);
  __syncthreads();
}
#endif

// The cone-unit contributions added to the root, slices of 32 targets (one a lane), warp w0 of nw: a
// target's contributions in their order, A_u' (G_u A_u) as d multiply-adds each. Four contributions'
// loads are in flight together, none under a condition (see sliceDot); one at a time cost two
// dependent loads from L2 each.
template <typename T>
__device__ __forceinline__ void addContributions(const Ctx& c, T* M, int64_t w0, int64_t nw) {
  const InstanceDesc& D = *c.D;
  const int lane = threadIdx.x & 31, nT = D.nTgt;
  const int *ci = c.contrib, *cj = ci + D.nContrib, *cd = cj + D.nContrib;
  for (int64_t sl = w0; sl < (nT + 31) / 32; sl += nw) {
    const int t = (int)(32 * sl) + lane;
    const int b0 = c.tgtBeg[min(t, nT)], len = c.tgtBeg[min(t + 1, nT)] - b0;
    const int64_t at = c.tgtIdx[min(t, nT - 1)];
    const int start = __shfl_sync(0xffffffffu, b0, 0), longest = __shfl_sync(0xffffffffu, len, 0);
    int base = start + lane;
    double acc = 0.0;
    for (int k = 0; k < longest; k += 4) {
      int oi[4], oj[4], d[4];
      double va[4], vt[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const bool on = k + u < len;
        const int q = on ? base : start;
        base += __popc(__ballot_sync(0xffffffffu, on));
        oi[u] = ci[q];
        oj[u] = cj[q];
        const int dq = cd[q];
        d[u] = on ? dq : 0;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        va[u] = c.Ad[oi[u]];
        vt[u] = c.T[oj[u]];
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (k + u >= longest) break;
        acc = fma(d[u] > 0 ? va[u] : 0.0, d[u] > 0 ? vt[u] : 0.0, acc);
        for (int r0 = 1; __any_sync(0xffffffffu, r0 < d[u]); r0 += 3) {
          double a[3], b[3];
#pragma unroll
          for (int e = 0; e < 3; ++e) {
            const int r = min(r0 + e, max(d[u] - 1, 0));
            a[e] = c.Ad[oi[u] + r];
            b[e] = c.T[oj[u] + r];
          }
#pragma unroll
          for (int e = 0; e < 3; ++e) {
            const bool on = r0 + e < d[u];
            if (__any_sync(0xffffffffu, on)) acc = fma(on ? a[e] : 0.0, on ? b[e] : 0.0, acc);
          }
        }
      }
    }
    if (t < nT) M[at] += (T)acc;
  }
}

// Root assembly spread over the grid, the same writes as the single-CTA assembly in
// assembleFactor: zero, then the distinct entries (padding identity, P diagonal + bump,
// strictly-upper P, Zero-row A, Zero-row diagonal), then the cone-unit contributions (one target
// root entry per thread, so no two threads add into the same entry).
template <typename T>
__device__ __noinline__ bool gridAssemble(GridCtl* g, const Ctx& c, const DevSettings& st, T* M, double ep, double ea) {
  const InstanceDesc& D = *c.D;
  const int n = c.n, nr = c.nr;
  const int64_t gt = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, gs = (int64_t)gridDim.x * blockDim.x;
  const int64_t rs = rootSize(nr);
  for (int64_t t = gt; t < rs; t += gs) M[t] = (T)0;
  if (!gridSync(g)) return false;
  for (int64_t i = nr + gt; i < (int64_t)rootTiles(nr) * kTile; i += gs) M[rootIdx(nr, (int)i, (int)i)] = (T)1;
  for (int64_t i = gt; i < n; i += gs) {
    const int src = c.pdiag[i];
    M[rootIdx(nr, (int)i, (int)i)] = (T)(((src >= 0) ? c.Pu[src] : 0.0) + st.static_reg_P + ep);
  }
  for (int64_t k = gt; k < D.nPlow; k += gs) M[c.plowIdx[k]] = (T)c.Pu[c.plowSrc[k]];
  for (int64_t k = gt; k < D.nAZ; k += gs) M[c.azIdx[k]] = (T)c.Av[c.azSrc[k]];
  for (int64_t r = gt; r < c.p; r += gs) M[rootIdx(nr, n + (int)r, n + (int)r)] = (T)(-(st.static_reg_A + ea));
  if (!gridSync(g)) return false;
  addContributions<T>(c, M, (int64_t)(threadIdx.x >> 5) * gridDim.x + blockIdx.x, (int64_t)gridDim.x * (blockDim.x >> 5));
  return gridSync(g);
}

// Asynchronous copy of one tile into shared memory (16-byte cp.async), thread t of nt; not committed.
template <typename T>
__device__ __forceinline__ void copyTileAsync(T* dst, const T* src, int t, int nt) {
  constexpr int nv = kTileElems * (int)sizeof(T) / 16;
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
#pragma unroll 4
  for (int v = t; v < nv; v += nt)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + 16u * v),
                 "l"(reinterpret_cast<const char*>(src) + 16 * v)
                 : "memory");
}

// Trailing update of tile column J on the CUDA cores (FP64 and double-float): C_IK -= L_IJ D_J L_KJ^T
// for the tiles J < K <= I but (J+1, J+1), one tile at a time and CTA (CTAs 1 .., 256 threads). The
// three tiles of the next product arrive by cp.async meanwhile; L_KJ is scaled by D_J once in shared
// memory; warp w takes columns 4 w .. 4 w + 3, a lane one row, with the tile routine's operations in its
// order. Single tiles rather than 128x128 super-blocks: a super-block holds one SM's FP64 units for
// 127 us (24 us of FP32 issue in double-float) while a root of some thousand rows has fewer
// super-blocks than the GPU has SMs; a tile takes 9 us (2 us). FP64 factor of 1020 rows in an iteration
// 5.4 -> 1.9 ms, of 6400 rows 111 -> 89 ms (its FP64 issue alone 72 ms); double-float of 1100 rows
// 1.64 -> 1.31 ms.
template <typename T>
__device__ __noinline__ void gridTileUpdate(T* M, int Tn, int J, T* sm) {
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, c0 = 4 * (tid >> 5);
  const int rem = Tn - J - 1, stride = (int)gridDim.x - 1;
  const long long tiles = (long long)rem * (rem + 1) / 2;
  const T* Ajj = M + tileBase(Tn, J, J);
  T* dg = sm;              // the diagonal of D_J
  T* bufs = sm + 32;       // two sets of L_IJ, L_KJ, C_IK
  // tile t (row order: t = i (i + 1) / 2 + k, tile (J+1+i, J+1+k)); t = 0 belongs to CTA 0
  auto where = [&](long long t, int& I, int& K) {
    int i = (int)((sqrtf(8.0f * (float)t + 1.0f) - 1.0f) * 0.5f);
    while ((long long)i * (i + 1) / 2 > t) --i;
    while ((long long)(i + 1) * (i + 2) / 2 <= t) ++i;
    I = J + 1 + i;
    K = J + 1 + (int)(t - (long long)i * (i + 1) / 2);
  };
  auto fetch = [&](long long t, int set) {
    if (t < tiles) {
      int I, K;
      where(t, I, K);
      T* b = bufs + set * 3 * kTileElems;
      copyTileAsync(b, M + tileBase(Tn, I, J), tid, nt);
      copyTileAsync(b + kTileElems, M + tileBase(Tn, K, J), tid, nt);
      copyTileAsync(b + 2 * kTileElems, M + tileBase(Tn, I, K), tid, nt);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  long long t = (long long)blockIdx.x;
  if (t >= tiles) return;
  fetch(t, 0);
  if (tid < 32) dg[tid] = Ajj[tid * kTileLd + tid];
  for (int set = 0; t < tiles; t += stride, set ^= 1) {
    fetch(t + stride, set ^ 1);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    T* A = bufs + set * 3 * kTileElems;
    T *B = A + kTileElems, *C = B + kTileElems;
    for (int e = tid; e < kTile * kTile; e += nt) {
      const int k = e >> 5, i = e & 31;
      B[k * kTileLd + i] = B[k * kTileLd + i] * dg[k];
    }
    __syncthreads();
    T acc[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[j] = (T)0;
#pragma unroll 4
    for (int k = 0; k < kTile; ++k) {
      const T av = A[k * kTileLd + lane];
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[j] = accT(acc[j], av, B[k * kTileLd + c0 + j]);
    }
    int I, K;
    where(t, I, K);
    T* out = M + tileBase(Tn, I, K);
#pragma unroll
    for (int j = 0; j < 4; ++j)
      out[(c0 + j) * kTileLd + lane] = C[(c0 + j) * kTileLd + lane] - accEnd(acc[j]);
    __syncthreads();  // this set of tiles is free for the copies after the next
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
}

// FP32 trailing update of tile column J on the tensor cores (tcgen05, kind::tf32): the same
// C_IK -= L_IJ D_J L_KJ^T as gridTileUpdate, over every super-block this CTA owns in the step
// (sb = blockIdx.x - 1, + gridDim.x - 1, ...). Each FP32 operand is split as hi + lo (hi = its
// TF32 rounding, lo = the TF32 rounding of the remainder) and the product taken as
// A_lo B_hi + A_hi B_lo + A_hi B_hi (3xTF32; the A_lo B_lo term is below FP32 rounding): twelve
// 128x128x8 MMAs accumulating in FP32 in TMEM, issued by one thread. Software pipeline: the C tiles
// of the next super-block arrive by bulk copies (TMA) into the other of two shared-memory buffers
// while the current super-block's panels are staged (generic loads, TF32 split), multiplied and
// its tiles updated from TMEM and written back by bulk copies. All bulk stores of the step are
// complete (and ordered before later generic accesses) when it returns.
// Shared memory `sm` (128-byte aligned, kGridTcStageBytes): the operand panels A_hi, A_lo, B_hi,
// B_lo (16 KB each, layout of cxg_tc.cuh), then two buffers of 16 C tiles. `tmem`: this CTA's 128
// accumulator columns; mbarriers: MMA completion and one per C buffer, with their phase parities.
// Returns false when a wait ran out (after waiting once more for the copies in flight).
constexpr int64_t kTcStageBytes = kGridTcStageBytes;
constexpr unsigned long long kTcWaitNs = 2ull * 1000ull * 1000ull * 1000ull;
constexpr uint32_t kTileBytes = (uint32_t)kTileElems * 4u;

struct SbGeo {
  int I0, K0, ni, nk;
  bool diag, skip00;
};

// the super-block sb of step J (row order: sb = r (r + 1) / 2 + k, tile rows J+1+4r.., tile
// columns J+1+4k..; super-block 0 without the tile (J+1, J+1), which CTA 0 updates)
__device__ __forceinline__ SbGeo sbGeo(long long sb, int J, int Tn) {
  int r = (int)((sqrtf(8.0f * (float)sb + 1.0f) - 1.0f) * 0.5f);
  while ((long long)r * (r + 1) / 2 > sb) --r;
  while ((long long)(r + 1) * (r + 2) / 2 <= sb) ++r;
  const int k = (int)(sb - (long long)r * (r + 1) / 2);
  SbGeo g;
  g.I0 = J + 1 + 4 * r;
  g.K0 = J + 1 + 4 * k;
  g.ni = min(4, Tn - g.I0);
  g.nk = min(4, Tn - g.K0);
  g.diag = r == k;
  g.skip00 = sb == 0;
  return g;
}

// tile t = 4a + b of the super-block is updated (and so loaded and stored) by it
__device__ __forceinline__ bool sbTile(const SbGeo& g, int t) {
  const int a = t >> 2, b = t & 3;
  return a < g.ni && b < g.nk && !(g.diag && b > a) && !(g.skip00 && t == 0);
}

static __device__ __noinline__ bool tcTrailingStep(float* M, int Tn, int J, long long nsb, unsigned char* sm,
                                                   uint32_t tmem, uint32_t mbarMma, uint32_t mbarLd0,
                                                   uint32_t mbarLd1, uint32_t& phMma, uint32_t& phLd0,
                                                   uint32_t& phLd1) {
  const int tid = threadIdx.x;
  const long long first = (long long)blockIdx.x - 1, stride = (long long)gridDim.x - 1;
  if (first >= nsb) return true;
  const float* Ajj = M + tileBase(Tn, J, J);
  const uint32_t opBase = tc::smemAddr(sm);
  const uint32_t cAddr[2] = {opBase + 4u * tc::kPanelBytes, opBase + 4u * tc::kPanelBytes + 16u * kTileBytes};
  float* cPtr[2] = {reinterpret_cast<float*>(sm + 4 * tc::kPanelBytes),
                    reinterpret_cast<float*>(sm + 4 * tc::kPanelBytes + 16 * kTileBytes)};
  const uint32_t mbarLd[2] = {mbarLd0, mbarLd1};
  // thread 0: the C tiles of super-block g into buffer buf, completing on that buffer's mbarrier
  auto issueLoads = [&](const SbGeo& g, int buf) {
    uint32_t bytes = 0;
    for (int t = 0; t < 16; ++t)
      if (sbTile(g, t)) bytes += kTileBytes;
    tc::mbarArriveExpectTx(mbarLd[buf], bytes);
    for (int t = 0; t < 16; ++t)
      if (sbTile(g, t))
        tc::bulkLoad(cAddr[buf] + (uint32_t)t * kTileBytes, M + tileBase(Tn, g.I0 + (t >> 2), g.K0 + (t & 3)),
                     kTileBytes, mbarLd[buf]);
  };
  if (tid == 0) {
    tc::fenceProxyAsyncGlobal();  // the previous step's generic writes before these async reads
    issueLoads(sbGeo(first, J, Tn), 0);
  }
  int buf = 0;
  for (long long sb = first; sb < nsb; sb += stride, buf ^= 1) {
    const SbGeo g = sbGeo(sb, J, Tn);
    if (tid == 0 && sb + stride < nsb) {
      tc::bulkWaitRead0();  // the previous super-block's stores have read the other buffer
      issueLoads(sbGeo(sb + stride, J, Tn), buf ^ 1);
    }
    // panels: thread tid stages row i = tid & 127 of A (L_IJ, tid < 128) or of B (D-scaled L_KJ),
    // four k at a time, as TF32 hi and lo parts; row m sits at byte (k / 4) * 2048 + m * 16 + (k % 4) * 4
    if (tid < 2 * tc::kRows) {
      const int i = tid & (tc::kRows - 1), isB = tid >> 7, a = i >> 5, rr = i & 31;
      const int nt = isB ? g.nk : g.ni;
      const float* src = (a < nt) ? M + tileBase(Tn, (isB ? g.K0 : g.I0) + a, J) + rr : nullptr;
      unsigned char* hiBase = sm + (isB ? 2 : 0) * tc::kPanelBytes;
      unsigned char* loBase = hiBase + tc::kPanelBytes;
#pragma unroll 2
      for (int kq = 0; kq < kTile / 4; ++kq) {
        float hi[4], lo[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const int k = 4 * kq + t;
          float x = src ? src[k * kTileLd] : 0.0f;
          if (isB) x = x * Ajj[k * kTileLd + k];
          hi[t] = tc::toTf32(x);
          lo[t] = tc::toTf32(x - hi[t]);
        }
        *reinterpret_cast<float4*>(hiBase + kq * 2048 + i * 16) = make_float4(hi[0], hi[1], hi[2], hi[3]);
        *reinterpret_cast<float4*>(loBase + kq * 2048 + i * 16) = make_float4(lo[0], lo[1], lo[2], lo[3]);
      }
    }
    tc::fenceProxyAsyncShared();
    __syncthreads();
    if (tid == 0) {
      tc::fenceAfterSync();
      const uint32_t aHi = opBase, aLo = opBase + tc::kPanelBytes, bHi = opBase + 2 * tc::kPanelBytes,
                     bLo = opBase + 3 * tc::kPanelBytes;
      constexpr uint32_t idesc = tc::idescTf32(tc::kRows, tc::kRows);
      for (int sK = 0; sK < kTile / 8; ++sK) {
        const uint32_t o = (uint32_t)sK * 4096u;
        tc::mmaTf32(tmem, tc::smemDesc(aLo + o), tc::smemDesc(bHi + o), idesc, sK > 0);
        tc::mmaTf32(tmem, tc::smemDesc(aHi + o), tc::smemDesc(bLo + o), idesc, true);
      }
      for (int sK = 0; sK < kTile / 8; ++sK) {
        const uint32_t o = (uint32_t)sK * 4096u;
        tc::mmaTf32(tmem, tc::smemDesc(aHi + o), tc::smemDesc(bHi + o), idesc, true);
      }
      tc::commitTo(mbarMma);
    }
    // the product and this buffer's C tiles (bounded waits; one vote for the whole CTA)
    uint32_t& phLd = buf ? phLd1 : phLd0;
    bool ok = tc::mbarWait(mbarMma, phMma, kTcWaitNs);
    ok = tc::mbarWait(mbarLd[buf], phLd, kTcWaitNs) && ok;
    phMma ^= 1u;
    phLd ^= 1u;
    tc::fenceAfterSync();
    if (!__syncthreads_and(ok)) {
      // a wait ran out: give the copies and MMAs in flight one more period, then give up
      tc::mbarWait(mbarMma, phMma ^ 1u, kTcWaitNs);
      tc::mbarWait(mbarLd[buf ^ 1], buf ? phLd0 : phLd1, kTcWaitNs);
      if (tid == 0) tc::bulkWait0();
      __syncthreads();
      return false;
    }
    // C -= product: warp w reads TMEM lanes 32 (w % 4) .. +31 (its rows), columns 64 (w / 4) ..
    // +63, sixteen at a time
    {
      float* Cs = cPtr[buf];
      const int warp = tid >> 5, lane = tid & 31;
      if (warp < 8) {
        const int q = warp & 3, h = warp >> 2;
        const int R = 32 * q + lane;
        for (int cb = 0; cb < 4; ++cb) {
          float d[16];
          const int c0 = 64 * h + 16 * cb;
          tc::tmemLoad16(tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)c0, d);
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const int Cc = c0 + j;
            float& cref = Cs[((R >> 5) * 4 + (Cc >> 5)) * kTileElems + (Cc & 31) * kTileLd + (R & 31)];
            cref = cref - d[j];
          }
        }
      }
    }
    tc::fenceProxyAsyncShared();  // the updated tiles visible to the bulk stores
    tc::fenceBeforeSync();
    __syncthreads();
    if (tid == 0) {
      for (int t = 0; t < 16; ++t)
        if (sbTile(g, t))
          tc::bulkStore(M + tileBase(Tn, g.I0 + (t >> 2), g.K0 + (t & 3)), cAddr[buf] + (uint32_t)t * kTileBytes,
                        kTileBytes);
      tc::bulkCommit();
    }
  }
  if (tid == 0) {
    tc::bulkWait0();
    tc::fenceProxyAsyncGlobal();  // the stores before the grid barrier's generic release
  }
  __syncthreads();
  return true;
}

// tensor-core state of a CTA for the length of one factorisation job
struct TcState {
  unsigned char* stage;  // kGridTcStageBytes, 128-byte aligned
  uint32_t tmem, mbar;   // TMEM base; three mbarriers at mbar, mbar + 8, mbar + 16
  uint32_t phMma, phLd0, phLd1;
};

// Double-float trailing update on the tensor cores (tcgen05, kind::f16 with BF16 operands), over a
// pair of tile columns (J0, J0 + 1) at once: C_IK -= L_I,pair D_pair L_K,pair^T, K = 64, by an
// error-free split of the double-float operands into BF16 slices (the splitting scheme of Ozaki,
// Ogita, Oishi and Rump, Numer. Algorithms 59, 2012, on BF16 tensor products with FP32
// accumulation):
//  - each 64-wide row of the panels A = [L_I,J0 L_I,J0+1] and B = A D (the double-float products
//    of the tile routine) is scaled by a power of two 2^-e (e = 1 + the exponent of its largest
//    entry), so that every entry r lies in [-1, 1], and split as r = a_0 + a_1 + ... + a_5 + rest
//    with a_s = round(r_s 2^(8 s + 8)) 2^(-8 s - 8), r_0 = r, r_(s+1) = r_s - a_s: each a_s has at
//    most eight significant bits (a BF16 value), every subtraction is exact (Sterbenz), and the
//    rest is below 2^-48, the resolution of the double-float value (sliceRowPair, once per tile
//    row, by the warp that computed the row's second tile);
//  - a slice product a_i b_j is an integer multiple of 2^(-8(i + j) - 16) of at most 2^16, so a
//    sum of 64 of them over one, two or three pairs of one order i + j stays below 2^24, exact in
//    an FP32 accumulator: orders 0, 1, 2 accumulate exactly in three 128 x 128 TMEM accumulators,
//    orders 3 to 5 (whose rounding lies below 2^-48 of the product) in a fourth; the pairs of
//    order 6 and above are below 2^-48 and left out. 84 MMAs of 128 x 128 x 16 per super-block,
//    issued by one thread;
//  - the four accumulators are summed in double-float (error-free sums), scaled back by
//    2^(e_A + e_B) and subtracted from the C tiles in place in global memory.
// Against the double-float product on the CUDA cores the error bound changes from 2^-48 times the
// sum of |a_k b_k| to about 2^-45 times (max_k |a_k|)(max_k |b_k|); on quasi-definite roots with
// pivots spread over 1e20 the factor's componentwise backward error stays near 3e-14 (FP64:
// 8e-16).
//
// Slice area (global, `slices`, dfSliceBytes): for operand o (0 = A, 1 = B), slice s and k-group
// kg (8 of the 64 columns), the 16 bytes of root row m at ((o * 6 + s) * 8 + kg) * rows * 16 +
// m * 16, i.e. each (o, s, kg) plane holds the canonical shared-memory layout of cxg_tc.cuh for
// every row, so the 128 rows of a super-block are one contiguous copy per plane; then the row
// exponents, int32, at 1536 * rows + (o * rows + m) * 4.
constexpr int kDfSlices = 6;
constexpr int kDfK = 2 * kTile;                                          // columns per C visit
constexpr uint32_t kDfPanelBytes = (uint32_t)tc::kRows * kDfK * 2;       // 16 KB: 128 x 64 BF16
constexpr uint32_t kDfTmemCols = 512;                                    // four FP32 accumulators
constexpr uint32_t kDfOpBytes = 2 * kDfSlices * kDfPanelBytes;           // 192 KB of operands
constexpr uint32_t kDfExpBytes = 2 * tc::kRows * 4;                      // row exponents, A and B
constexpr int64_t kDfStageBytes = (int64_t)kDfOpBytes + 2 * kDfExpBytes; // one operand + two exponent buffers
static_assert(kDfStageBytes + 128 <= kGridTcStageBytes, "double-float staging exceeds the stage area");

// x 2^ex, by one exact multiplication where 2^ex is a normal float (scalbnf otherwise)
__device__ __forceinline__ float pow2Scale(float x, int ex) {
  if (ex >= -126 && ex <= 127) return __fmul_rn(x, __int_as_float((ex + 127) << 23));
  return scalbnf(x, ex);
}

// Writes the slices of the 32 rows of tile row I over the tile columns J0, J0 + 1 and their
// exponents, from the finished tiles L0 = L_I,J0 and L1 = L_I,J0+1 and the diagonal tiles A0, A1 of
// the two columns (all in shared memory); part q of f (f = 1, 2, 4 warps a tile row: both operands,
// one each, or half of one operand's k-groups), one warp, lane rr takes row 32 I + rr.
static __device__ __noinline__ void sliceRowPair(const df64* L0, const df64* L1, const df64* A0, const df64* A1, int Tn,
                                                 int I, unsigned char* slices, int q, int f) {
  const int rr = threadIdx.x & 31;
  const int64_t rows = (int64_t)Tn * kTile, m = (int64_t)I * kTile + rr;
  const df64* src[2] = {L0 + rr, L1 + rr};
  const df64* dg[2] = {A0, A1};
  const int kgLo = (f == 4 && q >= 2) ? kDfK / 16 : 0, kgHi = (f == 4 && q < 2) ? kDfK / 16 : kDfK / 8;
  for (int o = (f == 1) ? 0 : (q & 1); o < ((f == 1) ? 2 : (q & 1) + 1); ++o) {
    auto value = [&](int k) -> df64 {
      const int t = k >> 5, kk = k & 31;
      df64 x = src[t][kk * kTileLd];
      if (o) x = x * dg[t][kk * kTileLd + kk];
      return x;
    };
    float mx = 0.0f;
#pragma unroll 8
    for (int k = 0; k < kDfK; ++k) mx = fmaxf(mx, fabsf(value(k).hi));
    const int e = (mx > 0.0f && mx <= 3.0e38f) ? ilogbf(mx) + 1 : 0;
    reinterpret_cast<int*>(slices + 1536 * rows)[o * rows + m] = e;
#pragma unroll 1
    for (int kg = kgLo; kg < kgHi; ++kg) {
      uint32_t w[kDfSlices][4];
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        const df64 v = value(8 * kg + t);
        float rh = pow2Scale(v.hi, -e), rl = pow2Scale(v.lo, -e);
        float p = 256.0f, pinv = 1.0f / 256.0f;
#pragma unroll
        for (int sl = 0; sl < kDfSlices; ++sl) {
          const float as = __fmul_rn(rintf(__fmul_rn(rh, p)), pinv);  // exact: <= 8 significant bits
          const uint32_t bits = __float_as_uint(as) >> 16;               // its BF16 pattern
          if (t & 1) w[sl][t >> 1] |= bits << 16;
          else w[sl][t >> 1] = bits;
          dfTwoSum(__fsub_rn(rh, as), rl, rh, rl);
          p = __fmul_rn(p, 256.0f);
          pinv = __fmul_rn(pinv, 1.0f / 256.0f);
        }
      }
#pragma unroll
      for (int sl = 0; sl < kDfSlices; ++sl)
        *reinterpret_cast<uint4*>(slices + ((int64_t)(o * kDfSlices + sl) * (kDfK / 8) + kg) * rows * 16 + m * 16) =
            make_uint4(w[sl][0], w[sl][1], w[sl][2], w[sl][3]);
    }
  }
}

// The trailing update of column pair (J - 1, J) over the super-blocks this CTA owns (sb =
// blockIdx.x - 1, + gridDim.x - 1, ...; tile rows and columns from J + 1). Per super-block: its
// slices and exponents arrive by bulk copies (TMA); one thread issues its 84 MMAs; once they are
// complete the operand buffer holds the super-block's C tiles instead (bulk copies from HBM),
// which are updated there from the accumulators and written back by bulk copies; once those have
// read the buffer, the next super-block's slices are issued into it (the exponents alternate
// between two buffers). Shared memory `sm` (128-byte aligned): kDfStageBytes. `tmem`: this CTA's
// 512 accumulator columns; mbarriers: MMA completion, slice copies and C copies, with their phase
// parities. Returns false when a wait ran out (after waiting once more for what is in flight).
static __device__ __noinline__ bool tcDfTrailingStep(df64* M, int Tn, int J, long long nsb, const unsigned char* slices,
                                                     unsigned char* sm, uint32_t tmem, uint32_t mbarMma,
                                                     uint32_t mbarLd, uint32_t mbarC, uint32_t& phMma, uint32_t& phLd,
                                                     uint32_t& phC) {
  const int tid = threadIdx.x;
  const long long first = (long long)blockIdx.x - 1, stride = (long long)gridDim.x - 1;
  if (first >= nsb) return true;
  const int64_t rows = (int64_t)Tn * kTile;
  const uint32_t opAddr = tc::smemAddr(sm);
  const uint32_t expAddr[2] = {opAddr + kDfOpBytes, opAddr + kDfOpBytes + kDfExpBytes};
  constexpr int kPlanes = kDfSlices * (kDfK / 8);  // per operand
  constexpr uint32_t kTileBytesDf = (uint32_t)kTileElems * 8u;
  df64* Cs = reinterpret_cast<df64*>(sm);  // the C tiles, where the operands were
  // thread 0: the slices of super-block g's A rows (tiles I0 ..) and B rows (K0 ..), exponents
  // into exponent buffer eb
  auto issueOps = [&](const SbGeo& g, int eb) {
    const int nt[2] = {g.ni, g.nk};
    const int64_t row0[2] = {(int64_t)g.I0 * kTile, (int64_t)g.K0 * kTile};
    uint32_t bytes = 0;
    for (int o = 0; o < 2; ++o) bytes += (uint32_t)nt[o] * (kPlanes * 512 + 128);
    tc::mbarArriveExpectTx(mbarLd, bytes);
    for (int o = 0; o < 2; ++o) {
      for (int sl = 0; sl < kDfSlices; ++sl)
        for (int kg = 0; kg < kDfK / 8; ++kg)
          tc::bulkLoad(opAddr + (uint32_t)(o * kDfSlices + sl) * kDfPanelBytes + (uint32_t)kg * 2048u,
                       slices + ((int64_t)(o * kDfSlices + sl) * (kDfK / 8) + kg) * rows * 16 + row0[o] * 16,
                       (uint32_t)nt[o] * 512u, mbarLd);
      tc::bulkLoad(expAddr[eb] + (uint32_t)o * tc::kRows * 4, slices + 1536 * rows + (o * rows + row0[o]) * 4,
                   (uint32_t)nt[o] * 128u, mbarLd);
    }
  };
  // thread 0: super-block g's C tiles (tile t = 4 a + b at t x 8448 bytes) into the operand buffer
  auto issueC = [&](const SbGeo& g) {
    uint32_t bytes = 0;
    for (int t = 0; t < 16; ++t)
      if (sbTile(g, t)) bytes += kTileBytesDf;
    tc::mbarArriveExpectTx(mbarC, bytes);
    for (int t = 0; t < 16; ++t)
      if (sbTile(g, t))
        tc::bulkLoad(opAddr + (uint32_t)t * kTileBytesDf, M + tileBase(Tn, g.I0 + (t >> 2), g.K0 + (t & 3)),
                     kTileBytesDf, mbarC);
  };
  if (tid == 0) {
    tc::fenceProxyAsyncGlobal();  // the slices and C written this step (generic stores) before the copies
    issueOps(sbGeo(first, J, Tn), 0);
  }
  int eb = 0;
  for (long long sb = first; sb < nsb; sb += stride, eb ^= 1) {
    const SbGeo g = sbGeo(sb, J, Tn);
    const bool okLd = tc::mbarWait(mbarLd, phLd, kTcWaitNs);
    phLd ^= 1u;
    if (!__syncthreads_and(okLd)) {
      tc::mbarWait(mbarLd, phLd ^ 1u, kTcWaitNs);  // the copies in flight, once more
      __syncthreads();
      return false;
    }
    // the slice products into four accumulators, by one thread
    if (tid == 0) {
      tc::fenceAfterSync();
      constexpr uint32_t idesc = tc::idescBf16(tc::kRows, tc::kRows);
      bool used[4] = {false, false, false, false};
      for (int si = 0; si < kDfSlices; ++si)
        for (int sj = 0; si + sj < kDfSlices; ++sj) {
          const int o = min(si + sj, 3);
          const uint32_t d = tmem + (uint32_t)(o * tc::kRows);
          const uint32_t aAddr = opAddr + (uint32_t)si * kDfPanelBytes;
          const uint32_t bAddr = opAddr + (uint32_t)(kDfSlices + sj) * kDfPanelBytes;
          for (int sK = 0; sK < kDfK / 16; ++sK) {
            const uint32_t off = (uint32_t)sK * 4096u;
            tc::mmaBf16(d, tc::smemDesc(aAddr + off), tc::smemDesc(bAddr + off), idesc, used[o] || sK > 0);
          }
          used[o] = true;
        }
      tc::commitTo(mbarMma);
      // the C tiles into the operand buffer once the MMAs have read it
      const bool okM = tc::mbarWait(mbarMma, phMma, kTcWaitNs);
      if (okM) issueC(g);
    }
    const bool ok = tc::mbarWait(mbarMma, phMma, kTcWaitNs);
    phMma ^= 1u;
    const bool okC = ok && tc::mbarWait(mbarC, phC, kTcWaitNs);
    if (ok) phC ^= 1u;
    tc::fenceAfterSync();
    if (!__syncthreads_and(ok && okC)) {
      tc::mbarWait(mbarMma, phMma ^ 1u, kTcWaitNs);  // the MMAs and copies in flight, once more
      if (ok) tc::mbarWait(mbarC, phC ^ 1u, kTcWaitNs);
      __syncthreads();
      return false;
    }
    // C -= scaled sum of the accumulators, in shared memory: warp w owns TMEM lanes 32 (w % 4) ..
    // +31 (its rows) and columns 64 (w / 4) .. +63, eight at a time
    {
      const int warp = tid >> 5, lane = tid & 31;
      const int q = warp & 3, hh = (warp >> 2) & 1;
      const int R = 32 * q + lane;
      const int* expA = reinterpret_cast<const int*>(sm + kDfOpBytes + (uint32_t)eb * kDfExpBytes);
      const int* expB = expA + tc::kRows;
      const int eR = expA[R];
      const uint32_t lanes = (uint32_t)(32 * q) << 16;
#pragma unroll 2
      for (int cb = 0; cb < 8; ++cb) {
        const int c0 = 64 * hh + 8 * cb;
        float d[4][8];
        tc::tmemLoad8x4(tmem + lanes + (uint32_t)c0, (uint32_t)tc::kRows, d);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int Cc = c0 + j;
          float h, e1, h2, e2;
          dfTwoSum(d[0][j], d[1][j], h, e1);
          dfTwoSum(h, d[2][j], h2, e2);
          e1 = __fadd_rn(e1, e2);
          dfTwoSum(h2, d[3][j], h, e2);
          e1 = __fadd_rn(e1, e2);
          float sh, sl;
          dfFastTwoSum(h, e1, sh, sl);
          // x 2^(eR + eB) as two exact power-of-two factors, each within the normal range
          const int ex = eR + expB[Cc];
          const int ex1 = min(max(ex >> 1, -126), 127), ex2 = min(max(ex - (ex >> 1), -126), 127);
          const float f1 = __int_as_float((ex1 + 127) << 23), f2 = __int_as_float((ex2 + 127) << 23);
          const int t = 4 * (R >> 5) + (Cc >> 5);
          if (sbTile(g, t)) {
            df64& cref = Cs[t * kTileElems + (Cc & 31) * kTileLd + (R & 31)];
            cref = cref - df64(__fmul_rn(__fmul_rn(sh, f1), f2), __fmul_rn(__fmul_rn(sl, f1), f2));
          }
        }
      }
    }
    tc::fenceProxyAsyncShared();  // the updated tiles visible to the bulk stores
    tc::fenceBeforeSync();
    __syncthreads();  // TMEM read, the C tiles updated, this exponent buffer consumed
    if (tid == 0) {
      for (int t = 0; t < 16; ++t)
        if (sbTile(g, t))
          tc::bulkStore(M + tileBase(Tn, g.I0 + (t >> 2), g.K0 + (t & 3)), opAddr + (uint32_t)t * kTileBytesDf,
                        kTileBytesDf);
      tc::bulkCommit();
      tc::bulkWaitRead0();  // the stores have read the buffer: the next slices may land in it
      if (sb + stride < nsb) issueOps(sbGeo(sb + stride, J, Tn), eb ^ 1);
    }
  }
  if (tid == 0) {
    tc::bulkWait0();
    tc::fenceProxyAsyncGlobal();  // the stores before the grid barrier's generic release
  }
  __syncthreads();
  return true;
}

// FP32 trailing update on the tensor cores over a pair of tile columns (J0, J0 + 1): C_IK -=
// L_I,pair D_pair L_K,pair^T with K = 64, as three TF32 products A_hi B_lo + A_lo B_hi + A_hi B_hi
// (each FP32 operand x split as hi = tf32(x), lo = tf32(x - hi)) into one FP32 TMEM accumulator:
// 24 MMAs of 128 x 128 x 8 per super-block, issued by one thread.
//
// Panel area (global, `slices`, within dfSliceBytes): for operand o (0 = A = L, 1 = B = L D), part
// p (0 = hi, 1 = lo) and k-group kg (4 of the 64 columns), the 16 bytes of root row m at
// ((o * 2 + p) * 16 + kg) * rows * 16 + m * 16: each (o, p, kg) plane is the canonical
// shared-memory layout of cxg_tc.cuh for every row, so the 128 rows of a super-block are one
// contiguous copy per plane.
constexpr int kF32Parts = 2;
constexpr int kF32Groups = kDfK / 4;                                     // 16-byte k-groups per row
constexpr uint32_t kF32PanelBytes = (uint32_t)tc::kRows * kDfK * 4;      // 32 KB: 128 x 64 TF32
constexpr uint32_t kF32OpBytes = 2 * kF32Parts * kF32PanelBytes;         // 128 KB of operands
constexpr int64_t kF32StageBytes = (int64_t)kF32OpBytes + 16 * (int64_t)kTileBytes;  // operands + C tiles
static_assert(kF32StageBytes + 128 <= kGridTcStageBytes, "FP32 pair staging exceeds the stage area");
static_assert(2 * kF32Parts * kF32Groups * 16 <= 2 * kDfSlices * (kDfK / 8) * 16, "FP32 panels exceed the slice area");

// Writes the TF32 parts of the 32 rows of tile row I over the tile columns J0, J0 + 1; arguments as
// for the double-float form.
static __device__ __noinline__ void sliceRowPair(const float* L0, const float* L1, const float* A0, const float* A1,
                                                 int Tn, int I, unsigned char* slices, int q, int f) {
  const int rr = threadIdx.x & 31;
  const int64_t rows = (int64_t)Tn * kTile, m = (int64_t)I * kTile + rr;
  const float* src[2] = {L0 + rr, L1 + rr};
  const float* dg[2] = {A0, A1};
  const int kgLo = (f == 4 && q >= 2) ? kF32Groups / 2 : 0, kgHi = (f == 4 && q < 2) ? kF32Groups / 2 : kF32Groups;
  for (int o = (f == 1) ? 0 : (q & 1); o < ((f == 1) ? 2 : (q & 1) + 1); ++o) {
#pragma unroll 2
    for (int kg = kgLo; kg < kgHi; ++kg) {
      float hi[4], lo[4];
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const int k = 4 * kg + t, tt = k >> 5, kk = k & 31;
        float x = src[tt][kk * kTileLd];
        if (o) x = x * dg[tt][kk * kTileLd + kk];
        hi[t] = tc::toTf32(x);
        lo[t] = tc::toTf32(x - hi[t]);
      }
      *reinterpret_cast<float4*>(slices + ((int64_t)(o * kF32Parts) * kF32Groups + kg) * rows * 16 + m * 16) =
          make_float4(hi[0], hi[1], hi[2], hi[3]);
      *reinterpret_cast<float4*>(slices + ((int64_t)(o * kF32Parts + 1) * kF32Groups + kg) * rows * 16 + m * 16) =
          make_float4(lo[0], lo[1], lo[2], lo[3]);
    }
  }
}

// The FP32 trailing update of column pair (J - 1, J) over the super-blocks this CTA owns (sb =
// blockIdx.x - 1, + gridDim.x - 1, ...). Shared memory `sm` (128-byte aligned, kF32StageBytes)
// holds an operand buffer (the TF32 parts, by bulk copies from the panel area) and a C buffer (the
// super-block's C tiles, by bulk copies from the root). Per super-block: one thread issues the 24
// MMAs; once they have read the operands, the next super-block's operands are issued into that
// buffer; the C tiles are updated from the accumulator and written back by bulk stores; once
// those have read the C buffer, the next super-block's C tiles are issued into it. So the operand
// copies overlap the epilogue and the C copies the next MMAs. `tmem`: this CTA's 128 accumulator
// columns. Returns false when a wait ran out (after waiting once more for what is in flight).
static __device__ __noinline__ bool tcF32PairTrailingStep(float* M, int Tn, int J, long long nsb,
                                                          const unsigned char* slices, unsigned char* sm, uint32_t tmem,
                                                          uint32_t mbarMma, uint32_t mbarLd, uint32_t mbarC,
                                                          uint32_t& phMma, uint32_t& phLd, uint32_t& phC) {
  const int tid = threadIdx.x;
  const long long first = (long long)blockIdx.x - 1, stride = (long long)gridDim.x - 1;
  if (first >= nsb) return true;
  const int64_t rows = (int64_t)Tn * kTile;
  const uint32_t opAddr = tc::smemAddr(sm), cAddr = opAddr + kF32OpBytes;
  float* Cs = reinterpret_cast<float*>(sm + kF32OpBytes);
  // thread 0: the TF32 parts of super-block g's A rows (tiles I0 ..) and B rows (K0 ..)
  auto issueOps = [&](const SbGeo& g) {
    const int nt[2] = {g.ni, g.nk};
    const int64_t row0[2] = {(int64_t)g.I0 * kTile, (int64_t)g.K0 * kTile};
    uint32_t bytes = 0;
    for (int o = 0; o < 2; ++o) bytes += (uint32_t)nt[o] * (uint32_t)(kF32Parts * kF32Groups * 512);
    tc::mbarArriveExpectTx(mbarLd, bytes);
    for (int o = 0; o < 2; ++o)
      for (int p = 0; p < kF32Parts; ++p)
        for (int kg = 0; kg < kF32Groups; ++kg)
          tc::bulkLoad(opAddr + (uint32_t)(o * kF32Parts + p) * kF32PanelBytes + (uint32_t)kg * 2048u,
                       slices + ((int64_t)(o * kF32Parts + p) * kF32Groups + kg) * rows * 16 + row0[o] * 16,
                       (uint32_t)nt[o] * 512u, mbarLd);
  };
  // thread 0: super-block g's C tiles (tile t = 4 a + b at t x kTileBytes) into the C buffer
  auto issueC = [&](const SbGeo& g) {
    uint32_t bytes = 0;
    for (int t = 0; t < 16; ++t)
      if (sbTile(g, t)) bytes += kTileBytes;
    tc::mbarArriveExpectTx(mbarC, bytes);
    for (int t = 0; t < 16; ++t)
      if (sbTile(g, t))
        tc::bulkLoad(cAddr + (uint32_t)t * kTileBytes, M + tileBase(Tn, g.I0 + (t >> 2), g.K0 + (t & 3)), kTileBytes,
                     mbarC);
  };
  if (tid == 0) {
    tc::fenceProxyAsyncGlobal();  // the panels and C written this step (generic stores) before the copies
    const SbGeo g0 = sbGeo(first, J, Tn);
    issueOps(g0);
    issueC(g0);
  }
  for (long long sb = first; sb < nsb; sb += stride) {
    const SbGeo g = sbGeo(sb, J, Tn);
    const bool more = sb + stride < nsb;
    const bool okLd = tc::mbarWait(mbarLd, phLd, kTcWaitNs);
    phLd ^= 1u;
    if (!__syncthreads_and(okLd)) {
      tc::mbarWait(mbarLd, phLd ^ 1u, kTcWaitNs);  // the copies in flight, once more
      tc::mbarWait(mbarC, phC, kTcWaitNs);
      __syncthreads();
      return false;
    }
    if (tid == 0) {
      tc::fenceAfterSync();
      constexpr uint32_t idesc = tc::idescTf32(tc::kRows, tc::kRows);
      const uint32_t aHi = opAddr, aLo = opAddr + kF32PanelBytes, bHi = opAddr + 2 * kF32PanelBytes,
                     bLo = opAddr + 3 * kF32PanelBytes;
      for (int sK = 0; sK < kDfK / 8; ++sK) {
        const uint32_t o = (uint32_t)sK * 4096u;
        tc::mmaTf32(tmem, tc::smemDesc(aLo + o), tc::smemDesc(bHi + o), idesc, sK > 0);
        tc::mmaTf32(tmem, tc::smemDesc(aHi + o), tc::smemDesc(bLo + o), idesc, true);
      }
      for (int sK = 0; sK < kDfK / 8; ++sK) {
        const uint32_t o = (uint32_t)sK * 4096u;
        tc::mmaTf32(tmem, tc::smemDesc(aHi + o), tc::smemDesc(bHi + o), idesc, true);
      }
      tc::commitTo(mbarMma);
      // the next super-block's operands once the MMAs have read this one's
      const bool okM = tc::mbarWait(mbarMma, phMma, kTcWaitNs);
      if (okM && more) issueOps(sbGeo(sb + stride, J, Tn));
    }
    const bool ok = tc::mbarWait(mbarMma, phMma, kTcWaitNs);
    phMma ^= 1u;
    const bool okC = ok && tc::mbarWait(mbarC, phC, kTcWaitNs);
    if (ok) phC ^= 1u;
    tc::fenceAfterSync();
    if (!__syncthreads_and(ok && okC)) {
      tc::mbarWait(mbarMma, phMma ^ 1u, kTcWaitNs);  // the MMAs and copies in flight, once more
      if (ok) tc::mbarWait(mbarC, phC ^ 1u, kTcWaitNs);
      if (ok && more) tc::mbarWait(mbarLd, phLd, kTcWaitNs);
      __syncthreads();
      return false;
    }
    // C -= product, in shared memory: warp w reads TMEM lanes 32 (w % 4) .. +31 (its rows),
    // columns 64 (w / 4) .. +63, sixteen at a time
    {
      const int warp = tid >> 5, lane = tid & 31;
      if (warp < 8) {
        const int q = warp & 3, h = warp >> 2;
        const int R = 32 * q + lane;
        for (int cb = 0; cb < 4; ++cb) {
          float d[16];
          const int c0 = 64 * h + 16 * cb;
          tc::tmemLoad16(tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)c0, d);
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const int Cc = c0 + j;
            float& cref = Cs[((R >> 5) * 4 + (Cc >> 5)) * kTileElems + (Cc & 31) * kTileLd + (R & 31)];
            cref = cref - d[j];
          }
        }
      }
    }
    tc::fenceProxyAsyncShared();  // the updated tiles visible to the bulk stores
    tc::fenceBeforeSync();
    __syncthreads();  // TMEM read, the C tiles updated
    if (tid == 0) {
      for (int t = 0; t < 16; ++t)
        if (sbTile(g, t))
          tc::bulkStore(M + tileBase(Tn, g.I0 + (t >> 2), g.K0 + (t & 3)), cAddr + (uint32_t)t * kTileBytes,
                        kTileBytes);
      tc::bulkCommit();
      tc::bulkWaitRead0();  // the stores have read the C buffer: the next C tiles may land in it
      if (more) issueC(sbGeo(sb + stride, J, Tn));
    }
  }
  if (tid == 0) {
    tc::bulkWait0();
    tc::fenceProxyAsyncGlobal();  // the stores before the grid barrier's generic release
  }
  __syncthreads();
  return true;
}

// Copies one tile between global and shared memory (16-byte vectors), thread t of nt.
template <typename T>
__device__ __forceinline__ void copyTile(T* dst, const T* src, int t, int nt) {
  constexpr int nv = kTileElems * (int)sizeof(T) / 16;
#pragma unroll 4
  for (int v = t; v < nv; v += nt) reinterpret_cast<uint4*>(dst)[v] = reinterpret_cast<const uint4*>(src)[v];
}

// Shared-memory tiles of a CTA in the whole-GPU factor's column phases: the pivot reciprocals of
// the diagonal tile(s), up to three tiles for the whole CTA, then two per team of warps.
template <typename T>
struct ColStage {
  T *inv0, *inv1, *t0, *t1, *t2, *team;
};
template <typename T>
__device__ __forceinline__ ColStage<T> colStage(T* stage) {
  T* t = stage + 64;
  return {stage, stage + 32, t, t + kTileElems, t + 2 * kTileElems, t + 3 * kTileElems};
}

// Warps per tile in a column phase with `rem` tiles on GW warps: four, two or one, as many as fit.
__device__ __forceinline__ int teamWarps(int rem, int GW) { return 4 * rem <= GW ? 4 : (2 * rem <= GW ? 2 : 1); }

// Named barrier of one team of f warps (ids 4 ..; f is 2 or 4, eight warps a CTA).
__device__ __forceinline__ void teamSync(int team, int f) {
  if (f == 1) __syncwarp();
  else asm volatile("bar.sync %0, %1;" ::"r"(4 + team), "r"(32 * f) : "memory");
}

// The column groups of warp q in a team of f: one (f = 4), two of together five units (f = 2) or
// all four, last first (f = 1); src and dst may be the same tile only for f = 1.
template <typename T>
__device__ __forceinline__ void teamOffDiag(const T* src, T* dst, const T* Ajj, const T* invD, int q, int f) {
#pragma unroll 1
  for (int i = 0; i < 4 / f; ++i) {
    const int g = (f == 4) ? q : (f == 2) ? (q ? 1 + i : 3 * i) : 3 - i;
    T o[8];
    tileOffDiagGroup(src, Ajj, invD, g, o);
    if (f == 1) __syncwarp();
    tileOffDiagStore(dst, g, o);
    if (f == 1) __syncwarp();
  }
}

// Column J's off-diagonal tiles I >= I0 on warps w0 .. GW-1 of the grid (gw this warp's number):
// the CTA's tiles are read into shared memory and the results written to global memory.
template <typename T>
__device__ __noinline__ void gridOffDiag(T* M, int Tn, int I0, int J, int w0, int gw, int GW, const ColStage<T>& cs) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int f = teamWarps(Tn - I0, GW - w0), first = (gw - warp - w0) / f;  // this CTA's first team
  if (gw - warp < w0 || I0 + first >= Tn) return;
  const T* Ajj = M + tileBase(Tn, J, J);
  copyTile(cs.t0, Ajj, (int)threadIdx.x, (int)blockDim.x);
  if (warp == 0) cs.inv0[lane] = recipT(Ajj[lane * kTileLd + lane]);
  const int team = warp / f, q = warp % f;
  T* A = cs.team + 2 * team * kTileElems;
  int I = I0 + first + team;
  if (I < Tn) copyTile(A, M + tileBase(Tn, I, J), q * 32 + lane, 32 * f);
  __syncthreads();
  for (; I < Tn; I += (GW - w0) / f) {
    T* dst = M + tileBase(Tn, I, J);
    if (f == 1) {
      for (int g = 3; g >= 0; --g) {
        T o[8];
        tileOffDiagGroup(A, cs.t0, cs.inv0, g, o);
        tileOffDiagStore(dst, g, o);
      }
      __syncwarp();
      const int In = I + (GW - w0);
      if (In < Tn) copyTile(A, M + tileBase(Tn, In, J), lane, 32);
      __syncwarp();
    } else {
      teamOffDiag(A, dst, cs.t0, cs.inv0, q, f);
    }
  }
  tc::fenceProxyAsyncShared();  // these accesses before the trailing update's bulk copies into the area
}

// CTA 0 with its eight warps: tile (J, J) of the root into cs.t2, updated by the columns whose
// off-diagonal tiles L_J,K and diagonal tiles A_KK are given (global; the second may be null),
// factored and written back.
template <typename T>
__device__ __noinline__ void gridNextDiag(T* M, int Tn, int J, const T* L0, const T* A0, const T* L1, const T* A1,
                                          int nr, int nx, const DevSettings& st, PivotStats* ps,
                                          const ColStage<T>& cs) {
  const int warp = threadIdx.x >> 5, tid = threadIdx.x, nt = blockDim.x;
  T* An = M + tileBase(Tn, J, J);
  copyTile(cs.t2, An, tid, nt);
  __syncthreads();
  for (int h = 0; h < 2; ++h) {
    const T* L = h ? L1 : L0;
    if (!L) break;
    copyTile(cs.t1, L, tid, nt);
    copyTile(cs.t0, h ? A1 : A0, tid, nt);
    __syncthreads();
    if (warp < 6) tileSyrkDiagUnit<T>(cs.t2, cs.t1, cs.t0, warp);
    __syncthreads();
  }
  if (warp < 4) tileFactorDiag<T>(cs.t2, J, nr, nx, st, ps, cs.inv0, 4);
  __syncthreads();
  copyTile(An, cs.t2, tid, nt);
  __syncthreads();
}

// Whole-GPU FP32 and double-float LDL' over pairs of tile columns (J0, J1 = J0 + 1), three grid
// barriers per pair; in the column phases a tile's work is shared by up to four warps, on copies
// in shared memory:
//  (A0) the off-diagonal tiles of column J0; CTA 0 takes L_J1,J0, then updates the diagonal tile
//       (J1, J1) with it and factors it;
//  (A1) column J1's tiles I > J1: the update by column J0 (tile routine), L_I,J1, and the
//       tensor-core operands of the row pair (sliceRowPair: TF32 parts for FP32, BF16 slices for
//       double-float);
//  (B)  the trailing update of both columns at once (tcF32PairTrailingStep / tcDfTrailingStep,
//       CTAs 1..), while CTA 0 updates the diagonal tile (J1 + 1, J1 + 1) with both columns and
//       factors it.
// Only CTA 0 factors diagonal tiles, so the pivot statistics stay in its shared memory.
template <typename T>
__device__ __noinline__ bool gridLdltPairs(GridCtl* g, int nr, int nx, const DevSettings& st, T* M, PivotStats* ps,
                                           T* stage, unsigned char* slices, int Tn, int warp, int gw, int GW, bool cta0,
                                           TcState& tcs) {
  const ColStage<T> cs = colStage(stage);
  const int W = blockDim.x >> 5, tid = threadIdx.x, lane = tid & 31;
  if (cta0) gridNextDiag<T>(M, Tn, 0, nullptr, nullptr, nullptr, nullptr, nr, nx, st, ps, cs);
  if (!gridSync(g)) return false;
  for (int J0 = 0; J0 + 1 < Tn; J0 += 2) {
    const int J1 = J0 + 1;
    const T* A0 = M + tileBase(Tn, J0, J0);
    const T* A1 = M + tileBase(Tn, J1, J1);
    // (A0)
    if (cta0) {
      T* L10 = M + tileBase(Tn, J1, J0);
      copyTile(cs.t0, A0, tid, (int)blockDim.x);
      copyTile(cs.t1, L10, tid, (int)blockDim.x);
      if (warp == 0) cs.inv0[lane] = recipT(A0[lane * kTileLd + lane]);
      __syncthreads();
      if (warp < 4) teamOffDiag(cs.t1, L10, cs.t0, cs.inv0, warp, 4);
      __syncthreads();
      gridNextDiag<T>(M, Tn, J1, L10, A0, nullptr, nullptr, nr, nx, st, ps, cs);
    } else {
      gridOffDiag<T>(M, Tn, J1 + 1, J0, W, gw, GW, cs);
    }
    if (!gridSync(g)) return false;
    // (A1)
    const int f = teamWarps(Tn - J1 - 1, GW), team = warp / f, q = warp % f, first = (gw - warp) / f;
    if (J1 + 1 + first < Tn) {
      T *C = cs.team + 2 * team * kTileElems, *L0 = C + kTileElems;
      copyTile(cs.t0, A0, tid, (int)blockDim.x);
      copyTile(cs.t1, A1, tid, (int)blockDim.x);
      copyTile(cs.t2, M + tileBase(Tn, J1, J0), tid, (int)blockDim.x);
      if (warp == 0) cs.inv1[lane] = recipT(A1[lane * kTileLd + lane]);
      __syncthreads();
      for (int I = J1 + 1 + first + team; I < Tn; I += GW / f) {
        T* dst = M + tileBase(Tn, I, J1);
        copyTile(C, dst, q * 32 + lane, 32 * f);
        copyTile(L0, M + tileBase(Tn, I, J0), q * 32 + lane, 32 * f);
        teamSync(team, f);
        for (int h = q; h < 2; h += f) tileSyrkHalf<T>(C, L0, cs.t2, cs.t0, h);
        teamSync(team, f);
        T o0[8], o1[8];
        if (f == 1) {
          teamOffDiag(C, C, cs.t1, cs.inv1, 0, 1);
        } else {
          const int g0 = (f == 4) ? q : (q ? 1 : 0), g1 = q ? 2 : 3;
          tileOffDiagGroup(C, cs.t1, cs.inv1, g0, o0);
          if (f == 2) tileOffDiagGroup(C, cs.t1, cs.inv1, g1, o1);
          teamSync(team, f);
          tileOffDiagStore(C, g0, o0);
          if (f == 2) tileOffDiagStore(C, g1, o1);
          teamSync(team, f);
        }
        copyTile(dst, C, q * 32 + lane, 32 * f);
        sliceRowPair(L0, C, cs.t0, cs.t1, Tn, I, slices, q, f);
        teamSync(team, f);
      }
      tc::fenceProxyAsyncShared();  // these accesses before the trailing update's bulk copies into the area
    }
    if (!gridSync(g)) return false;
    if (J1 + 1 >= Tn) break;
    // (B)
    const int rem = Tn - J1 - 1;
    const int nb = (rem + 3) >> 2;
    const long long nsb = (long long)nb * (nb + 1) / 2;
    if (cta0) {
      gridNextDiag<T>(M, Tn, J1 + 1, M + tileBase(Tn, J1 + 1, J0), A0, M + tileBase(Tn, J1 + 1, J1), A1, nr, nx, st, ps,
                      cs);
    } else {
      bool okT;
      if constexpr (sizeof(T) == 4)
        okT = tcF32PairTrailingStep(M, Tn, J1, nsb, slices, tcs.stage, tcs.tmem, tcs.mbar, tcs.mbar + 8u,
                                    tcs.mbar + 16u, tcs.phMma, tcs.phLd0, tcs.phLd1);
      else
        okT = tcDfTrailingStep(M, Tn, J1, nsb, slices, tcs.stage, tcs.tmem, tcs.mbar, tcs.mbar + 8u, tcs.mbar + 16u,
                               tcs.phMma, tcs.phLd0, tcs.phLd1);
      if (!okT) {
        if (threadIdx.x == 0) atomicExch(&g->error, 1);
        return false;
      }
    }
    if (!gridSync(g)) return false;
  }
  return true;
}

// Tiled right-looking LDL' of the root over the whole grid. Per tile column J:
//  (A) the off-diagonal tiles of column J, up to four warps each; barrier;
//  (B) the trailing update C_IK -= L_IJ D_J L_KJ^T, J < K <= I, on CTAs 1.. (FP32: super-blocks of 4x4
//      tiles on the tensor cores, tcTrailingStep; FP64 and double-float: tile by tile on the CUDA
//      cores, gridTileUpdate), while CTA 0 updates the tile (J+1, J+1) with the tile routine and
//      factors it (one-column lookahead); barrier.
// In FP64 every root entry receives its updates in increasing J with the same operations and
// rounding as the single-CTA factor, so both give the same bits. Only CTA 0 factors diagonal
// tiles, so the pivot statistics stay in its shared memory (ps). `stage` holds
// kGridStageBytes. Large FP32 and double-float roots run over column pairs instead (gridLdltPairs).
template <typename T>
__device__ __noinline__ bool gridLdltSteps(GridCtl* g, int nr, int nx, const DevSettings& st, T* M, PivotStats* ps,
                                           T* stage, unsigned char* slices, int Tn, int warp, int gw, int GW, bool cta0,
                                           TcState& tcs);

// Roots of at least this many tile columns factor over column pairs (gridLdltPairs): half the C
// traffic of the trailing update, but a longer serial chain per pair. Below it, one column at a
// time (gridLdltSteps: FP32 on the tensor cores, double-float on the CUDA cores). The thresholds
// were the measured crossovers of the two forms on GB300. Pairs win earlier now (double-float 5.6
// against 4.8 ms at 3072 rows, 2.8 against 3.1 ms at 2048; FP32 13.7 against 12.2 ms at 8192), but below
// the thresholds the one-column products' smaller error stays what it was.
constexpr int kPairMinTilesF32 = 352;  // 11264 rows
constexpr int kPairMinTilesDf = 160;   // 5120 rows
template <typename T>
__device__ __forceinline__ constexpr int pairMinTiles() {
  return (ArithOf<T>::v == 1) ? kPairMinTilesF32 : kPairMinTilesDf;
}

// `slices`: the tensor-core panel area of the FP32 and double-float pair forms (dfSliceBytes(nr),
// 16-byte aligned); unused by FP64.
template <typename T>
__device__ __noinline__ bool gridLdlt(GridCtl* g, int nr, int nx, const DevSettings& st, T* M, PivotStats* ps, T* stage,
                                      unsigned char* slices) {
  const int Tn = rootTiles(nr);
  const int warp = threadIdx.x >> 5, W = blockDim.x >> 5;
  const int gw = (int)blockIdx.x * W + warp, GW = (int)gridDim.x * W;
  const bool cta0 = blockIdx.x == 0;
  // FP32 and double-float: the super-blocks go to the tensor cores; every CTA but 0 holds TMEM
  // (128 columns for FP32, 512 for double-float) and the mbarriers for the length of the job
  constexpr bool kTc = ArithOf<T>::v != 0;
  constexpr uint32_t kCols = (ArithOf<T>::v == 2) ? kDfTmemCols : tc::kTmemCols;
  __shared__ __align__(8) unsigned long long sMbar[3];  // MMA completion, C buffer 0, C buffer 1
  __shared__ uint32_t sTmem;
  TcState tcs{};
  tcs.mbar = tc::smemAddr(&sMbar[0]);
  tcs.stage = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(stage) + 127) & ~static_cast<uintptr_t>(127));
  if (kTc && !cta0) {
    if (warp == 0) tc::tmemAlloc(tc::smemAddr(&sTmem), kCols);
    if (threadIdx.x == 32)
      for (int i = 0; i < 3; ++i) tc::mbarInit(tcs.mbar + 8u * i, 1);
    tc::fenceBeforeSync();
    __syncthreads();
    tc::fenceAfterSync();
    tcs.tmem = sTmem;
  }
  bool ok = false;
  if constexpr (kTc) {
    if (Tn >= pairMinTiles<T>()) ok = gridLdltPairs<T>(g, nr, nx, st, M, ps, stage, slices, Tn, warp, gw, GW, cta0, tcs);
  }
  if (!kTc || Tn < pairMinTiles<T>())
    ok = gridLdltSteps<T>(g, nr, nx, st, M, ps, stage, slices, Tn, warp, gw, GW, cta0, tcs);
  if (kTc && !cta0) {
    tc::fenceBeforeSync();
    __syncthreads();
    if (warp == 0) tc::tmemDealloc(tcs.tmem, kCols);
    if (threadIdx.x == 32)
      for (int i = 0; i < 3; ++i) tc::mbarInval(tcs.mbar + 8u * i);
  }
  return ok;
}

template <typename T>
__device__ __noinline__ bool gridLdltSteps(GridCtl* g, int nr, int nx, const DevSettings& st, T* M, PivotStats* ps,
                                           T* stage, unsigned char* slices, int Tn, int warp, int gw, int GW, bool cta0,
                                           TcState& tcs) {
  const ColStage<T> cs = colStage(stage);
  if (cta0) gridNextDiag<T>(M, Tn, 0, nullptr, nullptr, nullptr, nullptr, nr, nx, st, ps, cs);
  if (!gridSync(g)) return false;
  for (int J = 0; J + 1 < Tn; ++J) {
    T* Ajj = M + tileBase(Tn, J, J);
    gridOffDiag<T>(M, Tn, J + 1, J, 0, gw, GW, cs);
    if (!gridSync(g)) return false;
    const int rem = Tn - J - 1;
    const int nb = (rem + 3) >> 2;
    const long long nsb = (long long)nb * (nb + 1) / 2;
    // CTA 0 updates and factors the next diagonal tile (J+1, J+1), the critical path of the next
    // column; the rest of the update goes to CTAs 1.. cyclically
    if (cta0) {
      gridNextDiag<T>(M, Tn, J + 1, M + tileBase(Tn, J + 1, J), Ajj, nullptr, nullptr, nr, nx, st, ps, cs);
      if (!gridSync(g)) return false;
      continue;
    }
    if constexpr (sizeof(T) == 4) {
      if (!tcTrailingStep(M, Tn, J, nsb, tcs.stage, tcs.tmem, tcs.mbar, tcs.mbar + 8u, tcs.mbar + 16u, tcs.phMma,
                          tcs.phLd0, tcs.phLd1)) {
        if (threadIdx.x == 0) atomicExch(&g->error, 1);
        return false;
      }
    } else {
      gridTileUpdate<T>(M, Tn, J, stage);
    }
    if (!gridSync(g)) return false;
  }
  return true;
}

// ---- triangular solves over the grid --------------------------------------------------------------
// y <- M^-1 y as a dataflow over row tiles, without grid barriers inside. Each warp owns up to
// kSolveRows row tiles (a CTA a run of consecutive ones) and keeps their part of y in registers. It
// applies the solved tiles x_j to its rows in order (forward: j ascending, backward: descending), as
// they are published, solves its own tile when its turn comes and publishes it: within the CTA
// through shared memory, to the others in y with a flag per tile. Its tiles of the root arrive by
// asynchronous copies, two ahead of the one in use. So a tile step is one product and one diagonal
// solve, and only every eighth one a hand-over between SMs. Measured a step: FP32 1.5 us, double-float
// 2.9, FP64 3.4 (1020 rows, 2 x 32 steps: 94, 188 and 219 us; 6400 rows: 0.59, 1.14 and 1.37 ms), of
// which a product's arithmetic is a small part; in blocks of four tiles with a grid barrier each it was
// 17 us a block, mostly tiles read from L2 on the critical path.
// Every y tile takes its updates one source tile at a time in the same order as before.
constexpr int kSolveRows = 4;   // row tiles a warp owns at a time, at most
constexpr int kSolveBufs = 3;   // tile buffers of a warp
// FP64: four owners a CTA, one per sub-partition (a product holds the FP64 unit for 2000 cycles).
template <typename T>
__device__ __forceinline__ constexpr int solveWarps() { return ArithOf<T>::v == 0 ? 4 : 8; }

// Number of tiles solved in a row from tile j on (direction `step`, at most 32 and up to `last`
// exclusive), at least one: waits for tile j. The lanes read one flag each. 0 when the wait ran out or
// the launch has failed; bounded as gridSync is.
static __device__ __forceinline__ int waitTiles(GridCtl* g, const int* flags, int j, int last, int step, int epoch) {
  const int mine = j + step * (int)(threadIdx.x & 31);
  const bool in = step > 0 ? mine < last : mine > last;
  unsigned long long t0 = 0;
  for (int spin = 0;; ++spin) {
    int v = epoch - 1;
    if (in) asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(flags + mine) : "memory");
    const unsigned open = ~__ballot_sync(0xffffffffu, v == epoch);
    const int ready = open ? __ffs(open) - 1 : 32;
    if (ready > 0) {
      __syncwarp();  // what one lane's flag opens, the others read
      return ready;
    }
    if ((spin & 63) == 63) {
      volatile GridCtl* vg = g;
      const unsigned long long now = globalNs();
      unsigned long long limit = vg->waitNs;
      if (limit == 0) limit = kGridWaitNs;
      if (t0 == 0) t0 = now;
      const bool late = now - t0 > limit;
      if (late && (threadIdx.x & 31) == 0) atomicExch(&g->error, 1);
      if (__any_sync(0xffffffffu, late || vg->error)) return 0;
    }
    __nanosleep(20);
  }
}

// Publishes a solved tile: this lane's entry into y, then the tile's flag.
template <typename T>
__device__ __forceinline__ void publishTile(T* yJ, int* f, int epoch, T x) {
  const int lane = threadIdx.x & 31;
  yJ[lane] = x;
  __syncwarp();
  if (lane == 0) {
    __threadfence();
    asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(f), "r"(epoch) : "memory");
  }
}

__device__ __forceinline__ float loadL2(const float* p) { return __ldcg(p); }
__device__ __forceinline__ double loadL2(const double* p) { return __ldcg(p); }
__device__ __forceinline__ df64 loadL2(const df64* p) {
  const float2 v = __ldcg(reinterpret_cast<const float2*>(p));
  return df64(v.x, v.y);
}

// One row's part of Linv_JJ y_J (forward) or Linv_JJ^T y_J (backward): terms k < i or k > i in four
// sums of eight, added pairwise. A: the diagonal tile, yb: y_J (shared), lane = row i.
template <bool kForward, typename T>
__device__ __forceinline__ T diagPart(const T* A, const T* yb) {
  const int i = threadIdx.x & 31;
  T v[4];
#pragma unroll
  for (int p = 0; p < 4; ++p) v[p] = (T)0;
#pragma unroll 2
  for (int t = 0; t < 8; ++t) {
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const int k = 8 * p + t;
      const T a = kForward ? A[i * kTileLd + k] : A[k * kTileLd + i];
      if (kForward ? k < i : k > i) v[p] = accT(v[p], a, yb[k]);
    }
  }
  return (accEnd(v[0]) + accEnd(v[1])) + (accEnd(v[2]) + accEnd(v[3]));
}

// One pass (forward or backward) for the calling CTA's row tiles first .. end-1; yv: this lane's
// entries of the warp's rows. All warps of the CTA call it. xs (shared): two solved tiles of the CTA,
// the tile being solved, then one source tile per warp.
template <bool kForward, typename T>
__device__ __forceinline__ bool solvePass(GridCtl* g, int Tn, const T* M, T* y, int first, int end, int epoch, T* bufs,
                                          T* xs, T (&yv)[kSolveRows]) {
  constexpr int W = solveWarps<T>();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool owner = warp < W;
  int* flags = g->flags + (kForward ? 0 : kGridMaxTiles);
  T* buf = bufs + (int64_t)warp * kSolveBufs * kTileElems;
  auto rowOf = [&](int r) { return first + r * W + warp; };
  // this warp's tiles in the order it uses them: source j outermost (forward 0 .., backward Tn-1 ..),
  // then its rows from the one nearest to j on (j itself first: the diagonal tile)
  const int jEnd = kForward ? end : first - 1, jStep = kForward ? 1 : -1;
  auto uses = [&](int j, int r) {
    const int I = rowOf(r);
    return owner && I < end && (kForward ? I >= j : I <= j);
  };
  int nj = kForward ? 0 : Tn - 1, nrr = 0, issued = 0;  // the next tile to copy: source nj, row index nrr in order
  auto issueNext = [&]() {
    while (nj != jEnd) {
      const int r = kForward ? nrr : kSolveRows - 1 - nrr;
      const int j = nj;
      if (++nrr == kSolveRows) { nrr = 0; nj += jStep; }
      if (!uses(j, r)) continue;
      const int I = rowOf(r);
      const char* src = reinterpret_cast<const char*>(kForward ? M + tileBase(Tn, I, j) : M + tileBase(Tn, j, I));
      const unsigned dst = (unsigned)__cvta_generic_to_shared(buf + (issued % kSolveBufs) * kTileElems);
      constexpr int nv = kTileElems * (int)sizeof(T) / 16;
#pragma unroll 4
      for (int v = lane; v < nv; v += 32)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16u * v), "l"(src + 16 * v) : "memory");
      break;
    }
    ++issued;
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // the oldest tile copied; once read, its buffer is filled again (refill, off the critical path)
  int used = 0;
  auto oldest = [&]() -> const T* {
    asm volatile("cp.async.wait_group 2;" ::: "memory");
    __syncwarp();
    return buf + (used++ % kSolveBufs) * kTileElems;
  };
  auto refill = [&]() {
    __syncwarp();
    issueNext();
  };
  for (int i = 0; i < kSolveBufs; ++i) issueNext();
  T* xw = xs + 96 + 32 * warp;  // this warp's copy of a source tile from another CTA
  bool ok = true;
  int ready = 0;  // source tiles known to be solved from j on
  T xNext = (T)0;
  for (int j = kForward ? 0 : Tn - 1; j != jEnd; j += jStep) {
    const T* x;
    if (kForward ? j < first : j >= end) {
      if (!owner) continue;
      if (ready == 0) {
        ready = waitTiles(g, flags, j, kForward ? first : end - 1, jStep, epoch);
        if (ready == 0) {
          ok = false;
          ready = 1;
        }
        xNext = loadL2(y + (int64_t)j * 32 + lane);
      }
      __syncwarp();
      xw[lane] = xNext;
      __syncwarp();
      if (--ready > 0) xNext = loadL2(y + (int64_t)(j + jStep) * 32 + lane);
      x = xw;
    } else {
      const int t = j - first;
      T* xt = xs + (t & 1) * 32;
      T yI = (T)0, dI = (T)0;
      const bool mine = warp == t % W;
      const int r0 = t / W;
      if (mine) {
        T* yb = xs + 64;
        yI = yv[0];
#pragma unroll
        for (int r = 1; r < kSolveRows; ++r)
          if (r == r0) yI = yv[r];
        yb[lane] = yI;
        const T* A = oldest();
        if (kForward) dI = A[lane * kTileLd + lane];
        yI = yI + diagPart<kForward>(A, yb);
        xt[lane] = yI;
      }
      __syncthreads();
      if (mine) {  // the rest is not waited for by this CTA's other warps
        publishTile(y + (int64_t)j * 32, flags + j, epoch, yI);
        if (kForward) yI = yI / dI;  // the backward pass starts from y / D
#pragma unroll
        for (int r = 0; r < kSolveRows; ++r)
          if (r == r0) yv[r] = yI;
        refill();
      }
      x = xt;
    }
#pragma unroll
    for (int rr = 0; rr < kSolveRows; ++rr) {
      const int r = kForward ? rr : kSolveRows - 1 - rr;
      if (!uses(j, r) || rowOf(r) == j) continue;
      const T* A = oldest();
      T acc = (T)0;
#pragma unroll 8
      for (int k = 0; k < 32; ++k) acc = accT(acc, kForward ? A[k * kTileLd + lane] : A[lane * kTileLd + k], x[k]);
      yv[r] = yv[r] - accEnd(acc);
      refill();
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  return ok;
}

template <typename T>
__device__ __noinline__ bool gridSolve(GridCtl* g, int nr, const T* M, T* y, T* stage) {
  constexpr int W = solveWarps<T>();
  const int Tn = rootTiles(nr), warp = threadIdx.x >> 5, lane = threadIdx.x & 31, G = (int)gridDim.x;
  const int rows = min(kSolveRows, (Tn + W * G - 1) / (W * G));  // per warp
  const int run = W * rows;                                      // consecutive row tiles of a CTA
  // a root with more tiles than the grid's warps own at once: every G-th run, in order
  const int runs = (Tn + run * G - 1) / (run * G);
  const int epoch = reinterpret_cast<volatile GridCtl*>(g)->epoch;
  T* xs = stage;
  T* bufs = stage + 96 + 32 * 8;
  T yv[kSolveRows];
  bool ok = true;
  for (int k = 0; k < 2 * runs; ++k) {
    const bool forward = k < runs;
    const int first = ((forward ? k : 2 * runs - 1 - k) * G + (int)blockIdx.x) * run, end = min(Tn, first + run);
    if (first >= Tn) continue;
    if (forward || runs > 1) {
#pragma unroll
      for (int r = 0; r < kSolveRows; ++r) {
        const int I = first + r * W + warp;
        yv[r] = (T)0;
        if (warp < W && I < end) {
          yv[r] = loadL2(y + (int64_t)I * 32 + lane);
          if (!forward) yv[r] = yv[r] / M[tileBase(Tn, I, I) + lane * kTileLd + lane];
        }
      }
    }
    if (forward) ok = solvePass<true>(g, Tn, M, y, first, end, epoch, bufs, xs, yv) && ok;
    else ok = solvePass<false>(g, Tn, M, y, first, end, epoch, bufs, xs, yv) && ok;
  }
  tc::fenceProxyAsyncShared();  // these accesses before a factor's bulk copies into the area
  return gridSync(g) && ok;
}

// One posted job, run by every CTA (CTA 0 passes its pivot statistics).
template <typename T>
__device__ bool gridJobT(GridCtl* g, const DevSettings& st, int op, PivotStats* ps) {
  volatile GridCtl* vg = g;
  T* M = reinterpret_cast<T*>(vg->M);
  const Ctx& c = g->ctx;
  extern __shared__ __align__(16) unsigned char dynSmem[];
  T* stage = reinterpret_cast<T*>(dynSmem + vg->stageOff);
  if (op == kGridOpFactor)
    return gridAssemble<T>(g, c, st, M, vg->ep, vg->ea) && gridLdlt<T>(g, c.nr, c.n, st, M, ps, stage, c.slices);
  if (op == kGridOpSolve) return gridSolve<T>(g, c.nr, M, reinterpret_cast<T*>(vg->y), stage);
  return false;
}

// CTAs 1 .. of a whole-GPU launch: wait for a job, run it, until CTA 0 posts the exit.
template <typename FT>
__device__ __noinline__ void gridWorker(GridCtl* g, const DevSettings& st) {
  for (int job = 1;; ++job) {
    if (!gridSync(g)) return;
    volatile GridCtl* vg = g;
    const int op = vg->op, arith = vg->arith;
    if (op == kGridOpExit) return;
    if (blockIdx.x == 1 && vg->leaveJob == job) return;
#ifdef CXG_GRID_KERNELS
    if (op == kGridOpProducts) {
      gridProductsShare(g);
      if (!gridSync(g)) return;
      continue;
    }
    if (op == kGridOpSave) {
      gridSaveJob(g, (int)blockIdx.x, (int)gridDim.x);
      if (!gridSync(g)) return;
      continue;
    }
#endif
    bool ok;
    if constexpr (sizeof(FT) == 4)
      ok = (arith == 1) ? gridJobT<float>(g, st, op, nullptr) : gridJobT<df64>(g, st, op, nullptr);
    else
      ok = gridJobT<double>(g, st, op, nullptr);
    if (!ok) return;
  }
}

// CTA 0: post a job (the barrier publishes it) and run it with the other CTAs.
template <typename T>
__device__ bool gridPost(Ctx& c, const DevSettings& st, int op, T* M, T* y, double ep, double ea, PivotStats* ps) {
  GridCtl* g = c.grid;
  if (threadIdx.x == 0) {
    g->op = op;
    g->arith = ArithOf<T>::v;
    g->M = M;
    g->y = y;
    g->ep = ep;
    g->ea = ea;
    g->epoch += 1;
  }
  if (!gridSync(g)) return false;
  return gridJobT<T>(g, st, op, ps);
}

// ------------------------------------------------------------------------------------------
// reduced KKT: assembly + factorisation, and one solve through it
// ------------------------------------------------------------------------------------------
// Builds the root for the current cone scaling with extra diagonal bumps (ep on x rows, -ea on
// all cone rows, the regularisation ladder of kkt_system.cpp:152-168) and factors it in T.
template <typename T, bool G = false>
__device__ __noinline__ void assembleFactor(Ctx& c, const DevSettings& st, T* M, double ep, double ea,
                               int& fail, int& wrongSign, double& minAbsD) {
  const InstanceDesc& D = *c.D;
  const int n = c.n, nr = c.nr;
  const double epsA = st.static_reg_A + ea;
  const long long t0 = (st.record_timings && threadIdx.x == 0) ? clock64() : 0;
  // G_u = (Hs_u + epsA I)^-1 as eigenvalues (NN: cu[row]; SOC: sp.r0..r2), then
  // T_u = G_u Ad_u column by column
  FOR_T(u, c.nUnits) {  // the SOC blocks first (three divisions against one)
    if (u >= c.nsoc) {
      const int i = u - c.nsoc;
      const double w = c.cw[c.p + i];
      const double g = 1.0 / sqEps(w, epsA, true);
      c.cu[c.p + i] = g;
      for (int k = c.unitAd[i]; k < c.unitAd[i + 1]; ++k) c.T[k] = g * c.Ad[k];
    } else {
      socPrepareG(c.sp[u], c.cu + c.socOff[u], epsA);
    }
  }
  __syncthreads();
  FOR_T(k, D.nSocCols) {
    const int b = c.scUnit[k], o = c.scOff[k];
    socApplyG(c.sp[b], c.cu + c.socOff[b], c.socDim[b], c.Ad + o, c.T + o);
  }
  if constexpr (G) {
    // whole-GPU launch: the assembly and the LDL' run on every CTA
    PivotStats* ps = reinterpret_cast<PivotStats*>(c.sc + SC_COUNT);
    if (threadIdx.x == 0) {
      ps->nreg = 0;
      ps->zero = 0;
      ps->wrong = 0;
      ps->minAbs = INFINITY;
    }
    __syncthreads();
    const long long t1 = (st.record_timings && threadIdx.x == 0) ? clock64() : 0;
    // post the job, then run its two parts here (timed separately: assembly, LDL')
    GridCtl* g = c.grid;
    if (threadIdx.x == 0) {
      g->op = kGridOpFactor;
      g->arith = ArithOf<T>::v;
      g->M = M;
      g->y = nullptr;
      g->ep = ep;
      g->ea = ea;
    }
    extern __shared__ __align__(16) unsigned char dynSmem[];
    bool ok = gridSync(g) && gridAssemble<T>(g, g->ctx, st, M, ep, ea);
    const long long t2 = (st.record_timings && threadIdx.x == 0) ? clock64() : 0;
    ok = ok && gridLdlt<T>(g, nr, n, st, M, ps, reinterpret_cast<T*>(dynSmem + g->stageOff), c.slices);
    __syncthreads();
    const bool regularized = st.linear_solver == 2;
    fail = !ok ? 1 : (regularized ? (((double)ps->nreg > 0.05 * (double)nr) ? 1 : 0) : ps->zero);
    wrongSign = ps->wrong;
    minAbsD = ok ? ps->minAbs : NAN;
    __syncthreads();
    if (st.record_timings && threadIdx.x == 0) {
      timers(c)[TM_ASSEMBLE] += (t1 - t0) + (t2 - t1);
      timers(c)[TM_LDLT] += clock64() - t2;
    }
    return;
  }
  const int64_t rs = rootSize(nr);
#pragma unroll 1
  for (int64_t t = threadIdx.x; t < rs; t += blockDim.x) M[t] = (T)0;
  __syncthreads();
#pragma unroll 1
  for (int i = nr + (int)threadIdx.x; i < rootTiles(nr) * kTile; i += blockDim.x) M[rootIdx(nr, i, i)] = (T)1;
  FOR_T(i, n) {
    const int src = c.pdiag[i];
    M[rootIdx(nr, i, i)] = (T)(((src >= 0) ? c.Pu[src] : 0.0) + st.static_reg_P + ep);
  }
  FOR_T(k, D.nPlow) M[c.plowIdx[k]] = (T)c.Pu[c.plowSrc[k]];
  FOR_T(k, D.nAZ) M[c.azIdx[k]] = (T)c.Av[c.azSrc[k]];
  FOR_T(r, c.p) M[rootIdx(nr, n + r, n + r)] = (T)(-(st.static_reg_A + ea));
  __syncthreads();
  addContributions<T>(c, M, threadIdx.x >> 5, blockDim.x >> 5);
  __syncthreads();
  const long long t1 = (st.record_timings && threadIdx.x == 0) ? clock64() : 0;
  denseLdlt<T>(c, M, st, fail, wrongSign, minAbsD);
  if (st.record_timings && threadIdx.x == 0) {
    timers(c)[TM_ASSEMBLE] += t1 - t0;
    timers(c)[TM_LDLT] += clock64() - t1;
  }
}

// sol = Kreg^-1 rhs through the factored root (T) with the bump ea used at factorisation.
template <typename T, bool G = false>
__device__ __noinline__ void reducedSolve(Ctx& c, const DevSettings& st, const T* M, double ea,
                             const double* rhs, double* sol) {
  const int n = c.n, p = c.p, nr = c.nr;
  const double* r1 = rhs;
  const double* r2 = rhs + n;
  // u = G_C r2_C (eigenvalues of G prepared at factorisation time)
  coneApplyG(c, r2, c.tm, true);
  // t = [r1 + A_C' u ; r2_Z] in T precision
  T* y = reinterpret_cast<T*>(c.rr);
  FOR_T(r, p) y[n + r] = (T)r2[r];
#pragma unroll 1
  for (int i = nr + (int)threadIdx.x; i < rootTiles(nr) * kTile; i += blockDim.x) y[i] = (T)0;
  constexpr int kOut = ArithOf<T>::v == 1 ? kProdColsF32 : ArithOf<T>::v == 2 ? kProdColsDf : 0;
  sliceProducts(c, kProdCols | kProdInit | kOut, nullptr, c.tm, nullptr, y, nullptr, r1);
  const long long t0 = (st.record_timings && threadIdx.x == 0) ? clock64() : 0;
  if constexpr (G) {
    // whole-GPU launch; a failed barrier leaves a non-finite solution, which the caller's
    // finiteness test turns into NumericalError
    if (!gridPost<T>(c, st, kGridOpSolve, const_cast<T*>(M), y, 0.0, 0.0, nullptr) && threadIdx.x == 0)
      y[0] = (T)NAN;
    __syncthreads();
  } else {
    denseSolve<T>(c, M, y);
  }
  if (st.record_timings && threadIdx.x == 0) timers(c)[TM_DSOLVE] += clock64() - t0;
  FOR_T(j, n) sol[j] = (double)y[j];
  FOR_T(r, p) sol[n + r] = (double)y[n + r];
  __syncthreads();
  // z_C = G_C (A_C x - r2_C)
  sliceProducts(c, kProdRows | kProdInit, sol, nullptr, nullptr, nullptr, c.tm, r2);
  coneApplyG(c, c.tm, sol + n, false);
  (void)ea;
}

// Factorisation state of the current iteration.
struct FactState {
  int use64;      // the high-precision factor (in root64) is the one held
  double ep, ea;  // bumps of the held factor
};

template <typename FT>
__device__ __forceinline__ FT* rootT(Ctx& c) { return reinterpret_cast<FT*>(c.root); }

// Arithmetic of the high-precision factor held in root64: FP64 for the FP64 kernel, double-float
// (FP32 pipe, ~48 bits) as the fallback of the mixed-precision kernel.
template <typename FT> struct HighT { using type = double; };
template <> struct HighT<float> { using type = df64; };
template <typename FT>
__device__ __forceinline__ typename HighT<FT>::type* rootHigh(Ctx& c) {
  return reinterpret_cast<typename HighT<FT>::type*>(c.root64);
}

// factorizeWithRetry (kkt_system.cpp:242-264) on the reduced system. In MIXED precision an FP32
// factor with a wrong-signed pivot is replaced by the double-float factor (sticky).
template <typename FT, bool G = false>
__device__ __noinline__ bool factorizeWithRetryImpl(Ctx& c, const DevSettings& st, FactState& fs) {
  double ep = 0.0, ea = 0.0;
  // attempts below this level fail in the reference's dense SOC blocks (coneUpdateScaling)
  const int socLvl = (int)c.sc[SC_SOCLVL];
  for (int attempt = 0; attempt < 18; ++attempt) {
    int fail = 0, wrong = 0;
    double mind = 0.0;
    // fault injection (tests): this attempt reports failure before any work, as does an attempt
    // the reference's SOC-block pivots fail
    const bool injected = c.sc[SC_FAULTF] < (double)st.fault_factor_failures;
    __syncthreads();
    if (injected || attempt < socLvl) {
      if (threadIdx.x == 0) {
        c.sc[SC_ATTEMPTS] += 1.0;
        if (injected) c.sc[SC_FAULTF] += 1.0;
      }
      __syncthreads();
      ep = fmax(ep * 10.0, st.dynamic_reg_delta);
      ea = fmax(ea * 10.0, st.dynamic_reg_delta);
      continue;
    }
    if (!fs.use64) {
      assembleFactor<FT, G>(c, st, rootT<FT>(c), ep, ea, fail, wrong, mind);
      if (sizeof(FT) == 4 && (wrong || !isfinite(mind))) {
        fs.use64 = 1;
        if (threadIdx.x == 0) c.sc[SC_NFB] += 1.0;
        attempt -= 1;  // retry this attempt in FP64
        continue;
      }
    } else {
      assembleFactor<typename HighT<FT>::type, G>(c, st, rootHigh<FT>(c), ep, ea, fail, wrong, mind);
    }
    if (threadIdx.x == 0) c.sc[SC_ATTEMPTS] += 1.0;
    __syncthreads();
    if (!fail && isfinite(mind) && mind > st.dynamic_reg_eps) {
      fs.ep = ep;
      fs.ea = ea;
      return true;
    }
    ep = fmax(ep * 10.0, st.dynamic_reg_delta);
    ea = fmax(ea * 10.0, st.dynamic_reg_delta);
  }
  return false;
}

template <typename FT, bool G>
__device__ void solveOnce(Ctx& c, const DevSettings& st, const FactState& fs, const double* rhs, double* sol) {
  if (fs.use64)
    reducedSolve<typename HighT<FT>::type, G>(c, st, rootHigh<FT>(c), fs.ea, rhs, sol);
  else
    reducedSolve<FT, G>(c, st, rootT<FT>(c), fs.ea, rhs, sol);
  // fault injection (tests): this solve returns a non-finite vector
  if (st.fault_nonfinite_solves > 0) {
    const bool injected = c.sc[SC_FAULTS] < (double)st.fault_nonfinite_solves;
    __syncthreads();
    if (injected && threadIdx.x == 0) {
      c.sc[SC_FAULTS] += 1.0;
      sol[0] = NAN;
    }
    __syncthreads();
  }
}

static __device__ __noinline__ bool vecFinite(Ctx& c, const double* v, int len) {
  int bad = 0;
  FOR_T(i, len) bad |= !finiteBits(v[i]);
  return !blockAny(bad);
}

// Refinement of the whole-GPU form: restarted GMRES in FP64 on the statically regularised K
// (the matrix the reference refines against, kkt_system.cpp:296-311), right-preconditioned by
// the held factor (FP32, double-float or FP64 LDL' of the bumped reduced system). Where a
// large root is ill-conditioned enough that plain refinement x += K^-1 (rhs - K x) with that
// factor stalls or diverges (the factor's relative error times cond(K) near or above 1), GMRES
// still converges, in a few iterations per cluster of poorly resolved eigenvalues (the mixed
// precision GMRES-IR of Carson and Higham, SIAM J. Sci. Comput. 40(2), 2018). Each iteration is one
// solve with the factor (every SM), one K product and modified Gram-Schmidt (CTA 0). On entry
// sol is the first solve and c.res = rhs - K sol with relative norm rel; a cycle's correction is
// kept only if the true residual drops. Returns the final relative residual; counts iterations
// in SC_RSTEPS.
template <typename FT, bool G>
__device__ void solveOnce(Ctx& c, const DevSettings& st, const FactState& fs, const double* rhs, double* sol);

template <typename FT, bool G>
__device__ __noinline__ double gmresRefine(Ctx& c, const DevSettings& st, const FactState& fs, const double* rhs,
                                           double* sol, double rel, double rhsNorm, bool& pxOk) {
  const int N = c.n + c.m;
  const int64_t ld = ((int64_t)N + 1) & ~int64_t(1);
  constexpr int hl = kGmresDim + 1;  // leading dimension of H (column-major)
  double* V = c.kry;
  double* Z = V + (int64_t)(kGmresDim + 1) * ld;
  double* H = Z + (int64_t)kGmresDim * ld;
  double* cs = H + hl * kGmresDim;
  double* sn = cs + kGmresDim;
  double* g = sn + kGmresDim;
  double* y = g + kGmresDim + 1;
  int total = 0;
  for (int cyc = 0; cyc < kGmresCycles && rel > st.refine_tol; ++cyc) {
    const double beta = rel * rhsNorm;
    FOR_T(i, N) V[i] = c.res[i] / beta;
    if (threadIdx.x == 0) g[0] = beta;
    __syncthreads();
    int k = 0;
    for (int j = 0; j < kGmresDim; ++j) {
      double* vj = V + (int64_t)j * ld;
      double* zj = Z + (int64_t)j * ld;
      solveOnce<FT, G>(c, st, fs, vj, zj);
      double* w = V + (int64_t)(j + 1) * ld;
      kktApply(c, st, zj, w);
      for (int i = 0; i <= j; ++i) {
        const double* vi = V + (int64_t)i * ld;
        double d[1] = {0.0};
        FOR_V(t, N, c.vb) d[0] += w[t] * vi[t];
        blockSum<1>(d, c.red, c.vb);
        FOR_T(t, N) w[t] -= d[0] * vi[t];
        if (threadIdx.x == 0) H[j * hl + i] = d[0];
        __syncthreads();
      }
      double nn[1] = {0.0};
      FOR_V(t, N, c.vb) nn[0] += w[t] * w[t];
      blockSum<1>(nn, c.red, c.vb);
      const double hn = sqrt(nn[0]);
      if (threadIdx.x == 0) {
        double* h = H + j * hl;
        h[j + 1] = hn;
        for (int i = 0; i < j; ++i) {
          const double t = cs[i] * h[i] + sn[i] * h[i + 1];
          h[i + 1] = -sn[i] * h[i] + cs[i] * h[i + 1];
          h[i] = t;
        }
        const double den = hypot(h[j], h[j + 1]);
        const double cj = den > 0.0 ? h[j] / den : 1.0, sj = den > 0.0 ? h[j + 1] / den : 0.0;
        cs[j] = cj;
        sn[j] = sj;
        h[j] = den;
        h[j + 1] = 0.0;
        g[j + 1] = -sj * g[j];
        g[j] = cj * g[j];
        c.sc[SC_GMRES] = fabs(g[j + 1]) / rhsNorm;
      }
      __syncthreads();
      k = j + 1;
      // stop at a residual estimate well below the target (the true residual is checked below),
      // or at breakdown (the Krylov space holds the solution)
      if (!(hn > 0.0) || !(c.sc[SC_GMRES] > 0.25 * st.refine_tol)) break;
      const double inv = 1.0 / hn;
      FOR_T(t, N) w[t] *= inv;
      __syncthreads();
    }
    total += k;
    if (threadIdx.x == 0) {
      for (int i = k - 1; i >= 0; --i) {
        double acc = g[i];
        for (int l = i + 1; l < k; ++l) acc -= H[l * hl + i] * y[l];
        y[i] = acc / H[i * hl + i];
      }
    }
    __syncthreads();
    FOR_T(t, N) {
      double acc = sol[t];
      for (int l = 0; l < k; ++l) acc += y[l] * Z[(int64_t)l * ld + t];
      c.cor[t] = acc;
    }
    __syncthreads();
    double rn = rhsNorm;
    const double relNew = kktResidual(c, st, rhs, c.cor, c.res, rn, false);
    pxOk = relNew < rel;
    if (!pxOk) break;  // no progress (or a non-finite candidate): keep sol
    FOR_T(t, N) sol[t] = c.cor[t];
    __syncthreads();
    rel = relNew;
  }
  if (threadIdx.x == 0) c.sc[SC_RSTEPS] += total;
  __syncthreads();
  return rel;
}

// KktSystem::solve (kkt_system.cpp:296-311) incl. escalateAndResolve (:266-294), plus the
// MIXED-precision fallback to the double-float factor. Returns the final relative residual, and
// in SC_PXOK whether c.tn holds P sol (the last residual's product, of the solution kept).
template <typename FT, bool G = false>
__device__ bool factorizeWithRetry(Ctx& c, const DevSettings& st, FactState& fs);

template <typename FT, bool G = false>
__device__ __noinline__ double kktSolveImpl(Ctx& c, const DevSettings& st, FactState& fs, const double* rhs, double* sol) {
  const int N = c.n + c.m;
  for (int pass = 0; pass < 2; ++pass) {
    solveOnce<FT, G>(c, st, fs, rhs, sol);
    if (!vecFinite(c, sol, N)) {
      // escalate: x1000 bumps from the held factor's, up to 10 times
      double ep = fs.ep, ea = fs.ea;
      bool ok = false;
      const double socEa = ladderBump((int)c.sc[SC_SOCLVL], st.dynamic_reg_delta);
      for (int att = 0; att < 10 && !ok; ++att) {
        ep = fmax(ep * 1000.0, st.dynamic_reg_delta);
        ea = fmax(ea * 1000.0, st.dynamic_reg_delta);
        int fail = 0, wrong = 0;
        double mind = 0.0;
        if (threadIdx.x == 0) c.sc[SC_ESC] += 1.0;
        if (ea < socEa) continue;  // the reference's SOC-block pivots still fail at this bump
        if (fs.use64)
          assembleFactor<typename HighT<FT>::type, G>(c, st, rootHigh<FT>(c), ep, ea, fail, wrong, mind);
        else
          assembleFactor<FT, G>(c, st, rootT<FT>(c), ep, ea, fail, wrong, mind);
        if (fail || !isfinite(mind) || !(mind > st.dynamic_reg_eps)) continue;
        fs.ep = ep;
        fs.ea = ea;
        solveOnce<FT, G>(c, st, fs, rhs, sol);
        ok = vecFinite(c, sol, N);
      }
    }
    double rhsNorm = 1.0;
    bool pxOk = true;
    double rel = kktResidual(c, st, rhs, sol, c.res, rhsNorm, true);
    const bool fp32Factor = (sizeof(FT) == 4) && !fs.use64;
    const int maxRef = G ? 0 : (fp32Factor ? st.mixed_refine_max_iter : st.refine_max_iter);
    if constexpr (G) {
      if (rel > st.refine_tol) rel = gmresRefine<FT, G>(c, st, fs, rhs, sol, rel, rhsNorm, pxOk);
    }
    int steps = 0;
    for (int it = 0; it < maxRef && rel > st.refine_tol; ++it) {
      solveOnce<FT, G>(c, st, fs, c.res, c.cor);
      FOR_T(i, N) sol[i] += c.cor[i];
      __syncthreads();
      const double prev = rel;
      rel = kktResidual(c, st, rhs, sol, c.res, rhsNorm, false);
      ++steps;
      // an FP32 factor whose refinement contracts by less than 4x per step will not reach the
      // tolerance in the remaining steps: go to the high-precision factor now
      if (fp32Factor && !(rel <= st.mixed_fallback_tol) && !(rel <= 0.25 * prev)) break;
      // a step of the high-precision refinement that does not lower the residual: keep the
      // better solution and stop (further steps with the same factor do not converge either)
      if (!fp32Factor && !(rel < prev)) {
        FOR_T(i, N) sol[i] -= c.cor[i];
        __syncthreads();
        rel = prev;
        pxOk = false;
        break;
      }
    }
    if (threadIdx.x == 0) c.sc[SC_RSTEPS] += steps;
    const bool mixedFp32 = (sizeof(FT) == 4) && !fs.use64;
    if (mixedFp32 && !(rel <= st.mixed_fallback_tol)) {
      // sticky fallback: refactor in double-float (with the retry ladder) and redo this solve
      fs.use64 = 1;
      if (threadIdx.x == 0) c.sc[SC_NFB] += 1.0;
      if (!factorizeWithRetry<FT, G>(c, st, fs)) return INFINITY;
      continue;
    }
    if (threadIdx.x == 0) {
      c.sc[SC_PXOK] = pxOk ? 1.0 : 0.0;
      if (!(rel <= c.sc[SC_MAXREL])) c.sc[SC_MAXREL] = rel;
      if (!(rel <= c.sc[SC_ITREL])) c.sc[SC_ITREL] = rel;
    }
    __syncthreads();
    return rel;
  }
  return INFINITY;
}

template <typename FT, bool G>
__device__ bool factorizeWithRetry(Ctx& c, const DevSettings& st, FactState& fs) {
  const long long t0 = st.record_timings ? clock64() : 0;
  const bool ok = factorizeWithRetryImpl<FT, G>(c, st, fs);
  if (st.record_timings && threadIdx.x == 0) timers(c)[TM_FACTOR] += clock64() - t0;
  return ok;
}

template <typename FT, bool G = false>
__device__ double kktSolve(Ctx& c, const DevSettings& st, FactState& fs, const double* rhs, double* sol) {
  const long long t0 = st.record_timings ? clock64() : 0;
  const long long f0 = st.record_timings ? timers(c)[TM_FACTOR] : 0;
  if (threadIdx.x == 0) c.sc[SC_PXOK] = 0.0;
  __syncthreads();
  // a fallback refactorisation inside counts as factorisation time only
  const double r = kktSolveImpl<FT, G>(c, st, fs, rhs, sol);
  if (st.record_timings && threadIdx.x == 0) timers(c)[TM_SOLVE] += (clock64() - t0) - (timers(c)[TM_FACTOR] - f0);
  return r;
}

// ------------------------------------------------------------------------------------------
// the IPM driver for one instance (solver_impl.cpp SolverImpl::solve and helpers)
// ------------------------------------------------------------------------------------------
template <typename FT, bool G = false>
__device__ __noinline__ void solveInstance(Ctx& c, const LaunchArgs& a, int inst) {
  const DevSettings& st = a.st;
  const InstanceDesc& D = *c.D;
  const int n = c.n, m = c.m, N = n + m;
  const int degree = c.l + c.nsoc;
  FactState fs{0, 0.0, 0.0};
  double tau = 1.0, kappa = 1.0;
  int status = 4;  // MaxIterations
  int iterations = 0;
  double dqx = 0, dbz = 0, dsz = 0, dxPx = 0, rtau = 0;
  if (threadIdx.x < SC_COUNT) c.sc[threadIdx.x] = 0.0;
  if (threadIdx.x < TM_COUNT) timers(c)[threadIdx.x] = 0;
  const long long tStart = clock64();
  unsigned long long wallStart = 0;
  if (st.record_timings && threadIdx.x == 0) asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(wallStart));
  __syncthreads();

  const bool useWarm = st.warm_start && a.haveWarm && a.haveWarm[inst];
  bool initOk = true;
  if (useWarm) {
    FOR_T(j, n) c.x[j] = a.warmX[D.vQ + j];
    FOR_T(r, m) {
      c.s[r] = (r < c.p) ? 0.0 : a.warmS[D.vB + r];
      c.z[r] = a.warmZ[D.vB + r];
    }
    __syncthreads();
    ensureStrictlyInteriorWarm(c, c.s);
    ensureStrictlyInteriorWarm(c, c.z);
  } else {
    // computeInitialPoint: Hs = I scaling of the identity element, 1 or 2 KKT solves
    coneUpdateScaling(c, st, c.ev, c.ev);
    if (!factorizeWithRetry<FT, G>(c, st, fs)) {
      initOk = false;
    } else {
      if (D.pStoredNnz == 0) {
        FOR_T(j, n) c.rhs[j] = 0.0;
        FOR_T(r, m) c.rhs[n + r] = c.bs[r];
        __syncthreads();
        kktSolve<FT, G>(c, st, fs, c.rhs, c.sol);
        FOR_T(j, n) c.x[j] = c.sol[j];
        FOR_T(r, m) c.s[r] = -c.sol[n + r];
        FOR_T(j, n) c.rhs[j] = -c.qs[j];
        FOR_T(r, m) c.rhs[n + r] = 0.0;
        __syncthreads();
        kktSolve<FT, G>(c, st, fs, c.rhs, c.sol);
        FOR_T(r, m) c.z[r] = c.sol[n + r];
      } else {
        FOR_T(j, n) c.rhs[j] = -c.qs[j];
        FOR_T(r, m) c.rhs[n + r] = c.bs[r];
        __syncthreads();
        kktSolve<FT, G>(c, st, fs, c.rhs, c.sol);
        FOR_T(j, n) c.x[j] = c.sol[j];
        FOR_T(r, m) {
          c.z[r] = c.sol[n + r];
          c.s[r] = -c.sol[n + r];
        }
      }
      __syncthreads();
      FOR_T(r, c.p) c.s[r] = 0.0;
      __syncthreads();
      shiftToInteriorCold(c, c.s, degree);
      shiftToInteriorCold(c, c.z, degree);
      int bad = 0;
      FOR_T(j, n) bad |= !finiteBits(c.x[j]);
      FOR_T(r, m) bad |= !finiteBits(c.s[r]) | !finiteBits(c.z[r]);
      initOk = !blockAny(bad);
    }
  }
  if (!initOk) status = 5;

  // record_timings: one trace row per iteration (columns as kTraceCols), written by thread 0
  double* trow = nullptr;
  for (int iter = 0; initOk && iter < st.max_iter; ++iter) {
    iterations = iter + 1;
    trow = (a.trace && iter < a.traceRows) ? a.trace + ((int64_t)inst * a.traceRows + iter) * kTraceCols : nullptr;
    if (threadIdx.x == 0) {
      c.sc[SC_ITREL] = 0.0;
      if (trow)
        for (int k = 0; k < kTraceCols; ++k) trow[k] = 0.0;
    }
    const double att0 = c.sc[SC_ATTEMPTS];
    __syncthreads();
    // 1. refactorise for the current scaling
    coneUpdateScaling(c, st, c.s, c.z);
    if (!factorizeWithRetry<FT, G>(c, st, fs)) { status = 5; break; }
    if (trow && threadIdx.x == 0) trow[11] = c.sc[SC_ATTEMPTS] - att0;
    // 2. constant solve (-q, b) -> x1, z1; Px1
    FOR_T(j, n) c.rhs[j] = -c.qs[j];
    FOR_T(r, m) c.rhs[n + r] = c.bs[r];
    __syncthreads();
    kktSolve<FT, G>(c, st, fs, c.rhs, c.sol);
    FOR_T(j, n) c.x1[j] = c.sol[j];
    FOR_T(r, m) c.z1[r] = c.sol[n + r];
    __syncthreads();
    if (!vecFinite(c, c.sol, N)) { status = 5; break; }
    // P times a solution: what its last KKT residual formed, unless that solution was not kept
    if (c.sc[SC_PXOK] != 0.0) FOR_T(j, n) c.Px1[j] = c.tn[j];
    else pmul(c, c.x1, c.Px1);
    __syncthreads();
    // 3. residuals
    pmul(c, c.x, c.tn);  // Px
    {
      // A'z and A x (into dx and tm, free here)
      sliceProducts(c, kProdCols | kProdRows, c.x, c.z, nullptr, c.dx, c.tm, nullptr);
      double v[6] = {0, 0, 0, 0, 0, 0};
      FOR_V(t, n + m, c.vb) {
        if (t < n) {
          const double r = fma(-tau, c.qs[t], -c.dx[t] - c.tn[t]);
          c.rx[t] = r;
          v[0] += r * r;
          v[2] += c.qs[t] * c.x[t];
          v[5] += c.x[t] * c.tn[t];
        } else {
          const int r = t - n;
          const double rr = c.tm[r] + c.s[r] - tau * c.bs[r];
          c.rz[r] = rr;
          v[1] += rr * rr;
          v[3] += c.bs[r] * c.z[r];
          v[4] += c.s[r] * c.z[r];
        }
      }
      blockSum<6>(v, c.red, c.vb);
      dqx = v[2];
      dbz = v[3];
      dsz = v[4];
      dxPx = v[5];
      // The quotients of this stage side by side in the lanes of one division each (a division holds the
      // FP64 unit for some 600 cycles, whatever the number of lanes that want one). The scalars'
      // products are fused into their sums as written out here and below (the root's arithmetic decides
      // one of them), whatever the compiler finds around them.
      const int lane = threadIdx.x & 31;
      const double dkrA = __dmul_rn(tau, kappa);
      double quo;
      {
        const double root = sqrt((lane & 7) == 3 ? v[1] : v[0]), half = 0.5 * dxPx;
        const double num = (lane & 4) ? pick4(lane, half, tau, kappa, dkrA)
                                      : pick4(lane, dxPx, fma(tau, kappa, dsz), root, root);
        const double den = (lane & 4) ? pick4(lane, tau, fmax(kappa, 1e-30), tau, tau)
                                      : pick4(lane, tau, (double)(degree + 1), tau, tau);
        quo = num / den;
      }
      auto quotient = [&](int k) { return __shfl_sync(0xffffffffu, quo, k); };
      rtau = dqx + dbz + kappa + quotient(0);
      const double mu = quotient(1), nrx = quotient(2), nrz = quotient(3), halfTau = quotient(4);
      const double ratio = quotient(5), kappaTau = quotient(6), dkrTau = quotient(7);
      quo = ((lane & 1) ? -halfTau - dbz : halfTau + dqx) / tau;
      const double pobj = quotient(0), dobj = quotient(1);
      // 4. convergence / infeasibility (solver_impl.cpp checkConvergence / checkInfeasibility)
      if (trow && threadIdx.x == 0) {
        trow[0] = mu; trow[1] = nrx; trow[2] = nrz; trow[3] = pobj; trow[4] = dobj; trow[8] = tau; trow[9] = kappa;
      }
      const double gapAbs = fabs(pobj - dobj);
      const double gapTol = st.tol_gap_abs + st.tol_gap_rel * fmax(fabs(pobj), fabs(dobj));
      if (nrx < st.tol_feas && nrz < st.tol_feas && gapAbs < gapTol && tau > 1e-6) { status = 1; break; }
      if (ratio <= st.tol_infeas) {
        double w[2] = {0.0, 0.0};
        FOR_V(r, m, c.vb) w[0] += c.z[r] * c.z[r];
        FOR_V(j, n, c.vb) w[1] += c.x[j] * c.x[j];
        blockSum<2>(w, c.red, c.vb);
        if (dbz < -st.tol_infeas * fmax(1.0, sqrt(w[0]))) { status = 2; break; }
        if (dqx < -st.tol_infeas * fmax(1.0, sqrt(w[1]))) { status = 3; break; }
      }
      // tau_den is the same for the affine and the combined step (solver_impl.cpp:309-310,
      // 364-365): kappa/tau - q'x1 - b'z1 + (xi-x1)'P(xi-x1) - x1'Px1, xi = x/tau
      FOR_T(j, n) c.tn[j] = c.x[j] / tau - c.x1[j];
      __syncthreads();
      pmul(c, c.tn, c.dx);
      double td[4] = {0, 0, 0, 0};
      FOR_V(j, n, c.vb) {
        td[0] += c.qs[j] * c.x1[j];
        td[2] += c.tn[j] * c.dx[j];
        td[3] += c.x1[j] * c.Px1[j];
      }
      FOR_V(r, m, c.vb) td[1] += c.bs[r] * c.z1[r];
      blockSum<4>(td, c.red, c.vb);
      const double tauDen = kappaTau - td[0] - td[1] + td[2] - td[3];

      // 5. affine step: rhs (rx, s - rz)
      FOR_T(j, n) c.rhs[j] = c.rx[j];
      FOR_T(r, m) c.rhs[n + r] = c.s[r] - c.rz[r];
      __syncthreads();
      kktSolve<FT, G>(c, st, fs, c.rhs, c.sol);
      if (!vecFinite(c, c.sol, N)) { status = 5; break; }
      if (c.sc[SC_PXOK] == 0.0) pmul(c, c.sol, c.tn);  // P xv
      double tn3[4] = {0, 0, 0, 0};
      FOR_V(j, n, c.vb) {
        tn3[0] += c.qs[j] * c.sol[j];
        tn3[2] += (c.x[j] / tau) * c.tn[j];
      }
      FOR_V(r, m, c.vb) tn3[1] += c.bs[r] * c.sol[n + r];
      blockSum<4>(tn3, c.red, c.vb);
      const double tauNumA = rtau - dkrTau + tn3[0] + tn3[1] + 2.0 * tn3[2];
      if (tauDen == 0.0 || !isfinite(tauNumA) || !isfinite(tauDen)) { status = 5; break; }
      const double dtauA = tauNumA / tauDen;
      FOR_T(j, n) c.dx[j] = c.sol[j] + dtauA * c.x1[j];
      FOR_T(r, m) c.dz[r] = c.sol[n + r] + dtauA * c.z1[r];
      __syncthreads();
      coneApply(c, kHs, 0.0, c.dz, c.tm);
      FOR_T(r, m) c.ds[r] = -(c.tm[r] + c.s[r]);
      __syncthreads();
      // the batched FP64 kernel fuses the other product of the two
      const double dkappaNum =
          -((sizeof(FT) == 8 && !G) ? fma(tau, kappa, __dmul_rn(kappa, dtauA)) : fma(kappa, dtauA, dkrA));
      quo = ((lane & 1) ? -tau : dkappaNum) / ((lane & 1) ? dtauA : tau);
      const double dkappaA = quotient(0), toTau = quotient(1);
      {
        int bad = !finiteBits(dtauA) || !finiteBits(dkappaA);
        FOR_T(j, n) bad |= !finiteBits(c.dx[j]);
        FOR_T(r, m) bad |= !finiteBits(c.dz[r]) | !finiteBits(c.ds[r]);
        if (blockAny(bad)) { status = 5; break; }
      }
      // 6. affine step length (no fraction), mu_aff, sigma
      double aaff = 1.0;
      if (dtauA < 0) aaff = fmin(aaff, toTau);
      if (dkappaA < 0) aaff = fmin(aaff, -kappa / dkappaA);
      aaff = coneMaxStep2(c, aaff);
      double sa[2] = {0.0, 0.0};
      FOR_V(r, m, c.vb) sa[0] += (c.s[r] + aaff * c.ds[r]) * (c.z[r] + aaff * c.dz[r]);
      blockSum<2>(sa, c.red, c.vb);
      const double tauAff = fma(aaff, dtauA, tau);
      const double kappaAff = fma(aaff, dkappaA, kappa);
      const double muAff = fma(tauAff, kappaAff, sa[0]) / (double)(degree + 1);
      double sigma;
      if (mu > 0) {
        const double rt = fmax(muAff / mu, 0.0);
        sigma = fmin(fmax(rt * rt * rt, 0.0), 1.0);
      } else {
        sigma = 1.0;
      }
      if (trow && threadIdx.x == 0) { trow[5] = aaff; trow[6] = sigma; }
      // 7. combined step: lambda = W z; ds_comb = lambda o lambda + (W^-1 ds_aff) o (W dz_aff) - sigma mu e
      coneApply(c, kW, 0.0, c.z, c.lam);
      coneProduct(c, false, c.lam, c.lam, c.tm);           // lambda o lambda
      coneApply(c, kWinv, 0.0, c.ds, c.tm2);               // W^-1 ds_aff
      coneApply(c, kW, 0.0, c.dz, c.dcon);                 // W dz_aff (dcon as temp)
      coneProduct(c, false, c.tm2, c.dcon, c.rhs);         // corrector (rhs as temp, length m)
      FOR_T(r, m) c.tm2[r] = c.tm[r] + c.rhs[r] - sigma * mu * c.ev[r];
      __syncthreads();
      coneProduct(c, true, c.lam, c.tm2, c.tm);            // lambda \ ds_comb
      coneApply(c, kW, 0.0, c.tm, c.dcon);                 // ds_const = W (lambda \ ds_comb)
      FOR_T(j, n) c.rhs[j] = (1.0 - sigma) * c.rx[j];
      FOR_T(r, m) c.rhs[n + r] = c.dcon[r] - (1.0 - sigma) * c.rz[r];
      __syncthreads();
      kktSolve<FT, G>(c, st, fs, c.rhs, c.sol);
      if (!vecFinite(c, c.sol, N)) { status = 5; break; }
      if (c.sc[SC_PXOK] == 0.0) pmul(c, c.sol, c.tn);
      tn3[0] = tn3[1] = tn3[2] = 0.0;
      FOR_V(j, n, c.vb) {
        tn3[0] += c.qs[j] * c.sol[j];
        tn3[2] += (c.x[j] / tau) * c.tn[j];
      }
      FOR_V(r, m, c.vb) tn3[1] += c.bs[r] * c.sol[n + r];
      blockSum<4>(tn3, c.red, c.vb);
      const double dtrC = (1.0 - sigma) * rtau;
      const double dkrC = fma(-sigma, mu, fma(tau, kappa, __dmul_rn(dtauA, dkappaA)));
      const double tauNumC = dtrC - dkrC / tau + tn3[0] + tn3[1] + 2.0 * tn3[2];
      if (tauDen == 0.0 || !isfinite(tauNumC)) { status = 5; break; }
      const double dtau = tauNumC / tauDen;
      FOR_T(j, n) c.dx[j] = c.sol[j] + dtau * c.x1[j];
      FOR_T(r, m) c.dz[r] = c.sol[n + r] + dtau * c.z1[r];
      __syncthreads();
      coneApply(c, kHs, 0.0, c.dz, c.tm);
      FOR_T(r, m) c.ds[r] = -(c.tm[r] + c.dcon[r]);
      __syncthreads();
      quo = ((lane & 1) ? -tau : -fma(kappa, dtau, dkrC)) / ((lane & 1) ? dtau : tau);
      const double dkappa = quotient(0), toTauC = quotient(1);
      {
        int bad = !finiteBits(dtau) || !finiteBits(dkappa);
        FOR_T(j, n) bad |= !finiteBits(c.dx[j]);
        FOR_T(r, m) bad |= !finiteBits(c.dz[r]) | !finiteBits(c.ds[r]);
        if (blockAny(bad)) { status = 5; break; }
      }
      // 8. step length with the fraction-to-boundary factor
      double alpha = 1.0;
      if (dtau < 0) alpha = fmin(alpha, toTauC);
      if (dkappa < 0) alpha = fmin(alpha, -kappa / dkappa);
      alpha = coneMaxStep2(c, alpha);
      alpha *= st.max_step_fraction;
      if (trow && threadIdx.x == 0) { trow[7] = alpha; trow[10] = c.sc[SC_ITREL]; }
      if (!isfinite(alpha) || alpha <= 0.0) { status = 5; break; }
      // 9. update and rescale
      FOR_T(j, n) c.x[j] += alpha * c.dx[j];
      FOR_T(r, m) {
        c.s[r] += alpha * c.ds[r];
        c.z[r] += alpha * c.dz[r];
      }
      tau = fma(alpha, dtau, tau);
      kappa = fma(alpha, dkappa, kappa);
      __syncthreads();
      const double scl = fmax(tau, kappa);
      if (scl > 1e8 || scl < 1e-8) {
        const double inv = 1.0 / scl;
        FOR_T(j, n) c.x[j] *= inv;
        FOR_T(r, m) {
          c.s[r] *= inv;
          c.z[r] *= inv;
        }
        tau *= inv;
        kappa *= inv;
        __syncthreads();
      }
    }
  }
  if (trow && threadIdx.x == 0) trow[10] = c.sc[SC_ITREL];  // the last row, whichever way it ended

  // a wait that ran out: products may be old ones, whatever was concluded from them
  if constexpr (G) {
    if (gridFailed(c.grid)) status = 5;
  }

  // finalizeSolution (solver_impl.cpp:342-365 of the reference numbering)
  const bool infeas = (status == 2 || status == 3);
  const double scale = infeas ? 1.0 / fmax(kappa, 1e-30) : 1.0 / fmax(tau, 1e-30);
  const double* dvec = a.dpool + D.dD;
  const double* evec = a.dpool + D.dE;
  const double cs = D.cscale;
  const bool eq = st.equilibrate != 0;
  FOR_T(j, n) a.x[D.vX + j] = c.x[j] * scale * (eq ? dvec[j] : 1.0);
  FOR_T(r, m) {
    a.s[D.vS + r] = eq ? (c.s[r] * scale) / evec[r] : c.s[r] * scale;
    a.z[D.vZ + r] = eq ? (c.z[r] * scale) * evec[r] / cs : c.z[r] * scale;
  }
  if (a.bwd) {
    // final factorisation (as FP64), scaling and normalised iterate for the adjoint
    double* Bs = a.bwd + D.bwdOff;
    const BwdLayout bl = bwdLayout(c.nr, n, m, c.nsoc);
    const int64_t rs = rootSize(c.nr);
#ifdef CXG_GRID_KERNELS
    if constexpr (G) {
      if (fs.use64) gridSaveRoot(c, ArithOf<typename HighT<FT>::type>::v, c.root64, Bs + bl.root);
      else gridSaveRoot(c, ArithOf<FT>::v, c.root, Bs + bl.root);
    } else
#endif
    if (sizeof(FT) == 8) {
      const double* R = fs.use64 ? c.root64 : reinterpret_cast<const double*>(c.root);
#pragma unroll 1
      for (int64_t t = threadIdx.x; t < rs; t += blockDim.x) Bs[bl.root + t] = R[t];
    } else if (fs.use64) {
      const auto* R = rootHigh<FT>(c);
#pragma unroll 1
      for (int64_t t = threadIdx.x; t < rs; t += blockDim.x) Bs[bl.root + t] = (double)R[t];
    } else {
      const FT* R = rootT<FT>(c);
#pragma unroll 1
      for (int64_t t = threadIdx.x; t < rs; t += blockDim.x) Bs[bl.root + t] = (double)R[t];
    }
    FOR_T(r, m) {
      Bs[bl.cw + r] = c.cw[r];
      Bs[bl.cu + r] = c.cu[r];
      Bs[bl.zh + r] = c.z[r] / tau;
    }
    FOR_T(k, kSocScaleDoubles * c.nsoc) Bs[bl.sp + k] = reinterpret_cast<const double*>(c.sp)[k];
    FOR_T(j, n) Bs[bl.xh + j] = c.x[j] / tau;
    if (threadIdx.x == 0) {
      Bs[bl.sc + 0] = fs.ea;
      Bs[bl.sc + 1] = fs.ep;
      Bs[bl.sc + 2] = (double)status;
      Bs[bl.sc + 3] = tau;
    }
  }
  double nr2[2] = {0.0, 0.0};
  FOR_V(j, n, c.vb) nr2[0] += c.rx[j] * c.rx[j];
  FOR_V(r, m, c.vb) nr2[1] += c.rz[r] * c.rz[r];
  blockSum<2>(nr2, c.red, c.vb);
  if (status == 1 && st.warm_start && a.warmX) {
    FOR_T(j, n) a.warmX[D.vQ + j] = c.x[j];
    FOR_T(r, m) {
      a.warmS[D.vB + r] = c.s[r];
      a.warmZ[D.vB + r] = c.z[r];
    }
    if (threadIdx.x == 0 && a.haveWarm) a.haveWarm[inst] = 1;
  }
  if (threadIdx.x == 0) {
    DevResult R{};
    R.status = status;
    R.iterations = iterations;
    double pobj = (0.5 * dxPx / tau + dqx) / tau;
    double gap = dsz / (tau * tau);
    if (eq) {
      pobj /= cs;
      gap /= cs;
    }
    R.objective = pobj;
    R.duality_gap = gap;
    R.primal_residual = sqrt(nr2[1]) / fmax(tau, 1e-30);
    R.dual_residual = sqrt(nr2[0]) / fmax(tau, 1e-30);
    R.mu = (dsz + tau * kappa) / (double)(degree + 1);
    R.max_relres = c.sc[SC_MAXREL];
    R.fp64_fallbacks = (int)c.sc[SC_NFB];
    R.refine_steps = (int)c.sc[SC_RSTEPS];
    R.factor_attempts = (int)c.sc[SC_ATTEMPTS];
    R.escalations = (int)c.sc[SC_ESC];
    R.error_code = (G && reinterpret_cast<volatile GridCtl*>(c.grid)->error) ? 1 : 0;
    const long long tot = clock64() - tStart;
    R.cycles[0] = tot;
    if (st.record_timings) {
      unsigned long long wallEnd = 0;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(wallEnd));
      R.wall_ns[0] = (long long)wallStart;
      R.wall_ns[1] = (long long)wallEnd;
    }
    R.cycles[1] = timers(c)[TM_FACTOR];
    R.cycles[2] = timers(c)[TM_SOLVE];
    R.cycles[3] = tot - R.cycles[1] - R.cycles[2];
    R.cycles[4] = timers(c)[TM_ASSEMBLE];
    R.cycles[5] = timers(c)[TM_LDLT];
    R.cycles[6] = timers(c)[TM_DSOLVE];
    R.cycles[7] = timers(c)[TM_RESID];
    a.results[inst] = R;
  }
  __syncthreads();
}

// ------------------------------------------------------------------------------------------
// kernel: persistent CTAs over an atomic instance queue
// ------------------------------------------------------------------------------------------
// Points the per-instance context at shared memory, the CTA's scratch and the pools (thread 0).
static __device__ void setupCtx(Ctx& c, const LaunchArgs& a, int inst, unsigned char* smem, double* scratch, int* sRedi) {
  const SmemLayout& L = a.lay;
  const InstanceDesc& D = a.desc[inst];
  c.D = &D;
  c.vb = a.sumThreads;
  c.n = D.n; c.m = D.m; c.p = D.p; c.l = D.l; c.nsoc = D.nsoc; c.nr = D.nr; c.nUnits = D.nUnits;
  const int* I = a.ipool;
  c.pdiag = I + D.iPdiag;
  c.plowIdx = reinterpret_cast<const long long*>(I + D.iPlowIdx); c.plowSrc = I + D.iPlowSrc;
  c.ap = I + D.iAp; c.ai = I + D.iAi;
  c.arSrc = I + D.iArSrc;
  c.scUnit = I + D.iScUnit; c.scOff = I + D.iScOff;
  c.azIdx = reinterpret_cast<const long long*>(I + D.iAZIdx); c.azSrc = I + D.iAZSrc;
  c.socOff = I + D.iSocOff; c.socDim = I + D.iSocDim;
  c.unitAd = I + D.iUnitAd; c.unitSup = I + D.iUnitSup;
  c.tgtIdx = reinterpret_cast<const long long*>(I + D.iTgtIdx); c.tgtBeg = I + D.iTgtBeg; c.contrib = I + D.iContrib;
  // scratch carve-up for this instance (scaled P in user order, then its CSR-order copy)
  c.Pu = scratch + D.sPv;
  c.Pv = c.Pu + D.nnzPu;
  c.Av = scratch + D.sAv;
  c.gather = a.gatherA != 0;
  c.Avc = c.gather ? c.Av : scratch + D.sAc;
  c.Avr = c.gather ? c.Av : c.Avc + D.nnzA;
  c.sP = {c.Pv, I + D.iPsCol, I + D.iPsRow, I + D.iPsPerm, D.n, nullptr};
  c.sAc = {c.Avc, I + D.iAcCol, I + D.iAcRow, I + D.iAcPerm, D.n, I + D.iAcSrc};
  c.sAr = {c.Avr, I + D.iArCol, I + D.iArRow, I + D.iArPerm, D.m, I + D.iArSrc};
  c.Ad = scratch + D.sAd;
  c.T = scratch + D.sT;
  c.qs = scratch + D.sQ;
  c.bs = scratch + D.sB;
  c.root64 = L.root64InSmem ? reinterpret_cast<double*>(smem + L.rootOff) : scratch + D.sRoot64;
  // vectors: shared memory or scratch
  double* vb = L.vecInSmem ? reinterpret_cast<double*>(smem + L.vecOff) : scratch + D.sVec;
  const int nM = L.nMax, mM = L.mMax, NM = L.nMax + L.mMax, rM = rootTiles(L.nrMax) * kTile;
  double* q = vb;
  auto take = [&](int len) { double* r = q; q += (len + 1) & ~1; return r; };
  c.x = take(nM); c.rx = take(nM); c.x1 = take(nM); c.Px1 = take(nM); c.dx = take(nM); c.tn = take(nM);
  c.s = take(mM); c.z = take(mM); c.rz = take(mM); c.dz = take(mM); c.ds = take(mM);
  c.dcon = take(mM); c.lam = take(mM); c.tm = take(mM); c.tm2 = take(mM); c.cw = take(mM); c.cu = take(mM);
  c.rhs = take(NM); c.sol = take(NM); c.res = take(NM); c.cor = take(NM);
  c.rr = take(rM);
  c.sp = reinterpret_cast<SocScale*>(take(kSocScaleDoubles * L.nsocMax));
  // used once or twice per iteration: always in scratch (vecGlobalDoubles)
  c.ev = scratch + D.sVecG;
  c.z1 = c.ev + ((mM + 1) & ~1);
  c.root = L.rootInSmem ? reinterpret_cast<void*>(smem + L.rootOff) : reinterpret_cast<void*>(c.root64);
  c.red = reinterpret_cast<double*>(smem + L.redOff);
  c.sc = c.red + 128;
  c.kry = scratch + D.sKry;
  c.slices = reinterpret_cast<unsigned char*>(scratch + D.sSlice);
  c.redi = sRedi;
  c.grid = nullptr;
}

// ------------------------------------------------------------------------------------------
// kernel: persistent CTAs over an atomic instance queue
// ------------------------------------------------------------------------------------------
// kMaxThreads / kMinBlocks: the large-root form (up to 256 threads, registers for one CTA per
// SM) and the small-root form (up to 64 threads, at least 8 CTAs per SM: small instances are
// bound by FP64 latency, so more of them resident per SM is more throughput).

template <typename FT, int kMaxThreads, int kMinBlocks>
__global__ void __launch_bounds__(kMaxThreads, kMinBlocks) ipmKernel(LaunchArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int sInst;
  __shared__ int sRedi[4];
  __shared__ Ctx c;
  double* scratch = a.scratch + (int64_t)blockIdx.x * a.scratchStride;
  // the next size bucket's launch may begin once every CTA of this one is on an SM (LaunchArgs::after)
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  for (;;) {
    if (threadIdx.x == 0) sInst = atomicAdd(a.counter, 1);
    __syncthreads();
    const int slot = sInst;
    __syncthreads();
    if (slot >= a.count) break;
    const int inst = a.order[slot];
    if (threadIdx.x == 0) setupCtx(c, a, inst, smem, scratch, sRedi);
    __syncthreads();
    loadInstance(c, a);
    solveInstance<FT>(c, a, inst);
  }
  // What follows the last bucket in the stream must find all of them finished: a launch ends when its
  // first CTA has seen the one before it end, and so the last one after all. The other CTAs leave, so
  // that other streams have their SMs.
  if (blockIdx.x == 0) asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Whole-GPU form for one large instance (a.grid set): a cooperative launch with one CTA per SM.
// CTA 0 runs the iteration, the other CTAs run the root jobs it posts (see gridSync); the
// vectors, the root and the solve vector are in CTA 0's scratch (global memory) so every CTA can
// reach them. A kernel of its own, so that the batched kernels keep their register allocation.
template <typename FT>
__global__ void __launch_bounds__(256, 1) ipmGridKernel(LaunchArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int sRedi[4];
  __shared__ Ctx c;
  GridCtl* g = a.grid;
  if (blockIdx.x == 0) {
    const int inst = a.order[0];
    if (threadIdx.x == 0) {
      setupCtx(c, a, inst, smem, a.scratch, sRedi);
      c.grid = g;
      g->ctx = c;
      g->stageOff = a.lay.rootOff;  // the root itself is in scratch in this form
    }
    __syncthreads();
    loadInstance(c, a);
    solveInstance<FT, true>(c, a, inst);
    if (threadIdx.x == 0) g->op = kGridOpExit;
    gridSync(g);
  } else {
    gridWorker<FT>(g, a.st);
  }
}

// ------------------------------------------------------------------------------------------
// adjoint (new; no reference counterpart): differentiate the KKT conditions at the solution
// with one extra solve through the saved final factorisation,
//   K [u; v] = [D dL/dx; 0],  dL/dq = -u, dL/db = v, dL/dP = -(u x' + x u'), dL/dA = -(z u' + v x'),
// all in the equilibrated space and mapped back through D, E, c (P^ = c D P D, q^ = c D q,
// A^ = E A D, b^ = E b, x = D x^).
// ------------------------------------------------------------------------------------------
static __device__ __noinline__ void adjointInstance(Ctx& c, const LaunchArgs& a) {
  const InstanceDesc& D = *c.D;
  const double* Bs = a.bwd + D.bwdOff;
  const BwdLayout bl = bwdLayout(c.nr, c.n, c.m, c.nsoc);
  const int n = c.n, m = c.m;
  const int status = (int)Bs[bl.sc + 2];
  if (threadIdx.x < SC_COUNT) c.sc[threadIdx.x] = 0.0;
  FOR_T(r, m) {
    c.cw[r] = Bs[bl.cw + r];
    c.cu[r] = Bs[bl.cu + r];
  }
  FOR_T(k, kSocScaleDoubles * c.nsoc) reinterpret_cast<double*>(c.sp)[k] = Bs[bl.sp + k];
  if (a.lay.root64InSmem) {
    const int64_t rs = rootSize(c.nr);
#pragma unroll 1
    for (int64_t t = threadIdx.x; t < rs; t += blockDim.x) c.root64[t] = Bs[bl.root + t];
  } else if (threadIdx.x == 0) {
    c.root64 = const_cast<double*>(Bs + bl.root);
  }
  const double* dvec = a.dpool + D.dD;
  const double* evec = a.dpool + D.dE;
  const double cs = D.cscale;
  FOR_T(j, n) c.rhs[j] = dvec[j] * a.gx[D.vX + j];
  FOR_T(r, m) c.rhs[n + r] = 0.0;
  __syncthreads();
  const bool ok = status == 1;
  if (ok) {
    FactState fs{1, Bs[bl.sc + 1], Bs[bl.sc + 0]};
    kktSolve<double>(c, a.st, fs, c.rhs, c.sol);
  }
  const double* u = c.sol;
  const double* v = c.sol + n;
  const double* xh = Bs + bl.xh;
  const double* zh = Bs + bl.zh;
  const int* Pp = a.ipool + D.iPp;
  const int* Pi = a.ipool + D.iPi;
  FOR_T(j, n) {
    a.gq[D.vQ + j] = ok ? -u[j] * (cs * dvec[j]) : 0.0;
    for (int k = Pp[j]; k < Pp[j + 1]; ++k) {
      const int r = Pi[k];
      double g = 0.0;
      if (ok && r == j) g = -u[r] * xh[r];
      else if (ok && r < j) g = -(u[r] * xh[j] + u[j] * xh[r]);
      a.gP[D.vPx + k] = g * (cs * dvec[r] * dvec[j]);
    }
    for (int k = c.ap[j]; k < c.ap[j + 1]; ++k) {
      const int r = c.ai[k];
      a.gA[D.vAx + k] = ok ? -(zh[r] * u[j] + v[r] * xh[j]) * (evec[r] * dvec[j]) : 0.0;
    }
  }
  FOR_T(r, m) a.gb[D.vB + r] = ok ? v[r] * evec[r] : 0.0;
  __syncthreads();
}


// Host launchers of the kernels above, per root arithmetic FT (float: mixed precision, double:
// FP64) and launch form; explicitly instantiated in cxg_ipm_f32.cu, cxg_ipm_f32s.cu,
// cxg_ipm_f64.cu (batched forms) and cxg_ipm_gridf.cu, cxg_ipm_gridd.cu (whole-GPU form).
// Raises (never lowers) a kernel's dynamic shared-memory cap. The cap is one attribute of the
// function, while the size-bucket launches of one kernel form ask for different sizes: setting
// it to each launch's own size left the cap at the last bucket's, below what the earlier nodes of
// a captured graph carry, and a profiler replaying one of those nodes then failed to launch it.
// It also asks for the largest shared-memory carveout of the unified L1/shared array. An SM runs
// CTAs of different kernels side by side only while they share one carveout; with the driver's
// default choice the small-root forms (a few KB of shared memory) get a smaller carveout than the
// large ones, so the size buckets launched together could not share SMs and the small buckets
// started only once whole SMs had drained.
static inline cudaError_t raiseDynSmem(const void* k, size_t smem) {
  cudaFuncAttributes fa;
  cudaError_t e = cudaFuncGetAttributes(&fa, k);
  if (e != cudaSuccess) return e;
  if (fa.preferredShmemCarveout != (int)cudaSharedmemCarveoutMaxShared) {
    e = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return e;
  }
  if ((int)smem <= fa.maxDynamicSharedSizeBytes) return cudaSuccess;
  return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}

template <typename FT, int kMaxThreads, int kMinBlocks>
cudaError_t launchIpmFormT(const LaunchArgs& a, int grid, int block, size_t smem, cudaStream_t stream) {
  void (*k)(LaunchArgs) = ipmKernel<FT, kMaxThreads, kMinBlocks>;
  cudaError_t e = raiseDynSmem((const void*)k, smem);
  if (e != cudaSuccess) return e;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = &at;
  cfg.numAttrs = a.after ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, k, a);
}

template <typename FT, int kMaxThreads, int kMinBlocks>
cudaError_t ipmOccupancyFormT(int* blocksPerSM, int block, size_t smem) {
  void (*k)(LaunchArgs) = ipmKernel<FT, kMaxThreads, kMinBlocks>;
  cudaError_t e = raiseDynSmem((const void*)k, smem);
  if (e != cudaSuccess) return e;
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocksPerSM, k, block, smem);
}

template <typename FT>
cudaError_t launchIpmGridT(const LaunchArgs& a, GridCtl* g, int grid, size_t smem, cudaStream_t stream) {
  void (*k)(LaunchArgs) = ipmGridKernel<FT>;
  cudaError_t e = raiseDynSmem((const void*)k, smem);
  if (e != cudaSuccess) return e;
  LaunchArgs av = a;
  av.grid = g;
  void* args[] = {(void*)&av};
  return cudaLaunchCooperativeKernel((const void*)k, dim3(grid), dim3(256), args, smem, stream);
}

template <typename FT>
cudaError_t ipmGridOccupancyT(int* blocksPerSM, size_t smem) {
  void (*k)(LaunchArgs) = ipmGridKernel<FT>;
  cudaError_t e = raiseDynSmem((const void*)k, smem);
  if (e != cudaSuccess) return e;
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocksPerSM, k, 256, smem);
}

// Explicit instantiation (EXT empty) or declaration (EXT extern) of the launchers of one form.
#define CXG_IPM_FORM(EXT, FT, TH, MB)                                                            \
  EXT template cudaError_t launchIpmFormT<FT, TH, MB>(const LaunchArgs&, int, int, size_t, cudaStream_t); \
  EXT template cudaError_t ipmOccupancyFormT<FT, TH, MB>(int*, int, size_t);
#define CXG_IPM_GRID(EXT, FT)                                                                    \
  EXT template cudaError_t launchIpmGridT<FT>(const LaunchArgs&, GridCtl*, int, size_t, cudaStream_t); \
  EXT template cudaError_t ipmGridOccupancyT<FT>(int*, size_t);

}  // namespace cxg
