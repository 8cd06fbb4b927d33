// Device-side cone algebra (FP64), one cone unit per call.
//
// Semantics follow src/conicxx/cones/{nonnegative_cone,second_order_cone,zero_cone}.cpp and
// cone_set.cpp; the Nesterov-Todd scaling of a second-order block is held in eigen-form rather
// than as the dense W = beta (2 v v' - J) the reference caches (second_order_cone.cpp:132-158):
// W acts as beta * I off the plane span{e0, (0, u)} (u = v1/|v1|) and as beta * B in it,
// B = [[2v0^2-1, 2 v0 |v1|], [2 v0 |v1|, 2|v1|^2+1]] with eigenvalues lambda, 1/lambda
// (det B = 2 v'Jv - 1 = 1). Every operator the interior-point method needs -- W, W^-1,
// Hs = W^2, Hs + eps I and (Hs + eps I)^-1 -- is then f(W) for a scalar f, applied in O(dim)
// along the eigenvectors. Applying these near-singular operators as dense matrices loses all
// accuracy once cond(Hs) approaches 1/eps_machine (Hs * (Hs+eps)^-1 - I reaches O(0.1) in FP64),
// whereas the eigen-form round trip stays at FP64 rounding.
#pragma once

#include <cuda_runtime.h>
#include <math.h>

#include "cxg_layout.h"

namespace cxg {

// Finiteness and sign from the bits (integer tests: an FP64 comparison holds the FP64 unit of its
// sub-partition for 64 cycles).
__device__ __forceinline__ bool finiteBits(double v) {
  return ((__double_as_longlong(v) >> 52) & 0x7ff) != 0x7ff;
}
__device__ __forceinline__ bool negBits(double v) {  // v < 0
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  return b > 0x8000000000000000ull && b <= 0xfff0000000000000ull;
}

// Order of doubles as integers (NaN outside both infinities), and minima / maxima on it with fmin's
// and fmax's treatment of NaN.
__device__ __forceinline__ long long orderKey(double v) {
  const long long b = __double_as_longlong(v);
  return b ^ ((b >> 63) & 0x7fffffffffffffffll);
}
__device__ __forceinline__ bool nanBits(double v) {
  return (__double_as_longlong(v) & 0x7fffffffffffffffll) > 0x7ff0000000000000ll;
}
__device__ __forceinline__ double minBits(double a, double b) {
  if (nanBits(a)) return b;
  if (nanBits(b)) return a;
  return orderKey(b) < orderKey(a) ? b : a;
}
__device__ __forceinline__ double maxBits(double a, double b) {
  if (nanBits(a)) return b;
  if (nanBits(b)) return a;
  return orderKey(b) > orderKey(a) ? b : a;
}
__device__ __forceinline__ bool zeroBits(double v) { return (__double_as_longlong(v) << 1) == 0; }
// a < b (false when either is NaN)
__device__ __forceinline__ bool lessBits(double a, double b) {
  return !nanBits(a) && !nanBits(b) && orderKey(a) < orderKey(b) && !(zeroBits(a) && zeroBits(b));
}
__device__ __forceinline__ bool posBits(double v) {  // v > 0
  const long long b = __double_as_longlong(v);
  return b > 0 && b <= 0x7ff0000000000000ll;
}
__device__ __forceinline__ bool nonNegBits(double v) {  // v >= 0
  const long long b = __double_as_longlong(v);
  return (b >= 0 && b <= 0x7ff0000000000000ll) || b == (long long)0x8000000000000000ull;
}

constexpr double kTiny = 1e-12;                    // second_order_cone.cpp:23
constexpr double kDblMin = 2.2250738585072014e-308;
constexpr double kStepDegenerateEps = kDblMin * 1e4;  // second_order_cone.cpp:32
constexpr double kTinyRel = 1e-12;                 // second_order_cone.cpp:89
constexpr double kAbsFloor = kDblMin * 1e4;        // second_order_cone.cpp:90
constexpr double kBetaMax = 1e8;                   // second_order_cone.cpp:106
constexpr double kWMax = 1e8;                      // second_order_cone.cpp:152
// relative resolution of a dense FP64 Hs = W W (one ulp of its largest eigenvalue); see the
// reference dense form below
constexpr double kHsRes = 2.220446049250313e-16;

// Per-SOC-block scaling parameters (8 doubles in shared memory): beta, lam = lambda (plane) or
// a = 2v0^2-1 (diagonal), w2 = beta / lambda (plane), the small in-plane eigenvalue of W, kept since a
// division costs as much as nine multiply-adds and every application needs it, qc, qs (in-plane
// eigenvector of lambda), and the three eigenvalues of G = (Hs + eps I)^-1 prepared at factorisation
// time (socPrepareG). The unit vector u is kept in a row-indexed array at rows off+1 .. off+dim-1,
// whose row off holds the block's kind (socKind): 0 identity fallback, 1 diagonal, 2 plane, 3 plane
// with the small eigenvalue of Hs held at the dense form's resolution (hsSmall). A ninth double for
// the kind would move the sizes at which the vectors and the root fit in shared memory.
struct SocScale {
  double beta, lam, w2, qc, qs, r0, r1, r2;
};
__device__ __forceinline__ int socKind(const double* u) { return __double2loint(u[0]); }
__device__ __forceinline__ void setSocKind(double* u, int kind) { u[0] = __hiloint2double(0, kind); }
static_assert(sizeof(SocScale) == 8 * kSocScaleDoubles, "SocScale is kept in arrays of doubles");

// Computes the NT scaling of one SOC block from (s, z) (second_order_cone.cpp:70-159): the same
// clamps (margin floors, beta clamp, c floor, v0 floor) and the same identity fallback test on
// the entries of W = beta (2 v v' - J). DIM: the block's dimension where it is known when
// compiling (registers instead of loops), else 0. The sums are written as fused multiply-adds: an
// unrolled sum's first two products could otherwise be fused either way round.
template <int DIM>
__device__ __forceinline__ void socUpdateScalingDim(const double* s, const double* z, int dim, SocScale& sc, double* u) {
  const int d = DIM ? DIM : dim;
  double s1sq = 0, z1sq = 0, sz = 0;
#pragma unroll
  for (int i = 1; i < d; ++i) {
    s1sq = fma(s[i], s[i], s1sq);
    z1sq = fma(z[i], z[i], z1sq);
  }
#pragma unroll
  for (int i = 0; i < d; ++i) sz = fma(s[i], z[i], sz);
  const double s0 = s[0], z0 = z[0];
  const double a = sqrt(maxBits(maxBits(s0 * s0 - s1sq, kTinyRel * s0 * s0), kAbsFloor));
  const double b = sqrt(maxBits(maxBits(z0 * z0 - z1sq, kTinyRel * z0 * z0), kAbsFloor));
  const double beta = minBits(maxBits(sqrt(a / b), 1.0 / kBetaMax), kBetaMax);
  const double c = sqrt(maxBits((sz / (a * b) + 1.0) / 2.0, kTiny));
  // v = (s/a + J z / b) / (2c); v0 += 1; v0 = max(v0, tiny); v /= sqrt(2 v0)
  double v0 = (z0 / b + s0 / a) / (2.0 * c);
  v0 += 1.0;
  v0 = maxBits(v0, kTiny);
  const double nrm = sqrt(2.0 * v0);
  v0 /= nrm;
  double n1sq = 0.0, vmax1 = 0.0, vmax2 = 0.0, vdiagmax = 0.0;
  bool finite = finiteBits(v0) && finiteBits(beta);
#pragma unroll
  for (int i = 1; i < d; ++i) {
    const double vi = ((-z[i] / b + s[i] / a) / (2.0 * c)) / nrm;
    u[i] = vi;
    n1sq = fma(vi, vi, n1sq);
    const double av = fabs(vi);
    if (lessBits(vmax1, av)) { vmax2 = vmax1; vmax1 = av; } else if (lessBits(vmax2, av)) { vmax2 = av; }
    vdiagmax = maxBits(vdiagmax, fabs(2.0 * vi * vi + 1.0));
    finite = finite && finiteBits(vi);
  }
  // max |W_ij| / beta over the explicit W = beta (2 v v' - J)
  double wmax = fabs(2.0 * v0 * v0 - 1.0);
  wmax = maxBits(wmax, vdiagmax);
  wmax = maxBits(wmax, 2.0 * fabs(v0) * vmax1);
  if (d > 2) wmax = maxBits(wmax, 2.0 * vmax1 * vmax2);
  wmax *= beta;
  // Hs = W W has entries up to ~dim * wmax^2: finite whenever W is finite and wmax <= 1e8.
  if (!finite || nanBits(wmax) || lessBits(kWMax, wmax)) {
    setSocKind(u, 0);
    sc.beta = 1.0;
    sc.lam = 1.0;
    sc.w2 = 1.0;
    sc.qc = 1.0;
    sc.qs = 0.0;
    return;
  }
  const double n1 = sqrt(n1sq);
  sc.beta = beta;
  if (zeroBits(n1) || d == 1) {
    setSocKind(u, 1);
    sc.lam = 2.0 * v0 * v0 - 1.0;
    sc.w2 = beta;
    sc.qc = 1.0;
    sc.qs = 0.0;
#pragma unroll
    for (int i = 1; i < d; ++i) u[i] = 0.0;
    return;
  }
#pragma unroll
  for (int i = 1; i < d; ++i) u[i] /= n1;
  const double A = 2.0 * v0 * v0 - 1.0, C = 2.0 * v0 * n1, E = 2.0 * n1 * n1 + 1.0;
  const double h = 0.5 * (A + E);
  const double r = hypot(0.5 * (A - E), C);
  const double l1 = h + r;
  double qa, qb;
  if (!lessBits(A, E)) { qa = l1 - E; qb = C; } else { qa = C; qb = l1 - A; }
  const double qn = hypot(qa, qb);
  setSocKind(u, 2);
  sc.lam = l1;
  sc.w2 = beta / l1;
  sc.qc = qa / qn;
  sc.qs = qb / qn;
}

__device__ __forceinline__ void socUpdateScaling(const double* s, const double* z, int d, SocScale& sc, double* u) {
  if (d == 3) socUpdateScalingDim<3>(s, z, d, sc, u);
  else if (d == 4) socUpdateScalingDim<4>(s, z, d, sc, u);
  else socUpdateScalingDim<0>(s, z, d, sc, u);
}

// Scalar functions of W used by the method.
enum WFun { kW = 0, kWinv = 1, kHs = 2, kHsEps = 3, kGinv = 4 };

__device__ __forceinline__ double wfun(int f, double w, double eps) {
  switch (f) {
    case kW: return w;
    case kWinv: return 1.0 / w;
    case kHs: return w * w;
    case kHsEps: return w * w + eps;
    default: return 1.0 / (w * w + eps);
  }
}

// w^2 + eps, fused or with the square rounded first. Which of the two an expression takes is written
// out below, so that it does not depend on what the compiler finds in one basic block.
__device__ __forceinline__ double sqEps(double w, double eps, bool fused) {
  return fused ? __fma_rn(w, w, eps) : __dadd_rn(__dmul_rn(w, w), eps);
}
// wfun for an eigenvalue of a SOC block's W.
__device__ __forceinline__ double wfunSoc(int f, double w, double eps, bool fused) {
  switch (f) {
    case kW: return w;
    case kWinv: return 1.0 / w;
    case kHs: return w * w;
    case kHsEps: return sqEps(w, eps, fused);
    default: return 1.0 / sqEps(w, eps, fused);
  }
}

// Functions of Hs given one of its eigenvalues h (f = kHs, kHsEps, kGinv).
__device__ __forceinline__ double hsfun(int f, double h, double eps) {
  return f == kHs ? h : (f == kHsEps ? __dadd_rn(h, eps) : 1.0 / __dadd_rn(h, eps));
}

// The small in-plane eigenvalue of Hs of a kind-3 block: (beta / lambda)^2, held at no less than
// kHsRes (beta lambda)^2.
__device__ __forceinline__ double hsSmall(const SocScale& sc) {
  const double w1 = sc.beta * sc.lam, w2 = sc.w2;
  return maxBits(__dmul_rn(w2, w2), __dmul_rn(kHsRes, __dmul_rn(w1, w1)));
}

// y = f(W) x for one SOC block (x, y may alias only if identical).
template <int DIM>
__device__ __forceinline__ void socApplyDim(const SocScale& sc, const double* u, int dim, int f, double eps,
                                            const double* x, double* y) {
  const int d = DIM ? DIM : dim;
  const int kind = socKind(u);
  if (kind == 0) {
    const double g = wfun(f, 1.0, eps);
    for (int i = 0; i < d; ++i) y[i] = g * x[i];
    return;
  }
  if (kind == 1) {
    const double g0 = wfun(f, sc.beta * sc.lam, eps), g = wfun(f, sc.beta, eps);
    const double x0 = x[0];
    for (int i = 1; i < d; ++i) y[i] = g * x[i];
    y[0] = g0 * x0;
    return;
  }
  const double x0 = x[0];
  double xf = 0.0;
#pragma unroll
  for (int i = 1; i < d; ++i) xf = fma(u[i], x[i], xf);
  const double c1 = sc.qc * x0 + sc.qs * xf;
  const double c2 = -sc.qs * x0 + sc.qc * xf;
  const double f1 = wfunSoc(f, sc.beta * sc.lam, eps, true);
  const double f2 = (kind == 3 && f >= kHs) ? hsfun(f, hsSmall(sc), eps) : wfunSoc(f, sc.w2, eps, false);
  const double f3 = wfunSoc(f, sc.beta, eps, true);
  const double y0 = f1 * c1 * sc.qc - f2 * c2 * sc.qs;
  const double yF = f1 * c1 * sc.qs + f2 * c2 * sc.qc;
#pragma unroll
  for (int i = 1; i < d; ++i) y[i] = f3 * (x[i] - xf * u[i]) + yF * u[i];
  y[0] = y0;
}
__device__ __forceinline__ void socApply(const SocScale& sc, const double* u, int d, int f, double eps,
                                         const double* x, double* y) {
  if (d == 3) socApplyDim<3>(sc, u, d, f, eps, x, y);
  else if (d == 4) socApplyDim<4>(sc, u, d, f, eps, x, y);
  else socApplyDim<0>(sc, u, d, f, eps, x, y);
}

// G = (Hs + eps I)^-1 of one SOC block as its three eigenvalues (stored in sc.r0..r2).
__device__ __forceinline__ void socPrepareG(SocScale& sc, const double* u, double eps) {
  const int kind = socKind(u);
  if (kind == 0) {
    const double g = 1.0 / (1.0 + eps);
    sc.r0 = sc.r1 = sc.r2 = g;
  } else if (kind == 1) {
    const double w0 = sc.beta * sc.lam, w = sc.beta;
    sc.r0 = 1.0 / (w0 * w0 + eps);
    sc.r1 = sc.r2 = 1.0 / (w * w + eps);
  } else {
    const double w1 = sc.beta * sc.lam, w2 = sc.w2, w3 = sc.beta;
    sc.r0 = 1.0 / sqEps(w1, eps, false);
    sc.r1 = 1.0 / (kind == 3 ? __dadd_rn(hsSmall(sc), eps) : sqEps(w2, eps, false));
    sc.r2 = 1.0 / sqEps(w3, eps, true);
  }
}

// y = G x with the eigenvalues prepared by socPrepareG (same structure as socApply).
template <int DIM>
__device__ __forceinline__ void socApplyGDim(const SocScale& sc, const double* u, int dim, const double* x, double* y) {
  const int d = DIM ? DIM : dim;
  const int kind = socKind(u);
  if (kind == 0) {
    for (int i = 0; i < d; ++i) y[i] = sc.r0 * x[i];
    return;
  }
  if (kind == 1) {
    const double x0 = x[0];
    for (int i = 1; i < d; ++i) y[i] = sc.r1 * x[i];
    y[0] = sc.r0 * x0;
    return;
  }
  const double x0 = x[0];
  double xf = 0.0;
#pragma unroll
  for (int i = 1; i < d; ++i) xf = fma(u[i], x[i], xf);
  const double c1 = sc.qc * x0 + sc.qs * xf;
  const double c2 = -sc.qs * x0 + sc.qc * xf;
  const double y0 = sc.r0 * c1 * sc.qc - sc.r1 * c2 * sc.qs;
  const double yF = sc.r0 * c1 * sc.qs + sc.r1 * c2 * sc.qc;
#pragma unroll
  for (int i = 1; i < d; ++i) y[i] = sc.r2 * (x[i] - xf * u[i]) + yF * u[i];
  y[0] = y0;
}
__device__ __forceinline__ void socApplyG(const SocScale& sc, const double* u, int d, const double* x, double* y) {
  if (d == 3) socApplyGDim<3>(sc, u, d, x, y);
  else if (d == 4) socApplyGDim<4>(sc, u, d, x, y);
  else socApplyGDim<0>(sc, u, d, x, y);
}

// Jordan product (second_order_cone.cpp:43-48); out may alias neither u nor v.
__device__ __forceinline__ void socProduct(const double* u, const double* v, int d, double* out) {
  double dt = 0.0;
  for (int i = 0; i < d; ++i) dt += u[i] * v[i];
  const double u0 = u[0], v0 = v[0];
  for (int i = 1; i < d; ++i) out[i] = u0 * v[i] + v0 * u[i];
  out[0] = dt;
}

// Inverse Jordan product u \ w (second_order_cone.cpp:50-68).
__device__ __forceinline__ void socInverseProduct(const double* u, const double* w, int d, double* out) {
  double u0 = u[0];
  double u1sq = 0.0, nu = 0.0;
  for (int i = 1; i < d; ++i) {
    u1sq += u[i] * u[i];
    nu += u[i] * w[i];
  }
  double rho = u0 * u0 - u1sq;
  if (lessBits(fabs(rho), kTiny)) rho = (nonNegBits(rho) ? kTiny : -kTiny);
  if (lessBits(fabs(u0), kTiny)) u0 = kTiny;
  const double w0 = w[0];
  const double k1 = (nu / u0 - w0), k2 = (rho / u0);
  for (int i = 1; i < d; ++i) out[i] = (k1 * u[i] + k2 * w[i]) / rho;
  out[0] = (u0 * w0 - nu) / rho;
}

// Largest step in [0, amax] keeping x + a dx in the closed SOC (second_order_cone.cpp:174-215).
__device__ __forceinline__ double socMaxStep(const double* x, const double* dx, int d, double amax) {
  const double p0 = x[0], d0 = dx[0];
  double d1sq = 0, p1d1 = 0, p1sq = 0;
  for (int i = 1; i < d; ++i) {
    d1sq += dx[i] * dx[i];
    p1d1 += x[i] * dx[i];
    p1sq += x[i] * x[i];
  }
  const double a = d0 * d0 - d1sq;
  const double b = 2.0 * (p0 * d0 - p1d1);
  const double c = p0 * p0 - p1sq;
  double alpha = amax;
  if (lessBits(fabs(a), kStepDegenerateEps)) {
    if (lessBits(kStepDegenerateEps, fabs(b))) {
      const double r = -c / b;
      if (posBits(r) && nonNegBits(p0 + r * d0)) alpha = minBits(alpha, r);
    }
    return alpha;
  }
  const double disc = b * b - 4.0 * a * c;
  if (negBits(disc)) return alpha;
  const double sq = sqrt(disc);
  const double q = nonNegBits(b) ? -0.5 * (b + sq) : -0.5 * (b - sq);
  double r1, r2;
  if (lessBits(kStepDegenerateEps, fabs(q))) {
    r1 = q / a;
    r2 = c / q;
  } else {
    r1 = r2 = -b / (2.0 * a);
  }
  if (posBits(r1) && nonNegBits(p0 + r1 * d0)) alpha = minBits(alpha, r1);
  if (posBits(r2) && nonNegBits(p0 + r2 * d0)) alpha = minBits(alpha, r2);
  return alpha;
}

// ---- a second-order block in the reference's dense FP64 form -----------------------------
// The reference keeps a block's Hs = W W as a dense FP64 matrix, W = beta (2 v v' - J) formed
// entry by entry (second_order_cone.cpp:132-158). Near the cone boundary the in-plane eigenvalues
// of Hs, beta^2 lambda^2 and beta^2 / lambda^2, lie more than 1/eps_machine apart, and the dense
// entries no longer carry the small one: it is replaced by rounding of the order of
// eps_machine * beta^2 lambda^2. The eigen-form held here is exact to rounding. Two of the
// reference's decisions depend on that rounding, and both are reproduced from the dense entries
// in the reference's arithmetic (its operation order, no fused multiply-adds) for blocks of up to
// kRefDenseMaxDim rows:
//  - the sparse LDL' of K (qdldl_ldlt.cpp:58-69) takes a block's rows before the x rows they
//    couple to (a block row has degree dim - 1 + the nonzeros of its A row), so the block
//    -(Hs + eps I) is factored on its own; its last pivot comes out zero or below
//    dynamic_reg_eps and factorizeWithRetry (kkt_system.cpp:242-264) fails the attempt and raises
//    the bump x10 until the bump survives the block's rounding (socRefLadderLevel);
//  - Hs itself: from the first iteration in which that pivot test fails, the instance holds the
//    small in-plane eigenvalue of Hs at no less than kHsRes times the large one (kind 3 in
//    SocScale: Hs, Hs + eps I and G; W and W^-1 stay exact), the resolution of the dense form.
//    With the exact small eigenvalue the iteration drives the complementarity of such blocks to
//    zero ahead of primal feasibility and then stalls (configuration 2's family from 3000
//    variables on; the reference's own iteration with exact Hs products slows from 26 to 76
//    iterations there); at the dense form's resolution it converges as the reference does.
constexpr int kRefDenseMaxDim = 8;
constexpr int kLadderLevels = 18;  // factorizeWithRetry's attempts (kkt_system.cpp:242-264)

// the bump of ladder attempt `level`: 0, delta, 10 delta, ... (kkt_system.cpp:258-259)
__host__ __device__ __forceinline__ double ladderBump(int level, double delta) {
  double e = 0.0;
  for (int k = 0; k < level; ++k) e = fmax(e * 10.0, delta);
  return e;
}

// Dense Hs of one block (row-major d x d, d <= kRefDenseMaxDim) in the reference's arithmetic;
// false for the identity fallback (W non-finite or max |W_ij| > 1e8), where Hs = I (not written).
// W and Hs are symmetric to the last bit here (doubling is exact, products commute and the sums run
// over the same terms in the same order), so only their lower triangles are formed.
template <int DIM>
static __device__ __forceinline__ bool socRefHs(const double* s, const double* z, int dim, double* Hs) {
  constexpr int kMax = DIM ? DIM : kRefDenseMaxDim;
  const int d = DIM ? DIM : dim;
  double v[kMax];
  double s1sq = 0.0, z1sq = 0.0, sz = 0.0;
#pragma unroll
  for (int i = 1; i < d; ++i) {
    s1sq = __dadd_rn(s1sq, __dmul_rn(s[i], s[i]));
    z1sq = __dadd_rn(z1sq, __dmul_rn(z[i], z[i]));
  }
#pragma unroll
  for (int i = 0; i < d; ++i) sz = __dadd_rn(sz, __dmul_rn(s[i], z[i]));
  const double s0 = s[0], z0 = z[0];
  const double a = __dsqrt_rn(
      maxBits(maxBits(__dsub_rn(__dmul_rn(s0, s0), s1sq), __dmul_rn(__dmul_rn(kTinyRel, s0), s0)), kAbsFloor));
  const double b = __dsqrt_rn(
      maxBits(maxBits(__dsub_rn(__dmul_rn(z0, z0), z1sq), __dmul_rn(__dmul_rn(kTinyRel, z0), z0)), kAbsFloor));
  const double beta = minBits(maxBits(__dsqrt_rn(__ddiv_rn(a, b)), 1.0 / kBetaMax), kBetaMax);
  const double c = __dsqrt_rn(maxBits(__dmul_rn(__dadd_rn(__ddiv_rn(sz, __dmul_rn(a, b)), 1.0), 0.5), kTiny));
  v[0] = __dadd_rn(__ddiv_rn(z0, b), __ddiv_rn(s0, a));
#pragma unroll
  for (int i = 1; i < d; ++i) v[i] = __dadd_rn(__ddiv_rn(-z[i], b), __ddiv_rn(s[i], a));
  const double c2 = __dmul_rn(2.0, c);
#pragma unroll
  for (int i = 0; i < d; ++i) v[i] = __ddiv_rn(v[i], c2);
  v[0] = maxBits(__dadd_rn(v[0], 1.0), kTiny);
  const double nrm = __dsqrt_rn(__dmul_rn(2.0, v[0]));
#pragma unroll
  for (int i = 0; i < d; ++i) v[i] = __ddiv_rn(v[i], nrm);
  double W[kMax * kMax];
  double wmax = 0.0;
  bool finite = true;
#pragma unroll
  for (int r = 0; r < d; ++r)
#pragma unroll
    for (int cc = 0; cc <= r; ++cc) {
      double w = __dmul_rn(__dmul_rn(2.0, v[r]), v[cc]);
      if (r == cc) w = (r == 0) ? __dsub_rn(w, 1.0) : __dadd_rn(w, 1.0);
      w = __dmul_rn(w, beta);
      finite = finite && finiteBits(w);
      wmax = maxBits(wmax, fabs(w));
      W[r * kMax + cc] = W[cc * kMax + r] = w;
    }
  if (!finite || lessBits(kWMax, wmax)) return false;
#pragma unroll
  for (int r = 0; r < d; ++r)
#pragma unroll
    for (int cc = 0; cc <= r; ++cc) {
      double acc = 0.0;
#pragma unroll
      for (int k = 0; k < d; ++k) acc = __dadd_rn(acc, __dmul_rn(W[r * kMax + k], W[k * kMax + cc]));
      finite = finite && finiteBits(acc);
      Hs[r * kMax + cc] = acc;
    }
  return finite;
}

// Whether every dense pivot of a block passes at level 0 whatever the rounding, from a bound in
// FP32: the largest eigenvalue of Hs is at most (a / b)(s0 / a + z0 / b)^2, a^2 = s0^2 - |s1|^2, b^2 =
// z0^2 - |z1|^2. The dense entries and the LDL' of d <= 8 rows together change Hs by less than
// 1000 eps times it, and every pivot of an exact Hs + sregA I is at least sregA; so while 1000 eps
// |Hs| < sregA / 4 and deps < sregA / 4 the pivots pass. The FP32 values carry relative errors of
// about 1e-6 (the margins s0 - |s1| are used only above 1e-3 s0), far inside the factor four.
__device__ __forceinline__ bool socPivotsPass(const double* s, const double* z, int d, double sregA, double deps) {
  const float s0 = (float)s[0], z0 = (float)z[0];
  float s1 = 0.0f, z1 = 0.0f;
  for (int i = 1; i < d; ++i) {
    const float si = (float)s[i], zi = (float)z[i];
    s1 = fmaf(si, si, s1);
    z1 = fmaf(zi, zi, z1);
  }
  s1 = sqrtf(s1);
  z1 = sqrtf(z1);
  const float sm = s0 - s1, zm = z0 - z1;
  if (!(sm > 1e-3f * s0) || !(zm > 1e-3f * z0) || !(s0 > 1e-15f) || !(z0 > 1e-15f) || !(s0 < 1e15f) || !(z0 < 1e15f))
    return false;
  const float a = sqrtf(sm * (s0 + s1)), b = sqrtf(zm * (z0 + z1));
  const float t = s0 / a + z0 / b;
  const float hs = (a / b) * t * t, reg = (float)sregA;
  return hs * (1000.0f * 2.22e-16f) < 0.25f * reg && (float)deps < 0.25f * reg;
}

// The first ladder level (attempt index, 0..17) at which the block's dense pivots all pass, or
// 18 when none does; the search starts at startLevel (a block that passes there returns
// startLevel). Blocks of one row or above kRefDenseMaxDim rows: 0.
template <int DIM>
static __device__ __noinline__ int socRefLadderDim(const double* s, const double* z, int dim, double sregA, double deps,
                                                   double delta, int startLevel) {
  constexpr int kMax = DIM ? DIM : kRefDenseMaxDim;
  const int d = DIM ? DIM : dim;
  double Hs[kMax * kMax];
  if (!socRefHs<DIM>(s, z, d, Hs)) return 0;  // Hs = I: every pivot passes
  for (int level = startLevel; level < kLadderLevels; ++level) {
    const double ea = ladderBump(level, delta);
    // up-looking LDL' of -(Hs + sregA I) - ea I in natural order, QDLDL's operation order
    double L[kMax * kMax], Dinv[kMax], y[kMax];
    bool ok = true;
#pragma unroll
    for (int k = 0; k < d; ++k) {
      if (!ok) break;
      double Dk = __dsub_rn(-Hs[k * kMax + k], sregA);
      if (!zeroBits(ea)) Dk = __dsub_rn(Dk, ea);
#pragma unroll
      for (int r = 0; r < k; ++r) y[r] = -Hs[k * kMax + r];
#pragma unroll
      for (int cc = 0; cc < k; ++cc) {
        const double yc = y[cc];
#pragma unroll
        for (int r = cc + 1; r < k; ++r) y[r] = __dsub_rn(y[r], __dmul_rn(L[r * kMax + cc], yc));
        const double l = __dmul_rn(yc, Dinv[cc]);
        L[k * kMax + cc] = l;
        Dk = __dsub_rn(Dk, __dmul_rn(yc, l));
      }
      ok = finiteBits(Dk) && lessBits(deps, fabs(Dk));
      if (k + 1 < d) Dinv[k] = __ddiv_rn(1.0, Dk);
    }
    if (ok) return level;
  }
  return kLadderLevels;
}

__device__ __forceinline__ int socRefLadderExact(const double* s, const double* z, int d, double sregA, double deps,
                                                 double delta, int startLevel) {
  if (d == 2) return socRefLadderDim<2>(s, z, d, sregA, deps, delta, startLevel);
  if (d == 3) return socRefLadderDim<3>(s, z, d, sregA, deps, delta, startLevel);
  if (d == 4) return socRefLadderDim<4>(s, z, d, sregA, deps, delta, startLevel);
  return socRefLadderDim<0>(s, z, d, sregA, deps, delta, startLevel);
}

__device__ __forceinline__ int socRefLadderLevel(const double* s, const double* z, int d, double sregA, double deps,
                                                 double delta, int startLevel) {
  if (d > kRefDenseMaxDim || d < 2) return 0;
  if (socPivotsPass(s, z, d, sregA, deps)) return startLevel;
  return socRefLadderExact(s, z, d, sregA, deps, delta, startLevel);
}

__device__ __forceinline__ double socMargin(const double* x, int d) {
  double t = 0.0;
  for (int i = 1; i < d; ++i) t += x[i] * x[i];
  return x[0] - sqrt(t);
}

}  // namespace cxg
