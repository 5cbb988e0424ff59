// Per-state RMHD physics for the B200 step kernels: gamma-law EOS, P->U, flux and exact
// fast-magnetosonic speeds (quartic), the c2p Newton ladder, PLM / WENO5 reconstruction and
// the HLL / HLLC / HLLD Riemann solvers.
//
// Everything is templated on the bulk arithmetic type T.  With T = double and the
// translation unit compiled with --fmad=false, every expression is evaluated in the same
// IEEE operation order as the reference's gcc build (quotients by a shared divisor through its
// reciprocal, with the same bits), so the plain FP64 path reproduces the reference bit for bit
// except in two places: CUDA's pow/acos/cos/sin differ from glibc by an ulp (the quartic only),
// and the root of HLLD's eq. 48 is reached by fewer evaluations from a start that is inverted in
// FP32 (hlld_solve: the same root and the same fallbacks, the flux to rounding, 1e-12 at worst).
// With T = float the same algorithms run in FP32 with tolerances rescaled to FP32 resolution
// (RmhdTol<float>); the c2p starts in FP32 and ends in FP64, on the FP64 path's bound.
//
// Reference sources restated here (paths within the reference project):
//   EOS          Mara/eos.cpp:13-29                    P->U         Mara/rmhd.cpp:177-207
//   flux, speeds Mara/rmhd.cpp:208-310                 quartic      Mara/quartic.cpp:28-148
//   c2p          Mara/rmhd-c2p.c:132-376, Mara/rmhd.cpp:103-176
//   PLM / WENO5  Mara/weno.c:15-154                    HLL          Mara/riemann_hll.cpp:19-64
//   HLLC         Mara/riemann_hllc-rmhd.cpp:26-178
//   HLLD         Mara/riemann_hlld-rmhd.cpp:179-615, Newton Mara/nrsolver.cpp:89-152
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include "rmhd_types.cuh"

namespace mgpu {

// Tolerances of the Riemann solvers.  For double they are the reference's literals; the
// float set is scaled to FP32 resolution (the FP32 bulk path has no reference oracle and is
// compared with the FP64 path).
template <class T> struct RmhdTol;
template <> struct RmhdTol<double> {
  static constexpr double newton_eps = 1e-12;   // NewtonRaphesonSolver(15, 1e-12)
  static constexpr double jac_dp = 1e-8;        // HlldEquation48::Jacobian
  static constexpr double x_small = 1e-8;       // |X| < 1e-8 (eqs 23-25)
  static constexpr double k_small = 1e-10;      // |Kr-Kl|, |delK|, |Bc_x|, |denom|
  static constexpr double tol54 = 1e-14;        // TOL in ReconstructSolution
  static constexpr double contact = 1e-8;       // UnmatchedContactSpeed
  static constexpr double degenerate = 1e-8;    // |am - aL.v| etc.
  static constexpr double bx_small = 1e-8;      // |Bx| < 1e-8 -> eq. (55) guess only
  static constexpr double hllc_bx = 1e-12;      // SMALL_BX
  static constexpr double hllc_a = 1e-10;       // SMALL_A
};
template <> struct RmhdTol<float> {
  static constexpr float newton_eps = 2e-6f;
  static constexpr float jac_dp = 2e-3f;
  static constexpr float x_small = 1e-6f;
  static constexpr float k_small = 1e-6f;
  static constexpr float tol54 = 1e-6f;
  static constexpr float contact = 2e-4f;
  static constexpr float degenerate = 1e-6f;
  static constexpr float bx_small = 1e-6f;
#ifdef MGPU_HLLC_BX_F32
  static constexpr float hllc_bx = MGPU_HLLC_BX_F32;
#else
  static constexpr float hllc_bx = 1e-7f;
#endif
  static constexpr float hllc_a = 1e-6f;
};

__device__ __forceinline__ double m_sqrt(double x) { return sqrt(x); }
__device__ __forceinline__ float m_sqrt(float x) { return sqrtf(x); }
__device__ __forceinline__ double m_abs(double x) { return fabs(x); }
__device__ __forceinline__ float m_abs(float x) { return fabsf(x); }
// out of line: the one-real-root branch of the resolvent cubic is rare (no face of the turbulence
// states, 0.4% of the stress box's)
static __device__ __noinline__ double m_cbrt_pow(double x) { return pow(x, 1. / 3.); }
__device__ __forceinline__ float m_cbrt_pow(float x) { return cbrtf(x); }
__device__ __forceinline__ double m_acos(double x) { return acos(x); }
__device__ __forceinline__ float m_acos(float x) { return acosf(x); }
__device__ __forceinline__ double m_cos(double x) { return cos(x); }
__device__ __forceinline__ float m_cos(float x) { return cosf(x); }
__device__ __forceinline__ double m_sin(double x) { return sin(x); }
__device__ __forceinline__ float m_sin(float x) { return sinf(x); }

// Division by a denominator that several quotients share.  FP64: the correctly rounded quotient
// from the correctly rounded reciprocal and one exact remainder (Markstein, IBM J. Res. Dev.
// 34, 1990) -- the value a / b has, in three operations instead of a division's ten or so.  A
// non-finite quotient may come out as NaN instead of infinity.  FP32 multiplies by the
// reciprocal, as its fast division does.
template <class T> struct Recip {
  T b, r;
};
template <class T> __device__ __forceinline__ Recip<T> recip(T b) { return {b, T(1) / b}; }
__device__ __forceinline__ double operator/(double a, const Recip<double> &d)
{
  const double q = a * d.r;
  return fma(fma(-q, d.b, a), d.r, q);
}
__device__ __forceinline__ float operator/(float a, const Recip<float> &d) { return a * d.r; }

// ---- EOS (Mara/eos.cpp:13-29) -------------------------------------------------------
template <class T> __device__ __forceinline__ T eos_internal(T gamma, T p) { return p / recip(gamma - 1); }
template <class T> __device__ __forceinline__ T eos_cs2(T gamma, T r, T p)
{
  const T rhoh = r + eos_internal(gamma, p) + p;
  return gamma * p / rhoh;
}

// ---- P -> U (Mara/rmhd.cpp:177-207) ---------------------------------------------------
template <class T>
__device__ __forceinline__ int check_cons(const T *U)
{
  if (U[ddd] < T(0)) return C2P_CONS_NEG_DENSITY;
  if (U[tau] < T(0)) return C2P_CONS_NEG_ENERGY;
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if (isnan(U[i])) return C2P_CONS_NAN;
  return C2P_SUCCESS;
}

template <class T>
__device__ __forceinline__ int prim_to_cons(T gamma, const T *P, T *U)
{
  const T V2 = P[vx] * P[vx] + P[vy] * P[vy] + P[vz] * P[vz];
  const T B2 = P[Bx] * P[Bx] + P[By] * P[By] + P[Bz] * P[Bz];
  const T Bv = P[Bx] * P[vx] + P[By] * P[vy] + P[Bz] * P[vz];
  const T W2 = T(1) / (T(1) - V2);
  const T W = m_sqrt(W2);
  const Recip<T> iW = recip(W), ir = recip(P[rho]);
  const T b0 = W * Bv;
  const T b2 = (B2 + b0 * b0) / W2;
  const T bx = (P[Bx] + b0 * W * P[vx]) / iW;
  const T by = (P[By] + b0 * W * P[vy]) / iW;
  const T bz = (P[Bz] + b0 * W * P[vz]) / iW;
  const T e = eos_internal(gamma, P[pre]) / ir;
  const T e_ = e + T(0.5) * b2 / ir;
  const T p_ = P[pre] + T(0.5) * b2;
  const T h_ = T(1) + e_ + p_ / ir;
  U[ddd] = P[rho] * W;
  U[tau] = P[rho] * h_ * W2 - p_ - b0 * b0 - U[ddd];
  U[Sx] = P[rho] * h_ * W2 * P[vx] - b0 * bx;
  U[Sy] = P[rho] * h_ * W2 * P[vy] - b0 * by;
  U[Sz] = P[rho] * h_ * W2 * P[vz] - b0 * bz;
  U[Bx] = P[Bx];
  U[By] = P[By];
  U[Bz] = P[Bz];
  if (V2 >= T(1)) return C2P_PRIM_SUPERLUMINAL;
  return check_cons(U);
}

// ---- quartic (Mara/quartic.cpp:28-148) -------------------------------------------------
// x1 and the largest of the others (x3) of x^3 + c2 x^2 + c1 x + c0, as the quartic uses them; nr
// real roots (Mara/quartic.cpp:28-80).
template <class T>
__device__ __forceinline__ void cubic(T c2, T c1, T c0, T &x1, T &x3, int &nr)
{
  // c3 = 1: the reference divides by it, which is exact.
  const T a2 = c2, a1 = c1, a0 = c0;
  const Recip<T> i3 = recip(T(3));
  const T q = a1 / i3 - a2 * a2 / recip(T(9));
  const T r = (a1 * a2 - T(3) * a0) / recip(T(6)) - a2 * a2 * a2 / recip(T(27));
  const T delta = q * q * q + r * r;
  if (delta > T(0)) {
    T s1 = r + m_sqrt(delta);
    s1 = (s1 >= T(0)) ? m_cbrt_pow(s1) : -m_cbrt_pow(-s1);
    T s2 = r - m_sqrt(delta);
    s2 = (s2 >= T(0)) ? m_cbrt_pow(s2) : -m_cbrt_pow(-s2);
    x1 = (s1 + s2) - a2 / i3;
    x3 = T(-0.5) * (s1 + s2) - a2 / i3;
    nr = 1;
  } else if (delta < T(0)) {
    const T theta = m_acos(r / m_sqrt(-q * q * q)) / i3;
    const T costh = m_cos(theta), sq = m_sqrt(-q);
    x1 = T(2) * sq * costh - a2 / i3;
    // theta is in [0, pi/3], where 2 cos >= sqrt(3) sin - cos: x1 is the largest root, and only
    // next to pi/3 (cos = 1/2) can rounding put x3 above it
    x3 = x1;
    if (!(costh > T(0.5001))) {
      const T sinth = m_sin(theta);
      const T sqrt3 = T(1.7320508075688772);
      x3 = -sq * costh - a2 / i3 + sqrt3 * sq * sinth;
    }
    nr = 3;
  } else {
    const T s = (r >= T(0)) ? m_cbrt_pow(r) : -m_cbrt_pow(-r);
    x1 = T(2) * s - a2 / i3;
    x3 = -s - a2 / i3;
    nr = 3;
  }
}

// Returns (max root, min root) over the real roots of d4 x^4 + ... + d0 with the fold used
// by FluxAndEigenvalues: start at (-1, +1), then clamp to (1, -1) if either exceeds 1.
template <class T>
__device__ __forceinline__ void quartic_extreme_roots(T d4, T d3, T d2, T d1, T d0, T &ap, T &am)
{
  const Recip<T> i4 = recip(d4);
  const T a3 = d3 / i4, a2 = d2 / i4, a1 = d1 / i4, a0 = d0 / i4;
  const T au2 = -a2;
  const T au1 = (a1 * a3 - T(4) * a0);
  const T au0 = T(4) * a0 * a2 - a1 * a1 - a0 * a3 * a3;
  T x1, x3;
  int nr;
  cubic<T>(au2, au1, au0, x1, x3, nr);
  const T u1 = (nr == 1) ? x1 : ((x1 > x3) ? x1 : x3);
  const T R2 = T(0.25) * a3 * a3 + u1 - a2;
  const T R = (R2 > T(0)) ? m_sqrt(R2) : T(0);
  T D2, E2;
  if (R != T(0)) {
    const T foo1 = T(0.75) * a3 * a3 - R2 - T(2) * a2;
    const T foo2 = T(0.25) * (T(4) * a3 * a2 - T(8) * a1 - a3 * a3 * a3) / R;
    D2 = foo1 + foo2;
    E2 = foo1 - foo2;
  } else {
    const T foo1 = T(0.75) * a3 * a3 - T(2) * a2;
    const T foo2 = T(2) * m_sqrt(u1 * u1 - T(4) * a0);
    D2 = foo1 + foo2;
    E2 = foo1 - foo2;
  }
  ap = T(-1);
  am = T(1);
  if (D2 >= T(0)) {
    const T D = m_sqrt(D2);
    const T r1 = T(-0.25) * a3 + T(0.5) * R - T(0.5) * D;
    const T r2 = T(-0.25) * a3 + T(0.5) * R + T(0.5) * D;
    if (r1 > ap) ap = r1;
    if (r1 < am) am = r1;
    if (r2 > ap) ap = r2;
    if (r2 < am) am = r2;
  }
  if (E2 >= T(0)) {
    const T E = m_sqrt(E2);
    const T r3 = T(-0.25) * a3 - T(0.5) * R - T(0.5) * E;
    const T r4 = T(-0.25) * a3 - T(0.5) * R + T(0.5) * E;
    if (r3 > ap) ap = r3;
    if (r3 < am) am = r3;
    if (r4 > ap) ap = r4;
    if (r4 < am) am = r4;
  }
  if (m_abs(ap) > T(1) || m_abs(am) > T(1)) {
    ap = T(1);
    am = T(-1);
  }
}

// ---- fast magnetosonic speeds, FP32 --------------------------------------------------------------
// The quartic of Mara/rmhd.cpp:275-305 divided by rho h W^2 and written in d = lambda - v:
//   c4 d^4 + c3 d^3 + c2 d^2 + c1 d + c0.
// In this form nothing cancels (the expanded coefficients lose all their digits near
// degenerate roots and at high W, where FP32 Ferrari left errors of order one in the speed).
// A power of two then brings c2 to order one, so that no product below leaves the FP32 range
// down to p / (rho h) = 1e-34 (without it c4^2 left it at 1e-19); it changes no bit of the roots.
// hi, lo: the speeds at zero normal field, outside the fast roots.
struct FastQuartic {
  float c4, c3, c2, c1, c0, hi, lo;
};

__device__ __forceinline__ FastQuartic fast_quartic(float gamma, float p, float rh, float b2, float W2, float iW2,
                                                    float v, float vB, float B1)
{
  FastQuartic q;
  const float irh = 1.f / rh, ics2 = rh / (gamma * p);
  const float L0 = 1.f + b2 * irh * ics2;
  const float s = __int_as_float(0x7f000000 - (__float_as_int(L0) & 0x7f800000));   // 2^-exponent of L0
  const float M = W2 * (ics2 - 1.f) * s, L = L0 * s, k = irh * s;
  const float w = B1 * iW2;
  const float uu = vB * vB * k, uw = vB * w * k, ww = w * w * k;
  const float g0 = 1.f - v * v;
  q.c4 = M + L - uu;
  q.c3 = 2.f * (v * (L - uu) + uw);
  q.c2 = g0 * (uu - L) + 4.f * v * uw - ww;
  q.c1 = -2.f * (v * ww + uw * g0);
  q.c0 = ww * g0;
  const float r = sqrtf(L * (L + M * g0)), is = 1.f / (M + L);
  q.hi = (r - L * v) * is;
  q.lo = (-r - L * v) * is;
  return q;
}

// One Laguerre step toward the extreme root on side sg (+1 the largest, -1 the smallest): cubic
// convergence, monotone from outside since the quartic's roots are real.
__device__ __forceinline__ float laguerre_step(const FastQuartic &q, float d, float sg)
{
  float f = q.c4, f1 = q.c4, f2 = q.c4;
  f = f * d + q.c3; f1 = f1 * d + f; f2 = f2 * d + f1;
  f = f * d + q.c2; f1 = f1 * d + f; f2 = f2 * d + f1;
  f = f * d + q.c1; f1 = f1 * d + f;
  f = f * d + q.c0;
  const float D = fmaxf(9.f * f1 * f1 - 24.f * f * f2, 0.f);
  return 4.f * f / (f1 + sg * sqrtf(D));
}

// Both extreme roots from the starts hi and lo, which must lie outside them.  A step of s leaves an
// error of order s^3, so the step below 5e-4 is the last one.
__device__ __forceinline__ void laguerre_pair(const FastQuartic &q, float &hi, float &lo)
{
#pragma unroll 1
  for (int it = 0; it < 8; ++it) {
    const float a = laguerre_step(q, hi, 1.f), b = laguerre_step(q, lo, -1.f);
    hi -= a;
    lo -= b;
    if (!(fmaxf(fabsf(a), fabsf(b)) > 5e-4f)) break;
  }
}

// The speeds of a state outside the fluid's range (p <= 0 or rho <= 0, which reconstruction can
// produce and P->U accepts): the reference's closed form on the expanded coefficients.
static __device__ __noinline__ float2 irregular_speeds(float gamma, float r, float p, float v, float W2, float b0,
                                                       float b2, float bi)
{
  const float h = 1.f + p / (gamma - 1.f) / r + p / r;
  const float cs2 = eos_cs2(gamma, r, p);
  const float W4 = W2 * W2, v2 = v * v, v3 = v * v2, v4 = v * v3;
  const float K = r * h * (1.f / cs2 - 1.f) * W4;
  const float L = -(r * h + b2 / cs2) * W2;
  float2 o;
  quartic_extreme_roots<float>(K - L - b0 * b0, -4.f * K * v + L * v * 2.f + 2.f * b0 * bi,
                               6.f * K * v2 + L * (1.f - v2) + b0 * b0 - bi * bi,
                               -4.f * K * v3 - L * v * 2.f - 2.f * b0 * bi, K * v4 + L * v2 + bi * bi, o.x, o.y);
  return o;
}

// ---- flux and fast speeds (Mara/rmhd.cpp:208-310) ---------------------------------------
// dim is 1, 2 or 3.  Computes F (8) and, when want_speeds, (ap, am).
template <class T>
__device__ __forceinline__ void flux_and_eigenvalues(T gamma, const T *U, const T *P, T *F, T &ap,
                                                     T &am, int dim, bool want_speeds = true)
{
  const T V2 = P[vx] * P[vx] + P[vy] * P[vy] + P[vz] * P[vz];
  const T B2 = P[Bx] * P[Bx] + P[By] * P[By] + P[Bz] * P[Bz];
  const T Bv = P[Bx] * P[vx] + P[By] * P[vy] + P[Bz] * P[vz];
  const T W2 = T(1) / (T(1) - V2);
  const T W = m_sqrt(W2);
  const Recip<T> iW = recip(W), ir = recip(P[rho]);
  const T b0 = W * Bv;
  const T b2 = (B2 + b0 * b0) / W2;
  const T bx = (P[Bx] + b0 * W * P[vx]) / iW;
  const T by = (P[By] + b0 * W * P[vy]) / iW;
  const T bz = (P[Bz] + b0 * W * P[vz]) / iW;
  const T e = eos_internal(gamma, P[pre]) / ir;
  const T p_ = P[pre] + T(0.5) * b2;
  const T h = T(1) + e + P[pre] / ir;
  T vi, bi;
  if (dim == 1) {
    F[ddd] = U[ddd] * P[vx];
    F[tau] = U[tau] * P[vx] - b0 * P[Bx] / iW + p_ * P[vx];
    F[Sx] = U[Sx] * P[vx] - bx * P[Bx] / iW + p_;
    F[Sy] = U[Sy] * P[vx] - by * P[Bx] / iW;
    F[Sz] = U[Sz] * P[vx] - bz * P[Bx] / iW;
    F[Bx] = T(0);
    F[By] = P[vx] * P[By] - P[vy] * P[Bx];
    F[Bz] = P[vx] * P[Bz] - P[vz] * P[Bx];
    vi = P[vx];
    bi = bx;
  } else if (dim == 2) {
    F[ddd] = U[ddd] * P[vy];
    F[tau] = U[tau] * P[vy] - b0 * P[By] / iW + p_ * P[vy];
    F[Sx] = U[Sx] * P[vy] - bx * P[By] / iW;
    F[Sy] = U[Sy] * P[vy] - by * P[By] / iW + p_;
    F[Sz] = U[Sz] * P[vy] - bz * P[By] / iW;
    F[Bx] = P[vy] * P[Bx] - P[vx] * P[By];
    F[By] = T(0);
    F[Bz] = P[vy] * P[Bz] - P[vz] * P[By];
    vi = P[vy];
    bi = by;
  } else {
    F[ddd] = U[ddd] * P[vz];
    F[tau] = U[tau] * P[vz] - b0 * P[Bz] / iW + p_ * P[vz];
    F[Sx] = U[Sx] * P[vz] - bx * P[Bz] / iW;
    F[Sy] = U[Sy] * P[vz] - by * P[Bz] / iW;
    F[Sz] = U[Sz] * P[vz] - bz * P[Bz] / iW + p_;
    F[Bx] = P[vz] * P[Bx] - P[vx] * P[Bz];
    F[By] = P[vz] * P[By] - P[vy] * P[Bz];
    F[Bz] = T(0);
    vi = P[vz];
    bi = bz;
  }
  if (!want_speeds) return;
  if constexpr (sizeof(T) < sizeof(double)) {
    if (P[pre] > T(0) && P[rho] > T(0)) {
      const FastQuartic q = fast_quartic(gamma, P[pre], P[rho] * h, b2, W2, T(1) - V2, vi, Bv,
                                         dim == 1 ? P[Bx] : dim == 2 ? P[By] : P[Bz]);
      ap = q.hi;
      am = q.lo;
      laguerre_pair(q, ap, am);
      ap += vi;
      am += vi;
      if (!(ap <= T(1) && am >= T(-1))) {
        ap = T(1);
        am = T(-1);
      }
    } else {
      const float2 o = irregular_speeds(gamma, P[rho], P[pre], vi, W2, b0, b2, bi);
      ap = o.x;
      am = o.y;
    }
    return;
  }
  const T cs2 = eos_cs2(gamma, P[rho], P[pre]);
  const T W4 = W2 * W2, v2 = vi * vi, v3 = vi * v2, v4 = vi * v3;
  const Recip<T> ics = recip(cs2);
  const T K = P[rho] * h * (ics.r - T(1)) * W4;
  const T L = -(P[rho] * h + b2 / ics) * W2;
  const T A4 = K - L - b0 * b0;
  const T A3 = T(-4) * K * vi + L * vi * T(2) + T(2) * b0 * bi;
  const T A2 = T(6) * K * v2 + L * (T(1) - v2) + b0 * b0 - bi * bi;
  const T A1 = T(-4) * K * v3 - L * vi * T(2) - T(2) * b0 * bi;
  const T A0 = K * v4 + L * v2 + bi * bi;
  quartic_extreme_roots<T>(A4, A3, A2, A1, A0, ap, am);
}

// ---- c2p: Newton solvers and the four-attempt ladder (FP64; the FP32 bulk path starts in FP32) ----
struct C2PState {
  double D, Tau, S2, B2, BS, BS2, gamma, gamf, pfloor;
  double Sxyz[3], Bxyz[3];
};

__device__ __forceinline__ void c2p_new_state(C2PState &s, const double *U)
{
  s.D = U[ddd];
  s.Tau = U[tau];
  s.S2 = U[Sx] * U[Sx] + U[Sy] * U[Sy] + U[Sz] * U[Sz];
  s.B2 = U[Bx] * U[Bx] + U[By] * U[By] + U[Bz] * U[Bz];
  s.BS = U[Bx] * U[Sx] + U[By] * U[Sy] + U[Bz] * U[Sz];
  s.BS2 = s.BS * s.BS;
  s.Sxyz[0] = U[Sx]; s.Sxyz[1] = U[Sy]; s.Sxyz[2] = U[Sz];
  s.Bxyz[0] = U[Bx]; s.Bxyz[1] = U[By]; s.Bxyz[2] = U[Bz];
}

__device__ __forceinline__ void c2p_estimate(const C2PState &s, double &Z, double &W)
{
  Z = sqrt(s.S2 + s.D * s.D);
  W = Z / s.D;
}

__device__ __forceinline__ void c2p_from_prim(const C2PState &s, const double *P, double &Z, double &W)
{
  const double V2 = P[vx] * P[vx] + P[vy] * P[vy] + P[vz] * P[vz];
  const double W2 = 1.0 / (1.0 - V2);
  const double e = P[pre] / (P[rho] * (s.gamma - 1.0));
  const double h = 1.0 + e + P[pre] / P[rho];
  Z = P[rho] * h * W2;
  W = sqrt(W2);
}

template <class T>
__device__ __forceinline__ int check_prim(const T *P)
{
  const T v2 = P[vx] * P[vx] + P[vy] * P[vy] + P[vz] * P[vz];
  if (v2 >= T(1)) return C2P_PRIM_SUPERLUMINAL;
  if (P[pre] < T(0)) return C2P_PRIM_NEG_PRESSURE;
  if (P[rho] < T(0)) return C2P_PRIM_NEG_RESTMASS;
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if (isnan(P[i])) return C2P_PRIM_NAN;
  return C2P_SUCCESS;
}

__device__ __forceinline__ int c2p_reconstruct(const C2PState &s, double Z, double W, double *Pout)
{
  double P[8];
  const Recip<double> iW = recip(W), iZB = recip(Z + s.B2);
  const double b0 = s.BS * W / Z;
  P[rho] = s.D / iW;
  P[pre] = (s.D / iW) * (Z / (s.D * W) - 1.0) * s.gamf;
  P[vx] = (s.Sxyz[0] + b0 * s.Bxyz[0] / iW) / iZB;
  P[vy] = (s.Sxyz[1] + b0 * s.Bxyz[1] / iW) / iZB;
  P[vz] = (s.Sxyz[2] + b0 * s.Bxyz[2] / iW) / iZB;
  P[Bx] = s.Bxyz[0];
  P[By] = s.Bxyz[1];
  P[Bz] = s.Bxyz[2];
  if (P[pre] < s.pfloor && s.pfloor > 0.0) P[pre] = s.pfloor;
  const int e = check_prim(P);
  if (e) return e;
#pragma unroll
  for (int i = 0; i < 8; ++i) Pout[i] = P[i];
  return C2P_SUCCESS;
}

// The same reconstruction for the FP32-bulk path's Newton (c2p_anton2dzw_fast), from the
// reciprocals of W, Z and D it holds already: one FP64 division instead of nine.  Same
// formulas and checks; the primitives differ from c2p_reconstruct's at FP64 round-off.
__device__ __forceinline__ int c2p_reconstruct_fast(const C2PState &s, double Z, double W, double iZ, double iW,
                                                    double iD, double *Pout)
{
  double P[8];
  const double b0 = s.BS * W * iZ;
  const double iZB = 1.0 / (Z + s.B2);
  P[rho] = s.D * iW;
  P[pre] = P[rho] * (Z * iD * iW - 1.0) * s.gamf;
  P[vx] = (s.Sxyz[0] + b0 * s.Bxyz[0] * iW) * iZB;
  P[vy] = (s.Sxyz[1] + b0 * s.Bxyz[1] * iW) * iZB;
  P[vz] = (s.Sxyz[2] + b0 * s.Bxyz[2] * iW) * iZB;
  P[Bx] = s.Bxyz[0];
  P[By] = s.Bxyz[1];
  P[Bz] = s.Bxyz[2];
  if (P[pre] < s.pfloor && s.pfloor > 0.0) P[pre] = s.pfloor;
  const int e = check_prim(P);
  if (e) return e;
#pragma unroll
  for (int i = 0; i < 8; ++i) Pout[i] = P[i];
  return C2P_SUCCESS;
}

// Anton et al. (2006) eqs 84-85, 2-D Newton in (Z, W) (Mara/rmhd-c2p.c:232-303).
__device__ __forceinline__ int c2p_anton2dzw(const C2PState &s, double Z, double W, double *P, int &iters)
{
  const double D = s.D, B2 = s.B2, BS2 = s.BS2, S2 = s.S2, gamf = s.gamf, Tau = s.Tau;
  double error = 1.0;
  iters = 0;
  Recip<double> iW = recip(W);
  while (error > 1e-12) {
    const double Z2 = Z * Z, Z3 = Z * Z2, W2 = W * W, W3 = W * W2;
    const Recip<double> iW2 = recip(W2), iW3 = recip(W3), iZ2 = recip(Z2);
    const double Pre = (D / iW) * (Z / (D * W) - 1.0) * gamf;
    const double df0dZ = 2 * (B2 + Z) * (BS2 * W2 + (W2 - 1) * Z3) / (W2 * Z3);
    const double df0dW = 2 * (B2 + Z) * (B2 + Z) / iW3;
    const double df1dZ = 1.0 + BS2 / Z3 - gamf / iW2;
    const double df1dW = B2 / iW3 + (2 * Z - D * W) / iW3 * gamf;
    const double f0 = -S2 + (Z + B2) * (Z + B2) * (W2 - 1) / iW2 - (2 * Z + B2) * BS2 / iZ2;
    const double f1 = -Tau + Z + B2 - Pre - 0.5 * B2 / iW2 - 0.5 * BS2 / iZ2 - D;
    const Recip<double> idet = recip(df0dZ * df1dW - df0dW * df1dZ);
    const double G0 = df1dW / idet, G1 = -df0dW / idet, G2 = -df1dZ / idet, G3 = df0dZ / idet;
    const double dZ = -(G0 * f0 + G1 * f1);
    const double dW = -(G2 * f0 + G3 * f1);
    double Zn = Z + dZ, Wn = W + dW;
    Zn = (Zn > 0.0) ? Zn : -Zn;
    Zn = (Zn < 1e20) ? Zn : Z;
    Wn = (Wn > 1.0) ? Wn : 1.0;
    Wn = (Wn < 1e12) ? Wn : 1e12;
    Z = Zn;
    W = Wn;
    iW = recip(W);
    error = fabs(dZ / Z) + fabs(dW / iW);
    if (++iters == 250) return C2P_MAXITER;
  }
  return c2p_reconstruct(s, Z, W, P);
}

// An approximate reciprocal, also in the translation units built without fast math.
__device__ __forceinline__ float rcp32(float x) { return __fdividef(1.f, x); }

// The Anton et al. iteration in FP32 to a step of 1e-6, from and to (Z, W); E = tau + D.  Non-zero
// when it does not converge in `limit` iterations.
__device__ __forceinline__ int c2p_newton32(float D, float E, float S2, float B2, float BS2, float gamf, float &Z,
                                            float &W, int &iters, int limit)
{
  float iW = rcp32(W), iZ = rcp32(Z);
  iters = 0;
#pragma unroll 1
  for (;;) {
    const float W2 = W * W, iW2 = iW * iW, iW3 = iW2 * iW, iZ2 = iZ * iZ, iZ3 = iZ2 * iZ;
    const float T = BS2 * iZ2;
    const float BZ = B2 + Z, u2 = (W2 - 1.f) * iW2;
    const float Pre = (Z * iW2 - D * iW) * gamf;
    const float f0Z = 2.f * BZ * (BS2 * iZ3 + u2);
    const float f0W = 2.f * BZ * BZ * iW3;
    const float f1Z = 1.f + BS2 * iZ3 - gamf * iW2;
    const float f1W = (B2 + (2.f * Z - D * W) * gamf) * iW3;
    const float f0 = BZ * BZ * u2 - (2.f * Z + B2) * T - S2;
    const float f1 = Z + B2 - E - Pre - 0.5f * B2 * iW2 - 0.5f * T;
    const float idet = rcp32(f0Z * f1W - f0W * f1Z);
    const float dZ = -(f1W * f0 - f0W * f1) * idet;
    const float dW = -(f0Z * f1 - f1Z * f0) * idet;
    const float Zn = fabsf(Z + dZ);
    Z = (Zn < 1e20f) ? Zn : Z;
    W = fminf(fmaxf(W + dW, 1.f), 1e12f);
    iZ = rcp32(Z);
    iW = rcp32(W);
    const float err = fabsf(dZ * iZ) + fabsf(dW * iW);
    ++iters;
    if (!(err > 1e-6f)) return err == err ? 0 : 1;
    if (iters == limit) return 1;
  }
}

// The same Anton et al. Newton iteration with the divisions replaced by three reciprocals
// per iteration (1/W, 1/Z, 1/det); algebraically identical, rounded differently.  Used by
// the FP32-bulk path, whose c2p is an FP64 polish compared with the FP64 path rather than
// the reference's bit pattern.  The start is first brought to FP32 accuracy by the same
// iteration in FP32 (five iterations from the estimate, at a quarter of their FP64 cost).  The
// FP64 iteration keeps the reference's bound of 1e-12 on its last step: to end it on a first
// step below 1e-6 costs a tenth less (160^3 lean, RK3: 0.56 against 0.62 ms per step) but leaves
// up to 3e-10 of p at Lorentz factor 3 and p/rho 1e-3, as a step's error is its square times the
// state's condition.
__device__ __forceinline__ int c2p_anton2dzw_fast(const C2PState &s, double Z, double W, double *P, int &iters)
{
  const double D = s.D, B2 = s.B2, BS2 = s.BS2, S2 = s.S2, gamf = s.gamf, Tau = s.Tau;
  const double iD = 1.0 / D;
  iters = 0;
  {
    float z = float(Z), w = float(W);
    if (c2p_newton32(float(D), float(D + Tau), float(S2), float(B2), float(BS2), float(gamf), z, w, iters, 12) == 0) {
      Z = z;
      W = w;
    }
  }
  double iW = 1.0 / W, iZ = 1.0 / Z;
  double error = 1.0;
  while (error > 1e-12) {
    const double W2 = W * W, Z2 = Z * Z, Z3 = Z * Z2;
    const double iW2 = iW * iW, iW3 = iW2 * iW, iZ2 = iZ * iZ, iZ3 = iZ2 * iZ;
    const double Pre = D * iW * (Z * iD * iW - 1.0) * gamf;
    const double BZ = B2 + Z;
    const double df0dZ = 2 * BZ * (BS2 * W2 + (W2 - 1) * Z3) * iW2 * iZ3;
    const double df0dW = 2 * BZ * BZ * iW3;
    const double df1dZ = 1.0 + BS2 * iZ3 - gamf * iW2;
    const double df1dW = (B2 + (2 * Z - D * W) * gamf) * iW3;
    const double f0 = -S2 + BZ * BZ * (W2 - 1) * iW2 - (2 * Z + B2) * BS2 * iZ2;
    const double f1 = -Tau + Z + B2 - Pre - 0.5 * B2 * iW2 - 0.5 * BS2 * iZ2 - D;
    const double idet = 1.0 / (df0dZ * df1dW - df0dW * df1dZ);
    const double dZ = -(df1dW * f0 - df0dW * f1) * idet;
    const double dW = -(df0dZ * f1 - df1dZ * f0) * idet;
    double Zn = Z + dZ, Wn = W + dW;
    Zn = (Zn > 0.0) ? Zn : -Zn;
    Zn = (Zn < 1e20) ? Zn : Z;
    Wn = (Wn > 1.0) ? Wn : 1.0;
    Wn = (Wn < 1e12) ? Wn : 1e12;
    Z = Zn;
    W = Wn;
    iZ = 1.0 / Z;
    iW = 1.0 / W;
    error = fabs(dZ * iZ) + fabs(dW * iW);
    if (++iters >= 250) return C2P_MAXITER;
  }
  return c2p_reconstruct_fast(s, Z, W, iZ, iW, iD, P);
}

// Noble et al. (2006) 1-D Newton in Z (Mara/rmhd-c2p.c:311-376).
__device__ __forceinline__ int c2p_noble1dw(const C2PState &s, double Z, double *P, int &iters)
{
  const double D = s.D, B2 = s.B2, BS2 = s.BS2, S2 = s.S2, gamf = s.gamf, Tau = s.Tau;
  double error = 1.0;
  iters = 0;
  while (error > 1e-12) {
    const double Z2 = Z * Z, Z3 = Z * Z2;
    const double a = S2 * Z2 + BS2 * (B2 + 2 * Z);
    const double b = (B2 + Z) * (B2 + Z) * Z2;
    const double ap = 2 * (S2 * Z + BS2);
    const double bp = 2 * Z * (B2 + Z) * (B2 + 2 * Z);
    const double V2 = a / b;
    const double W2 = 1.0 / (1.0 - V2);
    const double W = sqrt(W2);
    const double W3 = W * W2;
    const double Pre = (D / W) * (Z / (D * W) - 1.0) * gamf;
    const double dv2dZ = (ap * b - bp * a) / (b * b);
    const double delPdelZ = gamf / W2;
    const double delPdelW = gamf * (D / W2 - 2 * Z / W3);
    const double dWdv2 = 0.5 * W3;
    const double dPdZ = delPdelW * dWdv2 * dv2dZ + delPdelZ;
    const double f = Tau + D - 0.5 * B2 * (1 + V2) + 0.5 * BS2 / Z2 - Z + Pre;
    const double g = -0.5 * B2 * dv2dZ - BS2 / Z3 - 1.0 + dPdZ;
    const double dZ = -f / g;
    double Zn = Z + dZ;
    Zn = (Zn > 0.0) ? Zn : -Zn;
    Zn = (Zn < 1e20) ? Zn : Z;
    Z = Zn;
    error = fabs(dZ / Z);
    if (++iters == 250) return C2P_MAXITER;
  }
  const double Z2 = Z * Z;
  const double a = S2 * Z2 + BS2 * (B2 + 2 * Z);
  const double b = (B2 + Z) * (B2 + Z) * Z2;
  const double V2 = a / b;
  const double W2 = 1.0 / (1.0 - V2);
  const double W = sqrt(W2);
  return c2p_reconstruct(s, Z, W, P);
}

// Per-call c2p statistics (iterations of the Newton that succeeded, attempts used).
struct C2PTally {
  int iters;      // Newton iterations summed over attempts
  int attempts;   // 1..4 (5 = learned guess rejected and ladder used)
};

// Optional learned initial guess: (Z, W) from the packed network; defined in c2p_mlp.cuh.
__device__ __forceinline__ bool c2p_learned_guess(const void *net, const C2PState &s, double &Z, double &W);

// The ladder's rungs 2-4 (previous prim -> Anton; estimate -> Noble; previous prim ->
// Noble), reached only when the first attempt fails: kept out of line, state by value.
struct C2PRungs {
  double P[8];
  int err, iters, attempt;
};
static __device__ __noinline__ C2PRungs c2p_rungs(const C2PState s, C2PRungs r)
{
  double Z, W;
  int it = 0;
  r.err = 1;
  r.iters = 0;
  c2p_from_prim(s, r.P, Z, W);
  r.err = c2p_anton2dzw(s, Z, W, r.P, it);
  r.iters += it;
  r.attempt = 2;
  if (r.err) {
    c2p_estimate(s, Z, W);
    r.err = c2p_noble1dw(s, Z, r.P, it);
    r.iters += it;
    r.attempt = 3;
  }
  if (r.err) {
    c2p_from_prim(s, r.P, Z, W);
    r.err = c2p_noble1dw(s, Z, r.P, it);
    r.iters += it;
    r.attempt = 4;
  }
  return r;
}

// AdiabaticIdealRmhd::ConsToPrim gamma-law ladder (Mara/rmhd.cpp:103-176).  P holds the
// previous primitive state on entry (second guess) and is written only on success.  With a
// learned network the first attempt starts from its guess instead, and the reference ladder
// follows unchanged if that attempt fails.  The first Anton attempt is inlined (one call
// site serves both the learned and the estimated starting point); the other rungs are not.
// Guess (compile time): 0 = the per-thread network when pp.learned; 1 = the given (Zg, Wg)
// when `have`; 2 = none (no network code is compiled in).  `prev` fills P with the previous
// primitive state when P does not hold it yet: it is called only on the paths that read P
// (the ladder's rungs) or leave it as the result (a failure), so a caller can defer that load.
struct C2PPrevInP {
  __device__ void operator()(double *) const {}
};
template <bool Fast = false, int Guess = 0, class Prev = C2PPrevInP>
__device__ __forceinline__ int cons_to_prim(const PhysParams &pp, const double *U, double *P,
                                            C2PTally *tally = nullptr, double Zg = 0.0, double Wg = 0.0,
                                            bool have = true, const Prev &prev = Prev())
{
  int error = check_cons(U);
  if (error) {
    prev(P);
    if (tally) { tally->iters = 0; tally->attempts = 0; }
    return error;
  }
  C2PState s;
  s.gamma = pp.gamma;
  s.gamf = (pp.gamma - 1.0) / pp.gamma;
  s.pfloor = pp.pfloor;
  c2p_new_state(s, U);
  int total = 0, attempts = 1;
  error = 1;
  const bool use_net = (Guess == 1 && have) || (Guess == 0 && pp.learned && pp.mlp);
  for (int a = use_net ? 0 : 1; a < 2 && error; ++a) {
    double Z, W;
    if (a == 0) {
      if (Guess == 1) {
        Z = Zg;
        W = Wg;
      } else if (Guess == 0) {
        if (!c2p_learned_guess(pp.mlp, s, Z, W)) continue;
      } else {
        continue;
      }
    } else {
      c2p_estimate(s, Z, W);
    }
    int it = 0;
    error = Fast ? c2p_anton2dzw_fast(s, Z, W, P, it) : c2p_anton2dzw(s, Z, W, P, it);
    total += it;
    if (error && a == 0) attempts = 5;
  }
  if (error) {
    prev(P);
    C2PRungs r;
#pragma unroll
    for (int i = 0; i < 8; ++i) r.P[i] = P[i];
    r = c2p_rungs(s, r);
    total += r.iters;
    error = r.err;
    if (attempts != 5) attempts = r.attempt;
    if (!error) {
#pragma unroll
      for (int i = 0; i < 8; ++i) P[i] = r.P[i];
    }
  }
  if (tally) { tally->iters = total; tally->attempts = attempts; }
  return error;
}

// ---- reconstruction (Mara/weno.c:85-154) ---------------------------------------------------
template <class T> __device__ __forceinline__ int sgn(T x) { return (x > T(0)) - (x < T(0)); }

template <class T>
__device__ __forceinline__ T min3(T a, T b, T c)
{
  const T x01 = a < b ? a : b;
  return x01 < c ? x01 : c;
}
template <class T>
__device__ __forceinline__ T max3(T a, T b, T c)
{
  const T x01 = a > b ? a : b;
  return x01 > c ? x01 : c;
}

// The smaller and the larger of two numbers, NaN when either is.
#ifdef __CUDA_ARCH__
__device__ __forceinline__ float min_nan(float a, float b)
{
  float r;
  asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float max_nan(float a, float b)
{
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
#else
__device__ __forceinline__ float min_nan(float a, float b) { return isnan(a) || isnan(b) ? a + b : fminf(a, b); }
__device__ __forceinline__ float max_nan(float a, float b) { return isnan(a) || isnan(b) ? a + b : fmaxf(a, b); }
#endif

// minmod of three slopes, as the reference's 0.25 |sgn a + sgn b| (sgn a + sgn c) min(|a|, |b|, |c|):
// the common sign times the smallest magnitude, or zero.  In FP32 by minima and maxima: c held
// between zero and the minmod of a and b (six operations without the integer signs and their
// conversions; the same value for every triple of finite numbers).  A NaN c gives NaN, as there,
// and NaN a and b (the far zone's, whose sign counts as zero) give zero.
template <class T>
__device__ __forceinline__ T minmod3(T a, T b, T c)
{
  if constexpr (sizeof(T) < sizeof(double)) {
    const float hi = fmaxf(fminf(a, b), 0.f), lo = fminf(fmaxf(a, b), 0.f);
    return min_nan(max_nan(c, lo), hi);
  } else {
    const int sa = sgn(a), sb = sgn(b), sc = sgn(c);
    return T(0.25) * T(abs(sa + sb)) * T(sa + sc) * min3(m_abs(a), m_abs(b), m_abs(c));
  }
}

// PLM minmod(theta): face value v0 + sgn * slope / 2
template <class T>
__device__ __forceinline__ T plm(T theta, T vm, T v0, T vp, T sg)
{
  return v0 + sg * T(0.5) * minmod3(theta * (v0 - vm), T(0.5) * (vp - vm), theta * (vp - v0));
}

// Both face values of the zone v0: toward vm (lo) and toward vp (hi), each as plm gives it.
template <class T>
__device__ __forceinline__ void plm_zone(T theta, T vm, T v0, T vp, T &lo, T &hi)
{
  const T h = T(0.5) * minmod3(theta * (v0 - vm), T(0.5) * (vp - vm), theta * (vp - v0));
  lo = v0 - h;
  hi = v0 + h;
}

// WENO5 smoothness indicators of the stencil v[-2..2], the same for both faces of the zone: for
// JS96 and SZ10 the squared denominators of the weights, for B08 the factors 1 + tau5 / (B + eps).
template <class T>
__device__ __forceinline__ void weno5_indicators(int is_mode, T sz10A, T vm2, T vm1, T v0, T vp1, T vp2, T *k)
{
  const T t0a = T(1) * v0 - T(2) * vp1 + T(1) * vp2, t0b = T(3) * v0 - T(4) * vp1 + T(1) * vp2;
  const T t1a = T(1) * vm1 - T(2) * v0 + T(1) * vp1, t1b = T(1) * vm1 - T(0) * v0 - T(1) * vp1;
  const T t2a = T(1) * vm2 - T(2) * vm1 + T(1) * v0, t2b = T(1) * vm2 - T(4) * vm1 + T(3) * v0;
  T B0 = T(13. / 12.) * (t0a * t0a) + T(1. / 4.) * (t0b * t0b);
  T B1 = T(13. / 12.) * (t1a * t1a) + T(1. / 4.) * (t1b * t1b);
  T B2 = T(13. / 12.) * (t2a * t2a) + T(1. / 4.) * (t2b * t2b);
  if (is_mode == IS_B08) {
    const T eps = T(1e-14);
    const T tau5 = m_abs(B0 - B2);
    k[0] = T(1) + (tau5 / (B0 + eps));
    k[1] = T(1) + (tau5 / (B1 + eps));
    k[2] = T(1) + (tau5 / (B2 + eps));
    return;
  }
  T epsp = T(1e-6);
  if (is_mode == IS_SZ10) {
    epsp = T(1e-10);
    const T minB = min3(B0, B1, B2), maxB = max3(B0, B1, B2);
    const T R0 = minB / (maxB + epsp);
    B0 = R0 * sz10A * minB + B0;
    B1 = R0 * sz10A * minB + B1;
    B2 = R0 * sz10A * minB + B2;
  }
  k[0] = (epsp + B0) * (epsp + B0);
  k[1] = (epsp + B1) * (epsp + B1);
  k[2] = (epsp + B2) * (epsp + B2);
}

// The face value on one side from the indicators: centre-to-right (c2r = true) or
// centre-to-left.
template <class T>
__device__ __forceinline__ T weno5_side(int is_mode, const T *k, T vm2, T vm1, T v0, T vp1, T vp2, bool c2r)
{
  // coefficient tables CeesC2R_FV / CeesC2L_FV and DeesC2R_FV / DeesC2L_FV (weno.c:21-28)
  T c00, c01, c02, c10, c11, c12, c20, c21, c22, d0, d1, d2;
  if (c2r) {
    c00 = T(3. / 8.);  c01 = T(3. / 4.);  c02 = T(-1. / 8.);
    c10 = T(-1. / 8.); c11 = T(3. / 4.);  c12 = T(3. / 8.);
    c20 = T(3. / 8.);  c21 = T(-5. / 4.); c22 = T(15. / 8.);
    d0 = T(5. / 16.); d1 = T(5. / 8.); d2 = T(1. / 16.);
  } else {
    c00 = T(15. / 8.); c01 = T(-5. / 4.); c02 = T(3. / 8.);
    c10 = T(3. / 8.);  c11 = T(3. / 4.);  c12 = T(-1. / 8.);
    c20 = T(-1. / 8.); c21 = T(3. / 4.);  c22 = T(3. / 8.);
    d0 = T(1. / 16.); d1 = T(5. / 8.); d2 = T(5. / 16.);
  }
  const T vs0 = c00 * v0 + c01 * vp1 + c02 * vp2;
  const T vs1 = c10 * vm1 + c11 * v0 + c12 * vp1;
  const T vs2 = c20 * vm2 + c21 * vm1 + c22 * v0;
  T w0, w1, w2;
  if (is_mode == IS_B08) {
    w0 = d0 * k[0];
    w1 = d1 * k[1];
    w2 = d2 * k[2];
  } else {
    w0 = d0 / k[0];
    w1 = d1 / k[1];
    w2 = d2 / k[2];
  }
  const T wtot = w0 + w1 + w2;
  return (w0 * vs0 + w1 * vs1 + w2 * vs2) / wtot;
}

// FP32 WENO5 of one zone, the same scheme from the four first differences D0..D3 of the stencil:
// the face values as v0 plus a weighted correction (each candidate two operations instead of
// three, and the correction's rounding instead of the value's), and the JS96 / SZ10 weights
// from the reciprocals of eps + B (three per zone instead of three per face).
struct Weno32 {
  float D0, D1, D2, D3, k0, k1, k2;
};
__device__ __forceinline__ Weno32 weno32(int is_mode, float sz10A, float vm2, float vm1, float v0, float vp1, float vp2)
{
  Weno32 w;
  w.D0 = vm1 - vm2;
  w.D1 = v0 - vm1;
  w.D2 = vp1 - v0;
  w.D3 = vp2 - vp1;
  const float a0 = w.D3 - w.D2, b0 = 3.f * w.D2 - w.D3, a1 = w.D2 - w.D1, b1 = w.D1 + w.D2, a2 = w.D1 - w.D0,
              b2 = 3.f * w.D1 - w.D0;
  float B0 = (13.f / 12.f) * (a0 * a0) + 0.25f * (b0 * b0);
  float B1 = (13.f / 12.f) * (a1 * a1) + 0.25f * (b1 * b1);
  float B2 = (13.f / 12.f) * (a2 * a2) + 0.25f * (b2 * b2);
  if (is_mode == IS_B08) {
    const float tau5 = fabsf(B0 - B2);
    w.k0 = 1.f + tau5 / (B0 + 1e-14f);
    w.k1 = 1.f + tau5 / (B1 + 1e-14f);
    w.k2 = 1.f + tau5 / (B2 + 1e-14f);
    return w;
  }
  float epsp = 1e-6f;
  if (is_mode == IS_SZ10) {
    epsp = 1e-10f;
    const float minB = min3(B0, B1, B2), maxB = max3(B0, B1, B2);
    const float c = minB / (maxB + epsp) * sz10A * minB;
    B0 += c;
    B1 += c;
    B2 += c;
  }
  const float i0 = 1.f / (epsp + B0), i1 = 1.f / (epsp + B1), i2 = 1.f / (epsp + B2);
  w.k0 = i0 * i0;
  w.k1 = i1 * i1;
  w.k2 = i2 * i2;
  return w;
}
__device__ __forceinline__ float weno32_hi(const Weno32 &w, float v0)
{
  const float e0 = 0.625f * w.D2 - 0.125f * w.D3, e1 = 0.125f * w.D1 + 0.375f * w.D2, e2 = 0.875f * w.D1 - 0.375f * w.D0;
  const float w0 = 0.3125f * w.k0, w1 = 0.625f * w.k1, w2 = 0.0625f * w.k2;
  return v0 + (w0 * e0 + w1 * e1 + w2 * e2) / (w0 + w1 + w2);
}
__device__ __forceinline__ float weno32_lo(const Weno32 &w, float v0)
{
  const float e0 = 0.375f * w.D3 - 0.875f * w.D2, e1 = -0.375f * w.D1 - 0.125f * w.D2, e2 = 0.125f * w.D0 - 0.625f * w.D1;
  const float w0 = 0.0625f * w.k0, w1 = 0.625f * w.k1, w2 = 0.3125f * w.k2;
  return v0 + (w0 * e0 + w1 * e1 + w2 * e2) / (w0 + w1 + w2);
}

// WENO5 finite-volume, centre-to-right (c2r = true) or centre-to-left face, on the stencil
// v[-2..2] given as (vm2, vm1, v0, vp1, vp2).
template <class T>
__device__ __forceinline__ T weno5(int is_mode, T sz10A, T vm2, T vm1, T v0, T vp1, T vp2, bool c2r)
{
  if constexpr (sizeof(T) < sizeof(double)) {
    const Weno32 w = weno32(is_mode, sz10A, vm2, vm1, v0, vp1, vp2);
    return c2r ? weno32_hi(w, v0) : weno32_lo(w, v0);
  } else {
    T k[3];
    weno5_indicators(is_mode, sz10A, vm2, vm1, v0, vp1, vp2, k);
    return weno5_side(is_mode, k, vm2, vm1, v0, vp1, vp2, c2r);
  }
}

// Both face values of the zone v0 (lo toward vm1, hi toward vp1) from one set of indicators.
template <class T>
__device__ __forceinline__ void weno5_zone(int is_mode, T sz10A, T vm2, T vm1, T v0, T vp1, T vp2, T &lo, T &hi)
{
  if constexpr (sizeof(T) < sizeof(double)) {
    const Weno32 w = weno32(is_mode, sz10A, vm2, vm1, v0, vp1, vp2);
    lo = weno32_lo(w, v0);
    hi = weno32_hi(w, v0);
  } else {
    T k[3];
    weno5_indicators(is_mode, sz10A, vm2, vm1, v0, vp1, vp2, k);
    lo = weno5_side(is_mode, k, vm2, vm1, v0, vp1, vp2, false);
    hi = weno5_side(is_mode, k, vm2, vm1, v0, vp1, vp2, true);
  }
}

// ---- Riemann solvers ------------------------------------------------------------------------
template <class T> struct RiemannCount {
  int hlld_ok, hlld_fallback;
};

// Index permutation of a sweep direction (compile time, so that the permuted state arrays
// stay in registers): (B1, B2, B3), (S1, S2, S3), (v1, v2, v3) as in the reference's
// IntercellFlux switch (e.g. Mara/riemann_hlld-rmhd.cpp:199-217).
template <int DIM> struct DimMap;
template <> struct DimMap<1> { enum { B1 = Bx, B2 = By, B3 = Bz, S1 = Sx, S2 = Sy, S3 = Sz, v1 = vx, v2 = vy, v3 = vz }; };
template <> struct DimMap<2> { enum { B1 = By, B2 = Bz, B3 = Bx, S1 = Sy, S2 = Sz, S3 = Sx, v1 = vy, v2 = vz, v3 = vx }; };
template <> struct DimMap<3> { enum { B1 = Bz, B2 = Bx, B3 = By, S1 = Sz, S2 = Sx, S3 = Sy, v1 = vz, v2 = vx, v3 = vy }; };

template <class T>
__device__ __forceinline__ T face_lambda(T ap, T am)
{
  return (m_abs(am) < m_abs(ap)) ? m_abs(ap) : m_abs(am);
}

// HllRiemannSolver::IntercellFlux at s = 0 (Mara/riemann_hll.cpp:19-64)
template <class T, int dim>
__device__ __forceinline__ int riemann_hll(T gamma, const T *Pl, const T *Pr, T *F, T &ml)
{
  T Ul[8], Ur[8], Fl[8], Fr[8], epl, eml, epr, emr;
  if (prim_to_cons(gamma, Pl, Ul)) return 1;
  if (prim_to_cons(gamma, Pr, Ur)) return 1;
  flux_and_eigenvalues(gamma, Ul, Pl, Fl, epl, eml, dim);
  flux_and_eigenvalues(gamma, Ur, Pr, Fr, epr, emr, dim);
  const T ap = (epl > epr) ? epl : epr;
  const T am = (eml < emr) ? eml : emr;
  const T l = face_lambda(ap, am);
  if (ml < l) ml = l;
  const T s = T(0);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const T Fh = (ap * Fl[i] - am * Fr[i] + ap * am * (Ur[i] - Ul[i])) / (ap - am);
    if (s <= am) F[i] = Fl[i];
    else if (am < s && s <= ap) F[i] = Fh;
    else if (ap < s) F[i] = Fr[i];
    else F[i] = T(0);   // unordered (NaN) speeds: the reference's zeroed flux stays
  }
  return 0;
}

// Contact speed of HLLC: the root (-b - sqrt(b^2 - 4ac)) / (2a) of a x^2 + b x + c, or -c/b
// when |a| is below SMALL_A (Mara/riemann_hllc-rmhd.cpp:96,134).  In FP64 the reference's
// expression is kept as written.  In FP32 it cancels catastrophically when a is small and
// b < 0 (an error of ~eps * |b| / a), so the FP32 path uses the algebraically identical
// 2c / (-b + sqrt(b^2 - 4ac)) there.
template <class T>
__device__ __forceinline__ T hllc_contact_speed(T a, T b, T c)
{
  using Tol = RmhdTol<T>;
  if (m_abs(a) < T(Tol::hllc_a)) return -c / b;
  if (sizeof(T) == sizeof(double)) return (-b - m_sqrt(b * b - T(4) * a * c)) / (T(2) * a);
  const T sq = m_sqrt(b * b - T(4) * a * c);
  return b <= T(0) ? T(2) * c / (-b + sq) : -(b + sq) / (T(2) * a);
}

// The HLL average, the HLLC star states and the flux at s = 0 from the two sides' states,
// fluxes (total-energy convention) and the outer speeds (FP64; FP32 faces take riemann_hllc32).
template <class C, int dim>
__device__ __forceinline__ void hllc_star_flux(const C *Pl, const C *Pr, const C *Ul, const C *Ur, const C *Fl,
                                               const C *Fr, C ap, C am, C *F)
{
  using T = C;
  using Tol = RmhdTol<T>;
  using M = DimMap<dim>;
  constexpr int B1 = M::B1, B2 = M::B2, B3 = M::B3, S1 = M::S1, S2 = M::S2, S3 = M::S3, v1 = M::v1;
  T Uh[8], Fh[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    Uh[i] = (ap * Ur[i] - am * Ul[i] + (Fl[i] - Fr[i])) / (ap - am);
    Fh[i] = (ap * Fl[i] - am * Fr[i] + ap * am * (Ur[i] - Ul[i])) / (ap - am);
  }
  T Ul_[8], Ur_[8], lc;
  if (m_abs(Uh[B1]) > T(Tol::hllc_bx)) {
    const T BdFB = Uh[B2] * Fh[B2] + Uh[B3] * Fh[B3];
    const T a = Fh[tau] - BdFB;
    const T b = -Fh[S1] - Uh[tau] + (Uh[B2] * Uh[B2] + Uh[B3] * Uh[B3]) + (Fh[B2] * Fh[B2] + Fh[B3] * Fh[B3]);
    const T c = Uh[S1] - BdFB;
    const T w1 = lc = hllc_contact_speed(a, b, c);
    const T w2 = (Uh[B2] * w1 - Fh[B2]) / Uh[B1];
    const T w3 = (Uh[B3] * w1 - Fh[B3]) / Uh[B1];
    const T b1 = Uh[B1], b2 = Uh[B2], b3 = Uh[B3];
    const T vdB = w1 * b1 + w2 * b2 + w3 * b3;
    const T vdv = w1 * w1 + w2 * w2 + w3 * w3;
    const T gm2 = T(1) / (T(1) - vdv);
    const T ps = Fh[S1] + b1 * b1 / gm2 - (Fh[tau] - b1 * vdB) * w1;
    Ul_[ddd] = (am - Pl[v1]) / (am - w1) * Ul[ddd];
    Ur_[ddd] = (ap - Pr[v1]) / (ap - w1) * Ur[ddd];
    Ul_[tau] = (am * Ul[tau] - Ul[S1] + ps * w1 - vdB * b1) / (am - w1);
    Ur_[tau] = (ap * Ur[tau] - Ur[S1] + ps * w1 - vdB * b1) / (ap - w1);
    Ul_[S1] = (Ul_[tau] + ps) * w1 - vdB * b1;
    Ur_[S1] = (Ur_[tau] + ps) * w1 - vdB * b1;
    Ul_[S2] = (-b1 * (b2 / gm2 + vdB * w2) + am * Ul[S2] - Fl[S2]) / (am - w1);
    Ur_[S2] = (-b1 * (b2 / gm2 + vdB * w2) + ap * Ur[S2] - Fr[S2]) / (ap - w1);
    Ul_[S3] = (-b1 * (b3 / gm2 + vdB * w3) + am * Ul[S3] - Fl[S3]) / (am - w1);
    Ur_[S3] = (-b1 * (b3 / gm2 + vdB * w3) + ap * Ur[S3] - Fr[S3]) / (ap - w1);
    Ul_[B1] = Ur_[B1] = b1;
    Ul_[B2] = Ur_[B2] = b2;
    Ul_[B3] = Ur_[B3] = b3;
  } else {
    const T a = Fh[tau];
    const T b = -Fh[S1] - Uh[tau];
    const T c = Uh[S1];
    const T v1_ = lc = hllc_contact_speed(a, b, c);
    const T p_ = -Fh[tau] * v1_ + Fh[S1];
    Ul_[ddd] = (am - Pl[v1]) / (am - v1_) * Ul[ddd];
    Ur_[ddd] = (ap - Pr[v1]) / (ap - v1_) * Ur[ddd];
    Ul_[tau] = (am * Ul[tau] - Ul[S1] + p_ * v1_) / (am - v1_);
    Ur_[tau] = (ap * Ur[tau] - Ur[S1] + p_ * v1_) / (ap - v1_);
    Ul_[S1] = (Ul_[tau] + p_) * v1_;
    Ur_[S1] = (Ur_[tau] + p_) * v1_;
    Ul_[S2] = (am - Pl[v1]) / (am - v1_) * Ul[S2];
    Ur_[S2] = (ap - Pr[v1]) / (ap - v1_) * Ur[S2];
    Ul_[S3] = (am - Pl[v1]) / (am - v1_) * Ul[S3];
    Ur_[S3] = (ap - Pr[v1]) / (ap - v1_) * Ur[S3];
    Ul_[B1] = Uh[B1];
    Ur_[B1] = Uh[B1];
    Ul_[B2] = (am - Pl[v1]) / (am - v1_) * Ul[B2];
    Ur_[B2] = (ap - Pr[v1]) / (ap - v1_) * Ur[B2];
    Ul_[B3] = (am - Pl[v1]) / (am - v1_) * Ul[B3];
    Ur_[B3] = (ap - Pr[v1]) / (ap - v1_) * Ur[B3];
  }
  const T s = T(0);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    if (s <= am) F[i] = Fl[i];
    else if (am < s && s <= lc) F[i] = Fl[i] + am * (Ul_[i] - Ul[i]);
    else if (lc < s && s <= ap) F[i] = Fr[i] + ap * (Ur_[i] - Ur[i]);
    else if (ap < s) F[i] = Fr[i];
    else F[i] = T(0);   // unordered (NaN) speeds: the reference's zeroed flux stays
  }
  F[tau] -= F[ddd];
}


// HllcRmhdRiemannSolver::IntercellFlux at s = 0 (Mara/riemann_hllc-rmhd.cpp:26-178)
template <class T, int dim>
__device__ __forceinline__ int riemann_hllc(T gamma, const T *pl, const T *pr, T *F, T &ml)
{
  using M = DimMap<dim>;
  constexpr int B1 = M::B1;
  T Pl[8], Pr[8], Ul[8], Ur[8], Fl[8], Fr[8], epl, eml, epr, emr;
#pragma unroll
  for (int i = 0; i < 8; ++i) { Pl[i] = pl[i]; Pr[i] = pr[i]; }
  Pl[B1] = Pr[B1] = T(0.5) * (Pl[B1] + Pr[B1]);
  if (prim_to_cons(gamma, Pl, Ul)) return 1;
  if (prim_to_cons(gamma, Pr, Ur)) return 1;
  flux_and_eigenvalues(gamma, Ul, Pl, Fl, epl, eml, dim);
  flux_and_eigenvalues(gamma, Ur, Pr, Fr, epr, emr, dim);
  Ul[tau] += Ul[ddd]; Fl[tau] += Fl[ddd];
  Ur[tau] += Ur[ddd]; Fr[tau] += Fr[ddd];
  const T ap = (epl > epr) ? epl : epr;
  const T am = (eml < emr) ? eml : emr;
  const T l = face_lambda(ap, am);
  if (ml < l) ml = l;
  hllc_star_flux<T, dim>(Pl, Pr, Ul, Ur, Fl, Fr, ap, am, F);
  return 0;
}

// Component of slot k of a state or flux in the normal frame of direction dim (1..3): density and
// energy (pressure), then the vector components from the normal one on, cyclically, as the
// reference's IntercellFlux switch orders them.
__host__ __device__ constexpr int frame_slot(int dim, int k)
{
  return k < 2 ? k : k < 5 ? 2 + (dim - 1 + k - 2) % 3 : 5 + (dim - 1 + k - 5) % 3;
}

// Out-of-line HLLC for the HLLD fallback (rare): arguments and result by value so that the
// caller's face states stay in registers on its hot path.  States in the reference's component
// order, the flux in the normal frame of dim.
template <class T> struct Face8 { T v[8]; };
template <class T> struct HllcOut { T F[8]; T ml; int err; };
template <class T>
static __device__ __noinline__ HllcOut<T> riemann_hllc_fallback(int dim, T gamma, Face8<T> pl, Face8<T> pr, T ml)
{
  HllcOut<T> o;
  o.ml = ml;
  T F[8];
  if (dim == 1) o.err = riemann_hllc<T, 1>(gamma, pl.v, pr.v, F, o.ml);
  else if (dim == 2) o.err = riemann_hllc<T, 2>(gamma, pl.v, pr.v, F, o.ml);
  else o.err = riemann_hllc<T, 3>(gamma, pl.v, pr.v, F, o.ml);
#pragma unroll
  for (int k = 0; k < 8; ++k) o.F[k] = F[frame_slot(dim, k)];
  return o;
}

// ---- columns in shared memory ------------------------------------------------------------------
// A thread's column of an array of shared memory (entry i at p[i * stride]): the stride is the
// block's width, so a warp's accesses to one entry are conflict-free.
template <class T> struct Column {
  T *p;
  int stride;
  __device__ __forceinline__ T &operator[](int i) const { return p[i * stride]; }
};

// ---- HLLD (Mignone, Ugliano & Bodo 2009; Mara/riemann_hlld-rmhd.cpp) -------------------------
template <class T> struct HlldJump { T E, D, B[3], m[3]; };
template <class T> struct HlldInner { T B[3], v[3]; };

// Equation 48: the outer speeds, the normal field (the same on both sides) and the jumps
// J = lambda U - F across the outer waves (normal frame, total-energy convention tau + D).
template <class T>
struct HlldEqn {
  T ap, am, bx;
  HlldJump<T> L, R;
};

template <class T> __device__ __forceinline__ T dot3(const T *v, const T *w) { return v[0] * w[0] + v[1] * w[1] + v[2] * w[2]; }
template <class T> __device__ __forceinline__ T dot1(const T *v) { return v[0] * v[0] + v[1] * v[1] + v[2] * v[2]; }

template <class T>
__device__ __forceinline__ void hlld_side(const HlldJump<T> &J, T a, T UBx, T p, HlldInner<T> &s, Recip<T> &ia)
{
  using Tol = RmhdTol<T>;
  const T A = J.m[0] - a * J.E + p * (T(1) - a * a);
  const T G = J.B[1] * J.B[1] + J.B[2] * J.B[2];
  const T C = J.B[1] * J.m[1] + J.B[2] * J.m[2];
  const T Q = -A - G + (UBx * UBx) * (T(1) - a * a);
  T X = UBx * (A * a * UBx + C) - (A + G) * (a * p + J.E);
  if (m_abs(X) < T(Tol::x_small)) X = T(Tol::x_small);
  const Recip<T> iX = recip(X);
  s.v[0] = (UBx * (A * UBx + a * C) - (A + G) * (p + J.m[0])) / iX;
  s.v[1] = (Q * J.m[1] + J.B[1] * (C + UBx * (a * J.m[0] - J.E))) / iX;
  s.v[2] = (Q * J.m[2] + J.B[2] * (C + UBx * (a * J.m[0] - J.E))) / iX;
  ia = recip(a - s.v[0]);
  s.B[0] = (J.B[0] - UBx * s.v[0]) / ia;
  s.B[1] = (J.B[1] - UBx * s.v[1]) / ia;
  s.B[2] = (J.B[2] - UBx * s.v[2]) / ia;
}

// The states between the fast waves at total pressure p.
template <class T> struct HlldFill {
  T Kl[3], Kr[3], Bc[3], etaL, etaR, wL, wR;
  HlldInner<T> aL, aR;
};

// FillInnerWaveStates (riemann_hlld-rmhd.cpp:357-420)
template <class T>
__device__ __forceinline__ void hlld_fill(const HlldEqn<T> &q, T p, HlldFill<T> &f)
{
  using Tol = RmhdTol<T>;
  HlldInner<T> &aL = f.aL, &aR = f.aR;
  Recip<T> il, ir;
  hlld_side(q.L, q.am, q.bx, p, aL, il);
  hlld_side(q.R, q.ap, q.bx, p, aR, ir);
  f.wL = p + (q.L.E - dot3(aL.v, q.L.m)) / il;
  f.wR = p + (q.R.E - dot3(aR.v, q.R.m)) / ir;
  if (f.wL < T(0)) f.wL *= T(-1);
  if (f.wR < T(0)) f.wR *= T(-1);
  f.etaL = T(-sgn(q.bx)) * m_sqrt(f.wL);
  f.etaR = T(+sgn(q.bx)) * m_sqrt(f.wR);
  const Recip<T> dl = recip(q.am * p + q.L.E + q.bx * f.etaL), dr = recip(q.ap * p + q.R.E + q.bx * f.etaR);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    f.Kl[k] = (q.L.m[k] + p * T(k == 0) + q.L.B[k] * f.etaL) / dl;
    f.Kr[k] = (q.R.m[k] + p * T(k == 0) + q.R.B[k] * f.etaR) / dr;
  }
  const Recip<T> dk = recip(f.Kr[0] - f.Kl[0]);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    f.Bc[k] = ((aR.B[k] * (f.Kr[0] - aR.v[0]) + aR.B[0] * aR.v[k]) -
               (aL.B[k] * (f.Kl[0] - aL.v[0]) + aL.B[0] * aL.v[k])) / dk;
    if (m_abs(f.Kr[0] - f.Kl[0]) < T(Tol::k_small)) f.Bc[k] = T(0);
  }
}

// The residual of eq. 48 from the states at its pressure.
template <class T>
__device__ __forceinline__ T hlld_residual(const HlldFill<T> &f)
{
  using Tol = RmhdTol<T>;
  const T delK = f.Kr[0] - f.Kl[0];
  const T Bch[3] = { f.Bc[0] * delK, f.Bc[1] * delK, f.Bc[2] * delK };
  const T Yl = (T(1) - dot1(f.Kl)) / (f.etaL * delK - dot3(f.Kl, Bch));
  const T Yr = (T(1) - dot1(f.Kr)) / (f.etaR * delK - dot3(f.Kr, Bch));
  if (m_abs(delK) < T(Tol::k_small)) return T(0);
  if (m_abs(f.Bc[0]) < T(Tol::k_small)) return delK;
  return delK * (T(1) - f.Bc[0] * (Yr - Yl));
}

// HlldEquation48::Function (riemann_hlld-rmhd.cpp:422-452); returns non-zero on "throw".
template <class T>
__device__ __forceinline__ int hlld_function(const HlldEqn<T> &q, T p, T &y)
{
  if (isinf(p)) return 1;   // (JumpInNormalBfield cannot occur: one normal field)
  HlldFill<T> f;
  hlld_fill(q, p, f);
  y = hlld_residual(f);
  return 0;
}

// NewtonRaphesonSolver::Solve, rank 1 (nrsolver.cpp:89-152) with the central-difference
// Jacobian of HlldEquation48::Jacobian.  At most 16 evaluations; bounded.
template <class T>
__device__ __forceinline__ int hlld_newton(const HlldEqn<T> &q, T &x)
{
  using Tol = RmhdTol<T>;
  const int MaxIterations = 15;
  const T dp = T(Tol::jac_dp);
  int worse = 0, it = 0;
  T eps = T(0), eps_last;
  do {
    eps_last = eps;
    // f(x), f(x - dp/2), f(x + dp/2): one evaluation site, three points
    T y = T(0), f0 = T(0), f1 = T(0);
#pragma unroll 1
    for (int e = 0; e < 3; ++e) {
      const T pe = e == 0 ? x : (e == 1 ? x - T(0.5) * dp : x + T(0.5) * dp);
      T r;
      if (hlld_function(q, pe, r)) return 1;
      if (e == 0) y = r;
      else if (e == 1) f0 = r;
      else f1 = r;
    }
    const T J = (f1 - f0) / dp;
    const T G = T(1) / J;
    T dx = T(0);
    dx += G * y;
    x -= dx;
    eps = T(0);
    eps += y > T(0) ? y : -y;
    worse += (eps > eps_last);
    if (worse >= 10 || it == MaxIterations) return 1;
    if (isnan(eps)) return 1;
  } while (eps > T(Tol::newton_eps) && ++it <= MaxIterations);
  return 0;
}

// The root of equation 48 that hlld_newton finds, with fewer evaluations: one difference slope
// at the starting pressure, then inverse interpolation through the points already there --
// Newton's first step and about its second from three evaluations, where the central
// differences of each Newton iteration take three -- and as in hlld_newton a last step from the
// point whose residual passes, repeated until it is short: the slope here is good to a few
// percent, so that a step of 4e-12 p leaves p off by 1e-13, hlld_newton's own accuracy.
//
// Faces on which the residual does not fall twentyfold in the first step and fiftyfold in the
// later ones (or is NaN) run hlld_newton from the start, out of line, and keep the reference's
// outcome: eq. 48 has other roots, and without this bound one face in 10^8 took one.  So do
// faces on which K_R and K_L meet on the way: the reference sets the residual to zero there, its
// Newton then divides by a zero slope and rejects the attempt, and the face falls back to HLLC
// (6% of the faces of magnetised jumps at Lorentz factor 50).
//
// Newton takes 6 to 12 evaluations on turbulence faces and this 4 or 5 (360,000 faces: fluxes
// within 1e-14 on 99.9%, the same branch on all).
struct HlldRoot {
  double p;
  int err;
};
static __device__ __noinline__ HlldRoot hlld_newton_cold(HlldEqn<double> q, double p)
{
  HlldRoot r;
  r.p = p;
  r.err = hlld_newton(q, r.p);
  return r;
}

// Walks p from the guess to the root of equation 48 (or, with `direct`, stays at it) and leaves
// the states at the final pressure in f: one evaluation site for the iteration and the flux.
// `guess` gives the reference's own starting pressure, for hlld_newton; with `own` that runs
// at once.
template <class Guess>
__device__ __forceinline__ int hlld_solve(const HlldEqn<double> &q, bool direct, bool own, double &p,
                                          HlldFill<double> &f, const Guess &guess)
{
  using Tol = RmhdTol<double>;
  const double dp = Tol::jac_dp;
  double x0 = p, y0 = 0.0, s0 = 0.0, sl = 0.0;   // the start, its residual and dx/dy; the latest dx/dy
  double x1 = 0.0, y1 = 0.0;             // the latest point
  bool last = direct;
#pragma unroll 1
  for (int it = 0;; ++it) {
    hlld_fill(q, p, f);
    if (last) return 0;
    const double y = hlld_residual(f);
    // where K_R and K_L agree the residual is zero by definition, not by convergence
    bool ok = !own && !(fabs(f.Kr[0] - f.Kl[0]) < Tol::k_small);
    if (it == 0) {
      y0 = y;
      p = x0 + dp;
      if (ok) continue;
    } else if (it == 1) {
      sl = s0 = dp / (y - y0);
      x1 = x0;
      y1 = y0;
      p = x0 - s0 * y0;
    } else {
      ok = ok && (fabs(y) <= (it == 2 ? 0.05 : 0.02) * fabs(y1) || fabs(y) <= Tol::newton_eps);
      double step;
      if (it == 2) {
        const double t = y0 / (y0 - y);
        step = s0 * y * t * t;
      } else {
        // below 1e-8 the residuals' rounding would enter the secant: keep the last slope
        if (fabs(y1) >= 1e-8) sl = (p - x1) / (y - y1);
        step = sl * y;
      }
      if (it == 2 && fabs(y0) >= 1e-8) sl = (p - x0) / (y - y0);
      x1 = p;
      y1 = y;
      p -= step;
    }
    // not the last where the residual passes with a step that the slope's last few percent matter
    // in: the residual's scale is that of the normal field, and 1e-12 of it can be 1e-9 of p.  The
    // bound on `it` ends faces whose residual is rounding by then; a flag that allowed one
    // evaluation more cost 3% of the sweeps instead of 1%.
    last = fabs(y1) <= Tol::newton_eps && (fabs(p - x1) <= 4e-12 * fabs(p) || it >= 8);
    if (!ok || !(fabs(p) < 1e300)) {
      const HlldRoot r = hlld_newton_cold(q, guess());
      if (r.err) return 1;
      p = r.p;
      last = true;
    }
  }
}

// ReconstructSolution (riemann_hlld-rmhd.cpp:453-575) at s = 0, flux only, from the states f at
// pressure p.
template <class T>
__device__ __forceinline__ int hlld_reconstruct(const HlldEqn<T> &q, T p, const HlldFill<T> &f, const Column<T> &col,
                                                T *F)
{
  using Tol = RmhdTol<T>;
  const T (&Kl)[3] = f.Kl, (&Kr)[3] = f.Kr, (&Bc)[3] = f.Bc;
  const T etaL = f.etaL, etaR = f.etaR, wL = f.wL, wR = f.wR;
  const HlldInner<T> &aL = f.aL, &aR = f.aR;
  const T am = q.am, ap = q.ap;
  const T denomL = etaL - dot3(Kl, Bc);
  const T denomR = etaR - dot3(Kr, Bc);
  T cLv[3], cRv[3];
  const Recip<T> iL = recip(denomL), iR = recip(denomR);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    cLv[k] = Kl[k] - Bc[k] * (T(1) - dot1(Kl)) / iL;
    cRv[k] = Kr[k] - Bc[k] * (T(1) - dot1(Kr)) / iR;
    if (m_abs(denomL) < T(Tol::k_small)) cLv[k] = aL.v[k];
    if (m_abs(denomR) < T(Tol::k_small)) cRv[k] = aR.v[k];
  }
  const T lamC = cRv[0], lmaL = Kl[0], lmaR = Kr[0], TOL = T(Tol::tol54);
  if (p < T(0)) return 1;
  if (lmaL < T(-1) || lmaR > T(1) || m_abs(lamC) > T(1)) return 1;
  if (!((wL > p) && (aL.v[0] > am - TOL) && (cLv[0] > lmaL - TOL))) return 1;
  if (!((wR > p) && (aR.v[0] < ap + TOL) && (cRv[0] < lmaR + TOL))) return 1;
  if (m_abs(cRv[0] - cLv[0]) > T(Tol::contact)) return 1;

  const T s = T(0);
  // The flux needs only the states of the region containing s = 0 and those between it and
  // the outer fast wave; the region test below is the reference's, evaluated first.
  int region;
  if (s <= am) region = 0;
  else if (am < s && s <= lmaL) region = 1;
  else if (lmaL < s && s <= lamC) region = 2;
  else if (lamC < s && s <= lmaR) region = 3;
  else if (lmaR < s && s <= ap) region = 4;
  else if (ap < s) region = 5;
  else region = 6;   // unordered (NaN) speeds: the reference leaves F unset
  if (region == 6) {
#pragma unroll
    for (int i = 0; i < 8; ++i) F[i] = T(0);
    return 0;
  }
  const bool left = region <= 2;
  const HlldJump<T> &J = left ? q.L : q.R;
  const HlldInner<T> &a = left ? aL : aR;
  const T wave = left ? am : ap;
  T Uo[8], Fo[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    Uo[i] = col[(left ? 0 : 8) + i];
    Fo[i] = col[(left ? 16 : 24) + i];
  }
  if (region == 0 || region == 5) {
#pragma unroll
    for (int i = 0; i < 8; ++i) F[i] = Fo[i];
    F[tau] -= F[ddd];
    return 0;
  }
  // States between the fast and Alfven waves (aL / aR)
  T aU[8];
  T denom;
  if (m_abs(denom = wave - a.v[0]) < T(Tol::degenerate)) {
#pragma unroll
    for (int i = 0; i < 8; ++i) aU[i] = Uo[i];
  } else {
    const T vB = dot3(a.v, a.B);
    aU[ddd] = J.D / denom;
    aU[tau] = (J.E + p * a.v[0] - vB * a.B[0]) / denom;
    aU[Sx] = (aU[tau] + p) * a.v[0] - vB * a.B[0];
    aU[Sy] = (aU[tau] + p) * a.v[1] - vB * a.B[1];
    aU[Sz] = (aU[tau] + p) * a.v[2] - vB * a.B[2];
    aU[Bx] = a.B[0];
    aU[By] = a.B[1];
    aU[Bz] = a.B[2];
  }
  if (region == 1 || region == 4) {
#pragma unroll
    for (int i = 0; i < 8; ++i) F[i] = Fo[i] + wave * (aU[i] - Uo[i]);
    F[tau] -= F[ddd];
    return 0;
  }
  // States between the Alfven and contact waves (cL / cR)
  const T lma = left ? lmaL : lmaR;
  const T *cv = left ? cLv : cRv;
  T cU[8];
  if (m_abs(denom = lma - lamC) < T(Tol::degenerate)) {
#pragma unroll
    for (int i = 0; i < 8; ++i) cU[i] = aU[i];
  } else {
    const T vBc = dot3(cv, Bc);
    cU[ddd] = aU[ddd] * (lma - a.v[0]) / denom;
    cU[tau] = (lma * aU[tau] - aU[Sx] + p * lamC - vBc * Bc[0]) / denom;
    cU[Sx] = (cU[tau] + p) * cv[0] - vBc * Bc[0];
    cU[Sy] = (cU[tau] + p) * cv[1] - vBc * Bc[1];
    cU[Sz] = (cU[tau] + p) * cv[2] - vBc * Bc[2];
    cU[Bx] = Bc[0];
    cU[By] = Bc[1];
    cU[Bz] = Bc[2];
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) F[i] = Fo[i] + wave * (aU[i] - Uo[i]) + lma * (cU[i] - aU[i]);
  F[tau] -= F[ddd];
  return 0;
}

// HLL total pressure, EstimateSolution(0) (riemann_hlld-rmhd.cpp:543-553), from the HLL
// state's primitives.
template <class T>
__device__ __forceinline__ T hlld_estimate0(const T *P)
{
  const T V2 = P[vx] * P[vx] + P[vy] * P[vy] + P[vz] * P[vz];
  const T B2 = P[Bx] * P[Bx] + P[By] * P[By] + P[Bz] * P[Bz];
  const T Bv = P[Bx] * P[vx] + P[By] * P[vy] + P[Bz] * P[vz];
  const T W2 = T(1) / (T(1) - V2);
  const T W = m_sqrt(W2);
  const T b0 = W * Bv;
  const T b2 = (B2 + b0 * b0) / W2;
  return P[pre] + T(0.5) * b2;
}

// Eq. (55), EstimateSolution(1) (riemann_hlld-rmhd.cpp:557-574): the smaller root of
// p^2 + (E - Fm) p + (FE m - E Fm) = 0 from the HLL state's total energy E, normal momentum m
// and their fluxes.
template <class T>
__device__ __forceinline__ T hlld_estimate1(T E, T FE, T m, T Fm)
{
  const T a = T(1);
  const T b = E - Fm;
  const T c = FE * m - E * Fm;
  const T p1 = m_abs((-b + m_sqrt(b * b - T(4) * a * c)) / (T(2) * a));
  const T p2 = m_abs((-b - m_sqrt(b * b - T(4) * a * c)) / (T(2) * a));
  return (p1 < p2) ? p1 : p2;
}

// The HLL state's total pressure by the reference's ladder (P: the average face state, its
// previous state), out of line.
struct HllState64 {
  double U[8], P[8];
};
struct HllGuess64 {
  double p;
  int err, iters, attempts;
};
static __device__ __noinline__ HllGuess64 hll_guess64(PhysParams pp, HllState64 s)
{
  C2PTally t{0, 0};
  HllGuess64 o;
  o.err = cons_to_prim<false, 2>(pp, s.U, s.P, &t);
  o.iters = t.iters;
  o.attempts = t.attempts;
  o.p = hlld_estimate0(s.P);
  return o;
}

// Total pressure of the HLL state, the first pressure guess, by the Anton et al. 2-D Newton in
// FP32 from (Z, W) of the average face state, to a step of 1e-6 (the guess only seeds the
// secants, and is kept in FP32): U as D, E, S0..S2, Bx, B1, B2.  Non-zero when the state fails
// check_cons, Newton does not converge in 32 iterations, or the primitives fail check_prim, with
// `margin` (of Z for the pressure, of 1 for 1 - v^2) on the last; the caller then takes the FP64
// ladder.
__device__ __forceinline__ int hll_pressure32(float gamma, float pfloor, float D, float E, float S0, float S1,
                                              float S2_, float Bx, float B1, float B2_, float Z, float W, float &pt,
                                              int &iters, float margin = 0.f)
{
  iters = 0;
  if (!(D >= 0.f) || !(E - D >= 0.f)) return 1;
  const float gamf = (gamma - 1.f) / gamma;
  const float S2 = S0 * S0 + S1 * S1 + S2_ * S2_;
  const float B2 = Bx * Bx + B1 * B1 + B2_ * B2_;
  const float BS = Bx * S0 + B1 * S1 + B2_ * S2_;
  const float BS2 = BS * BS;
  if (c2p_newton32(D, E, S2, B2, BS2, gamf, Z, W, iters, 32)) return 1;
  const float iD = rcp32(D), iW = rcp32(W), iZ = rcp32(Z);
  const float r = D * iW;
  float p = r * (Z * iD * iW - 1.f) * gamf;
  if (pfloor > 0.f && p < pfloor) p = pfloor;
  const float vB = BS * iZ, iZB = rcp32(Z + B2);
  const float v2 = (S2 + vB * (2.f * BS + vB * B2)) * iZB * iZB;
  if (!(v2 < 1.f - margin) || !(p >= margin * Z) || !(r >= 0.f)) return 1;
  pt = p + 0.5f * (B2 * (1.f - v2) + vB * vB);
  return 0;
}

// HlldRmhdRiemannSolver::IntercellFlux at s = 0 (riemann_hlld-rmhd.cpp:179-313), FP64 (FP32 faces
// take riemann_hlld32, rmhd_face32.cuh).  The face's states come in the first 16 entries of
// this thread's column -- left, then right, in the normal frame of dim -- and the column then
// holds both sides' U (0..15) and F (16..31): they are needed again only for the
// outermost flux, and in registers they would halve the resident warps.  One copy of the side's
// code serves both sides, and one of the inner states' code serves the pressure iteration and
// the flux: with every copy inlined the kernel was 520 KB, and up to a third of its warps'
// waiting was for instructions.
// Returns 1 when a face state is unphysical (the caller retries with PCM states); `used_hllc`
// reports the fallback; `src` gives the two face states again, in the reference's component
// order, on the rare paths.  The flux f is in the normal frame.
template <class Src>
__device__ __forceinline__ int riemann_hlld64(const PhysParams &pp, int dim, const Column<double> &col, double *f,
                                              double &ml, int &used_hllc, C2PTally *tally, const Src &src)
{
  using T = double;
  using Tol = RmhdTol<T>;
  const T gamma = T(pp.gamma);
  HlldEqn<T> q;
  q.bx = T(0.5) * (col[Bx] + col[8 + Bx]);
  used_hllc = 0;
  if (tally) { tally->iters = 0; tally->attempts = 0; }
  T ap = T(0), am = T(0);
  float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f, a4 = 0.f;   // the average face state: rho, p, v
#pragma unroll 1
  for (int side = 0; side < 2; ++side) {
    const Column<T> u{col.p + 8 * side * col.stride, col.stride}, w{col.p + (16 + 8 * side) * col.stride, col.stride};
    T P[8], U[8], F[8], ep, em;
#pragma unroll
    for (int i = 0; i < 8; ++i) P[i] = u[i];
    P[Bx] = q.bx;
    a0 += 0.5f * float(P[rho]);
    a1 += 0.5f * float(P[pre]);
    a2 += 0.5f * float(P[vx]);
    a3 += 0.5f * float(P[vy]);
    a4 += 0.5f * float(P[vz]);
    if (prim_to_cons(gamma, P, U)) return 1;
    flux_and_eigenvalues(gamma, U, P, F, ep, em, 1);
    am = (side == 0 || em < am) ? em : am;
    ap = (side == 0 || ep > ap) ? ep : ap;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      u[i] = U[i];
      w[i] = F[i];
    }
  }
  const T l = face_lambda(ap, am);
  if (ml < l) ml = l;
  // The HLL state and flux, and from them the first pressure guess.  The iteration converges to
  // the same root from a guess good to 1e-6, so the HLL state is inverted in FP32 where its
  // pressure and velocity are clear of the checks the reference's inversion makes; elsewhere,
  // and for the faces that run the reference's own Newton, in FP64 (hll_guess64).  Among those
  // are the faces of a weak normal field, |Bx| < 1e-5 sqrt(p): the residual there is of the
  // order of Bx (K_R - K_L), so that it passes within a step of any guess and the result would
  // keep what the FP32 guess is off by (fluxes up to 1e-6 off at |Bx| = 1e-7).  So are those of a
  // total pressure above 1e4 or below 1e-5: the reference's difference step is an absolute 1e-8,
  // whose slope is rounding up there and not local down here, and whether the iteration passes
  // depends on its every step.
  T U_hll[8], F_hll[3];
  {
    const Recip<T> iS = recip(ap - am);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const T ul = col[i], ur = col[8 + i], fl = col[16 + i], fr = col[24 + i];
      U_hll[i] = (ap * ur - am * ul + (fl - fr)) / iS;
      if (i < 3) F_hll[i] = (ap * fl - am * fr + ap * am * (ur - ul)) / iS;
    }
  }
  const auto guess64 = [&](double &p) {
    double ql[8], qr[8];
    src(ql, qr);
    HllState64 h;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      h.U[i] = U_hll[i];
      h.P[i] = T(0.5) * (ql[frame_slot(dim, i)] + qr[frame_slot(dim, i)]);
    }
    h.P[Bx] = q.bx;
    const HllGuess64 o = hll_guess64(pp, h);
    p = o.p;
    if (tally) { tally->iters = o.iters; tally->attempts = o.attempts; }
    return o.err;
  };
  const bool direct = m_abs(q.bx) < T(Tol::bx_small);
  T p_est0;
  int hll_c2p_failed;
  {
    const float g = float(gamma), i2 = 1.f - (a2 * a2 + a3 * a3 + a4 * a4);
    const float W2 = rcp32(i2);
    float pt = 0.f;
    int it = 0;
    hll_c2p_failed = !(i2 > 0.f && a0 > 0.f && a1 > 0.f) ||
                     hll_pressure32(g, float(pp.pfloor), float(U_hll[ddd]), float(U_hll[tau] + U_hll[ddd]),
                                    float(U_hll[Sx]), float(U_hll[Sy]), float(U_hll[Sz]), float(U_hll[Bx]),
                                    float(U_hll[By]), float(U_hll[Bz]), (a0 + g * rcp32(g - 1.f) * a1) * W2,
                                    sqrtf(W2), pt, it, 1e-3f);
    p_est0 = T(pt);
    if (tally) { tally->iters = it; tally->attempts = 1; }
    if (hll_c2p_failed) hll_c2p_failed = guess64(p_est0);
  }
  const bool own = q.bx * q.bx < T(1e-10) * p_est0 || !(p_est0 > T(1e-5) && p_est0 < T(1e4));
  // HlldEquation48 constructor (riemann_hlld-rmhd.cpp:315-345)
  q.ap = ap;
  q.am = am;
  {
    const T El = col[tau] + col[ddd], FEl = col[16 + tau] + col[16 + ddd];
    const T Er = col[8 + tau] + col[8 + ddd], FEr = col[24 + tau] + col[24 + ddd];
    col[tau] = El;
    col[16 + tau] = FEl;
    col[8 + tau] = Er;
    col[24 + tau] = FEr;
    q.L.E = am * El - FEl;
    q.R.E = ap * Er - FEr;
    q.L.D = am * col[ddd] - col[16 + ddd];
    q.R.D = ap * col[8 + ddd] - col[24 + ddd];
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    q.L.B[k] = am * col[Bx + k] - col[16 + Bx + k];
    q.R.B[k] = ap * col[8 + Bx + k] - col[24 + Bx + k];
    q.L.m[k] = am * col[Sx + k] - col[16 + Sx + k];
    q.R.m[k] = ap * col[8 + Sx + k] - col[24 + Sx + k];
  }
  T F[8];
  int attempt = 0, success = 0;
#pragma unroll 1
  while (!hll_c2p_failed && attempt < 3 && !success) {
    T p_star;
    const int est = direct ? 1 : attempt;
    if (est == 0) {
      p_star = p_est0;
    } else if (est == 1) {   // EstimateSolution(1) shifts tau and restores it afterwards
      F_hll[tau] += F_hll[ddd];
      U_hll[tau] += U_hll[ddd];
      p_star = hlld_estimate1(U_hll[tau], F_hll[tau], U_hll[Sx], F_hll[Sx]);
      F_hll[tau] -= F_hll[ddd];
      U_hll[tau] -= U_hll[ddd];
    } else {
      p_star = T(0);
    }
    const T p_star0 = p_star;
    HlldFill<T> fill;
    const auto start = [&]() {
      double p = p_star0;
      if (est == 0) guess64(p);
      return p;
    };
    int rc = hlld_solve(q, direct, own, p_star, fill, start);
    if (rc == 0) rc = hlld_reconstruct(q, p_star, fill, col, F);
    success = (rc == 0);
    ++attempt;
  }
  if (success) {
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] = F[i];
    return 0;
  }
  used_hllc = 1;
  Face8<T> a, b;
  src(a.v, b.v);
  const HllcOut<T> o = riemann_hllc_fallback<T>(dim, gamma, a, b, ml);
  ml = o.ml;
#pragma unroll
  for (int i = 0; i < 8; ++i) f[i] = o.F[i];
  return o.err;
}

}  // namespace mgpu
