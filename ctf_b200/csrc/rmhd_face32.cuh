// The FP32-bulk HLLC and HLLD faces, written for FP32 (the FP64 path keeps the reference's expressions in
// rmhd_physics.cuh).
//
// The sweeps are bound by instruction issue and latency, so this file spends as few
// instructions and live registers per face as the algorithm allows:
//  * the energy is carried as the total energy E = tau + D throughout, whose flux is the
//    momentum density;
//  * the fast speeds come from two or three Laguerre steps (rmhd_physics.cuh) instead of the
//    closed form, whose two branches the rounding chose between within every warp;
//  * the HLL state and the jumps share one set of values: J = lambda U - F on both sides gives
//    U_hll = (J_R - J_L) / (ap - am), so U and F are dead before the pressure iteration;
//  * the normal field is the same on both sides and through all waves (Bx), so the x
//    components of the field jumps and of the contact field are never formed;
//  * eq. 48 needs the contact field only as its numerator Bch = Bc (K_R - K_L);
//  * the flux is built from the pressure iteration's last evaluation.
//
// Reference formulas: Mara/riemann_hlld-rmhd.cpp:179-615 (HLLD), Mara/rmhd.cpp:177-310 (P->U,
// flux, quartic coefficients).
#pragma once
#include "rmhd_physics.cuh"

namespace mgpu {

// ---- one side of a face --------------------------------------------------------------------------
// Normal frame: component 0 along the sweep.  Conserved state (E total energy) and flux; the
// normal field is Bx on both sides.
struct SideState {
  float D, E, S0, S1, S2, B1, B2;      // U
  float FD, FS0, FS1, FS2, FB1, FB2;   // F (F[E] = S0)
};

// The fast speeds of a side.
struct FastPair {
  float hi, lo;
};

// Fills U, F and the side's fast speeds.  Returns non-zero where P->U fails its checks
// (Mara/rmhd.cpp:177-207).  Each side's iteration starts from its own speeds at zero normal
// field.  A start taken from the other side is a step closer in smooth flow, but it can lie inside
// the fast root, next to the slow one, and needs a check against that which costs more than the
// step (160^3 lean PLM sweeps per RK3 step: 3.31 ms with it, 3.25 without).
__device__ __forceinline__ int side_state(float gamma, float rh_p, float r, float p, float v0, float v1, float v2,
                                          float Bx, float B1, float B2, SideState &s, FastPair &o)
{
  const float V2 = v0 * v0 + v1 * v1 + v2 * v2;
  const float BB = Bx * Bx + B1 * B1 + B2 * B2;
  const float vB = v0 * Bx + v1 * B1 + v2 * B2;
  const float iW2 = 1.f - V2;
  const float W = rsqrtf(iW2);
  const float W2 = W * W;
  const float rh = r + rh_p * p;               // rho h
  const float b2 = BB * iW2 + vB * vB;
  const float wt = rh * W2 + BB;
  const float pt = p + 0.5f * b2;
  s.D = r * W;
  s.E = wt - pt;
  s.S0 = wt * v0 - vB * Bx;
  s.S1 = wt * v1 - vB * B1;
  s.S2 = wt * v2 - vB * B2;
  s.B1 = B1;
  s.B2 = B2;
  if (!(V2 < 1.f)) return 1;
  if (!(s.D >= 0.f) || !(s.E - s.D >= 0.f) || isnan(s.S0 + s.S1 + s.S2 + BB)) return 1;
  s.FD = s.D * v0;
  s.FS0 = s.S0 * v0 - (Bx * iW2 + vB * v0) * Bx + pt;
  s.FS1 = s.S1 * v0 - (B1 * iW2 + vB * v1) * Bx;
  s.FS2 = s.S2 * v0 - (B2 * iW2 + vB * v2) * Bx;
  s.FB1 = v0 * B1 - v1 * Bx;
  s.FB2 = v0 * B2 - v2 * Bx;
  if (!(p > 0.f && r > 0.f)) {
    const float2 q = irregular_speeds(gamma, r, p, v0, W2, W * vB, b2, Bx * iW2 * W + W * vB * v0);
    o.hi = q.x;
    o.lo = q.y;
    return 0;
  }
  const FastQuartic q = fast_quartic(gamma, p, rh, b2, W2, iW2, v0, vB, Bx);
  float a = q.hi, b = q.lo;
  laguerre_pair(q, a, b);
  o.hi = a + v0;
  o.lo = b + v0;
  return 0;
}

// One side's outer speed and the jump J = lam U - F across it (the normal field's is lam Bx).
struct HlldSide32 {
  float lam, D, E, m0, m1, m2, B1, B2;
};

__device__ __forceinline__ HlldSide32 side_jump(const SideState &s, float lam)
{
  return {lam, lam * s.D - s.FD, lam * s.E - s.S0, lam * s.S0 - s.FS0, lam * s.S1 - s.FS1, lam * s.S2 - s.FS2,
          lam * s.B1 - s.FB1, lam * s.B2 - s.FB2};
}

// Both sides of a face from its states pl, pr in the normal frame, the outer speeds and their
// fold into ml.  Non-zero when a face state is unphysical.
__device__ __forceinline__ int face_sides(float gamma, const float *pl, const float *pr, float bx, SideState &s,
                                          SideState &t, float &ap, float &am, float &ml)
{
  const float rh_p = gamma / (gamma - 1.f);
  FastPair fl, fr;
  if (side_state(gamma, rh_p, pl[rho], pl[pre], pl[vx], pl[vy], pl[vz], bx, pl[By], pl[Bz], s, fl)) return 1;
  if (side_state(gamma, rh_p, pr[rho], pr[pre], pr[vx], pr[vy], pr[vz], bx, pr[By], pr[Bz], t, fr)) return 1;
  ap = fmaxf(fl.hi, fr.hi);
  am = fminf(fl.lo, fr.lo);
  if (!(ap <= 1.f && am >= -1.f)) {
    ap = 1.f;
    am = -1.f;
  }
  ml = fmaxf(ml, fmaxf(fabsf(ap), fabsf(am)));
  return 0;
}

// ---- HLLC ------------------------------------------------------------------------------------------
// HllcRmhdRiemannSolver::IntercellFlux at s = 0 (Mara/riemann_hllc-rmhd.cpp:26-178) from the
// jumps: U_hll = (J_R - J_L) / (ap - am), and the flux lam U* - J of the side of the contact that holds s = 0 (the other side's star state is not
// formed).  A contact or star state that FP32 made non-finite takes the HLL flux.  pl, pr and f
// in the normal frame.
__device__ __forceinline__ int riemann_hllc32(float gamma, const float *pl, const float *pr, float *f, float &ml)
{
  using Tol = RmhdTol<float>;
  const float bx = 0.5f * (pl[Bx] + pr[Bx]);
  SideState s, t;
  float ap, am;
  if (face_sides(gamma, pl, pr, bx, s, t, ap, am, ml)) return 1;
  f[Bx] = 0.f;
  if (am >= 0.f || ap < 0.f) {
    const bool left = am >= 0.f;
    f[ddd] = left ? s.FD : t.FD;
    f[tau] = (left ? s.S0 : t.S0) - f[ddd];
    f[Sx] = left ? s.FS0 : t.FS0;
    f[Sy] = left ? s.FS1 : t.FS1;
    f[Sz] = left ? s.FS2 : t.FS2;
    f[By] = left ? s.FB1 : t.FB1;
    f[Bz] = left ? s.FB2 : t.FB2;
    return 0;
  }
  const HlldSide32 L = side_jump(s, am), R = side_jump(t, ap);
  const float is = 1.f / (ap - am);
  const float UE = (R.E - L.E) * is, U0 = (R.m0 - L.m0) * is, U1 = (R.B1 - L.B1) * is, U2 = (R.B2 - L.B2) * is;
  // not from the jumps: their difference would cancel ap am U, and w2, w3 divide F1, F2 by bx
  const float q = ap * am;
  const float FE = (ap * s.S0 - am * t.S0 + q * (t.E - s.E)) * is, F0 = (ap * s.FS0 - am * t.FS0 + q * (t.S0 - s.S0)) * is,
              F1 = (ap * s.FB1 - am * t.FB1 + q * (t.B1 - s.B1)) * is,
              F2 = (ap * s.FB2 - am * t.FB2 + q * (t.B2 - s.B2)) * is;
  float w1, w2 = 0.f, w3 = 0.f, vdB = 0.f, g2 = 1.f, b1 = 0.f, ps;
  const bool field = fabsf(bx) > Tol::hllc_bx;
  if (field) {
    const float BdFB = U1 * F1 + U2 * F2;
    w1 = hllc_contact_speed(FE - BdFB, -F0 - UE + (U1 * U1 + U2 * U2) + (F1 * F1 + F2 * F2), U0 - BdFB);
    const float ib = 1.f / bx;
    w2 = (U1 * w1 - F1) * ib;
    w3 = (U2 * w1 - F2) * ib;
    b1 = bx;
    vdB = w1 * b1 + w2 * U1 + w3 * U2;
    g2 = 1.f - (w1 * w1 + w2 * w2 + w3 * w3);
    ps = F0 + b1 * b1 * g2 - (FE - b1 * vdB) * w1;
  } else {
    w1 = hllc_contact_speed(FE, -F0 - UE, U0);
    ps = F0 - FE * w1;
  }
  const bool left = w1 >= 0.f;
  const float lam = left ? am : ap;
  const float JD = left ? L.D : R.D, JE = left ? L.E : R.E, J0 = left ? L.m0 : R.m0, J1 = left ? L.m1 : R.m1,
              J2 = left ? L.m2 : R.m2, JB1 = left ? L.B1 : R.B1, JB2 = left ? L.B2 : R.B2;
  const float k = 1.f / (lam - w1);
  const float D = JD * k, E = (JE + ps * w1 - vdB * b1) * k;
  const float m0 = (E + ps) * w1 - vdB * b1;
  const float m1 = (J1 - b1 * (U1 * g2 + vdB * w2)) * k, m2 = (J2 - b1 * (U2 * g2 + vdB * w3)) * k;
  const float c1 = field ? U1 : JB1 * k, c2 = field ? U2 : JB2 * k;
  if (isfinite(w1) && isfinite(ps) && isfinite(D) && isfinite(E) && isfinite(m1) && isfinite(m2) && isfinite(m0) &&
      isfinite(c1) && isfinite(c2)) {
    f[ddd] = lam * D - JD;
    f[tau] = (lam * E - JE) - f[ddd];
    f[Sx] = lam * m0 - J0;
    f[Sy] = lam * m1 - J1;
    f[Sz] = lam * m2 - J2;
    f[By] = lam * c1 - JB1;
    f[Bz] = lam * c2 - JB2;
  } else {
    f[ddd] = (am * R.D - ap * L.D) * is;
    f[tau] = FE - f[ddd];
    f[Sx] = F0;
    f[Sy] = (am * R.m1 - ap * L.m1) * is;
    f[Sz] = (am * R.m2 - ap * L.m2) * is;
    f[By] = F1;
    f[Bz] = F2;
  }
  return 0;
}

// The HLLD solver's fallback, out of line (rare); states in the reference's component order.
static __device__ __noinline__ HllcOut<float> riemann_hllc32_fallback(int dim, float gamma, Face8<float> pl,
                                                                      Face8<float> pr, float ml)
{
  float l[8], r[8];
  for (int k = 0; k < 8; ++k) {
    l[k] = pl.v[frame_slot(dim, k)];
    r[k] = pr.v[frame_slot(dim, k)];
  }
  HllcOut<float> o;
  o.ml = ml;
  o.err = riemann_hllc32(gamma, l, r, o.F, o.ml);
  return o;
}

// ---- HLLD ------------------------------------------------------------------------------------------
struct HlldInner32 {
  float v0, v1, v2, b1, b2;   // between the fast and Alfven waves
  float ia, w;                // 1 / (lam - v0), total enthalpy
  float K0, K1, K2;
};

struct HlldEval32 {
  HlldInner32 l, r;
  float dK, c1, c2;           // K_R - K_L and the contact field times it (normal part Bx dK)
  float nl, nr;               // eta dK - K . Bch
};

__device__ __forceinline__ void hlld_inner32(const HlldSide32 &q, float Bx, float p, float sgn_eta, HlldInner32 &s,
                                             float &eta)
{
  using Tol = RmhdTol<float>;
  const float ol = 1.f - q.lam * q.lam, Bx2 = Bx * Bx;
  const float G = q.B1 * q.B1 + q.B2 * q.B2;
  const float C = Bx * (q.B1 * q.m1 + q.B2 * q.m2);
  const float A = q.m0 - q.lam * q.E + p * ol;
  const float AG = A + G;
  const float lpE = q.lam * p + q.E;
  float X = A * (q.lam * Bx2) + C - AG * lpE;
  if (fabsf(X) < Tol::x_small) X = Tol::x_small;
  const float iX = 1.f / X;
  const float Q = Bx2 * ol - AG;
  const float t = (q.B1 * q.m1 + q.B2 * q.m2) + Bx * (q.lam * q.m0 - q.E);
  const float pm = p + q.m0;
  s.v0 = (A * Bx2 + q.lam * C - AG * pm) * iX;
  s.v1 = (Q * q.m1 + q.B1 * t) * iX;
  s.v2 = (Q * q.m2 + q.B2 * t) * iX;
  s.ia = 1.f / (q.lam - s.v0);
  s.b1 = (q.B1 - Bx * s.v1) * s.ia;
  s.b2 = (q.B2 - Bx * s.v2) * s.ia;
  s.w = fabsf(p + (q.E - (s.v0 * q.m0 + s.v1 * q.m1 + s.v2 * q.m2)) * s.ia);
  eta = sgn_eta * sqrtf(s.w);
  const float id = 1.f / (lpE + Bx * eta);
  s.K0 = (pm + q.lam * Bx * eta) * id;
  s.K1 = (q.m1 + q.B1 * eta) * id;
  s.K2 = (q.m2 + q.B2 * eta) * id;
}

// Eq. 48 at p: the residual, and everything the flux needs in `e`.
__device__ __forceinline__ float hlld_eval32(const HlldSide32 &L, const HlldSide32 &R, float Bx, float p,
                                             HlldEval32 &e)
{
  using Tol = RmhdTol<float>;
  const float sg = copysignf(Bx == 0.f ? 0.f : 1.f, Bx);
  float el, er;
  hlld_inner32(L, Bx, p, -sg, e.l, el);
  hlld_inner32(R, Bx, p, sg, e.r, er);
  e.dK = e.r.K0 - e.l.K0;
  const float kl = e.l.K0 - e.l.v0, kr = e.r.K0 - e.r.v0;
  e.c1 = (e.r.b1 * kr + Bx * e.r.v1) - (e.l.b1 * kl + Bx * e.l.v1);
  e.c2 = (e.r.b2 * kr + Bx * e.r.v2) - (e.l.b2 * kl + Bx * e.l.v2);
  const float c0 = Bx * e.dK;
  e.nl = el * e.dK - (e.l.K0 * c0 + e.l.K1 * e.c1 + e.l.K2 * e.c2);
  e.nr = er * e.dK - (e.r.K0 * c0 + e.r.K1 * e.c1 + e.r.K2 * e.c2);
  const float yl = (1.f - (e.l.K0 * e.l.K0 + e.l.K1 * e.l.K1 + e.l.K2 * e.l.K2)) / e.nl;
  const float yr = (1.f - (e.r.K0 * e.r.K0 + e.r.K1 * e.r.K1 + e.r.K2 * e.r.K2)) / e.nr;
  const float y = e.dK * (1.f - Bx * (yr - yl));
  return fabsf(e.dK) < Tol::k_small ? 0.f : y;
}


// The root of eq. 48 from p, by secants: the first step takes the slope of the unmagnetised
// problem, d(v_R - v_L)/dp, scaled by the 0.85 that it lies below the full slope on turbulence
// faces (0.76-0.92 between the 10th and 90th percentile).  Where that step is longer than the
// difference step jac_dp, the second point is p + jac_dp, which keeps the iteration on the root
// of the local slope (eq. 48 has others).  `e` is left at the returned p.  Non-zero when it does
// not converge.
__device__ __forceinline__ int hlld_root32(const HlldSide32 &L, const HlldSide32 &R, float Bx, bool direct, float &p,
                                           HlldEval32 &e)
{
  using Tol = RmhdTol<float>;
  const int MaxIterations = 15;
  float p0 = p, y0 = 0.f;
  int worse = 0;
#pragma unroll 1
  for (int it = 0; it <= MaxIterations + 2; ++it) {
    const float y = hlld_eval32(L, R, Bx, p, e);
    if (direct) return 0;               // no normal field: the guess is the solution
    if (isnan(y)) return 1;
    // the first step converges linearly: hold it to a quarter of the tolerance
    if (fabsf(y) <= (it == 1 ? 0.25f : 1.f) * Tol::newton_eps) return 0;
    float dp;
    if (it == 0) {
      const float sl = (1.f - R.lam * e.r.v0) / (R.E + R.lam * p) - (1.f - L.lam * e.l.v0) / (L.E + L.lam * p);
      dp = -0.85f * y / sl;
      if (!(fabsf(dp) <= Tol::jac_dp)) dp = Tol::jac_dp;
    } else {
      worse += fabsf(y) > fabsf(y0);
      if (worse >= 10) return 1;
      dp = -y * (p - p0) / (y - y0);
    }
    p0 = p;
    y0 = y;
    p += dp;
  }
  return 1;
}

// ReconstructSolution at s = 0 (flux only) from the evaluation at p: F as D, tau, S0, S1, S2,
// B1, B2.  Non-zero when the solution fails the reference's checks.  `outer` refetches the
// conserved state outside the fast wave where the state behind it is degenerate.
template <class Outer>
__device__ __forceinline__ int hlld_flux32(const HlldSide32 &L, const HlldSide32 &R, float Bx, float p,
                                           const HlldEval32 &e, float *F, const Outer &outer)
{
  using Tol = RmhdTol<float>;
  // contact velocities: K - Bc (1 - K^2) / (eta - K . Bc) on each side
  const float idK = 1.f / e.dK;
  const bool flat = fabsf(e.dK) < Tol::k_small;      // the contact field counts as zero
  const float c0 = flat ? 0.f : Bx * e.dK, c1 = flat ? 0.f : e.c1, c2 = flat ? 0.f : e.c2;
  const float yl = (1.f - (e.l.K0 * e.l.K0 + e.l.K1 * e.l.K1 + e.l.K2 * e.l.K2)) / e.nl;
  const float yr = (1.f - (e.r.K0 * e.r.K0 + e.r.K1 * e.r.K1 + e.r.K2 * e.r.K2)) / e.nr;
  const bool sl = !(fabsf(e.nl) >= Tol::k_small * fabsf(e.dK)), sr = !(fabsf(e.nr) >= Tol::k_small * fabsf(e.dK));
  const float cl0 = sl ? e.l.v0 : (flat ? e.l.K0 : e.l.K0 - c0 * yl);
  const float cr0 = sr ? e.r.v0 : (flat ? e.r.K0 : e.r.K0 - c0 * yr);
  const float lamC = cr0, TOL = Tol::tol54;
  if (p < 0.f) return 1;
  if (e.l.K0 < -1.f || e.r.K0 > 1.f || fabsf(lamC) > 1.f) return 1;
  if (!((e.l.w > p) && (e.l.v0 > L.lam - TOL) && (cl0 > e.l.K0 - TOL))) return 1;
  if (!((e.r.w > p) && (e.r.v0 < R.lam + TOL) && (cr0 < e.r.K0 + TOL))) return 1;
  if (fabsf(cr0 - cl0) > Tol::contact) return 1;
  const bool left = lamC >= 0.f;
  const float lam = left ? L.lam : R.lam;
  const float JD = left ? L.D : R.D, JE = left ? L.E : R.E, m0 = left ? L.m0 : R.m0, m1 = left ? L.m1 : R.m1,
              m2 = left ? L.m2 : R.m2, JB1 = left ? L.B1 : R.B1, JB2 = left ? L.B2 : R.B2;
  const float v0 = left ? e.l.v0 : e.r.v0, v1 = left ? e.l.v1 : e.r.v1, v2 = left ? e.l.v2 : e.r.v2;
  const float b1 = left ? e.l.b1 : e.r.b1, b2 = left ? e.l.b2 : e.r.b2, ia = left ? e.l.ia : e.r.ia;
  const float K0 = left ? e.l.K0 : e.r.K0;
  const bool outside = left ? L.lam >= 0.f : R.lam < 0.f;
  // between the fast and the Alfven wave: F = lam U_a - J
  const float vb = v0 * Bx + v1 * b1 + v2 * b2;
  float aD = JD * ia, aE = (JE + p * v0 - vb * Bx) * ia;
  float a0 = (aE + p) * v0 - vb * Bx, a1 = (aE + p) * v1 - vb * b1, a2 = (aE + p) * v2 - vb * b2;
  float aB1 = b1, aB2 = b2;
  if (outside || fabsf(lam - v0) < Tol::degenerate) {   // the state outside the fast wave
    float U[7];
    outer(left, U);
    aD = U[0]; aE = U[1]; a0 = U[2]; a1 = U[3]; a2 = U[4]; aB1 = U[5]; aB2 = U[6];
  }
  float f0 = lam * aD - JD, f1 = lam * aE - JE, f2 = lam * a0 - m0, f3 = lam * a1 - m1, f4 = lam * a2 - m2,
        f5 = lam * aB1 - JB1, f6 = lam * aB2 - JB2;
  const bool inner = !outside && (left ? K0 < 0.f : K0 >= 0.f);
  if (inner) {   // between the Alfven wave and the contact: + K0 (U_c - U_a)
    const float B1 = c1 * idK, B2 = c2 * idK;
    const float B0 = flat ? 0.f : Bx, t1 = flat ? 0.f : B1, t2 = flat ? 0.f : B2;
    const bool s = left ? sl : sr;
    const float y = left ? yl : yr;
    const float cv0 = left ? cl0 : cr0;
    const float K1 = left ? e.l.K1 : e.r.K1, K2 = left ? e.l.K2 : e.r.K2;
    const float cv1 = s ? v1 : (flat ? K1 : K1 - c1 * y), cv2 = s ? v2 : (flat ? K2 : K2 - c2 * y);
    const float den = K0 - lamC;
    if (!(fabsf(den) < Tol::degenerate)) {
      const float id = 1.f / den;
      const float vB = cv0 * B0 + cv1 * t1 + cv2 * t2;
      const float cD = aD * (K0 - v0) * id;
      const float cE = (K0 * aE - a0 + p * lamC - vB * B0) * id;
      f0 += K0 * (cD - aD);
      f1 += K0 * (cE - aE);
      f2 += K0 * ((cE + p) * cv0 - vB * B0 - a0);
      f3 += K0 * ((cE + p) * cv1 - vB * t1 - a1);
      f4 += K0 * ((cE + p) * cv2 - vB * t2 - a2);
      f5 += K0 * (t1 - aB1);
      f6 += K0 * (t2 - aB2);
    }
  }
  F[0] = f0;
  F[1] = f1 - f0;
  F[2] = f2;
  F[3] = f3;
  F[4] = f4;
  F[5] = f5;
  F[6] = f6;
  return 0;
}

// The FP64 form of the same, for the faces where FP32 does not converge: Newton from the
// average face state, then the reference's ladder.  Out of line (rare, and its FP64 state
// would set the register budget of the sweeps).
struct HllPressure64 {
  float pt;
  int err, iters, attempts;
};
struct HllState32 {
  float U[8], P[8];   // D tau S B, and the average primitives
};
static __device__ __noinline__ HllPressure64 hll_pressure64(PhysParams pp, HllState32 s)
{
  double U[8], P[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) { U[i] = double(s.U[i]); P[i] = double(s.P[i]); }
  const double V2 = P[vx] * P[vx] + P[vy] * P[vy] + P[vz] * P[vz];
  const double W2 = 1.0 / (1.0 - V2);
  const double h = 1.0 + P[pre] / P[rho] * (1.0 / (pp.gamma - 1.0) + 1.0);
  const bool usable = V2 < 1.0 && P[rho] > 0.0 && P[pre] > 0.0;
  C2PTally t{0, 0};
  HllPressure64 o;
  o.err = cons_to_prim<true, 1>(pp, U, P, &t, P[rho] * h * W2, sqrt(W2), usable);
  o.iters = t.iters;
  o.attempts = t.attempts;
  float Pf[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) Pf[i] = float(P[i]);
  o.pt = hlld_estimate0(Pf);
  return o;
}

// HlldRmhdRiemannSolver::IntercellFlux at s = 0 in FP32 (riemann_hlld-rmhd.cpp:179-313).  pl, pr
// and the flux f are in the normal frame of dim.  `src` gives the two face states (reference
// component order) again where a rare path needs them, so that they need not stay live through
// the pressure iteration.  Returns 1 when a face state is
// unphysical (the caller retries with the zone states); used_hllc reports the fallback.
template <class Src>
__device__ __forceinline__ int riemann_hlld32(const PhysParams &pp, int dim, const float *pl, const float *pr,
                                              float *f, float &ml, int &used_hllc, C2PTally *tally, const Src &src)
{
  using Tol = RmhdTol<float>;
  const float gamma = float(pp.gamma), rh_p = gamma / (gamma - 1.f);
  const float bx = 0.5f * (pl[Bx] + pr[Bx]);
  used_hllc = 0;
  if (tally) { tally->iters = 0; tally->attempts = 0; }
  SideState s, t;
  float ap, am;
  if (face_sides(gamma, pl, pr, bx, s, t, ap, am, ml)) return 1;
  // (Z, W) of the average face state
  float Z0, W0;
  bool usable;
  {
    const float ar = 0.5f * (pl[rho] + pr[rho]), apr = 0.5f * (pl[pre] + pr[pre]);
    const float a1 = 0.5f * (pl[vx] + pr[vx]), a2 = 0.5f * (pl[vy] + pr[vy]), a3 = 0.5f * (pl[vz] + pr[vz]);
    const float i2 = 1.f - (a1 * a1 + a2 * a2 + a3 * a3);
    usable = i2 > 0.f && ar > 0.f && apr > 0.f;
    W0 = rsqrtf(i2);
    Z0 = (ar + rh_p * apr) * W0 * W0;
  }
  const HlldSide32 L = side_jump(s, am), R = side_jump(t, ap);
  float p0 = 0.f;
  int failed;
  {
    const float is = 1.f / (ap - am);
    const float D = (R.D - L.D) * is, E = (R.E - L.E) * is, m0 = (R.m0 - L.m0) * is, m1 = (R.m1 - L.m1) * is,
                m2 = (R.m2 - L.m2) * is, b1 = (R.B1 - L.B1) * is, b2 = (R.B2 - L.B2) * is;
    int it = 0;
    failed = usable ? hll_pressure32(gamma, float(pp.pfloor), D, E, m0, m1, m2, bx, b1, b2, Z0, W0, p0, it) : 1;
    int att = 1;
    if (failed) {
      float ql[8], qr[8];
      src(ql, qr);
      HllState32 h;
      h.U[ddd] = D; h.U[tau] = E - D; h.U[Sx] = m0; h.U[Sy] = m1; h.U[Sz] = m2;
      h.U[Bx] = bx; h.U[By] = b1; h.U[Bz] = b2;
#pragma unroll
      for (int i = 0; i < 8; ++i) h.P[i] = 0.5f * (ql[frame_slot(dim, i)] + qr[frame_slot(dim, i)]);
      h.P[Bx] = bx;
      const HllPressure64 o = hll_pressure64(pp, h);
      failed = o.err;
      p0 = o.pt;
      it = o.iters;
      att = o.attempts;
    }
    if (tally) { tally->iters = it; tally->attempts = att; }
  }
  const bool direct = fabsf(bx) < Tol::bx_small;
  if (!failed) {
#pragma unroll 1
    for (int attempt = 0; attempt < 3; ++attempt) {
      float p = attempt == 0 ? p0 : 0.f;
      if (direct || attempt == 1) {   // eq. 55: the HLL state without its field
        const float is = 1.f / (ap - am);
        const float E = (R.E - L.E) * is, m = (R.m0 - L.m0) * is;
        p = hlld_estimate1(E, (am * R.E - ap * L.E) * is, m, (am * R.m0 - ap * L.m0) * is);
      }
      HlldEval32 e;
      float F[7];
      const auto outer = [&](bool left, float *U) {
        float ql[8], qr[8];
        src(ql, qr);
        SideState o;
        FastPair fp;
        const float *q = left ? ql : qr;
        const auto at = [&](int k) { return q[frame_slot(dim, k)]; };
        side_state(gamma, rh_p, q[rho], q[pre], at(vx), at(vy), at(vz), bx, at(By), at(Bz), o, fp);
        U[0] = o.D; U[1] = o.E; U[2] = o.S0; U[3] = o.S1; U[4] = o.S2; U[5] = o.B1; U[6] = o.B2;
      };
      if (hlld_root32(L, R, bx, direct, p, e) == 0 && hlld_flux32(L, R, bx, p, e, F, outer) == 0) {
#pragma unroll
        for (int i = 0; i < 5; ++i) f[i] = F[i];
        f[Bx] = 0.f;
        f[By] = F[5];
        f[Bz] = F[6];
        return 0;
      }
      if (direct) break;
    }
  }
  used_hllc = 1;
  Face8<float> a, b;
  src(a.v, b.v);
  const HllcOut<float> o = riemann_hllc32_fallback(dim, gamma, a, b, ml);
  ml = o.ml;
#pragma unroll
  for (int i = 0; i < 8; ++i) f[i] = o.F[i];
  return o.err;
}

}  // namespace mgpu
