// mbm_math.cuh -- per-cell and per-face FP64 arithmetic of the Grad-13 Heun stage,
// in namespace mbm::MBM_ARITH (bitwise by default, fastmath under MBM_FAST_ARITH).
//
// Bitwise mode: every expression keeps the operand order and association of the
// reference expression it restates (file:line cited per function), the file is
// compiled with -fmad=false, and double division and sqrt are IEEE round-to-
// nearest on sm_100a, so results agree bit for bit with the reference compiled
// by gcc on x86-64 (SSE2, no contraction).
#pragma once

#include <cuda_runtime.h>
#include <math.h>

#include "mbm_internal.h"

#ifndef MBM_ARITH
#define MBM_ARITH bitwise
#endif
#ifndef MBM_FAST_ARITH
#define MBM_FAST_ARITH 0
#endif
#if MBM_FAST_ARITH
#define MBM_HD __host__ __device__ __forceinline__
#include "mbm_adjoint_math.cuh"   // primitive-form Conservative and Grad-13 flux
#endif
#include "mbm_div.cuh"
#include "mbm_newton.cuh"

namespace mbm {
namespace MBM_ARITH {

// the reference's max/min/sgn (src/tools.h:3-17): a > b ? a : b etc.
__device__ __forceinline__ double rmax(double a, double b) { return a > b ? a : b; }
__device__ __forceinline__ double rmin(double a, double b) { return a < b ? a : b; }
__device__ __forceinline__ double rsgn(double a) { return a == 0 ? 0.0 : (a < 0 ? -1.0 : 1.0); }

// Reciprocal, square root and lone quotients.  Bitwise: the exact division of mbm_div.cuh,
// IEEE division and sqrt.
//
// Fast arithmetic (MBM_FAST_ARITH, MBM_MODE_FAST): the refined hardware approximations of
// mbm_newton.cuh; the quotient is RN(x*r) without the correction, within one unit in the last
// place of x/y, and nothing is checked.  Its multiply-adds are written out, not left to the
// compiler's contraction, so that every kernel that evaluates these functions (row march, tiles)
// gets the same bits.
#if MBM_FAST_ARITH
using mbm_newton::frcp;
using mbm_newton::fsqrt;
__device__ __forceinline__ double fdiv(double x, double y) { return x * frcp(y); }
#else
__device__ __forceinline__ double fdiv(double x, double y) { return x / y; }
__device__ __forceinline__ double fsqrt(double x) { return sqrt(x); }
#endif

struct Recip {        // 1/y for a denominator shared by several quotients
  double y, r;
#if MBM_FAST_ARITH
  __device__ __forceinline__ explicit Recip(double y_) : y(y_), r(frcp(y_)) {}
  __device__ __forceinline__ Recip(double y_, double r_) : y(y_), r(r_) {}
#else
  bool bad;           // y outside what mk_rcp and mk_div admit
  __device__ __forceinline__ explicit Recip(double y_) : y(y_), r(mk_rcp_all(y_)), bad(mk_bad_den(y_)) {}
  __device__ __forceinline__ Recip(double y_, double r_) : y(y_), r(r_), bad(false) {}   // r_ = RN(1/y_), y_ in range
#endif
};

// q[n] = x[n] / D.y
template <int N>
__device__ __forceinline__ void quotients(const double (&x)[N], const Recip& D, double (&q)[N]) {
#if MBM_FAST_ARITH
#pragma unroll
  for (int n = 0; n < N; n++) q[n] = x[n] * D.r;
#else
  MkRange g;
#pragma unroll
  for (int n = 0; n < N; n++) {
    g.add(x[n]);
    q[n] = mk_div(x[n], D.y, D.r);
  }
  if (__builtin_expect(g.bad() || D.bad, 0)) {
#pragma unroll
    for (int n = 0; n < N; n++) q[n] = div_ieee(x[n], D.y);
  }
#endif
}

__device__ __forceinline__ double quotient(double x, const Recip& D) {
  const double a[1] = {x};
  double q[1];
  quotients(a, D, q);
  return q[0];
}

#if MBM_FAST_ARITH
// Primitive (src/Flux.c:30-56)
__device__ __forceinline__ void primitive(const double (&U)[NV], double (&P)[NV]) {
  const double rho = U[0], r = frcp(rho), E = U[3];
  const double v1 = U[1] * r, v2 = U[2] * r;
  const double a = v1 * v1, b = v2 * v2;
  const double T11 = fma(U[4], r, -a), T12 = fma(U[5], r, -(v1 * v2)), T22 = fma(U[6], r, -b);
  P[0] = rho; P[1] = v1; P[2] = v2;
  P[3] = fma(2 * E, r, -(a + b)) * (1.0 / 3);
  P[4] = T11; P[5] = T12; P[6] = T22;
  P[7] = fma(-rho, fma(T11, v1, T12 * v2), fma(-E, v1, U[7]));
  P[8] = fma(-rho, fma(T12, v1, T22 * v2), fma(-E, v2, U[8]));
}
#else
// Primitive (src/Flux.c:30-56)
__device__ __forceinline__ void primitive(const double (&U)[NV], double (&P)[NV]) {
  const double rho = U[0];
  const Recip R(rho), third(3.0, 1.0 / 3.0);
  const double x[6] = {U[1], U[2], 2 * U[3], U[4], U[5], U[6]};
  double q[6];
  quotients(x, R, q);
  const double v1 = q[0], v2 = q[1];
  const double vs = v1 * v1 + v2 * v2;
  const double th = quotient(q[2] - vs, third);
  const double E = U[3];
  const double T11 = q[3] - v1 * v1;
  const double T12 = q[4] - v1 * v2;
  const double T22 = q[5] - v2 * v2;
  P[0] = rho; P[1] = v1; P[2] = v2; P[3] = th;
  P[4] = T11; P[5] = T12; P[6] = T22;
  P[7] = U[7] - E * v1 - rho * (T11 * v1 + T12 * v2);
  P[8] = U[8] - E * v2 - rho * (T12 * v1 + T22 * v2);
}
#endif

#if !MBM_FAST_ARITH
// moments with an explicit energy (src/Flux.c:65-73, 255-263)
__device__ __forceinline__ void moments_e(double rho, double v1, double v2, double E, double T11,
                                          double T12, double T22, double q1, double q2,
                                          double (&U)[NV]) {
  U[0] = rho;
  U[1] = rho * v1;
  U[2] = rho * v2;
  U[3] = E;
  U[4] = rho * (T11 + v1 * v1);
  U[5] = rho * (T12 + v1 * v2);
  U[6] = rho * (T22 + v2 * v2);
  U[7] = q1 + E * v1 + rho * (T11 * v1 + T12 * v2);
  U[8] = q2 + E * v2 + rho * (T12 * v1 + T22 * v2);
}

// Conservative (src/Flux.c:61-74 with src/primDef.h:9-20)
__device__ __forceinline__ void conservative(const double (&P)[NV], double (&U)[NV]) {
  const double vs = P[1] * P[1] + P[2] * P[2];
  const double E = 0.5 * P[0] * vs + 1.5 * P[0] * P[3];
  moments_e(P[0], P[1], P[2], E, P[4], P[5], P[6], P[7], P[8], U);
}

// Grad-13 flux along x of a moment vector (src/Flux.c:79-119)
__device__ __forceinline__ void grad13_flux_x(const double (&U)[NV], double (&F)[NV]) {
  const double rho = U[0];
  const Recip R(rho), third(3.0, 1.0 / 3.0);
  const double x[6] = {U[1], U[2], 2 * U[3], U[4], U[5], U[6]};
  double q[6];
  quotients(x, R, q);
  const double v1 = q[0], v2 = q[1];
  const double vs = v1 * v1 + v2 * v2;
  const double th = quotient(q[2] - vs, third);
  const double E = U[3];
  const double T11 = q[3] - v1 * v1;
  const double T12 = q[4] - v1 * v2;
  const double T22 = q[5] - v2 * v2;
  const double q1 = U[7] - E * v1 - rho * (T11 * v1 + T12 * v2);
  const double q2 = U[8] - E * v2 - rho * (T12 * v1 + T22 * v2);
  const double y[3] = {1.2 * q1, 0.4 * q2, 0.4 * q1};
  double M[3];
  quotients(y, R, M);
  const double M111 = M[0], M121 = M[1], M112 = M[1], M221 = M[2], M122 = M[2];
  const double R11 = 5 * th * th + 7 * th * (T11 - th);
  const double R12 = 7 * th * T12;
  F[0] = rho * v1;
  F[1] = rho * (T11 + v1 * v1);
  F[2] = rho * (T12 + v1 * v2);
  F[3] = E * v1 + rho * (T11 * v1 + T12 * v2) + q1;
  F[4] = rho * (M111 + 3 * T11 * v1 + v1 * v1 * v1);
  F[5] = rho * (M121 + T11 * v2 + 2 * T12 * v1 + v1 * v2 * v1);
  F[6] = rho * (M221 + T22 * v1 + 2 * T12 * v2 + v2 * v2 * v1);
  F[7] = 2 * (q1 + rho * (T11 * v1 + T12 * v2)) * v1 + E * v1 * v1 +
         rho * (M111 * v1 + M112 * v2) + 0.5 * rho * (T11 * vs + R11);
  F[8] = q2 * v1 + q1 * v2 + rho * (v1 * v2 * (T11 + T22) + 1.5 * T12 * vs) + E * v1 * v2 +
         rho * (M121 * v1 + M122 * v2) + 0.5 * rho * R12;
}
#endif

#if !MBM_FAST_ARITH
// Damping factors of the direct production integration (src/Flux.c:213-223) at one
// argument: flags 0 (= -1) and 1 share a denominator, hence one reciprocal; flag 2 is
// (1 + z/2) / (1 + z/2), which is 1 in any rounding; flag 3 is a reciprocal.  For
// 0 <= z < 2^200 every numerator is 0 or in the range of mk_div; otherwise (NaN, a negative
// or huge z) IEEE division.
__device__ __forceinline__ bool damp_in(double z) { return (unsigned)__double2hiint(z) < (1223u << 20); }

__device__ __forceinline__ void damp01(double z, double& r0, double& r1) {
  const double s = 0.25 * z * z, n0 = 1 + 0.5 * z - s, n1 = 1 + z;
  const Recip D(n1 + s);
  r0 = mk_div(n0, D.y, D.r);
  r1 = mk_div(n1, D.y, D.r);
  if (__builtin_expect(D.bad || !damp_in(z), 0)) {
    r0 = div_ieee(n0, D.y);
    r1 = div_ieee(n1, D.y);
  }
}

__device__ __forceinline__ void damp23(double z, double& r2, double& r3) {
  const Recip D(1 + 0.5 * z);
  r2 = 1.0;
  r3 = D.r;
  if (__builtin_expect(D.bad || !damp_in(z), 0)) {
    r2 = div_ieee(D.y, D.y);
    r3 = div_ieee(1.0, D.y);
  }
}
#endif

// The collision number z = dt nu0 rho sqrt(theta) / Kn of ProductionsDirect
// (src/Flux.c:230-267 with CollFreq, src/Scenario.c:28-42; nu0 = 1): the same
// expression for every flag, so one evaluation serves all of a cell's flags.
__device__ __forceinline__ double coll_of(const double (&P)[NV], double dt, const Recip& Kn) {
  const double nu0 = 1.0;
  return quotient(nu0 * P[0] * fsqrt(P[3]), Kn) * dt;
}

#if !MBM_FAST_ARITH
// ProductionsDirect (src/Flux.c:230-267) with ExternalForce (src/Scenario.c:28-42;
// force (F, 0)), starting from the primitives P of the input moments, given its damping
// factors d1 = rdamp<FLAG>(z), d2 = rdamp<FLAG>(2z/3).  Writes the relaxed moments.
template <int FLAG>
__device__ __forceinline__ void relax_d(const double (&P)[NV], double (&Out)[NV], double dt, double F,
                                        double d1, double d2) {
  const double rho = P[0], th = P[3];
  double v1 = P[1], v2 = P[2];
  double vs = v1 * v1 + v2 * v2;
  double E = 0.5 * rho * vs + 1.5 * rho * th;
  if (FLAG == 0 || FLAG == 2) {
    const double g0 = F, g1 = 0.0;
    v1 += dt * g0;
    v2 += dt * g1;
    vs = v1 * v1 + v2 * v2;
    E = 0.5 * rho * vs + 1.5 * rho * th;
  }
  const double T11 = d1 * (P[4] - th) + th;
  const double T12 = d1 * P[5];
  const double T22 = d1 * (P[6] - th) + th;
  moments_e(rho, v1, v2, E, T11, T12, T22, d2 * P[7], d2 * P[8], Out);
}

// ProductionsDirect of flag -1 from the primitives P: writes the relaxed moments
__device__ __forceinline__ void relax_m1(const double (&P)[NV], double (&Out)[NV], double dt,
                                         const Recip& Kn, double F) {
  const double coll = coll_of(P, dt, Kn);
  double d1, d2, unused;
  damp01(coll, d1, unused);
  damp01(2.0 / 3 * coll, d2, unused);
  relax_d<-1>(P, Out, dt, F, d1, d2);
}
#endif

#if MBM_FAST_ARITH
// The projection of stage 2 (flag 3) in primitive form: rho, theta and the velocity kept,
// T_ij - theta delta_ij scaled by 1/(1 + z/2), q by 1/(1 + z/3) -- without forming the
// moments and dividing by rho again
__device__ __forceinline__ void project3(double (&P)[NV], double z) {
  const double th = P[3];
  const double d1 = frcp(fma(0.5, z, 1.0)), d2 = frcp(fma(0.5, 2.0 / 3 * z, 1.0));
  P[4] = fma(d1, P[4] - th, th);
  P[5] = d1 * P[5];
  P[6] = fma(d1, P[6] - th, th);
  P[7] = d2 * P[7];
  P[8] = d2 * P[8];
}
#endif

#if MBM_FAST_ARITH
// The damping factors of flags 0 (= -1) and 1 at z and 2z/3 (src/Flux.c:213-223) from
// one reciprocal per argument (fast arithmetic): both share the denominator
// 1 + z + z^2/4 = (1 + z/2)^2, so with w = 1/(1 + z/2)
//   R_0(z) = (1 + z/2 - z^2/4) w^2,   R_1(z) = (1 + z) w^2.
struct Damp01 {
  double d1_0, d2_0;   // flag 0 / -1: R(z), R(2z/3)
  double d1_1, d2_1;   // flag 1
  __device__ __forceinline__ explicit Damp01(double z) {
    const double z2 = 2.0 / 3 * z;
    const double w1 = frcp(fma(0.5, z, 1.0)), w2 = frcp(fma(0.5, z2, 1.0));
    const double s1 = w1 * w1, s2 = w2 * w2;
    d1_0 = fma(z, fma(-0.25, z, 0.5), 1.0) * s1;
    d2_0 = fma(z2, fma(-0.25, z2, 0.5), 1.0) * s2;
    d1_1 = (1.0 + z) * s1;
    d2_1 = (1.0 + z2) * s2;
  }
};

// the moments of relax<-1>(P) (ProductionsDirect without the force, src/Flux.c:230-267)
// given its damping factors d1 = R(z), d2 = R(2z/3) (fast arithmetic)
__device__ __forceinline__ void relaxed_moments(const double (&P)[NV], double d1, double d2,
                                                double (&Out)[NV]) {
  const double rho = P[0], v1 = P[1], v2 = P[2], th = P[3];
  const double E = rho * fma(0.5, fma(v1, v1, v2 * v2), 1.5 * th);
  const double T11 = fma(d1, P[4] - th, th), T12 = d1 * P[5], T22 = fma(d1, P[6] - th, th);
  Out[0] = rho;
  Out[1] = rho * v1;
  Out[2] = rho * v2;
  Out[3] = E;
  Out[4] = rho * (T11 + v1 * v1);
  Out[5] = rho * (T12 + v1 * v2);
  Out[6] = rho * (T22 + v2 * v2);
  Out[7] = fma(rho, fma(T11, v1, T12 * v2), fma(E, v1, d2 * P[7]));
  Out[8] = fma(rho, fma(T12, v1, T22 * v2), fma(E, v2, d2 * P[8]));
}

__device__ __forceinline__ void relax_m1(const double (&P)[NV], double (&Out)[NV], double dt,
                                         const Recip& Kn, double) {
  const Damp01 dm(coll_of(P, dt, Kn));
  relaxed_moments(P, dm.d1_0, dm.d2_0, Out);
}

// relax<2>(Primitive(U)) in moment form (fast arithmetic): flag 2 leaves T and q as
// they are (R = 1), so only the push of the velocity by g = dt F changes the moments:
//   U1 + rho g,  E + g (U1 + rho g/2),  U4 + g (2 U1 + rho g),  U5 + g U2,
//   U7 + g (E + U4 + g (3 U1 + rho g)/2),  U8 + g (U5 + g U2/2)   (E = U3)
// -- no Primitive, no division
__device__ __forceinline__ void push_moments(const double (&U)[NV], double g, double (&R)[NV]) {
  const double rg = U[0] * g;
  R[0] = U[0];
  R[1] = U[1] + rg;
  R[2] = U[2];
  R[3] = fma(g, fma(0.5, rg, U[1]), U[3]);
  R[4] = fma(g, fma(2.0, U[1], rg), U[4]);
  R[5] = fma(g, U[2], U[5]);
  R[6] = U[6];
  R[7] = fma(g, fma(0.5 * g, fma(3.0, U[1], rg), U[3] + U[4]), U[7]);
  R[8] = fma(g, fma(0.5 * g, U[2], U[5]), U[8]);
}
// The same push applies to any moment vector whose temperature and heat flux stay
// fixed: relax<0>(P) = push_moments(relax<-1>(P), dt F), flag 0 differing from flag
// -1 only by the force acting on the velocity before the moments are formed.
#endif

// A cell's update from its relaxation terms and its faces' fluxes, in the order of the
// reference's face loop (src/Main.c:353-384)
__device__ __forceinline__ double accumulate(double R, double dtdx, double dtdy, double Fm, double Gm, double G,
                                             double F) {
#if MBM_FAST_ARITH
  return fma(-dtdx, F, fma(-dtdy, G, fma(dtdy, Gm, fma(dtdx, Fm, R))));
#else
  return (((R + dtdx * Fm) + dtdy * Gm) - dtdy * G) - dtdx * F;
#endif
}

// Limit1 (src/Limiter.c:26-59)
__device__ __forceinline__ double superbee_phi(double r) {
  if (r < 0.0) return 0.0;
  if (r < 0.5) return 2 * r;
  if (r < 1.0) return 1.0;
  if (r < 2.0) return r;
  return 2.0;
}

template <int LIM>
__device__ __forceinline__ double limit(double d1, double d2) {
  if (LIM == 0) return 0.0;
  if (LIM == 1) return 0.5 * (d1 + d2);
  if (LIM == 2) return 0.5 * (rsgn(d1) + rsgn(d2)) * rmin(fabs(d1), fabs(d2));
  if (LIM == 3) return d1 * superbee_phi(fdiv(d2, d1));
  const double eps = 1.0e-10;
  const double w1 = fabs(d1) + eps, w2 = fabs(d2) + eps;
#if MBM_FAST_ARITH
  return fdiv(fma(w1, d2, w2 * d1), w1 + w2);
#else
  return fdiv(w1 * d2 + w2 * d1, w1 + w2);
#endif
}

#if MBM_FAST_ARITH
// S = Limit1(d1, d2) of N components by limiter LIM, or by lim if LIM is LIM_ANY
template <int LIM, int N>
__device__ __forceinline__ void limits(const double (&d1)[N], const double (&d2)[N], int lim, double (&S)[N]) {
  if constexpr (LIM == LIM_ANY) {
    switch (lim) {
      case 0: limits<0>(d1, d2, lim, S); return;
      case 1: limits<1>(d1, d2, lim, S); return;
      case 2: limits<2>(d1, d2, lim, S); return;
      case 3: limits<3>(d1, d2, lim, S); return;
      default: limits<4>(d1, d2, lim, S); return;
    }
  } else {
#pragma unroll
    for (int n = 0; n < N; n++) S[n] = limit<LIM>(d1[n], d2[n]);
  }
}
#endif

#if !MBM_FAST_ARITH
// L = Limit1(d1, d2) and the slope L / h of N components (src/Main.c:346-349), D =
// Recip(h), h in the safe range.  The harmonic limiter's quotient has a denominator of its
// own, |d1| + |d2| + 2e-10: reciprocals without a branch, and one check of the set
// (numerators within 2^+-400 or zero, denominators below 2^80, so that L itself is within
// the range the division by h admits).
template <int LIM, int N>
__device__ __forceinline__ void slopes(const double (&d1)[N], const double (&d2)[N], const Recip& D,
                                       double (&S)[N]) {
  if (LIM == 0) {
#pragma unroll
    for (int n = 0; n < N; n++) S[n] = 0.0;      // 0 / h
    return;
  }
  double L[N];
  if (LIM != 4) {
#pragma unroll
    for (int n = 0; n < N; n++) L[n] = limit<LIM>(d1[n], d2[n]);
    quotients(L, D, S);
    return;
  }
  const double eps = 1.0e-10;
  MkRange g;
  unsigned md = 0u;
  int ones = 0;
#pragma unroll
  for (int n = 0; n < N; n++) {
    const double w1 = fabs(d1[n]) + eps, w2 = fabs(d2[n]) + eps;
    const double x = w1 * d2[n] + w2 * d1[n], y = w1 + w2;
    g.add(x);
    md = max(md, (unsigned)__double2hiint(y));
    ones |= __double2loint(y) == -1;
    L[n] = mk_div(x, y, mk_rcp(y));
    S[n] = mk_div(L[n], D.y, D.r);
  }
  if (__builtin_expect(g.lo < (623u << 21) || g.hi >= (1424u << 21) || md >= (1103u << 20) || ones || D.bad, 0)) {
#pragma unroll
    for (int n = 0; n < N; n++) S[n] = div_ieee(limit<LIM>(d1[n], d2[n]), D.y);
  }
}

// the same by the limiter LIM, or by lim if LIM is LIM_ANY
template <int LIM, int N>
__device__ __forceinline__ void slopes_of(const double (&d1)[N], const double (&d2)[N], const Recip& D, int lim,
                                          double (&S)[N]) {
  if constexpr (LIM != LIM_ANY) {
    slopes<LIM>(d1, d2, D, S);
  } else {
    switch (lim) {
      case 0: slopes<0>(d1, d2, D, S); return;
      case 1: slopes<1>(d1, d2, D, S); return;
      case 2: slopes<2>(d1, d2, D, S); return;
      case 3: slopes<3>(d1, d2, D, S); return;
      default: slopes<4>(d1, d2, D, S); return;
    }
  }
}
#endif

#if MBM_FAST_ARITH
// Conservative(P) and the Grad-13 flux along x of the same state (src/Flux.c:61-119
// in primitive variables; fast arithmetic).  The flux's first four components are
// moments (F0..F3 = U1, U4, U5, U7) and the others are regrouped around them:
//   F4 = U1 (3 T11 + u^2) + 6/5 q1
//   F5 = v U4 + 2 u rho T12 + 2/5 q2,   F6 = u U6 + 2 v rho T12 + 2/5 q1
//   F7 = u (2 U7 - E u + 6/5 q1) + 2/5 q2 v + rho/2 (T11 (|v|^2 + 7 theta) - 2 theta^2)
//   F8 = 7/5 (q2 u + q1 v) + u v (rho (T11 + T22) + E) + rho T12 (3/2 |v|^2 + 7/2 theta)
// (E = U3; M111 = 6/5 q1/rho, M112 = M121 = 2/5 q2/rho, M122 = M221 = 2/5 q1/rho).
__device__ __forceinline__ void cons_flux_x(const double (&P)[NV], double (&U)[NV], double (&F)[NV]) {
  const double r = P[0], u = P[1], v = P[2], th = P[3];
  const double T11 = P[4], T12 = P[5], T22 = P[6], q1 = P[7], q2 = P[8];
  const double uu = u * u, vs = fma(v, v, uu);
  const double E = fma(1.5 * r, th, 0.5 * r * vs);
  U[0] = r;
  U[1] = r * u;
  U[2] = r * v;
  U[3] = E;
  U[4] = r * (T11 + uu);
  U[5] = r * (T12 + u * v);
  U[6] = r * fma(v, v, T22);
  U[7] = fma(r, fma(T11, u, T12 * v), fma(E, u, q1));
  U[8] = fma(r, fma(T12, u, T22 * v), fma(E, v, q2));
  const double q1a = 1.2 * q1, q1b = 0.4 * q1, q2b = 0.4 * q2;
  const double rT12 = r * T12, t2 = rT12 + rT12;
  F[0] = U[1];
  F[1] = U[4];
  F[2] = U[5];
  F[3] = U[7];
  F[4] = fma(U[1], fma(3.0, T11, uu), q1a);
  F[5] = fma(v, U[4], fma(u, t2, q2b));
  F[6] = fma(u, U[6], fma(v, t2, q1b));
  F[7] = fma(u, fma(-E, u, 2.0 * U[7]) + q1a,
             fma(q2b, v, 0.5 * r * fma(T11, fma(7.0, th, vs), -2.0 * th * th)));
  F[8] = fma(1.4, fma(q2, u, q1 * v), fma(u * v, fma(r, T11 + T22, E), rT12 * fma(1.5, vs, 3.5 * th)));
}

// FnumHLLE (src/Flux.c:308-379) in primitive form (fast arithmetic): the Grad-13
// flux straight from the face states -- no Conservative -> Primitive round trip and
// no rotations (a y face swaps the x and y components, which is what the rotation
// to the normal (0,1) amounts to); c = 2 sqrt(5/3 theta) as sqrt(20/3 theta).  The
// wave speeds and the coefficients of
//   (lamR fL - lamL fR + lamL lamR (UR - UL)) / alpha
// come first, then each side's moments and flux are formed and added in turn, so one
// side's vectors are live at a time (alpha = 0, both speeds 0: the mean of the two
// fluxes, coefficients 1/2, -1/2, 0).  Mathematically hll_swapped below; the
// rounding differs.
template <int DIR>
__device__ __forceinline__ double hll(const double (&PL_)[NV], const double (&PR_)[NV],
                                      double (&flx)[NV]) {
  double PL[NV], PR[NV];
  if (DIR == 2) {
    mbm_adj::swap_xy(PL_, PL);
    mbm_adj::swap_xy(PR_, PR);
  } else {
#pragma unroll
    for (int n = 0; n < NV; n++) { PL[n] = PL_[n]; PR[n] = PR_[n]; }
  }
  const double cR = fsqrt(20.0 / 3 * PR[3]);
  const double cL = fsqrt(20.0 / 3 * PL[3]);
  const double vR = PR[1], vL = PL[1];
  const double cMax = fabs(0.5 * (vL + vR)) + rmax(cR, cL);
  const double lamL = rmin(vL - cL, 0.0);
  const double lamR = rmax(vR + cR, 0.0);
  const double alph = lamR - lamL;
  const double ra = frcp(alph);
  const bool pos = alph > 0.0;
  const double a = lamR * ra, b = lamL * ra;
  const double ca = pos ? a : 0.5, cb = pos ? b : -0.5, cc = pos ? lamL * a : 0.0;
  double U[NV], F[NV], f[NV];
  cons_flux_x(PL, U, F);
#pragma unroll
  for (int n = 0; n < NV; n++) f[n] = fma(-cc, U[n], ca * F[n]);
  cons_flux_x(PR, U, F);
#pragma unroll
  for (int n = 0; n < NV; n++) f[n] = fma(cc, U[n], fma(-cb, F[n], f[n]));
  if (DIR == 2) {
    mbm_adj::swap_xy(f, flx);
  } else {
#pragma unroll
    for (int n = 0; n < NV; n++) flx[n] = f[n];
  }
  return cMax;
}
#else
// v, or -v where sg is the sign bit
__device__ __forceinline__ double signed_by(double v, unsigned sg) {
  return __hiloint2double(__double2hiint(v) ^ (int)sg, __double2loint(v));
}

// Flux through a face: rotate to the normal, x-flux, rotate back (src/Flux.c:126-172), with the
// direction a run-time value: U and F of a y face come with x and y swapped, so that both
// directions run the same operations.  The reference forms each rotated component as a*c + b*d
// with one of c, d +-1 and the other +-0; the product with +-1 is exact, so one FMA rounds like
// the two products and the sum (signs of zeros included).  An x face has normal (1, 0) and
// tangent (0, -1), a y face (0, 1) and (1, -0): in the swapped order the two differ by the sign of
// the second component (sg: the sign bit for x faces) and by the sign of the zero products (z:
// +0 for x, -0 for y faces), which fix the signs of zeros as the reference computes them.
__device__ __forceinline__ void flux_swapped(const double (&U)[NV], bool y, unsigned sg, double z,
                                             double (&F)[NV]) {
  double W[NV], G[NV];
  W[0] = U[0];
  W[1] = fma(U[2], 0.0, U[1]);
  W[2] = fma(U[1], z, signed_by(U[2], sg));
  W[3] = U[3];
  const double a = fma(U[5], 0.0, U[4]), b = fma(U[6], 0.0, U[5]);
  W[4] = fma(b, 0.0, a);
  W[5] = fma(a, z, signed_by(b, sg));
  const double a2 = fma(U[4], z, signed_by(U[5], sg)), b2 = fma(U[5], z, signed_by(U[6], sg));
  W[6] = fma(a2, z, signed_by(b2, sg));
  W[7] = fma(U[8], 0.0, U[7]);
  W[8] = fma(U[7], z, signed_by(U[8], sg));
  grad13_flux_x(W, G);
  F[0] = G[0];
  F[1] = fma(G[2], z, G[1]);
  F[2] = fma(G[1], 0.0, signed_by(G[2], sg));
  F[3] = G[3];
  const double a3 = fma(G[5], z, G[4]), b3 = fma(G[6], z, G[5]);
  F[4] = fma(b3, z, a3);
  const double g4 = y ? G[6] : G[4], g6 = y ? G[4] : G[6];
  const double p = fma(g6, 0.0, G[5]), r = fma(G[5], 0.0, g4);
  F[5] = fma(r, z, signed_by(p, sg));
  const double a4 = fma(G[4], 0.0, signed_by(G[5], sg)), b4 = fma(G[5], 0.0, signed_by(G[6], sg));
  F[6] = fma(a4, 0.0, signed_by(b4, sg));
  F[7] = fma(G[8], z, G[7]);
  F[8] = fma(G[7], 0.0, signed_by(G[8], sg));
}

// FnumHLLE (src/Flux.c:308-379) for a face with left/right primitives, the direction a run-time
// value: states and flux of a y face with x and y swapped (Conservative commutes with the swap
// bit for bit).  The diffusive scale FFlux/GFlux return is 0, so lamDiff(0/(cMax*dx)) is 1 for
// every cMax and cMax/1.0 == cMax: the division is omitted without changing a bit.  The left
// side is reduced to lamR fL and UL before the right side is formed, so that one side's vectors
// are live at a time (alpha <= 0: the mean of the fluxes, with factor 1 in place of lamR).
__device__ __forceinline__ double hll_swapped(const double (&PL)[NV], const double (&PR)[NV], bool y,
                                              double (&flx)[NV]) {
  const unsigned sg = y ? 0u : 0x80000000u;
  const double z = __hiloint2double(y ? (int)0x80000000u : 0, 0);
  const double cR = 2.0 * sqrt(5.0 / 3 * PR[3]);
  const double cL = 2.0 * sqrt(5.0 / 3 * PL[3]);
  const double vR = PR[1], vL = PL[1];
  const double cMax = fabs(0.5 * (vL + vR)) + rmax(cR, cL);
  const double lamL = rmin(vL - cL, 0.0);
  const double lamR = rmax(vR + cR, 0.0);
  const double alph = lamR - lamL;
  const bool pos = alph > 0.0;
  double UL[NV], UR[NV], f[NV], A[NV];
  conservative(PL, UL);
  flux_swapped(UL, y, sg, z, f);
  const double kL = pos ? lamR : 1.0;
#pragma unroll
  for (int n = 0; n < NV; n++) A[n] = kL * f[n];
  conservative(PR, UR);
  flux_swapped(UR, y, sg, z, f);
  if (pos) {
    const Recip D(alph);
    double num[NV];
#pragma unroll
    for (int n = 0; n < NV; n++) num[n] = A[n] - lamL * f[n] + lamL * lamR * (UR[n] - UL[n]);
    quotients(num, D, flx);
  } else {
#pragma unroll
    for (int n = 0; n < NV; n++) flx[n] = 0.5 * (A[n] + f[n]);
  }
  return cMax;
}
#endif

}  // namespace MBM_ARITH
}  // namespace mbm
