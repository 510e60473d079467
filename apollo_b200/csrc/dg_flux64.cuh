// Pointwise float64 fluxes and sources of the float64 kernels.
#pragma once

#include <cuda_runtime.h>

#include "dg_device.cuh"

namespace apollo {

// Reciprocal and square root of numbers well inside the normal range, without
// the range checks and branches of the general operations: the hardware's
// approximation (PTX rcp.approx.ftz.f64, rsqrt.approx.ftz.f64; relative error
// e of some 2^-20) corrected once by the third-order iteration that the series
// of 1/(1-e) and (1-e)^(-1/2) give (Householder, The Numerical Treatment of a
// Single Nonlinear Equation, 1970), which leaves e^3.  Error measured against the
// correctly rounded operations over 1.5e9 numbers between 2^-400 and 2^400: at
// most one unit in the last place (two for the reciprocal root, against the
// rounded reciprocal of the rounded root); the test suite holds these bounds from
// 2^-1000 to 2^1000.  Together with the tile prefetch and
// one branch for a lane's two points they took a right-hand side of Euler N = 4,
// K = 130,050 from 256 to 199 us, of HLL with 5 fields, N = 3, K = 32,258 from
// 122 to 67.
__device__ __forceinline__ double recip_normal(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x, y, 1.0);
  return fma(y, fma(e, e, e), y);
}
__device__ __forceinline__ double sqrt_normal(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double g = x * y, e = fma(-g, y, 1.0);
  return fma(g, e * fma(e, 0.375, 0.5), g);
}

__device__ __forceinline__ double rsqrt_normal(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-(x * y), y, 1.0);
  return fma(y, e * fma(e, 0.375, 0.5), y);
}

// A float64 whose divisions and roots are the ones above.  The equation's own code,
// its clamps, checks and quirks included, runs on it for states that need a clamp but
// lie inside quick_ok's range (the root of a number below 2^-1020 is zero; negative
// ones give NaN).  On doubles that code is a chain of some twenty divisions and roots
// a point: with 2 % of the elements below the density floor a right-hand side took,
// 4 fields, Lax-Friedrichs, N = 5, K = 2,048 58 us, K = 16,200 89; so 41 and 71 (no
// floors: 30, 61).
struct Quick {
  double v;
  __device__ __forceinline__ Quick() {}
  __device__ __forceinline__ Quick(double x) : v(x) {}
  __device__ __forceinline__ friend Quick operator+(Quick a, Quick b) { return a.v + b.v; }
  __device__ __forceinline__ friend Quick operator-(Quick a, Quick b) { return a.v - b.v; }
  __device__ __forceinline__ friend Quick operator-(Quick a) { return -a.v; }
  __device__ __forceinline__ friend Quick operator*(Quick a, Quick b) { return a.v * b.v; }
  __device__ __forceinline__ friend Quick operator/(Quick a, Quick b) { return a.v * recip_normal(b.v); }
  __device__ __forceinline__ friend bool operator<(Quick a, Quick b) { return a.v < b.v; }
  __device__ __forceinline__ friend bool operator<=(Quick a, Quick b) { return a.v <= b.v; }
  __device__ __forceinline__ friend bool operator>(Quick a, Quick b) { return a.v > b.v; }
  __device__ __forceinline__ friend bool operator>=(Quick a, Quick b) { return a.v >= b.v; }
  __device__ __forceinline__ friend bool operator==(Quick a, Quick b) { return a.v == b.v; }
  __device__ __forceinline__ friend Quick sqrt(Quick a) {
    const double r = sqrt_normal(a.v);
    return (__double2hiint(a.v) & 0x7fffffff) < 0x00300000 ? 0.0 : r;
  }
  __device__ __forceinline__ friend Quick fabs(Quick a) { return ::fabs(a.v); }
  __device__ __forceinline__ friend Quick abs_int(Quick a) { return ::apollo::abs_int(a.v); }
};

// Euler fluxes in float64 with one reciprocal of the density per state and
// the flux formed along a direction directly (a n.F + b n.G in one pass): the
// same quantities as WxEulerEqn's flux and Lax-Friedrichs flux
// (wxeulereqn.cc:809-871, :1097-1117) to round-off, for states that need none
// of the reference's clamps and whose density and pressure lie between 2^-400
// and 2^400 (checked on the high words, so that the float64 pipe does not
// compare; their quotient, the square of the sound speed up to gamma, then lies
// far above the 1e-300 that keeps the flow speed's root off zero); any other state takes the equation's own code, which applies the
// clamps and raises its error flags.  The density's bound comes from the host:
// formed here from the floor's high word, four of the kernels (HLL with 4 fields
// at order 2 and with 5 at order 5, the tangent with 5 fields at orders 4 and 5)
// found sound states below it and ran at half their rate.
template <int MF> struct EulerFast64 {
  static constexpr int IE = MF - 1;
  static constexpr int LO = kWordLo, HI = kWordHi;
  struct Side {
    double rho, ir, vx, vy, vz, v2, p;
    bool clean;
  };
  __device__ __forceinline__ static bool within(double v, int lo) {
    return (unsigned)(__double2hiint(v) - lo) < (unsigned)(HI - lo);
  }
  __device__ __forceinline__ static Side side(const EqParams& P, const double* q) {
    const double g1 = P.p[0] - 1.0;
    Side s;
    s.rho = q[0];
    s.ir = recip_normal(s.rho);
    s.vx = q[1] * s.ir;
    s.vy = q[2] * s.ir;
    s.vz = MF == 5 ? q[3] * s.ir : 0.0;
    // 1e-300 keeps the speed's square root off zero and, with p / rho above
    // 2^-800, changes no other sum
    s.v2 = fma(s.vx, s.vx, fma(s.vy, s.vy, MF == 5 ? fma(s.vz, s.vz, 1e-300) : 1e-300));
    s.p = g1 * fma(-0.5 * s.rho, s.v2, q[IE]);
    s.clean = within(s.rho, P.rho_lo) && within(s.p, LO);
    return s;
  }
  // whether the equation's own code may run on Quick: a density between 2^-200 and
  // 2^200, momenta and energy below 2^250 (squared speeds then stay finite), floors
  // to match (quick_floors, on the host)
  __device__ __forceinline__ static bool quick_ok(const EqParams& P, const double* q) {
    int top = 0;
#pragma unroll
    for (int f = 1; f < MF; ++f) top = max(top, __double2hiint(q[f]) & 0x7fffffff);
    return P.quick && (unsigned)(__double2hiint(q[0]) - 0x33700000) < 0x19000000u && top < 0x4f900000;
  }
  // the flux along (ax, ay): ax F + ay G
  __device__ __forceinline__ static void along(const Side& s, const double* q, double ax, double ay, double* R) {
    const double ua = s.vx * ax + s.vy * ay;
    R[0] = s.rho * ua;
    R[1] = fma(q[1], ua, s.p * ax);
    R[2] = fma(q[2], ua, s.p * ay);
    if (MF == 5) R[3] = q[3] * ua;
    R[IE] = (q[IE] + s.p) * ua;
  }
  // twice the Lax-Friedrichs flux of two clean states times w (nxw, nyw: the
  // normal times w); returns its speed
  __device__ __forceinline__ static double lf2(const EqParams& P, const Side& a, const Side& b, const double* qM,
                                               const double* qP, double nxw, double nyw, double w, double* nf) {
    double FM[MF], FP[MF];
    along(a, qM, nxw, nyw, FM);
    along(b, qP, nxw, nyw, FP);
    const double cM = speed(P, a), cP = speed(P, b);
    const double lam = cM > cP ? cM : cP, wl = w * lam;
#pragma unroll
    for (int c = 0; c < MF; ++c) nf[c] = fma(wl, qM[c] - qP[c], FM[c] + FP[c]);
    return lam;
  }
  // twice Apollo's HLL flux of two clean states times w (wxeulereqn.cc:1121-1202:
  // in the face's normal-tangent frame, |S_R| truncated, no z-momentum flux);
  // false where the averaged sound speed leaves the checked range
  __device__ __forceinline__ static bool hll2(const EqParams& P, const Side& a, const Side& b, const double* qM,
                                              const double* qP, double nx, double ny, double w, double* nf,
                                              double* lam) {
    const double gamma = P.p[0];
    const double ua = nx * a.vx + ny * a.vy, ub = nx * b.vx + ny * b.vy;
    const double ta = nx * a.vy - ny * a.vx, tb = nx * b.vy - ny * b.vx;
    const double ca = sqrt_normal(gamma * a.p * a.ir), cb = sqrt_normal(gamma * b.p * b.ir);
    const double ra = sqrt_normal(a.rho), rb = sqrt_normal(b.rho), ri = recip_normal(ra + rb);
    const double ea = qM[IE] + a.p, eb = qP[IE] + b.p;
    const double u = (ra * ua + rb * ub) * ri, t = (ra * ta + rb * tb) * ri;
    const double z = MF == 5 ? (ra * a.vz + rb * b.vz) * ri : 0.0;
    const double H = (ra * (ea * a.ir) + rb * (eb * b.ir)) * ri;
    const double c2 = (gamma - 1.0) * (H - 0.5 * (u * u + t * t + z * z));
    if (!within(c2, LO)) return false;
    const double c = sqrt_normal(c2);
    const double SL = fmin(ua - ca, u - c), SR = fmax(ub + cb, u + c);
    const double D = (2.0 * w) * recip_normal(SR - SL);
    const double t1 = (fmin(SR, 0.0) - fmin(SL, 0.0)) * D, t2 = 2.0 * w - t1;
    const double t3 = 0.5 * (SR * fabs(SL) - SL * abs_int(SR)) * D;
    const double na = nx * qM[1] + ny * qM[2], nb = nx * qP[1] + ny * qP[2];
    const double sa = nx * qM[2] - ny * qM[1], sb = nx * qP[2] - ny * qP[1];
    nf[0] = t1 * nb + t2 * na - t3 * (qP[0] - qM[0]);
    const double f1 = t1 * fma(nb, ub, b.p) + t2 * fma(na, ua, a.p) - t3 * (nb - na);
    const double f2 = t1 * (sb * ub) + t2 * (sa * ua) - t3 * (sb - sa);
    nf[1] = nx * f1 - ny * f2;
    nf[2] = ny * f1 + nx * f2;
    if (MF == 5) nf[3] = 0.0;
    nf[IE] = t1 * (eb * ub) + t2 * (ea * ua) - t3 * (qP[IE] - qM[IE]);
    const double la = sqrt_normal(a.v2) + ca, lb = sqrt_normal(b.v2) + cb;
    *lam = la > lb ? la : lb;
    return true;
  }
  // twice Apollo's Roe flux of two clean states times w (wxeulereqn.cc:1206-1275:
  // the first momentum component assigned twice, no second and no z one); false
  // as for hll2
  __device__ __forceinline__ static bool roe2(const EqParams& P, const Side& a, const Side& b, const double* qM,
                                              const double* qP, double nx, double ny, double w, double* nf,
                                              double* lam) {
    const double gamma = P.p[0];
    const double ua = nx * a.vx + ny * a.vy, ub = nx * b.vx + ny * b.vy;
    const double ta = nx * a.vy - ny * a.vx, tb = nx * b.vy - ny * b.vx;
    const double ra = sqrt_normal(a.rho), rb = sqrt_normal(b.rho), ri = recip_normal(ra + rb);
    const double ea = qM[IE] + a.p, eb = qP[IE] + b.p;
    const double u = (ra * ua + rb * ub) * ri, t = (ra * ta + rb * tb) * ri;
    const double z = MF == 5 ? (ra * a.vz + rb * b.vz) * ri : 0.0;
    const double H = (ra * (ea * a.ir) + rb * (eb * b.ir)) * ri;
    const double c2 = (gamma - 1.0) * (H - 0.5 * (u * u + t * t + z * z));
    if (!within(c2, LO)) return false;
    const double ic = rsqrt_normal(c2), c = c2 * ic, rho = ra * rb;
    const double du = 0.5 * rho * (ub - ua) * ic, dp = 0.5 * (b.p - a.p) * (ic * ic);
    const double w1 = fabs(u - c) * (dp - du), w2 = fabs(u) * ((b.rho - a.rho) - 2.0 * dp);
    const double w3 = fabs(u) * (rho * (tb - ta)), w4 = fabs(u + c) * (dp + du), ws = w1 + w2 + w4;
    const double na = nx * qM[1] + ny * qM[2], nb = nx * qP[1] + ny * qP[2];
    const double sa = nx * qM[2] - ny * qM[1], sb = nx * qP[2] - ny * qP[1];
    const double f1 = (fma(na, ua, a.p) + fma(nb, ub, b.p)) - (w1 * (u - c) + w2 * u + w4 * (u + c));
    const double f2 = (sa * ua + sb * ub) - (ws * t + w3);
    nf[0] = w * ((na + nb) - ws);
    nf[1] = w * (ny * f1 + nx * f2);
    nf[2] = 0.0;
    if (MF == 5) nf[3] = 0.0;
    nf[IE] = w * ((ea * ua + eb * ub) -
                  (w1 * (H - u * c) + w2 * (0.5 * (u * u + t * t)) + w3 * t + w4 * (H + u * c)));
    const double la = speed(P, a), lb = speed(P, b);
    *lam = la > lb ? la : lb;
    return true;
  }
  // twice what remains of Apollo's Wave flux (wxeulereqn.cc:888-892, :1279-1322)
  // of two clean states times w: Lax-Friedrichs of the rotated traces with the
  // unrotated normal; its checks and its pressure floor do not touch states that
  // pass wave_ok
  __device__ __forceinline__ static bool wave_ok(const EqParams& P, const Side& s, const double* q) {
    // a pressure 2^40 below the energy is rounding, and so are the checks on it
    return s.p >= P.p[1] && __double2hiint(q[IE]) - __double2hiint(s.p) < (40 << 20);
  }
  __device__ __forceinline__ static double wave2(const EqParams& P, Side a, Side b, const double* qM, const double* qP,
                                                 double nx, double ny, double w, double* nf) {
    double rM[MF], rP[MF];
    rotate(a, qM, nx, ny, rM);
    rotate(b, qP, nx, ny, rP);
    return lf2(P, a, b, rM, rP, w * nx, w * ny, w, nf);
  }
  __device__ __forceinline__ static void rotate(Side& s, const double* q, double nx, double ny, double* r) {
#pragma unroll
    for (int f = 0; f < MF; ++f) r[f] = q[f];
    r[1] = nx * q[1] + ny * q[2];
    r[2] = nx * q[2] - ny * q[1];
    const double u = nx * s.vx + ny * s.vy;
    s.vy = nx * s.vy - ny * s.vx;
    s.vx = u;
  }
  // qb = (d (aR . R + aS . S) / d q)^T of the fluxes R along (rx, ry), S along
  // (sx, sy): with cF = rx aR + sx aS, cG = ry aR + sy aS the reverse sweep of
  // cF . F + cG . G, F = (m1, m1 vx + p, m1 vy, (E + p) vx) and so on
  __device__ __forceinline__ static void vol_t(const EqParams& P, const Side& s, const double* q, double rx, double ry,
                                               double sx, double sy, const double* aR, const double* aS, double* qb) {
    const double g1 = P.p[0] - 1.0;
    double cF[MF], cG[MF];
#pragma unroll
    for (int f = 0; f < MF; ++f) {
      cF[f] = rx * aR[f] + sx * aS[f];
      cG[f] = ry * aR[f] + sy * aS[f];
    }
    const double Hp = q[IE] + s.p;
    const double eb = cF[IE] * s.vx + cG[IE] * s.vy, pb = g1 * (cF[1] + cG[2] + eb);
    const double xb = cF[1] * q[1] + cG[1] * q[2] + cF[IE] * Hp, yb = cF[2] * q[1] + cG[2] * q[2] + cG[IE] * Hp;
    double zb = 0.0;
    if (MF == 5) zb = cF[3] * q[1] + cG[3] * q[2];
    qb[0] = fma(0.5 * pb, s.v2, -(xb * s.vx + yb * s.vy + zb * s.vz) * s.ir);
    qb[1] = cF[0] + cF[1] * s.vx + cF[2] * s.vy + (MF == 5 ? cF[3] * s.vz : 0.0) + xb * s.ir - pb * s.vx;
    qb[2] = cG[0] + cG[1] * s.vx + cG[2] * s.vy + (MF == 5 ? cG[3] * s.vz : 0.0) + yb * s.ir - pb * s.vy;
    if (MF == 5) qb[3] = zb * s.ir - pb * s.vz;
    qb[IE] = eb + pb;
  }
  // qb = (d (n . F) / d q)^T r
  __device__ __forceinline__ static void along_t(const EqParams& P, const Side& s, const double* q, double nx,
                                                 double ny, const double* r, double* qb) {
    const double g1 = P.p[0] - 1.0, un = s.vx * nx + s.vy * ny;
    const double ub = (r[1] * q[1] + r[2] * q[2] + (MF == 5 ? r[3] * q[3] : 0.0) + r[IE] * (q[IE] + s.p)) * s.ir;
    const double pb = g1 * (r[1] * nx + r[2] * ny + r[IE] * un), t = r[0] + ub;
    qb[0] = fma(0.5 * pb, s.v2, -ub * un);
    qb[1] = r[1] * un + t * nx - pb * s.vx;
    qb[2] = r[2] * un + t * ny - pb * s.vy;
    if (MF == 5) qb[3] = r[3] * un - pb * s.vz;
    qb[IE] = r[IE] * un + pb;
  }
  // flow speed + sound speed, and with the reciprocals of both the gradient
  struct Speed {
    double c, cs, rv, rc;  // sum, sound speed, 1 / flow speed, 1 / sound speed
  };
  __device__ __forceinline__ static Speed speeds(const EqParams& P, const Side& s) {
    Speed r;
    const double c2 = P.p[0] * s.p * s.ir;
    r.rv = rsqrt_normal(s.v2);
    r.rc = rsqrt_normal(c2);
    r.cs = c2 * r.rc;
    r.c = s.v2 * r.rv + r.cs;
    return r;
  }
  // g += w grad c
  __device__ __forceinline__ static void add_speed_grad(const EqParams& P, const Side& s, const Speed& v, double w,
                                                        double* g) {
    const double g1 = P.p[0] - 1.0;
    const double kc = 0.5 * P.p[0] * s.ir * v.rc * g1, k = w * (v.rv * s.ir - kc);
    g[0] += w * (0.5 * kc * s.v2 - (s.v2 * v.rv + 0.5 * v.cs) * s.ir);
    g[1] += k * s.vx;
    g[2] += k * s.vy;
    if (MF == 5) g[3] += k * s.vz;
    g[IE] += w * kc;
  }
  // (d f*/d a)^T dv and, with want_b, (d f*/d b)^T dv of twice the
  // Lax-Friedrichs flux f* = Fn(a) + Fn(b) + max(c(a), c(b)) (a - b)
  __device__ __forceinline__ static void lf2_t(const EqParams& P, const Side& a, const Side& b, const double* qM,
                                               const double* qP, double nx, double ny, const double* dv, bool want_b,
                                               double* ab, double* bb) {
    const Speed ca = speeds(P, a), cb = speeds(P, b);
    const bool a_wins = ca.c > cb.c;  // the branch the forward flux takes
    const double lam = a_wins ? ca.c : cb.c;
    double jump = 0.0;
#pragma unroll
    for (int f = 0; f < MF; ++f) jump += dv[f] * (qM[f] - qP[f]);
    along_t(P, a, qM, nx, ny, dv, ab);
#pragma unroll
    for (int f = 0; f < MF; ++f) ab[f] += lam * dv[f];
    if (a_wins) add_speed_grad(P, a, ca, jump, ab);
    if (want_b) {
      along_t(P, b, qP, nx, ny, dv, bb);
#pragma unroll
      for (int f = 0; f < MF; ++f) bb[f] -= lam * dv[f];
      if (!a_wins) add_speed_grad(P, b, cb, jump, bb);
    }
  }
  // derivatives along dq: of velocity and pressure, of the flux along (ax, ay),
  // of the speed
  struct Rate {
    double vx, vy, vz, p;
  };
  __device__ __forceinline__ static Rate rate(const EqParams& P, const Side& s, const double* dq) {
    const double g1 = P.p[0] - 1.0;
    Rate r;
    r.vx = (dq[1] - s.vx * dq[0]) * s.ir;
    r.vy = (dq[2] - s.vy * dq[0]) * s.ir;
    r.vz = MF == 5 ? (dq[3] - s.vz * dq[0]) * s.ir : 0.0;
    double m = s.vx * dq[1] + s.vy * dq[2];
    if (MF == 5) m += s.vz * dq[3];
    r.p = g1 * (dq[IE] - m + 0.5 * s.v2 * dq[0]);
    return r;
  }
  __device__ __forceinline__ static void along_d(const Side& s, const Rate& r, const double* q, const double* dq,
                                                 double ax, double ay, double* R) {
    const double un = s.vx * ax + s.vy * ay, du = r.vx * ax + r.vy * ay;
    R[0] = dq[0] * un + s.rho * du;
    R[1] = dq[1] * un + q[1] * du + r.p * ax;
    R[2] = dq[2] * un + q[2] * du + r.p * ay;
    if (MF == 5) R[3] = dq[3] * un + q[3] * du;
    R[IE] = (dq[IE] + r.p) * un + (q[IE] + s.p) * du;
  }
  __device__ __forceinline__ static double speed_d(const EqParams& P, const Side& s, const Rate& r, const Speed& v,
                                                   double drho) {
    const double dv2 = s.vx * r.vx + s.vy * r.vy + (MF == 5 ? s.vz * r.vz : 0.0);
    // cs^2 = gamma p / rho
    return dv2 * v.rv + 0.5 * (P.p[0] * r.p * v.rc - v.cs * drho) * s.ir;
  }
  // derivative of twice the Lax-Friedrichs flux, times w
  __device__ __forceinline__ static void lf2_d(const EqParams& P, const Side& a, const Side& b, const double* qM,
                                               const double* qP, const double* dM, const double* dP, double nxw,
                                               double nyw, double w, double* nf) {
    const Rate ra = rate(P, a, dM), rb = rate(P, b, dP);
    const Speed ca = speeds(P, a), cb = speeds(P, b);
    const bool a_wins = ca.c > cb.c;
    const double lam = w * (a_wins ? ca.c : cb.c);
    const double dlam = w * (a_wins ? speed_d(P, a, ra, ca, dM[0]) : speed_d(P, b, rb, cb, dP[0]));
    double FM[MF], FP[MF];
    along_d(a, ra, qM, dM, nxw, nyw, FM);
    along_d(b, rb, qP, dP, nxw, nyw, FP);
#pragma unroll
    for (int c = 0; c < MF; ++c) nf[c] = fma(dlam, qM[c] - qP[c], fma(lam, dM[c] - dP[c], FM[c] + FP[c]));
  }
  // flow speed + sound speed
  __device__ __forceinline__ static double speed(const EqParams& P, const Side& s) {
    return sqrt_normal(s.v2) + sqrt_normal(P.p[0] * s.p * s.ir);
  }
};

template <int EQ> constexpr bool kEulerEq = EQ == EQ_EULER || EQ == EQ_EULER2D;

template <int EQ> constexpr bool kLinearEq = EQ == EQ_ADVECTION || EQ == EQ_MAXWELL || EQ == EQ_MAXWELL_TM;

// The linear equations' flux along (ax, ay), ax F + ay G, written out, and
// their numerical flux as the flux of the sum of the two traces plus the
// dissipation of their difference (wxadvectioneqn.cc:176-208,
// wxphmaxwelleqn.cc:450-522; the upwind extensions as in dg_physics.cuh): the
// plugins' values to round-off.
template <int EQ> struct LinearFast64 {
  static constexpr int M = Eq<EQ>::M;
  __device__ __forceinline__ static void along(const EqParams& P, const double* q, double ax, double ay, double* R) {
    if constexpr (EQ == EQ_ADVECTION) {
      R[0] = (ax * P.p[0] + ay * P.p[1]) * q[0];
    } else {
      const double c2 = P.p[0] * P.p[0];
      if constexpr (EQ == EQ_MAXWELL_TM) {
        R[0] = c2 * (ay * q[1] - ax * q[2]);
        R[1] = ay * q[0];
        R[2] = -ax * q[0];
      } else {
        const double gm = P.p[1], chi = P.p[2], cp = chi * q[6], gp = gm * q[7];
        R[0] = c2 * (ax * cp - ay * q[5]);
        R[1] = c2 * (ax * q[5] + ay * cp);
        R[2] = c2 * (ay * q[3] - ax * q[4]);
        R[3] = ax * gp + ay * q[2];
        R[4] = ay * gp - ax * q[2];
        R[5] = ax * q[1] - ay * q[0];
        R[6] = chi * (ax * q[0] + ay * q[1]);
        R[7] = gm * c2 * (ax * q[3] + ay * q[4]);
      }
    }
  }
  // qb = (d along / d q)^T r
  __device__ __forceinline__ static void along_t(const EqParams& P, const double* r, double ax, double ay,
                                                 double* qb) {
    if constexpr (EQ == EQ_ADVECTION) {
      qb[0] = (ax * P.p[0] + ay * P.p[1]) * r[0];
    } else {
      const double c2 = P.p[0] * P.p[0];
      if constexpr (EQ == EQ_MAXWELL_TM) {
        qb[0] = ay * r[1] - ax * r[2];
        qb[1] = c2 * ay * r[0];
        qb[2] = -c2 * ax * r[0];
      } else {
        const double gm = P.p[1], chi = P.p[2], c6 = chi * r[6], c7 = gm * c2 * r[7];
        qb[0] = ax * c6 - ay * r[5];
        qb[1] = ax * r[5] + ay * c6;
        qb[2] = ay * r[3] - ax * r[4];
        qb[3] = c2 * ay * r[2] + ax * c7;
        qb[4] = ay * c7 - c2 * ax * r[2];
        qb[5] = c2 * (ax * r[1] - ay * r[0]);
        qb[6] = chi * c2 * (ax * r[0] + ay * r[1]);
        qb[7] = gm * (ax * r[3] + ay * r[4]);
      }
    }
  }
  // dissipation of a jump, as face2 applies it (symmetric)
  __device__ __forceinline__ static void dissipate(const EqParams& P, double nx, double ny, const double* dq,
                                                   double* out) {
    if constexpr (EQ == EQ_ADVECTION) {
      const double lam = dmax2(fabs(P.p[0]), fabs(P.p[1]));
      out[0] = ((int)P.p[3] == NF_UPWIND ? fabs(nx * P.p[0] + ny * P.p[1]) : lam) * dq[0];
    } else {
      const double lam = EQ == EQ_MAXWELL_TM ? P.p[0] : dmax3(P.p[2] * P.p[0], P.p[1] * P.p[0], P.p[0]);
#pragma unroll
      for (int f = 0; f < M; ++f) out[f] = lam * dq[f];
      if (EQ == EQ_MAXWELL_TM && (int)P.p[3] == NF_UPWIND) {
        const double bn = lam * (nx * dq[1] + ny * dq[2]);
        out[1] -= bn * nx;
        out[2] -= bn * ny;
      }
    }
  }
  // twice the numerical flux times w; returns its speed
  __device__ __forceinline__ static double face2(const EqParams& P, double nx, double ny, double w, const double* qM,
                                                 const double* qP, double* nf) {
    double s[M], dq[M];
#pragma unroll
    for (int f = 0; f < M; ++f) {
      s[f] = qM[f] + qP[f];
      dq[f] = qM[f] - qP[f];
    }
    along(P, s, w * nx, w * ny, nf);
    double lam;
    if constexpr (EQ == EQ_ADVECTION) {
      lam = dmax2(fabs(P.p[0]), fabs(P.p[1]));
      const double diss = (int)P.p[3] == NF_UPWIND ? fabs(nx * P.p[0] + ny * P.p[1]) : lam;
      nf[0] = fma(w * diss, dq[0], nf[0]);
    } else {
      lam = EQ == EQ_MAXWELL_TM ? P.p[0] : dmax3(P.p[2] * P.p[0], P.p[1] * P.p[0], P.p[0]);
      const double wl = w * lam;
      if (EQ == EQ_MAXWELL_TM && (int)P.p[3] == NF_UPWIND) {
        const double bn = nx * dq[1] + ny * dq[2];
        dq[1] -= bn * nx;
        dq[2] -= bn * ny;
      }
#pragma unroll
      for (int f = 0; f < M; ++f) nf[f] = fma(wl, dq[f], nf[f]);
    }
    return lam;
  }
};

// R = rx F + ry G, S = sx F + sy G of one state
template <int EQ>
__device__ __forceinline__ void volume_flux(const EqParams& P, const double* q, double rx, double ry, double sx,
                                            double sy, double* R, double* S, int* err) {
  constexpr int M = Eq<EQ>::M;
  if constexpr (kEulerEq<EQ>) {
    using X = EulerFast64<M>;
    const typename X::Side sd = X::side(P, q);
    if (sd.clean) {
      X::along(sd, q, rx, ry, R);
      X::along(sd, q, sx, sy, S);
      return;
    }
    if (X::quick_ok(P, q)) {
      Quick a[M], F[M], G[M];
#pragma unroll
      for (int f = 0; f < M; ++f) a[f] = q[f];
      Eq<EQ>::flux2(P, a, F, G, err);
#pragma unroll
      for (int f = 0; f < M; ++f) {
        R[f] = rx * F[f].v + ry * G[f].v;
        S[f] = sx * F[f].v + sy * G[f].v;
      }
      return;
    }
  }
  double F[M], G[M];
  Eq<EQ>::flux2(P, q, F, G, err);
#pragma unroll
  for (int f = 0; f < M; ++f) {
    R[f] = rx * F[f] + ry * G[f];
    S[f] = sx * F[f] + sy * G[f];
  }
}

// The same for two points: one branch for both, so that the two chains of
// dependent operations run side by side
template <int EQ>
__device__ __forceinline__ void volume_flux_pair(const EqParams& P, const double (*q)[Eq<EQ>::M], double rx, double ry,
                                                 double sx, double sy, double (*R)[Eq<EQ>::M], double (*S)[Eq<EQ>::M],
                                                 int* err) {
  if constexpr (kEulerEq<EQ>) {
    using X = EulerFast64<Eq<EQ>::M>;
    const typename X::Side a = X::side(P, q[0]), b = X::side(P, q[1]);
    if (a.clean && b.clean) {
      X::along(a, q[0], rx, ry, R[0]);
      X::along(b, q[1], rx, ry, R[1]);
      X::along(a, q[0], sx, sy, S[0]);
      X::along(b, q[1], sx, sy, S[1]);
      return;
    }
  }
#pragma unroll
  for (int j = 0; j < 2; ++j) volume_flux<EQ>(P, q[j], rx, ry, sx, sy, R[j], S[j], err);
}

// Twice the numerical flux of one face point (qM, qP may be modified as the
// reference modifies them) times w, by the equation's own code but for
// Lax-Friedrichs of two clean states.  KIND: the numerical flux, or kAnyFlux.
constexpr int kAnyFlux = -1;
template <int EQ, int KIND>
__device__ __forceinline__ double face_flux2(const EqParams& P, double nx, double ny, double w, double* qM, double* qP,
                                             double* nf, int* err) {
  constexpr int M = Eq<EQ>::M;
  double lam;
  if constexpr (kEulerEq<EQ> && KIND != kAnyFlux) {
    if (EulerFast64<M>::quick_ok(P, qM) && EulerFast64<M>::quick_ok(P, qP)) {
      Quick a[M], b[M], r[M], l;
#pragma unroll
      for (int f = 0; f < M; ++f) {
        a[f] = qM[f];
        b[f] = qP[f];
      }
      if constexpr (KIND == NF_HLL) {
        l = Eq<EQ>::hll(P, Quick(nx), Quick(ny), a, b, r, err);
      } else if constexpr (KIND == NF_ROE) {
        l = Eq<EQ>::roe(P, Quick(nx), Quick(ny), a, b, r, err);
      } else {
        if constexpr (KIND == NF_WAVE) Eq<EQ>::wave_prelude(P, Quick(nx), Quick(ny), a, b, err);
        l = Eq<EQ>::lf(P, Quick(nx), Quick(ny), a, b, r, err);
      }
#pragma unroll
      for (int c = 0; c < M; ++c) nf[c] = r[c].v * (2.0 * w);
      return l.v;
    }
    if constexpr (KIND == NF_HLL) {
      lam = Eq<EQ>::hll(P, nx, ny, qM, qP, nf, err);
    } else if constexpr (KIND == NF_ROE) {
      lam = Eq<EQ>::roe(P, nx, ny, qM, qP, nf, err);
    } else {
      if constexpr (KIND == NF_WAVE) {
        Eq<EQ>::wave_prelude(P, nx, ny, qM, qP, err);
      } else {
        using X = EulerFast64<M>;
        const typename X::Side a = X::side(P, qM), b = X::side(P, qP);
        if (a.clean && b.clean) return X::lf2(P, a, b, qM, qP, w * nx, w * ny, w, nf);
      }
      lam = Eq<EQ>::lf(P, nx, ny, qM, qP, nf, err);
    }
  } else {
    lam = Eq<EQ>::numflux(P, nx, ny, qM, qP, nf, err);
  }
#pragma unroll
  for (int c = 0; c < M; ++c) nf[c] *= 2.0 * w;
  return lam;
}

// The same for two points of one face: one branch for both
template <int EQ, int KIND>
__device__ __forceinline__ void face_flux2_pair(const EqParams& P, double nx, double ny, double w,
                                                double (*qM)[Eq<EQ>::M], double (*qP)[Eq<EQ>::M],
                                                double (*nf)[Eq<EQ>::M], double* lam, int* err) {
  if constexpr (kEulerEq<EQ>) {
    using X = EulerFast64<Eq<EQ>::M>;
    const typename X::Side a0 = X::side(P, qM[0]), b0 = X::side(P, qP[0]);
    const typename X::Side a1 = X::side(P, qM[1]), b1 = X::side(P, qP[1]);
    const bool clean = a0.clean && b0.clean && a1.clean && b1.clean;
    if constexpr (KIND == NF_HLL) {
      if (clean && (X::hll2(P, a0, b0, qM[0], qP[0], nx, ny, w, nf[0], &lam[0]) &
                    X::hll2(P, a1, b1, qM[1], qP[1], nx, ny, w, nf[1], &lam[1])))
        return;
    } else if constexpr (KIND == NF_ROE) {
      if (clean && (X::roe2(P, a0, b0, qM[0], qP[0], nx, ny, w, nf[0], &lam[0]) &
                    X::roe2(P, a1, b1, qM[1], qP[1], nx, ny, w, nf[1], &lam[1])))
        return;
    } else if constexpr (KIND == NF_WAVE) {
      if (clean && X::wave_ok(P, a0, qM[0]) && X::wave_ok(P, b0, qP[0]) && X::wave_ok(P, a1, qM[1]) &&
          X::wave_ok(P, b1, qP[1])) {
        lam[0] = X::wave2(P, a0, b0, qM[0], qP[0], nx, ny, w, nf[0]);
        lam[1] = X::wave2(P, a1, b1, qM[1], qP[1], nx, ny, w, nf[1]);
        return;
      }
    } else {
      if (clean) {
        const double nxw = w * nx, nyw = w * ny;
        lam[0] = X::lf2(P, a0, b0, qM[0], qP[0], nxw, nyw, w, nf[0]);
        lam[1] = X::lf2(P, a1, b1, qM[1], qP[1], nxw, nyw, w, nf[1]);
        return;
      }
    }
  }
#pragma unroll
  for (int j = 0; j < 2; ++j) lam[j] = face_flux2<EQ, KIND>(P, nx, ny, w, qM[j], qP[j], nf[j], err);
}

// The source plugins at one point (Apollo adds each into its output field,
// WxHyperbolicSrc::compSource, src/hyper/wxhyperbolicsrc.cc:64-80).
template <int M>
__device__ __forceinline__ void source_terms(const SrcTable& T, double t, double x, double y, double* s) {
  for (int i = 0; i < T.n; ++i) {
    const double* p = T.p[i];
    double v = 0.0;
    if (T.kind[i] == SRC_TM) {
      v = exp(t) * (x * (1 - x) * y * (1 - y) + 2. * x * (1 - x) + 2 * y * (1 - y));
    } else if (T.kind[i] == SRC_POINT) {
      const double qbyme = p[6] / (p[7] * p[8]);
      if (sqrt((x - p[0]) * (x - p[0]) + (y - p[1]) * (y - p[1])) < p[2]) v = p[3] * qbyme * sin(p[4] * t + p[5]);
    }
#pragma unroll
    for (int f = 0; f < M; ++f)
      if (T.out[i] == f) s[f] += v;
  }
}

}  // namespace apollo
