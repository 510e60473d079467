// Reverse sweeps of the Euler fluxes with the reference's clamps, all inline
// (no calls, so a kernel's stack size is static).
#pragma once

#include <cuda_runtime.h>

#include "dg_device.cuh"

namespace apollo {

template <int MF> struct EulerAdj {
  static constexpr int IE = MF - 1;
  // qbar += (dR/dq)^T r for the flux R along (ax, ay): reverse sweep of the
  // flux's own graph with its clamps (rho = max(q0, minD) as a constant when
  // clamped; p = minP as a constant when clamped),
  // rho, v = m / rho, p = g1 (E - rho |v|^2 / 2), u = v . a,
  // R = (rho u, rho vx u + p ax, rho vy u + p ay, [rho vz u], (E + p) u)
  __device__ __forceinline__ static void dir(const EqParams& P, const double* q, double ax, double ay,
                                             const double* r, double* qbar, int* err) {
    const double g1 = P.p[0] - 1.0, minP = P.p[1], minD = P.p[2];
    double rho = q[0];
    if (minD == 0.0 && rho <= 0.0) *err |= ERRB_NONPHYS;
    const bool rho_c = rho < minD;
    if (rho_c) rho = minD;
    const double ir = 1.0 / rho;
    const double vx = q[1] * ir, vy = q[2] * ir, vz = MF == 5 ? q[3] * ir : 0.0, E = q[IE];
    const double v2 = vx * vx + vy * vy + vz * vz;
    double p = g1 * (E - 0.5 * rho * v2);
    bool p_c = false;
    if (p <= 0.0) {
      if (minP == 0.0) *err |= ERRB_NONPHYS;
      else { p = minP; p_c = true; }
    }
    const double u = vx * ax + vy * ay;
    const double r3 = MF == 5 ? r[3] : 0.0;
    const double ub = r[0] * rho + r[1] * rho * vx + r[2] * rho * vy + r3 * rho * vz + r[IE] * (E + p);
    const double pb = p_c ? 0.0 : r[1] * ax + r[2] * ay + r[IE] * u;
    double rhob = (r[0] + r[1] * vx + r[2] * vy + r3 * vz) * u - 0.5 * g1 * v2 * pb;
    const double vxb = r[1] * rho * u + ub * ax - g1 * rho * vx * pb;
    const double vyb = r[2] * rho * u + ub * ay - g1 * rho * vy * pb;
    const double vzb = r3 * rho * u - g1 * rho * vz * pb;
    rhob -= (vxb * vx + vyb * vy + vzb * vz) * ir;
    if (!rho_c) qbar[0] += rhob;
    qbar[1] += vxb * ir;
    qbar[2] += vyb * ir;
    if (MF == 5) qbar[3] += vzb * ir;
    qbar[IE] += r[IE] * u + g1 * pb;
  }
  // Lax-Friedrichs wave speed of the primitive variables and its gradient.
  // Where the primitive variables clamp (non-physical states) the gradient is
  // taken as zero and NONPHYS is flagged.
  __device__ __forceinline__ static double speed(const EqParams& P, const double* q, double* grad, int* err) {
    const double gamma = P.p[0], g1 = gamma - 1.0, minP = P.p[1], minD = P.p[2];
    const double q3 = MF == 5 ? q[3] : 0.0;
    if (!(q[0] > 0.0)) {
      *err |= ERRB_NONPHYS;
#pragma unroll
      for (int j = 0; j < MF; ++j) grad[j] = 0.0;
      return sqrt(gamma * minP / minD);
    }
    const double rho = q[0], ir = 1.0 / rho;
    const double u = q[1] / rho, v = q[2] / rho, w = q3 / rho;
    double p = g1 * (q[IE] - 0.5 * (q[1] * q[1] + q[2] * q[2] + q3 * q3) / q[0]);
    const double sp = sqrt(u * u + v * v + w * w);
    if (p <= 0.0) {
      *err |= ERRB_NONPHYS;
#pragma unroll
      for (int j = 0; j < MF; ++j) grad[j] = 0.0;
      return sp + sqrt(gamma * minP / rho);
    }
    const double cs = sqrt(gamma * p / rho);
    const double ks = sp > 0.0 ? ir / sp : 0.0;  // d|v|/dm = v / (|v| rho)
    const double kc = 0.5 * gamma / (cs * rho);   // dcs/dp = kc, dcs/drho = -kc p / rho
    grad[0] = -sp * ir + kc * (0.5 * g1 * (u * u + v * v + w * w) - p * ir);
    grad[1] = u * ks - kc * g1 * u;
    grad[2] = v * ks - kc * g1 * v;
    if (MF == 5) grad[3] = w * ks - kc * g1 * w;
    grad[IE] = kc * g1;
    return sp + cs;
  }
  // (d f/d a)^T dv and, with want_b, (d f/d b)^T dv of twice the
  // Lax-Friedrichs flux, f = Fn(a) + Fn(b) + lambda (a - b), lambda =
  // max(c(a), c(b))
  __device__ __forceinline__ static void lf2_t(const EqParams& P, double nx, double ny, const double* a,
                                               const double* b, const double* dv, double* abar, double* bbar,
                                               bool want_b, int* err) {
    double ga[MF], gb[MF];
    const double ca = speed(P, a, ga, err), cb = speed(P, b, gb, err);
    const bool a_wins = ca > cb;  // the branch the forward flux takes
    const double lam = a_wins ? ca : cb;
    double jump = 0.0;
#pragma unroll
    for (int f = 0; f < MF; ++f) jump += dv[f] * (a[f] - b[f]);
#pragma unroll
    for (int j = 0; j < MF; ++j) abar[j] = lam * dv[j] + (a_wins ? jump * ga[j] : 0.0);
    dir(P, a, nx, ny, dv, abar, err);
    if (want_b) {
#pragma unroll
      for (int j = 0; j < MF; ++j) bbar[j] = (a_wins ? 0.0 : jump * gb[j]) - lam * dv[j];
      dir(P, b, nx, ny, dv, bbar, err);
    }
  }
};

}  // namespace apollo
