// Pointwise float64 fluxes and sources of the float64 kernels.
#pragma once

#include <cuda_runtime.h>

#include "dg_device.cuh"

namespace apollo {

// Euler fluxes in float64 with one reciprocal of the density per state and
// the flux formed along a direction directly (a n.F + b n.G in one pass): the
// same quantities as WxEulerEqn's flux and Lax-Friedrichs flux
// (wxeulereqn.cc:809-871, :1097-1117) to round-off, for states that need none
// of the reference's clamps; a state that does (density below its floor or
// not positive, pressure not positive) takes the equation's own code, which
// applies them and raises its error flags.
template <int MF> struct EulerFast64 {
  static constexpr int IE = MF - 1;
  struct Side {
    double rho, ir, vx, vy, vz, p;
    bool clean;
  };
  __device__ __forceinline__ static Side side(const EqParams& P, const double* q) {
    const double g1 = P.p[0] - 1.0, minD = P.p[2];
    Side s;
    s.rho = q[0];
    s.ir = 1.0 / s.rho;
    s.vx = q[1] * s.ir;
    s.vy = q[2] * s.ir;
    s.vz = MF == 5 ? q[3] * s.ir : 0.0;
    s.p = g1 * (q[IE] - 0.5 * s.rho * (s.vx * s.vx + s.vy * s.vy + s.vz * s.vz));
    s.clean = s.rho > 0.0 && s.rho >= minD && s.p > 0.0;
    return s;
  }
  // the flux along (ax, ay): ax F + ay G
  __device__ __forceinline__ static void along(const Side& s, const double* q, double ax, double ay, double* R) {
    const double ua = s.vx * ax + s.vy * ay;
    R[0] = s.rho * ua;
    R[1] = s.rho * s.vx * ua + s.p * ax;
    R[2] = s.rho * s.vy * ua + s.p * ay;
    if (MF == 5) R[3] = s.rho * s.vz * ua;
    R[IE] = (q[IE] + s.p) * ua;
  }
};

template <int EQ> constexpr bool kEulerEq = EQ == EQ_EULER || EQ == EQ_EULER2D;

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
  }
  double F[M], G[M];
  Eq<EQ>::flux2(P, q, F, G, err);
#pragma unroll
  for (int f = 0; f < M; ++f) {
    R[f] = rx * F[f] + ry * G[f];
    S[f] = sx * F[f] + sy * G[f];
  }
}

// The numerical flux of one face point (qM, qP may be modified as the
// reference modifies them); the Euler Lax-Friedrichs flux of two clean states
// through EulerFast64
template <int EQ>
__device__ __forceinline__ double face_flux(const EqParams& P, double nx, double ny, double* qM, double* qP,
                                            double* nf, int* err) {
  constexpr int M = Eq<EQ>::M;
  if constexpr (kEulerEq<EQ>) {
    const int kind = (int)P.p[3];
    if (kind != NF_HLL && kind != NF_ROE && kind != NF_WAVE) {
      using X = EulerFast64<M>;
      const typename X::Side a = X::side(P, qM), b = X::side(P, qP);
      if (a.clean && b.clean) {
        double FM[M], FP[M];
        X::along(a, qM, nx, ny, FM);
        X::along(b, qP, nx, ny, FP);
        const double gamma = P.p[0];
        const double cM = sqrt(a.vx * a.vx + a.vy * a.vy + a.vz * a.vz) + sqrt(gamma * a.p * a.ir);
        const double cP = sqrt(b.vx * b.vx + b.vy * b.vy + b.vz * b.vz) + sqrt(gamma * b.p * b.ir);
        const double lam = cM > cP ? cM : cP;
#pragma unroll
        for (int c = 0; c < M; ++c) nf[c] = 0.5 * (FM[c] + FP[c] + lam * (qM[c] - qP[c]));
        return lam;
      }
    }
  }
  return Eq<EQ>::numflux(P, nx, ny, qM, qP, nf, err);
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
