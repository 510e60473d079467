// Apollo's slope limiters "eulerLimiterHW" and "tuAliabadiLimiter"
// (WxHestavenWarburtonEulerLimiter::applyLimiter,
// src/hyperapps/euler/wxhesthavenwarburtoneulerlimiter.cc:44-330), float64, in
// two passes:
//   pass 1: the element's four-element patch (centroids, areas), cell averages
//           of the conserved and primitive variables, averages of the face
//           traces at the patch's edge ends, and the primitive-variable
//           gradients of the three sub-triangles and of the element;
//   pass 2: gradients weighted from the neighbours' (or, on a boundary, the
//           element's own edge gradient), and the linear reconstruction of
//           the conserved variables with Apollo's density and pressure fixes.
// The arithmetic follows the reference line by line, including what it does
// that a textbook limiter would not: the patch "centroid" weights the vertex
// coordinates with the averaging weights of nodes 0..2, the third edge's
// gradient uses the second edge's vertex differences, and the face averages
// are read at positions given by element node ids.
//
// tuAliabadiLimiter (WxTuAliabadiLimiter::applyLimiter,
// src/hyperapps/multifluid/aptualiabadilimiter.cc:75-410) runs the same patch
// procedure through the equation set: for Euler the primitive variables come
// from the equation (with its density and pressure floors, which rewrite the
// averages they are given) and the equation's gas_gamma, minPressure and
// minDensity drive the reconstruction; for phMaxwellEqn the reconstruction
// returns the cell averages, so every node takes its element's average.
#include "dg_device.cuh"

namespace apollo {
namespace {

template <int M>
__device__ __forceinline__ void lim_prim(double gamma, const double* c, double* p) {
  // the limiter's primitiveVariables (no floors), 5-field order with rho w = 0 for 4 fields
  const double c3 = M == 5 ? c[3] : 0.0;
  p[0] = c[0];
  p[1] = c[1] / c[0];
  p[2] = c[2] / c[0];
  p[3] = c3 / c[0];
  p[4] = (gamma - 1.) * (c[M - 1] - 0.5 * (c[1] * c[1] + c[2] * c[2] + c3 * c3) / c[0]);
}

// The equation's primitive variables as Apollo's tuAliabadiLimiter obtains
// them (WxEulerEqn::primitiveVariables, src/hyperapps/euler/wxeulereqn.cc:1326-1341):
// density and pressure floors, which also rewrite the conserved values given.
__device__ __forceinline__ void ta_prim(double gamma, double minP, double minD, double* c, double* p) {
  p[0] = c[0];
  if (p[0] <= 0.) {
    c[0] = minD;
    p[0] = minD;
  }
  p[1] = c[1] / c[0];
  p[2] = c[2] / c[0];
  p[3] = c[3] / c[0];
  p[4] = (gamma - 1.) * (c[4] - 0.5 * (c[1] * c[1] + c[2] * c[2] + c[3] * c[3]) / c[0]);
  if (p[4] <= 0.) {
    p[4] = minP;
    c[4] = minP / (gamma - 1.) + 0.5 * p[0] * (p[1] * p[1] + p[2] * p[2] + p[3] * p[3]);
  }
}

// per element: E1x E1y E2x E2y E3x E3y C0x C0y (5 each), cons average, prim average
constexpr int kLimStride = 10 * 5;

// Both passes work on kLimE elements per block, the independent pieces of an
// element (patch members, edge ends, variables, nodes) on threads of their own:
// one thread per element left most of the GPU idle on the meshes in use
// (K = 8,192, N = 3: 23.8 and 12.0 us; so 11.4 and 7.5).
constexpr int kLimE = 16, kLimThreads = 128;

template <int EQ, int N>
__global__ void __launch_bounds__(kLimThreads) k_limiter_grad(DgDev d, LimArgs L, const double* __restrict__ x,
                                                              const double* __restrict__ xn,
                                                              const double* __restrict__ yn,
                                                              double* __restrict__ work) {
  constexpr int M = Eq<EQ>::M;
  constexpr int NP = Sizes<N>::NP, NPF = N + 1;
  __shared__ int sNb[kLimE][3], sNf[kLimE][3];
  // averages of the patch members as summed, and with their floors; primitive
  // variables; patch centroids and areas; edge-end averages
  __shared__ double sRaw[kLimE][4][5], sCons[kLimE][5], sPrim[kLimE][4][5], sXc[kLimE][4], sYc[kLimE][4], sA[kLimE][4],
      sFp[kLimE][6][5];
  const int e0 = blockIdx.x * kLimE, ne = min(kLimE, d.K - e0), tid = threadIdx.x;
  auto to5 = [&](const double* a, double* b) {
    b[0] = a[0]; b[1] = a[1]; b[2] = a[2]; b[3] = M == 5 ? a[3] : 0.0; b[4] = a[M - 1];
  };
  // eulerLimiterHW: the limiter's own primitive variables; tuAliabadiLimiter:
  // the equation's, whose floors rewrite the averages they are given
  const bool ta = L.kind == 1;
  auto prim_of = [&](double* c, double* p) {
    if (ta) ta_prim(L.gamma, L.minP, L.minD, c, p);
    else lim_prim<5>(L.gamma, c, p);
  };
  for (int i = tid; i < ne * 3; i += kLimThreads) {
    const int2 c = *reinterpret_cast<const int2*>(d.conn + (size_t)e0 * 6 + 2 * i);
    sNb[i / 3][i % 3] = c.x;
    sNf[i / 3][i % 3] = c.y;
  }
  __syncthreads();
  // Step 2: cell averages of the patch (5-field order), a thread per member and field
  for (int i = tid; i < ne * 4 * M; i += kLimThreads) {
    const int e = i / (4 * M), r = i - e * 4 * M, m = r / M, f = r - m * M;
    const int k = m == 0 ? e0 + e : sNb[e][m - 1];
    if (k < 0) continue;  // a boundary: the ghost average below
    const double* q = x + (size_t)k * NP * M + f;
    double acc = 0.;
#pragma unroll
    for (int n = 0; n < NP; ++n) acc += L.ave[n] * q[n * M];
    sRaw[e][m][f == M - 1 ? 4 : f] = acc;
    if (M == 4 && f == 0) sRaw[e][m][3] = 0.0;
  }
  __syncthreads();
  // Step 1: patch geometry, and the members' primitive variables
  for (int i = tid; i < ne * 4; i += kLimThreads) {
    const int e = i >> 2, m = i & 3, k = e0 + e;
    const ElemGeo& g = d.geo[k];
    double xc0 = 0, yc0 = 0, A0 = 0, c0[5], p0[5];
    for (int kk = 0; kk < 3; ++kk) {
      xc0 += L.ave[kk] * xn[(size_t)k * NP + L.fmask[kk * NPF]];
      yc0 += L.ave[kk] * yn[(size_t)k * NP + L.fmask[kk * NPF]];
      A0 += 2. / 3. * L.ave[kk] * g.J;
    }
    for (int c = 0; c < 5; ++c) c0[c] = sRaw[e][0][c];
    prim_of(c0, p0);
    if (m == 0) {
      sXc[e][0] = xc0;
      sYc[e][0] = yc0;
      for (int c = 0; c < 5; ++c) {
        sCons[e][c] = c0[c];
        sPrim[e][0][c] = p0[c];
      }
      continue;
    }
    const int f = m - 1, nb = sNb[e][f];
    double xc = 0, yc = 0, A = 0, c5[5], p5[5];
    if (nb < 0) {
      const double H1 = 2.0 * A0 / g.sJ[f];
      xc = xc0 + 2.0 * g.nx[f] * H1;
      yc = yc0 + 2.0 * g.ny[f] * H1;
      double qa[M], qb[M];
      qa[0] = c0[0]; qa[1] = c0[1]; qa[2] = c0[2];
      if (M == 5) qa[3] = c0[3];
      qa[M - 1] = c0[4];
      apply_bc<EQ, double>(d.bcs, -nb, xc, yc, 0.0, g.nx[f], g.ny[f], qa, qb);
      to5(qb, c5);
    } else {
      const double Jn = d.geo[nb].J;
      for (int node = 0; node < 3; ++node) {
        xc += L.ave[node] * xn[(size_t)nb * NP + L.fmask[node * NPF]];
        yc += L.ave[node] * yn[(size_t)nb * NP + L.fmask[node * NPF]];
        A += 2. / 3. * L.ave[node] * Jn;
      }
      for (int c = 0; c < 5; ++c) c5[c] = sRaw[e][m][c];
    }
    prim_of(c5, p5);
    sXc[e][m] = xc;
    sYc[e][m] = yc;
    sA[e][m] = A + A0;
    for (int c = 0; c < 5; ++c) sPrim[e][m][c] = p5[c];
  }
  // Step 3: face averages at the six positions Apollo reads (fConsA at index
  // endIDs[n], an element node id, taken as a face-node position)
  for (int i = tid; i < ne * 6; i += kLimThreads) {
    const int e = i / 6, n = i - e * 6, k = e0 + e;
    const ElemGeo& g = d.geo[k];
    const double* q = x + (size_t)k * NP * M;
    const int end_id = L.fmask[n == 0 ? 0 : n == 1 ? NPF - 1 : n == 2 ? NPF : n == 3 ? 2 * NPF - 1 : n == 4 ? 2 * NPF : 3 * NPF - 1];
    const int edge = end_id / NPF, nd = end_id - edge * NPF;
    const int node = L.fmask[edge * NPF + nd], nb = sNb[e][edge];
    double qm[M], qp[M];
    for (int f = 0; f < M; ++f) qm[f] = q[node * M + f];
    if (nb < 0) {
      // Apollo reads the patch neighbours through the pointer that held this
      // element's nodes and never points it back, so the condition sees the
      // nodes of the last neighbour read before this face (faces in order;
      // this element's own where none): wxhesthavenwarburtoneulerlimiter.cc
      // :158, 221, aptualiabadilimiter.cc:170, 233
      const double* qs = q;
      for (int j = 0; j < edge; ++j)
        if (sNb[e][j] >= 0) qs = x + (size_t)sNb[e][j] * NP * M;
      double qin[M];
      for (int f = 0; f < M; ++f) qin[f] = qs[node * M + f];
      apply_bc<EQ, double>(d.bcs, -nb, xn[(size_t)k * NP + node], yn[(size_t)k * NP + node], 0.0, g.nx[edge], g.ny[edge],
                           qin, qp);
    } else {
      const double* qn = x + (size_t)nb * NP * M + L.fmask[sNf[e][edge] * NPF + NPF - 1 - nd] * M;
      for (int f = 0; f < M; ++f) qp[f] = qn[f];
    }
    double fa[M], c5[5], p5[5];
    for (int f = 0; f < M; ++f) fa[f] = 0.5 * (qp[f] + qm[f]);
    to5(fa, c5);
    if (ta) {
      ta_prim(L.gamma, L.minP, L.minD, c5, p5);
    } else {
      const double rho = c5[0], rhou = c5[1], rhov = c5[2], rhow = c5[3], en = c5[4];
      p5[0] = rho;
      p5[1] = rhou / rho;
      p5[2] = rhov / rho;
      p5[3] = rhow / rho;
      p5[4] = (L.gamma - 1.) * (en - 0.5 * (rhou * rhou + rhov * rhov + rhow * rhow) / rho);
    }
    for (int c = 0; c < 5; ++c) sFp[e][n][c] = p5[c];
  }
  __syncthreads();
  // Step 4: gradients, a thread per variable
  for (int i = tid; i < ne * 5; i += kLimThreads) {
    const int e = i / 5, c = i - e * 5, k = e0 + e;
    const double *xe = xn + (size_t)k * NP, *ye = yn + (size_t)k * NP;
    const double xv1 = xe[L.fmask[0]], yv1 = ye[L.fmask[0]];
    const double xv2 = xe[L.fmask[NPF]], yv2 = ye[L.fmask[NPF]];
    const double xv3 = xe[L.fmask[2 * NPF]], yv3 = ye[L.fmask[2 * NPF]];
    const double *xc = sXc[e], *yc = sYc[e], *A0 = sA[e];
    const double prim[4] = {sPrim[e][0][c], sPrim[e][1][c], sPrim[e][2][c], sPrim[e][3][c]};
    double fp[6];
    for (int n = 0; n < 6; ++n) fp[n] = sFp[e][n][c];
    double* w = work + (size_t)k * kLimStride;
    const double ex1 = 0.5 * ((prim[1] - prim[0]) * (yv2 - yv1) + (fp[0] - fp[1]) * (yc[1] - yc[0])) / A0[1];
    const double ey1 = -0.5 * ((prim[1] - prim[0]) * (xv2 - xv1) + (fp[0] - fp[1]) * (xc[1] - xc[0])) / A0[1];
    const double ex2 = 0.5 * ((prim[2] - prim[0]) * (yv3 - yv2) + (fp[2] - fp[3]) * (yc[2] - yc[0])) / A0[2];
    const double ey2 = -0.5 * ((prim[2] - prim[0]) * (xv3 - xv2) + (fp[2] - fp[3]) * (xc[2] - xc[0])) / A0[2];
    // (the reference's third edge repeats the second edge's vertex differences)
    const double ex3 = 0.5 * ((prim[3] - prim[0]) * (yv3 - yv2) + (fp[4] - fp[5]) * (yc[3] - yc[0])) / A0[3];
    const double ey3 = -0.5 * ((prim[3] - prim[0]) * (xv3 - xv2) + (fp[4] - fp[5]) * (xc[3] - xc[0])) / A0[3];
    w[0 * 5 + c] = ex1; w[1 * 5 + c] = ey1;
    w[2 * 5 + c] = ex2; w[3 * 5 + c] = ey2;
    w[4 * 5 + c] = ex3; w[5 * 5 + c] = ey3;
    w[6 * 5 + c] = (A0[1] * ex1 + A0[2] * ex2 + A0[3] * ex3) / (A0[1] + A0[2] + A0[3]);
    w[7 * 5 + c] = (A0[1] * ey1 + A0[2] * ey2 + A0[3] * ey3) / (A0[1] + A0[2] + A0[3]);
    w[8 * 5 + c] = sCons[e][c];
    w[9 * 5 + c] = prim[0];
  }
}

template <int EQ, int N>
__global__ void __launch_bounds__(kLimThreads) k_limiter_apply(DgDev d, LimArgs L, const double* __restrict__ xn,
                                                               const double* __restrict__ yn,
                                                               const double* __restrict__ work,
                                                               double* __restrict__ out) {
  constexpr int M = Eq<EQ>::M;
  constexpr int NP = Sizes<N>::NP;
  __shared__ double sLx[kLimE][5], sLy[kLimE][5];
  const int e0 = blockIdx.x * kLimE, ne = min(kLimE, d.K - e0), tid = threadIdx.x;
  // the weighted gradients, a thread per variable
  for (int i = tid; i < ne * 5; i += kLimThreads) {
    const int e = i / 5, c = i - e * 5, k = e0 + e;
    const double* w = work + (size_t)k * kLimStride;
    double gx[3], gy[3];
    for (int edge = 0; edge < 3; ++edge) {
      const int nbr = d.conn[(size_t)k * 6 + 2 * edge];
      if (nbr < 0) {
        gx[edge] = w[(2 * edge) * 5 + c];
        gy[edge] = w[(2 * edge + 1) * 5 + c];
      } else {
        const double* wn = work + (size_t)nbr * kLimStride;
        gx[edge] = wn[6 * 5 + c];
        gy[edge] = wn[7 * 5 + c];
      }
    }
    const double g1 = (gx[0] * gx[0] + gy[0] * gy[0]);
    const double g2 = (gx[1] * gx[1] + gy[1] * gy[1]);
    const double g3 = (gx[2] * gx[2] + gy[2] * gy[2]);
    const double fac = g1 * g1 + g2 * g2 + g3 * g3;
    const double epse = 1.e-14;
    const double fac3e = fac + 3.0 * epse;
    const double w1 = (g2 * g3 + epse) / fac3e;
    const double w2 = (g1 * g3 + epse) / fac3e;
    const double w3 = (g1 * g2 + epse) / fac3e;
    sLx[e][c] = w1 * gx[0] + w2 * gx[1] + w3 * gx[2];
    sLy[e][c] = w1 * gy[0] + w2 * gy[1] + w3 * gy[2];
  }
  __syncthreads();
  const double gamma = L.gamma, minD = L.minD, minP = L.minP;
  int err = 0;
  // the reconstruction, a thread per node
  for (int i = tid; i < ne * NP; i += kLimThreads) {
    const int e = i / NP, n = i - e * NP, k = e0 + e;
    const double* w = work + (size_t)k * kLimStride;
    const double *xe = xn + (size_t)k * NP, *ye = yn + (size_t)k * NP;
    double ldx = 0.0, ldy = 0.0;
#pragma unroll
    for (int j = 0; j < NP; ++j) {
      double drop = -L.ave[j];
      if (n == j) drop += 1.;
      ldx += drop * xe[j];
      ldy += drop * ye[j];
    }
    const double *Lx = sLx[e], *Ly = sLy[e], *cons = w + 40;
    const double averho = w[45 + 0], aveu = w[45 + 1], avev = w[45 + 2], avew = w[45 + 3], avep = w[45 + 4];
    double drho = ldx * Lx[0] + ldy * Ly[0];
    const double du = ldx * Lx[1] + ldy * Ly[1];
    const double dv = ldx * Lx[2] + ldy * Ly[2];
    const double dw = ldx * Lx[3] + ldy * Ly[3];
    double dp = ldx * Lx[4] + ldy * Ly[4];
    double Lrho = averho + drho;
    if (Lrho < minD) {
      for (int it = 0; it < 4; ++it) {
        drho *= 0.5;
        Lrho = averho + drho;
        if (Lrho > minD) break;
        else if (it == 3) Lrho = cons[0];
      }
    }
    const double Lrhou = cons[1] + averho * du + drho * aveu;
    const double Lrhov = cons[2] + averho * dv + drho * avev;
    const double Lrhow = cons[3] + averho * dw + drho * avew;
    double dEner = dp / (gamma - 1.) + 0.5 * drho * (aveu * aveu + avev * avev + avew * avew) +
                   averho * (aveu * du + avev * dv + avew * dw);
    double LEner = cons[4] + dEner;
    double Lp = (gamma - 1.) * (LEner - 0.5 * (Lrhou * Lrhou + Lrhov * Lrhov + Lrhow * Lrhow) / Lrho);
    if (Lp < minP) {
      for (int it = 0; it < 4; ++it) {
        dp *= 0.5;
        dEner = dp / (gamma - 1.) + 0.5 * drho * (aveu * aveu + avev * avev + avew * avew) +
                averho * (aveu * du + avev * dv + avew * dw);
        LEner = cons[4] + dEner;
        Lp = (gamma - 1.) * (LEner - 0.5 * (Lrhou * Lrhou + Lrhov * Lrhov + Lrhow * Lrhow) / Lrho);
        if (Lp > minP) break;
        else if (it == 3) LEner = avep / (gamma - 1.) + 0.5 * (Lrhou * Lrhou + Lrhov * Lrhov + Lrhow * Lrhow) / Lrho;
      }
    }
    if (!isfinite(Lrho) || !isfinite(Lrhou) || !isfinite(Lrhov) || !isfinite(LEner)) err |= ERRB_NAN;
    // tuAliabadiLimiter's reconstruction (WxEulerEqn::limiterTuAndAliabadi)
    // also stops on a non-positive density
    if (L.kind == 1 && Lrho <= 0.) err |= ERRB_NONPHYS;
    double* o = out + ((size_t)k * NP + n) * M;
    o[0] = Lrho;
    o[1] = Lrhou;
    o[2] = Lrhov;
    if (M == 5) o[3] = Lrhow;
    o[M - 1] = LEner;
  }
  if (err) atomicOr(&d.st->err, err);
}

// tuAliabadiLimiter for phMaxwellEqn (WxPHMaxwellEqn::limiterTuAndAliabadi,
// src/hyperapps/maxwell/wxphmaxwelleqn.cc:740-755, returns the cell averages):
// every node of an element takes the element average, field by field, summed
// in node order.  One thread per (element, field); it reads its row before it
// writes it, so out may be x.
template <int M, int N>
__global__ void __launch_bounds__(128) k_limiter_average(int K, LimArgs L, const double* x, double* out) {
  constexpr int NP = Sizes<N>::NP;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)K * M) return;
  const long long e = t / M;
  const int f = (int)(t - e * M);
  double s = 0.0;
  for (int n = 0; n < NP; ++n) s += L.ave[n] * x[(e * NP + n) * M + f];
  for (int n = 0; n < NP; ++n) out[(e * NP + n) * M + f] = s;
}

template <int M>
cudaError_t average_n(const DgDev& d, const LimArgs& L, const double* x, double* out, cudaStream_t s) {
  const long long n = (long long)d.K * M;
  const int blocks = (int)((n + 127) / 128);
  switch (d.N) {
    case 2: k_limiter_average<M, 2><<<blocks, 128, 0, s>>>(d.K, L, x, out); break;
    case 3: k_limiter_average<M, 3><<<blocks, 128, 0, s>>>(d.K, L, x, out); break;
    case 4: k_limiter_average<M, 4><<<blocks, 128, 0, s>>>(d.K, L, x, out); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

template <int EQ, int N>
cudaError_t limiter_t(const DgDev& d, const LimArgs& L, const double* x, double* out, const double* xn,
                      const double* yn, double* work, cudaStream_t s) {
  const int blocks = (d.K + kLimE - 1) / kLimE;
  k_limiter_grad<EQ, N><<<blocks, kLimThreads, 0, s>>>(d, L, x, xn, yn, work);
  k_limiter_apply<EQ, N><<<blocks, kLimThreads, 0, s>>>(d, L, xn, yn, work, out);
  return cudaGetLastError();
}

template <int EQ>
cudaError_t limiter_n(const DgDev& d, const LimArgs& L, const double* x, double* out, const double* xn,
                      const double* yn, double* work, cudaStream_t s) {
  switch (d.N) {
    case 2: return limiter_t<EQ, 2>(d, L, x, out, xn, yn, work, s);
    case 3: return limiter_t<EQ, 3>(d, L, x, out, xn, yn, work, s);
    case 4: return limiter_t<EQ, 4>(d, L, x, out, xn, yn, work, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace

size_t limiter_work_doubles(int K) { return (size_t)K * kLimStride; }

cudaError_t launch_limiter(int eq, const DgDev& d, const LimArgs& L, const double* x, double* out, const double* xn,
                           const double* yn, double* work, cudaStream_t s) {
  if (eq == EQ_EULER) return limiter_n<EQ_EULER>(d, L, x, out, xn, yn, work, s);
  if (eq == EQ_EULER2D) return limiter_n<EQ_EULER2D>(d, L, x, out, xn, yn, work, s);
  if (L.kind == 1 && eq == EQ_MAXWELL) return average_n<Eq<EQ_MAXWELL>::M>(d, L, x, out, s);
  if (L.kind == 1 && eq == EQ_MAXWELL_TM) return average_n<Eq<EQ_MAXWELL_TM>::M>(d, L, x, out, s);
  return cudaErrorInvalidValue;
}

}  // namespace apollo
