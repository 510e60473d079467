// Float64 nodal-DG right-hand side on sm_100a: one volume kernel, one face
// kernel and one LIFT kernel with the SSP stage update fused in, per stage.
//
//  k_volume  : per element tile, q -> cubature values (V), physical flux at
//              every cubature point, volume contraction with the weighted
//              derivative operators (Dr, Ds) and the face traces (I q).
//              Apollo: wxnodaldg2dmethod.cc:346-394 with
//              wxcubature2d.cc:290-363.
//  k_face    : per face Gauss point, both traces through the face map (the
//              partner in reversed Gauss order), boundary hook, Lax-Friedrichs
//              flux, times sJ and the Gauss weight, written to both sides, and
//              the max wave speed.  Apollo: wxnodaldg2dmethod.cc:396-469.
//  k_lift    : per element tile, surface contraction (L = VVT I^T), 1/J,
//              combination with the volume term and the stage update.
//              Apollo: wxcubature2d.cc:367-382, wxnodaldggeometry2d.cc:444-456,
//              wxnodaldg2dmethod.cc:475-504; PETSc TSSSP RK_2 update.
#include <cuda_runtime.h>
#include <stdint.h>

#include "dg_chain64.cuh"
#include "dg_device.cuh"
#include "dg_dmma.cuh"
#include "dg_flux64.cuh"
#include "dg_stage64.h"

namespace apollo {

namespace {

constexpr int kThreads = 256;

// Tile of elements for the float64 volume kernel.  Columns of every GEMM are
// (element, field) pairs; rows are cubature points, Gauss points or nodes.
template <int N, int M> struct VolTile {
  static constexpr int NP = Sizes<N>::NP, NC = Sizes<N>::NC, NF = Sizes<N>::NF;
  // 16 elements per tile (8 for 8 fields or N >= 5), 64 for scalar advection,
  // keeping the tile near 110 KB of shared memory (two blocks per SM)
  static constexpr int E = M == 1 ? 64 : ((M == 8 || N >= 5) ? 8 : 16);
  static constexpr int COLS = round_up(E * M, 8);
  static constexpr int LDB = pad_ld(COLS);
  static constexpr int NPK = round_up(NP, 4);    // K of V*q and I*q
  static constexpr int LDA1 = pad_ld(NPK);
  static constexpr int NCR = round_up(NC, 8);    // rows of V*q
  static constexpr int NFR = round_up(NF, 8);    // rows of I*q
  static constexpr int NPR = round_up(NP, 8);    // rows of D*[R;S]
  static constexpr int K2 = round_up(2 * NC, 4); // K of D*[R;S]
  static constexpr int LDA2 = pad_ld(K2);
  static constexpr int RSR = K2 > NCR ? K2 : NCR;
  static constexpr int OFF_V = 0;
  static constexpr int OFF_D = OFF_V + NCR * LDA1;
  static constexpr int OFF_I = OFF_D + NPR * LDA2;
  static constexpr int OFF_Q = OFF_I + NFR * LDA1;
  static constexpr int OFF_RS = OFF_Q + NPK * LDB;
  static constexpr int TOTAL = OFF_RS + RSR * LDB;
  static constexpr size_t BYTES = sizeof(double) * TOTAL;
};

template <int EQ, int N>
__global__ void __launch_bounds__(kThreads) k_volume(DgDev d, StageArgs a) {
  using P = Eq<EQ>;
  constexpr int M = P::M;
  using T = VolTile<N, M>;
  constexpr int NP = T::NP, NC = T::NC, NF = T::NF, E = T::E, LDB = T::LDB;
  constexpr int NWARPS = kThreads / 32;
  extern __shared__ double smem[];
  double* sV = smem + T::OFF_V;
  double* sD = smem + T::OFF_D;
  double* sI = smem + T::OFF_I;
  double* sQ = smem + T::OFF_Q;
  double* sRS = smem + T::OFF_RS;
  const int tid = threadIdx.x;
  if (a.reset_lambda && blockIdx.x == 0)
    for (int i = tid; i < d.ninst; i += kThreads) d.st[i].lam_bits = 0ull;
  // operators, zero-padded: V [NCR][NPK], D = [Dr | Ds] [NPR][K2], I [NFR][NPK]
  for (int i = tid; i < T::NCR * T::LDA1; i += kThreads) {
    const int r = i / T::LDA1, c = i % T::LDA1;
    sV[i] = (r < NC && c < NP) ? d.V[r * NP + c] : 0.0;
  }
  for (int i = tid; i < T::NPR * T::LDA2; i += kThreads) {
    const int r = i / T::LDA2, c = i % T::LDA2;
    double v = 0.0;
    if (r < NP && c < NC) v = d.Dr[r * NC + c];
    else if (r < NP && c >= NC && c < 2 * NC) v = d.Ds[r * NC + c - NC];
    sD[i] = v;
  }
  for (int i = tid; i < T::NFR * T::LDA1; i += kThreads) {
    const int r = i / T::LDA1, c = i % T::LDA1;
    sI[i] = (r < NF && c < NP) ? d.I[r * NP + c] : 0.0;
  }
  // padding rows of the right-hand operands stay zero
  for (int i = tid; i < T::NPK * LDB; i += kThreads) sQ[i] = 0.0;
  for (int i = tid; i < T::RSR * LDB; i += kThreads) sRS[i] = 0.0;
  int err = 0;
  const int ntiles = (d.K + E - 1) / E;
  // q tile, [e][node][field] -> Q[node][e*M + field]: the first tile here, each
  // next one loaded into registers while this one's fluxes are evaluated and
  // stored after them (Q is read only by the first two contractions)
  constexpr int NQ = E * NP * M, QPT = (NQ + kThreads - 1) / kThreads;
  auto put_q = [&](int i, double v) {
    const int e = i / (NP * M), r = i - e * NP * M, j = r / M, f = r - j * M;
    sQ[j * LDB + e * M + f] = v;
  };
  __syncthreads();  // the zero padding above is written before the first tile
  if ((int)blockIdx.x < ntiles) {
    const int k0 = blockIdx.x * E, nq = min(E, d.K - k0) * NP * M;
    const double* src = a.x + (size_t)k0 * NP * M;
    for (int i = tid; i < nq; i += kThreads) put_q(i, src[i]);
  }
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int k0 = tile * E;
    const int ne = min(E, d.K - k0);
    __syncthreads();
    // cubature values Qc = V Q (into the R/S buffer) and face traces I Q (to HBM)
    block_dgemm<T::NCR, T::COLS, T::NPK, T::LDA1, LDB, NWARPS>(
        sV, sQ, [&](int r, int c, double v) { sRS[r * LDB + c] = v; });
    block_dgemm<T::NFR, T::COLS, T::NPK, T::LDA1, LDB, NWARPS>(sI, sQ, [&](int r, int c, double v) {
      const int e = c / M, f = c - e * M;
      if (r < NF && e < ne) d.trace[((size_t)(k0 + e) * NF + r) * M + f] = v;
    });
    __syncthreads();
    // the next tile's states, in flight during the flux evaluation
    const int nxt = tile + (int)gridDim.x;
    const int nq_next = nxt < ntiles ? min(E, d.K - nxt * E) * NP * M : 0;
    double qn[QPT];
#pragma unroll
    for (int u = 0; u < QPT; ++u) {
      const int i = tid + u * kThreads;
      qn[u] = i < nq_next ? a.x[(size_t)nxt * E * NP * M + i] : 0.0;
    }
    // physical flux at every cubature point; R = rx F + ry G into row c,
    // S = sx F + sy G into row NC + c (row c is overwritten by its reader only)
    for (int idx = tid; idx < ne * NC; idx += kThreads) {
      const int e = idx / NC, c = idx - e * NC;
      double qc[M], R[M], S[M];
#pragma unroll
      for (int f = 0; f < M; ++f) qc[f] = sRS[c * LDB + e * M + f];
      const ElemGeo& g = d.geo[k0 + e];
      volume_flux<EQ>(d.eqp, qc, g.rx, g.ry, g.sx, g.sy, R, S, &err);
#pragma unroll
      for (int f = 0; f < M; ++f) {
        sRS[c * LDB + e * M + f] = R[f];
        sRS[(NC + c) * LDB + e * M + f] = S[f];
      }
    }
#pragma unroll
    for (int u = 0; u < QPT; ++u) {
      const int i = tid + u * kThreads;
      if (i < nq_next) put_q(i, qn[u]);
    }
    __syncthreads();
    // volume term: [Dr | Ds] [R; S]
    block_dgemm<T::NPR, T::COLS, T::K2, T::LDA2, LDB, NWARPS, 4>(sD, sRS, [&](int r, int c, double v) {
      const int e = c / M, f = c - e * M;
      if (r < NP && e < ne) d.vol[((size_t)(k0 + e) * NP + r) * M + f] = v;
    });
  }
  if (err) atomicOr(&d.st->err, err);
}

// M consecutive doubles of one Gauss point (a trace or a face flux): 16-byte
// vector accesses when M is even (every point's block then starts on a
// 16-byte boundary), scalar ones otherwise.
template <int M>
__device__ __forceinline__ void load_point(const double* __restrict__ p, double* q) {
  if constexpr (M % 2 == 0) {
#pragma unroll
    for (int f = 0; f < M; f += 2) {
      const double2 v = __ldg(reinterpret_cast<const double2*>(p + f));
      q[f] = v.x;
      q[f + 1] = v.y;
    }
  } else {
#pragma unroll
    for (int f = 0; f < M; ++f) q[f] = __ldg(p + f);
  }
}
template <int M>
__device__ __forceinline__ void store_point(double* __restrict__ p, const double* q, double w) {
  if constexpr (M % 2 == 0) {
#pragma unroll
    for (int f = 0; f < M; f += 2) *reinterpret_cast<double2*>(p + f) = make_double2(q[f] * w, q[f + 1] * w);
  } else {
#pragma unroll
    for (int f = 0; f < M; ++f) p[f] = q[f] * w;
  }
}

template <int EQ, int N>
__global__ void __launch_bounds__(kThreads) k_face(DgDev d, StageArgs a) {
  using P = Eq<EQ>;
  constexpr int M = P::M;
  constexpr int NG = Sizes<N>::NG, NF = Sizes<N>::NF;
  int err = 0;
  LamAcc lam_acc;
  // each block takes a contiguous range of face points, so a thread's points
  // stay within one instance of a batched ensemble
  const bool two_sided = flux_two_sided<EQ>(d.eqp);
  const int total = d.nfaces * NG;
  const int per_block = (total + gridDim.x - 1) / gridDim.x;
  const int i0 = blockIdx.x * per_block, i1 = min(total, i0 + per_block);
  for (int idx = i0 + threadIdx.x; idx < i1; idx += blockDim.x) {
    const int fi = idx / NG, gq = idx - fi * NG;
    const FaceRec fr = d.faces[fi];
    const int inst = inst_of(d, fr.k1);
    const double t = a.time_from_state ? d.st[inst].t + d.st[inst].dt * a.frac : a.t_arg;
    const ElemGeo& g = d.geo[fr.k1];
    const double nx = g.nx[fr.f1], ny = g.ny[fr.f1], sJ = g.sJ[fr.f1];
    double qM[M], qP[M], nf[M];
    const double* tm = d.trace + ((size_t)fr.k1 * NF + fr.f1 * NG + gq) * M;
    load_point<M>(tm, qM);
    if (fr.k2 >= 0) {
      load_point<M>(d.trace + ((size_t)fr.k2 * NF + fr.f2 * NG + (NG - 1 - gq)) * M, qP);
    } else {
      // Gauss point coordinates on face f1: the affine map of the face
      // parametrisation (wxcubature2d.cc:118-124)
      const double z = d.gz[gq];
      double r, s;
      if (fr.f1 == 0) { r = z; s = -1.0; }
      else if (fr.f1 == 1) { r = -z; s = z; }
      else { r = -1.0; s = -z; }
      const double x = 0.5 * (-g.vx[0] * (r + s) + g.vx[1] * (1. + r) + g.vx[2] * (1. + s));
      const double y = 0.5 * (-g.vy[0] * (r + s) + g.vy[1] * (1. + r) + g.vy[2] * (1. + s));
      apply_bc<EQ, double>(d.bcs, -fr.k2, t, x, y, nx, ny, qM, qP);
    }
    const int kind = (int)d.eqp.p[3];
    const double lam = kind == NF_HLL || kind == NF_ROE || kind == NF_WAVE
                           ? face_flux2<EQ, kAnyFlux>(d.eqp, nx, ny, 0.5, qM, qP, nf, &err)
                           : face_flux2<EQ, NF_LF>(d.eqp, nx, ny, 0.5, qM, qP, nf, &err);
    lam_acc.add(d.st, inst, fabs(lam));
    const double w = d.gw[gq] * sJ;
    store_point<M>(d.flux + ((size_t)fr.k1 * NF + fr.f1 * NG + gq) * M, nf, w);
    if (fr.k2 >= 0) {
      const int g2 = NG - 1 - gq;
      double* op = d.flux + ((size_t)fr.k2 * NF + fr.f2 * NG + g2) * M;
      if (two_sided) {
        // the partner's own evaluation: its normal, weight and trace as "-"
        const ElemGeo& h2 = d.geo[fr.k2];
        load_point<M>(d.trace + ((size_t)fr.k2 * NF + fr.f2 * NG + g2) * M, qM);
        load_point<M>(tm, qP);
        const double lam2 = P::numflux(d.eqp, h2.nx[fr.f2], h2.ny[fr.f2], qM, qP, nf, &err);
        lam_acc.add(d.st, inst, fabs(lam2));
        store_point<M>(op, nf, d.gw[g2] * h2.sJ[fr.f2]);
      } else {
        store_point<M>(op, nf, -w);
      }
    }
  }
  lam_acc.flush_warp(d.st);
  if (err) atomicOr(&d.st->err, err);
}

template <int N, int M> struct LiftTile {
  static constexpr int NP = Sizes<N>::NP, NF = Sizes<N>::NF;
  static constexpr int E = M == 1 ? 64 : (M == 8 ? 8 : 16);
  static constexpr int COLS = round_up(E * M, 8);
  static constexpr int LDB = pad_ld(COLS);
  static constexpr int NFK = round_up(NF, 4);  // K: face Gauss points
  static constexpr int LDA = pad_ld(NFK);
  static constexpr int NPR = round_up(NP, 8);
  static constexpr int OFF_L = 0;
  static constexpr int OFF_F = NPR * LDA;
  static constexpr size_t BYTES = sizeof(double) * (OFF_F + NFK * LDB);
};

template <int EQ, int N>
__global__ void __launch_bounds__(kThreads) k_lift(DgDev d, StageArgs a) {
  constexpr int M = Eq<EQ>::M;
  using T = LiftTile<N, M>;
  constexpr int NP = T::NP, NF = T::NF, E = T::E, LDB = T::LDB;
  constexpr int NWARPS = kThreads / 32;
  extern __shared__ double smem[];
  double* sL = smem + T::OFF_L;
  double* sF = smem + T::OFF_F;
  const int tid = threadIdx.x;
  for (int i = tid; i < T::NPR * T::LDA; i += kThreads) {
    const int r = i / T::LDA, c = i % T::LDA;
    sL[i] = (r < NP && c < NF) ? d.L[r * NF + c] : 0.0;
  }
  for (int i = tid; i < T::NFK * LDB; i += kThreads) sF[i] = 0.0;
  int err = 0;
  const int ntiles = (d.K + E - 1) / E;
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int k0 = tile * E;
    const int ne = min(E, d.K - k0);
    __syncthreads();
    // numerical-flux tile, [e][gauss][field] -> F[gauss][e*M + field]
    const double* src = d.flux + (size_t)k0 * NF * M;
    for (int i = tid; i < ne * NF * M; i += kThreads) {
      const int e = i / (NF * M), r = i - e * NF * M, g = r / M, f = r - g * M;
      sF[g * LDB + e * M + f] = src[i];
    }
    __syncthreads();
    block_dgemm<T::NPR, T::COLS, T::NFK, T::LDA, LDB, NWARPS>(sL, sF, [&](int i, int c, double v) {
      const int e = c / M, f = c - e * M;
      if (i >= NP || e >= ne) return;
      const int k = k0 + e;
      const size_t off = ((size_t)k * NP + i) * M + f;
      const double dt = a.time_from_state ? d.st[inst_of(d, k)].dt : a.dt_arg;
      const double c_stage = dt / 4.0;  // dt/(s-1), s = 5
      const double c_al = 4.0 / 5.0, c_be = dt / 5.0, c_ga = 1.0 / 5.0;
      const double r = d.vol[off] - d.geo[k].invJ * v;
      if (r != r) err |= ERRB_NAN;
      double o;
      if (a.mode == MODE_RHS) o = r;
      else if (a.mode == MODE_STAGE) o = a.x[off] + c_stage * r;
      else o = c_al * a.x[off] + c_be * r + c_ga * a.u0[off];
      a.out[off] = o;
    });
  }
  if (err) atomicOr(&d.st->err, err);
}

template <int EQ>
__global__ void k_init_speed(DgDev d, const double* u, int nnodes) {
  constexpr int M = Eq<EQ>::M;
  LamAcc lam_acc;
  const int per_block = (nnodes + gridDim.x - 1) / gridDim.x;
  const int i0 = blockIdx.x * per_block, i1 = min(nnodes, i0 + per_block);
  const int np = nnodes / d.K;
  for (int i = i0 + threadIdx.x; i < i1; i += blockDim.x) {
    double q[M];
#pragma unroll
    for (int f = 0; f < M; ++f) q[f] = u[(size_t)i * M + f];
    double s2 = Eq<EQ>::speed2(d.eqp, q);
    lam_acc.add(d.st, inst_of(d, i / np), sqrt(s2 > 0.0 ? s2 : 0.0));
  }
  lam_acc.flush_warp(d.st);
}

// After a step: t += dt; dt = min(dt, suggestion of the last stage), clipped
// to the end time (ApSolver::ComputeRHSforTS + MonitorVTK,
// src/solvers/apsolver.cc:421-480).
__global__ void k_finalize(DgDev d) {
  wait_previous();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.ninst) return;
  DevState* st = d.st + i;
  const double lam = __longlong_as_double((long long)st->lam_bits);
  const double sugg = (st->dtfac > 0.0 ? st->dtfac : d.dtfac) * (d.rmin / lam);
  st->last_sugg = sugg;
  const double dt = st->dt;
  const double t = st->t + dt;
  double nd = fmin(sugg, dt);
  if (st->tend > 0.0 && fabs(st->tend - t) < nd) nd = fabs(st->tend - t);
  st->t = t;
  st->dt = nd;
  st->steps += 1;
  st->lam_bits = 0ull;  // the next step's last stage reduces into it afresh
}

template <int EQ>
__global__ void k_integrals(DgDev d, const double* u, const double* wmass, int NP) {
  constexpr int M = Eq<EQ>::M;
  double acc[M];
#pragma unroll
  for (int f = 0; f < M; ++f) acc[f] = 0.0;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < d.K; k += gridDim.x * blockDim.x) {
    const double J = d.geo[k].J;
    for (int j = 0; j < NP; ++j) {
      const double w = wmass[j] * J;
#pragma unroll
      for (int f = 0; f < M; ++f) acc[f] += w * u[((size_t)k * NP + j) * M + f];
    }
  }
#pragma unroll
  for (int f = 0; f < M; ++f) {
    double v = acc[f];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(&d.st->sums[f], v);
  }
}

// Per-field integrals of u^2 over the mesh: sum_k J_k u_k^T Mref u_k with the
// reference-element mass matrix Mref = (V V^T)^-1 (the inverse of Apollo's
// VVT, wxnodaldggeometry2d.cc:71-75), one thread per element.
template <int EQ>
__global__ void k_energy(DgDev d, const double* __restrict__ u, const double* __restrict__ mass, int NP) {
  constexpr int M = Eq<EQ>::M;
  double acc[M];
#pragma unroll
  for (int f = 0; f < M; ++f) acc[f] = 0.0;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < d.K; k += gridDim.x * blockDim.x) {
    const double J = d.geo[k].J;
    const double* uk = u + (size_t)k * NP * M;
    for (int i = 0; i < NP; ++i) {
      double mu[M];
#pragma unroll
      for (int f = 0; f < M; ++f) mu[f] = 0.0;
      for (int j = 0; j < NP; ++j) {
        const double w = mass[i * NP + j];
#pragma unroll
        for (int f = 0; f < M; ++f) mu[f] += w * uk[j * M + f];
      }
#pragma unroll
      for (int f = 0; f < M; ++f) acc[f] += J * uk[i * M + f] * mu[f];
    }
  }
#pragma unroll
  for (int f = 0; f < M; ++f) {
    double v = acc[f];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(&d.st->sums[f], v);
  }
}

// Source contribution of a block of kSrcE elements: the sources at every
// cubature point (physical coordinates from the element's affine map), then
// VS times them per (element, node, field).
constexpr int kSrcE = 4;
template <int EQ, int N>
__global__ void __launch_bounds__(128) k_source(DgDev d, StageArgs a, double* __restrict__ dst, int accumulate) {
  constexpr int M = Eq<EQ>::M, NP = Sizes<N>::NP, NC = Sizes<N>::NC;
  __shared__ double S[kSrcE][NC][M];
  const int k0 = blockIdx.x * kSrcE;
  for (int i = threadIdx.x; i < kSrcE * NC; i += blockDim.x) {
    const int e = i / NC, c = i - e * NC, k = k0 + e;
    double sv[M];
#pragma unroll
    for (int f = 0; f < M; ++f) sv[f] = 0.0;
    if (k < d.K) {
      const ElemGeo& g = d.geo[k];
      const double r = d.cub_r[c], q = d.cub_s[c];
      const double x = 0.5 * (-g.vx[0] * (r + q) + g.vx[1] * (1. + r) + g.vx[2] * (1. + q));
      const double y = 0.5 * (-g.vy[0] * (r + q) + g.vy[1] * (1. + r) + g.vy[2] * (1. + q));
      const DevState& st = d.st[inst_of(d, k)];
      const double t = a.time_from_state ? st.t + st.dt * a.frac : a.t_arg;
      source_terms<M>(d.src, t, x, y, sv);
    }
#pragma unroll
    for (int f = 0; f < M; ++f) S[e][c][f] = sv[f];
  }
  __syncthreads();
  unsigned fmask = 0;
  for (int i = 0; i < d.src.n; ++i) fmask |= 1u << d.src.out[i];
  for (int i = threadIdx.x; i < kSrcE * NP * M; i += blockDim.x) {
    const int e = i / (NP * M), r = i - e * NP * M, n = r / M, f = r - n * M, k = k0 + e;
    if (k >= d.K) continue;
    double v = 0.0;
    if (fmask & (1u << f))
      for (int c = 0; c < NC; ++c) v += d.VS[n * NC + c] * S[e][c][f];
    double* o = dst + ((size_t)k * NP + n) * M + f;
    if (accumulate) {
      if (fmask & (1u << f)) *o += v;
    } else {
      *o = v;
    }
  }
}

template <int EQ>
cudaError_t source_dispatch(const DgDev& d, const StageArgs& a, double* dst, int acc, cudaStream_t s) {
  const unsigned g = (unsigned)((d.K + kSrcE - 1) / kSrcE);
  if (g == 0) return cudaSuccess;
  switch (d.N) {
    case 2: k_source<EQ, 2><<<g, 128, 0, s>>>(d, a, dst, acc); break;
    case 3: k_source<EQ, 3><<<g, 128, 0, s>>>(d, a, dst, acc); break;
    case 4: k_source<EQ, 4><<<g, 128, 0, s>>>(d, a, dst, acc); break;
    case 5: k_source<EQ, 5><<<g, 128, 0, s>>>(d, a, dst, acc); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

int g_num_sms = 0;
int num_sms() {
  if (g_num_sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev);
    if (g_num_sms <= 0) g_num_sms = 148;
  }
  return g_num_sms;
}

template <int EQ, int N>
cudaError_t launch_rhs_t(const DgDev& d, const StageArgs& a, cudaStream_t s, cudaEvent_t* ev) {
  constexpr int M = Eq<EQ>::M;
  using VT = VolTile<N, M>;
  using LT = LiftTile<N, M>;
  static unsigned configured = 0;  // bit per device
  static int vol_res = 1, lift_res = 1;  // resident blocks per SM
  int dev = 0;
  cudaGetDevice(&dev);
  if (!(configured & (1u << (dev & 31)))) {
    cudaError_t e = cudaFuncSetAttribute(k_volume<EQ, N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)VT::BYTES);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(k_lift<EQ, N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)LT::BYTES);
    if (e != cudaSuccess) return e;
    // persistent grids of the blocks that are resident at once (registers
    // and shared memory): a block beyond them would start a late second wave
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&vol_res, k_volume<EQ, N>, kThreads, VT::BYTES);
    if (e != cudaSuccess) return e;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&lift_res, k_lift<EQ, N>, kThreads, LT::BYTES);
    if (e != cudaSuccess) return e;
    configured |= 1u << (dev & 31);
  }
  const int sms = d.grid_div > 1 ? (num_sms() + d.grid_div - 1) / d.grid_div : num_sms();
  const int vt = (d.K + VT::E - 1) / VT::E;
  int per_sm = vol_res < 1 ? 1 : (vol_res > 8 ? 8 : vol_res);
  int gv = sms * per_sm;
  if (gv > vt) gv = vt;
  if (ev) cudaEventRecord(ev[0], s);
  k_volume<EQ, N><<<gv, kThreads, VT::BYTES, s>>>(d, a);
  // sources enter the volume term (wxcubature2d.cc:297-325: VT (w J S))
  if (d.src.n > 0) {
    cudaError_t e = source_dispatch<EQ>(d, a, d.vol, 1, s);
    if (e != cudaSuccess) return e;
  }
  if (ev) cudaEventRecord(ev[1], s);
  const int fthreads = d.nfaces * Sizes<N>::NG;
  int gf = (fthreads + kThreads - 1) / kThreads;
  if (gf > sms * 8) gf = sms * 8;
  if (gf < 1) gf = 1;
  if (fthreads > 0) k_face<EQ, N><<<gf, kThreads, 0, s>>>(d, a);
  if (ev) cudaEventRecord(ev[2], s);
  const int lt = (d.K + LT::E - 1) / LT::E;
  int lper = lift_res < 1 ? 1 : (lift_res > 8 ? 8 : lift_res);
  int gl = sms * lper;
  if (gl > lt) gl = lt;
  k_lift<EQ, N><<<gl, kThreads, LT::BYTES, s>>>(d, a);
  if (ev) cudaEventRecord(ev[3], s);
  return cudaGetLastError();
}

// The LIFT kernel alone (surface contraction, 1/J, stage update) on the given
// volume and face-flux buffers: the lift and the stage update are linear, so
// the tangent of a stage applies it to the tangent buffers unchanged.
template <int EQ, int N>
cudaError_t launch_lift_t(const DgDev& d, const StageArgs& a, cudaStream_t s) {
  constexpr int M = Eq<EQ>::M;
  using LT = LiftTile<N, M>;
  static unsigned configured = 0;  // bit per device
  static int lift_res = 1;          // resident blocks per SM
  int dev = 0;
  cudaGetDevice(&dev);
  if (!(configured & (1u << (dev & 31)))) {
    cudaError_t e = cudaFuncSetAttribute(k_lift<EQ, N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)LT::BYTES);
    if (e != cudaSuccess) return e;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&lift_res, k_lift<EQ, N>, kThreads, LT::BYTES);
    if (e != cudaSuccess) return e;
    configured |= 1u << (dev & 31);
  }
  const int lt = (d.K + LT::E - 1) / LT::E;
  int lper = lift_res < 1 ? 1 : (lift_res > 8 ? 8 : lift_res);
  int gl = num_sms() * lper;
  if (gl > lt) gl = lt;
  k_lift<EQ, N><<<gl, kThreads, LT::BYTES, s>>>(d, a);
  return cudaGetLastError();
}

template <int EQ>
cudaError_t lift_dispatch_n(const DgDev& d, const StageArgs& a, cudaStream_t s) {
  switch (d.N) {
    case 2: return launch_lift_t<EQ, 2>(d, a, s);
    case 3: return launch_lift_t<EQ, 3>(d, a, s);
    case 4: return launch_lift_t<EQ, 4>(d, a, s);
    case 5: return launch_lift_t<EQ, 5>(d, a, s);
    default: return cudaErrorInvalidValue;
  }
}

template <int EQ>
cudaError_t dispatch_n(const DgDev& d, const StageArgs& a, cudaStream_t s, cudaEvent_t* ev) {
  switch (d.N) {
    case 2: return launch_rhs_t<EQ, 2>(d, a, s, ev);
    case 3: return launch_rhs_t<EQ, 3>(d, a, s, ev);
    case 4: return launch_rhs_t<EQ, 4>(d, a, s, ev);
    case 5: return launch_rhs_t<EQ, 5>(d, a, s, ev);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace

int device_sms() { return num_sms(); }

static int eq_fields(int eq) {
  switch (eq) {
    case EQ_ADVECTION: return 1;
    case EQ_EULER: return 5;
    case EQ_MAXWELL: return 8;
    case EQ_EULER2D: return 4;
    default: return 3;
  }
}

int fp64_supported(int eq, int N) { return eq >= 0 && eq <= 4 && N >= 2 && N <= 5; }

// The fused stage where it applies: an output that does not overlap the input
// (it reads the neighbours' states while other warps write theirs), and arrays
// that start on a 16-byte boundary (its copies and vector accesses).  The
// rule knows no mesh size or flux, so that batches and partitions compute the
// whole mesh's bits.  A right-hand side, three kernels and fused: Euler N = 2,
// K = 130,050 168 and 87 us, N = 5 572 and 329; 8 fields N = 3, K = 32,258 129
// and 39; K = 2,048, 16,200 and 50,562 with 5 fields, N = 3: HLL 43, 94, 260 and
// 24, 40, 84; Roe 38, 84, 213 and 24, 40, 83; Wave 47, 106, 306 and 25, 38, 77.  Over
// fluxes, orders and field counts it takes 0.84 of the three kernels' time at most;
// with floored states on meshes below a wave of tiles about their time.
static bool fused_applies(int eq, const DgDev& d, const StageArgs& a) {
  if (d.fp64_fused == 0) return false;
  if (d.fp64_fused == 2 && (d.K + 7) / 8 > stage64_wave_tiles(eq, d, num_sms())) return false;
  if (((uintptr_t)a.x | (uintptr_t)a.out | (uintptr_t)a.u0) % 16) return false;
  const size_t nbytes = (size_t)d.K * ((d.N + 1) * (d.N + 2) / 2) * eq_fields(eq) * sizeof(double);
  const char *xb = (const char*)a.x, *ob = (const char*)a.out;
  return ob + nbytes <= xb || xb + nbytes <= ob;
}

cudaError_t launch_rhs_fp64(int eq, const DgDev& d, const StageArgs& a, cudaStream_t s, cudaEvent_t* ev) {
  if (fused_applies(eq, d, a)) {
    if (ev) cudaEventRecord(ev[0], s);
    cudaError_t e = cudaSuccess;
    if (a.reset_lambda && a.mode == MODE_RHS) e = launch_reset_lambda(d, s);
    if (e == cudaSuccess) e = launch_stage64(eq, d, a, nullptr, 0, s);
    if (ev)
      for (int i = 1; i < 4; ++i) cudaEventRecord(ev[i], s);
    return e;
  }
  switch (eq) {
    case EQ_ADVECTION: return dispatch_n<EQ_ADVECTION>(d, a, s, ev);
    case EQ_EULER: return dispatch_n<EQ_EULER>(d, a, s, ev);
    case EQ_MAXWELL: return dispatch_n<EQ_MAXWELL>(d, a, s, ev);
    case EQ_EULER2D: return dispatch_n<EQ_EULER2D>(d, a, s, ev);
    case EQ_MAXWELL_TM: return dispatch_n<EQ_MAXWELL_TM>(d, a, s, ev);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_source(int eq, const DgDev& d, const StageArgs& a, double* dst, int accumulate, cudaStream_t s) {
  switch (eq) {
    case EQ_ADVECTION: return source_dispatch<EQ_ADVECTION>(d, a, dst, accumulate, s);
    case EQ_EULER: return source_dispatch<EQ_EULER>(d, a, dst, accumulate, s);
    case EQ_MAXWELL: return source_dispatch<EQ_MAXWELL>(d, a, dst, accumulate, s);
    case EQ_EULER2D: return source_dispatch<EQ_EULER2D>(d, a, dst, accumulate, s);
    case EQ_MAXWELL_TM: return source_dispatch<EQ_MAXWELL_TM>(d, a, dst, accumulate, s);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_lift_fp64(int eq, const DgDev& d, const StageArgs& a, cudaStream_t s) {
  switch (eq) {
    case EQ_ADVECTION: return lift_dispatch_n<EQ_ADVECTION>(d, a, s);
    case EQ_EULER: return lift_dispatch_n<EQ_EULER>(d, a, s);
    case EQ_MAXWELL: return lift_dispatch_n<EQ_MAXWELL>(d, a, s);
    case EQ_EULER2D: return lift_dispatch_n<EQ_EULER2D>(d, a, s);
    case EQ_MAXWELL_TM: return lift_dispatch_n<EQ_MAXWELL_TM>(d, a, s);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_init_speed(int eq, const DgDev& d, const double* u, cudaStream_t s) {
  const int np = (d.N + 1) * (d.N + 2) / 2;
  const int nn = d.K * np;
  int g = (nn + 255) / 256;
  if (g > num_sms() * 8) g = num_sms() * 8;
  if (g < 1) g = 1;
  switch (eq) {
    case EQ_ADVECTION: k_init_speed<EQ_ADVECTION><<<g, 256, 0, s>>>(d, u, nn); break;
    case EQ_EULER: k_init_speed<EQ_EULER><<<g, 256, 0, s>>>(d, u, nn); break;
    case EQ_MAXWELL: k_init_speed<EQ_MAXWELL><<<g, 256, 0, s>>>(d, u, nn); break;
    case EQ_EULER2D: k_init_speed<EQ_EULER2D><<<g, 256, 0, s>>>(d, u, nn); break;
    case EQ_MAXWELL_TM: k_init_speed<EQ_MAXWELL_TM><<<g, 256, 0, s>>>(d, u, nn); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

__global__ void k_reset_lambda(DevState* st, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) st[i].lam_bits = 0ull;
}

cudaError_t launch_finalize(const DgDev& d, cudaStream_t s, bool overlap) {
  return launch_kernel(k_finalize, (d.ninst + 127) / 128, 128, 0, s, overlap, d);
}

cudaError_t launch_reset_lambda(const DgDev& d, cudaStream_t s) {
  k_reset_lambda<<<(d.ninst + 127) / 128, 128, 0, s>>>(d.st, d.ninst);
  return cudaGetLastError();
}

// the value travels as a kernel argument, captured at launch: the caller's
// host copy may change before the stream reaches the write
__global__ void k_put_state(DevState* st, DevState v) {
  if (threadIdx.x == 0 && blockIdx.x == 0) *st = v;
}

cudaError_t launch_put_state(DevState* st, const DevState& v, cudaStream_t s) {
  k_put_state<<<1, 32, 0, s>>>(st, v);
  return cudaGetLastError();
}

cudaError_t launch_integrals(int eq, const DgDev& d, const double* u, const double* wmass, cudaStream_t s) {
  const int np = (d.N + 1) * (d.N + 2) / 2;
  int g = (d.K + 255) / 256;
  if (g > num_sms() * 4) g = num_sms() * 4;
  if (g < 1) g = 1;
  switch (eq) {
    case EQ_ADVECTION: k_integrals<EQ_ADVECTION><<<g, 256, 0, s>>>(d, u, wmass, np); break;
    case EQ_EULER: k_integrals<EQ_EULER><<<g, 256, 0, s>>>(d, u, wmass, np); break;
    case EQ_MAXWELL: k_integrals<EQ_MAXWELL><<<g, 256, 0, s>>>(d, u, wmass, np); break;
    case EQ_EULER2D: k_integrals<EQ_EULER2D><<<g, 256, 0, s>>>(d, u, wmass, np); break;
    case EQ_MAXWELL_TM: k_integrals<EQ_MAXWELL_TM><<<g, 256, 0, s>>>(d, u, wmass, np); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launch_energy(int eq, const DgDev& d, const double* u, const double* mass, cudaStream_t s) {
  const int np = (d.N + 1) * (d.N + 2) / 2;
  int g = (d.K + 127) / 128;
  if (g > num_sms() * 8) g = num_sms() * 8;
  if (g < 1) g = 1;
  switch (eq) {
    case EQ_ADVECTION: k_energy<EQ_ADVECTION><<<g, 128, 0, s>>>(d, u, mass, np); break;
    case EQ_EULER: k_energy<EQ_EULER><<<g, 128, 0, s>>>(d, u, mass, np); break;
    case EQ_MAXWELL: k_energy<EQ_MAXWELL><<<g, 128, 0, s>>>(d, u, mass, np); break;
    case EQ_EULER2D: k_energy<EQ_EULER2D><<<g, 128, 0, s>>>(d, u, mass, np); break;
    case EQ_MAXWELL_TM: k_energy<EQ_MAXWELL_TM><<<g, 128, 0, s>>>(d, u, mass, np); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

}  // namespace apollo
