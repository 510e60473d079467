// Tangent and adjoint of one float64 stage in the fragment chain of
// dg_stage64.cu (a warp per eight elements, the fields of a point in one lane,
// contractions chained in registers), for the Lax-Friedrichs and the linear
// equations' fluxes; Apollo's HLL, Roe and Wave fluxes keep the general kernels
// of dg_adjoint.cu.
//
// Adjoint: the lift is V V^T I^T, so with y = -(1/J) V V^T w per element
// (k_adj_y) the weighted lifted adjoint at a face point is the trace of y, and a
// neighbour contributes the N + 1 nodes of the shared face of x and of y, as in
// the forward stage.  One pass then holds [Dr Ds]^T w, the transposed flux
// Jacobians, V^T, the face terms and the stage combination
// out = alpha w + beta L'(x)^T w + gamma z.  Every supported boundary state is
// affine in the trace with a symmetric matrix A (mirror, copy or constant), so
// A^T v is the boundary hook at v minus the hook at zero.
//
// Tangent: the forward stage on the pair (x, v).
//
// What bounds them: the float64 pipe and the latency of the pointwise
// derivatives, as the forward stage (Euler N = 3, K = 32,258: 53 % of the pipe
// busy).  Euler N = 3, K = 32,258, before (trace and face kernels of their own,
// block-wide contractions) and now: adjoint right-hand side 22 + 120 and
// 10 + 51 us, tangent 57 + 43 us and the LIFT kernel, and 53 us.
#include <cuda_runtime.h>

#include "dg_adjoint.h"
#include "dg_chain64.cuh"
#include "dg_dmma.cuh"
#include "dg_dual.cuh"
#include "dg_euler_adj.cuh"
#include "dg_flux64.cuh"
#include "dg_stage64.h"

namespace apollo {

namespace {

// Shared memory of the two kernels (doubles).  Per warp: arrays A and B are
// x and y (adjoint) or x and v (tangent), with the neighbours' face nodes; the
// linear equations need only the second.
template <int EQ, int N> struct Deriv {
  static constexpr int M = Eq<EQ>::M;
  static constexpr int NP = Sizes<N>::NP, NG = Sizes<N>::NG, NF = Sizes<N>::NF;
  static constexpr bool LIN = kLinearEq<EQ>;
  using P = Pack64<N>;
  static constexpr int ADJ_OPS = LIN ? P::W_SIZE + P::Q_SIZE : P::E_SIZE + P::V_SIZE + P::DT_SIZE + P::VT_SIZE + P::ET_SIZE;
  static constexpr int TAN_OPS = LIN ? P::S_OFF - P::Q_OFF : P::Q_OFF;
  static constexpr int TABS = NG + (3 * (N + 1) + 1) / 2;
  static constexpr int ES = elem_stride(NP * M, M), FS = face_stride(3 * (N + 1) * M, M);
  static constexpr int X = 8 * ES, PN = 8 * FS, G = 8 * kGeoStride, C = 24;
  static constexpr int WARP = (LIN ? 1 : 2) * (X + PN) + G + C;
  static constexpr size_t bytes(int ops, int warps) {
    return sizeof(double) * (size_t)(round_up(ops + TABS, 2) + warps * WARP);
  }
  static constexpr int fit(int ops, int w) { return bytes(ops, w) <= 227 * 1024 ? w : fit(ops, w - 1); }
  // Eight warps have 255 registers a lane; the Euler tangent still spills 16 to 52
  // bytes (4 fields, orders 3-5) and 72 to 168 (5 fields), the adjoint of 5 and of 8
  // fields at order 5 some 155.  Twelve have 168, and the Euler kernels then
  // spill 40 to 470 bytes a lane: the gradient of ten steps, N = 3,
  // K = 6,962 2,605 us with twelve and 2,192 with eight, N = 4, K = 32,258 9,495
  // and 8,990, N = 3, K = 32,258 6,000 and 5,890.  The linear equations (but for
  // eight fields) fit in 168.
  static constexpr int WMAX = LIN && M != 8 ? 12 : 8;
  static constexpr int ADJ_WARPS = fit(ADJ_OPS, WMAX), TAN_WARPS = fit(TAN_OPS, WMAX);
};

// y = -(1/J) V V^T w
template <int M, int N>
__global__ void __launch_bounds__(128) k_adj_y(DgDev d, const double* __restrict__ w, double* __restrict__ y) {
  using PK = Pack64<N>;
  constexpr int NP = PK::NP;
  const int lane = threadIdx.x & 31, lr = lane >> 2, lc = lane & 3;
  const int row = (blockIdx.x * 4 + (threadIdx.x >> 5)) * 8 + lr;
  const int k = min(row, d.K - 1);
  allow_next();
  wait_previous();
  const double* we = w + (size_t)k * NP * M;
  const double s = -d.geo[k].invJ;
  Nodes<M, PK> acc;
  acc.zero();
#pragma unroll
  for (int ks = 0; ks < PK::KS; ++ks) {
    const int node = min(PK::node(ks, lc), NP - 1);  // past the last node the operator is zero
    double q[M];
#pragma unroll
    for (int f = 0; f < M; ++f) q[f] = we[node * M + f];
    acc.add1(d.pack64 + PK::Y_OFF + ks * PK::NS, lane, q);
  }
  acc.finish();
  if (row >= d.K) return;
#pragma unroll
  for (int b = 0; b < PK::NBT; ++b) {
    double v[M][2];
    acc.get(b, lc, v);
#pragma unroll
    for (int f = 0; f < M; ++f) {
      v[f][0] *= s;
      v[f][1] *= s;
    }
    store_block<M, PK>(y + (size_t)k * NP * M, b, lc, v);
  }
}

// The face nodes of array x that the tile's elements see across their faces,
// in this side's order, into dst [8][FS] (a boundary face: its own).
template <int N, int M, int FS>
__device__ __forceinline__ void copy_face_nodes(double* dst, const double* __restrict__ x, const int2* sC,
                                                const int* sFm, int ke, int lr, int lc) {
  using PK = Pack64<N>;
#pragma unroll
  for (int fc = 0; fc < 3; ++fc) {
    const int2 cn = sC[lr * 3 + fc];
    const double* from = x + (size_t)(cn.y < 0 ? ke : cn.x) * PK::NP * M;
#pragma unroll
    for (int k = 0; k < (N + 4) / 4; ++k) {
      const int m = 4 * k + lc;
      if (m > N) continue;
      cp_async_node<M>(dst + lr * FS + (fc * (N + 1) + m) * M,
                       from + sFm[cn.y < 0 ? fc * (N + 1) + m : cn.y * (N + 1) + N - m] * M);
    }
  }
}

// What both kernels share: the operator copy, the tile's copies, boundary
// states and the final contraction.
template <int EQ, int N> struct Warp {
  using T = Deriv<EQ, N>;
  using PK = Pack64<N>;
  static constexpr int M = T::M, NP = T::NP;
  int lane, lr, lc;
  double *sGz, *sA, *sB, *sPA, *sPB, *sG;
  int* sFm;
  int2* sC;

  __device__ __forceinline__ void init(const DgDev& d, double* smem, int ops) {
    const int tid = threadIdx.x;
    lane = tid & 31;
    lr = lane >> 2;
    lc = lane & 3;
    sGz = smem + ops;
    sFm = (int*)(sGz + T::NG);
    double* w = smem + round_up(ops + T::TABS, 2) + (tid >> 5) * T::WARP;
    sB = w;
    sPB = sB + T::X;
    sG = sPB + T::PN;
    sC = (int2*)(sG + T::G);
    sA = sG + T::G + T::C;
    sPA = sA + T::X;
    for (int i = tid; i < T::NG; i += blockDim.x) sGz[i] = d.gz[i];
    for (int i = tid; i < PK::NFN; i += blockDim.x) sFm[i] = PK::face_node(i / (N + 1), i % (N + 1));
  }
  // lane's entry of a tile's connectivity
  __device__ __forceinline__ int2 load_conn(const DgDev& d, int tile) const {
    const int l = min(lane, 23);
    return *reinterpret_cast<const int2*>(d.conn + (size_t)min(tile * 8 + l / 3, d.K - 1) * 6 + 2 * (l % 3));
  }
  // a tile's own arrays; the neighbours' nodes arrive during the volume term
  // (faces_here), and the next tile's connectivity replaces conn
  __device__ __forceinline__ void load(const DgDev& d, int tile, const double* a, const double* b) {
    const int ke = min(tile * 8 + lr, d.K - 1);
    __syncwarp();  // the previous tile's reads are done
    if (lane < 24) sC[lane] = load_conn(d, tile);
    copy_tile<NP * M, T::ES>(sB, b, tile, d.K, lane);
    if (!T::LIN) copy_tile<NP * M, T::ES>(sA, a, tile, d.K, lane);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int i = lane + 32 * u, e = i >> 3, q = i & 7;
      cp_async16(sG + kGeoStride * e + 2 * q, reinterpret_cast<const double*>(d.geo + min(tile * 8 + e, d.K - 1)) + 2 * q);
    }
    cp_async_commit();
    __syncwarp();
    copy_face_nodes<N, M, T::FS>(sPB, b, sC, sFm, ke, lr, lc);
    if (!T::LIN) copy_face_nodes<N, M, T::FS>(sPA, a, sC, sFm, ke, lr, lc);
    cp_async_commit();
    cp_async_wait<1>();
    __syncwarp();
  }
  __device__ __forceinline__ void faces_here() const {
    cp_async_wait<0>();
    __syncwarp();
  }
  // boundary hook of face fc at face coordinate z
  __device__ __forceinline__ void hook(const DgDev& d, int ke, int tag, int fc, double z, double t, const double* q,
                                       double* qb) const {
    const ElemGeo& g = d.geo[ke];
    const double* ge = sG + kGeoStride * lr;
    const double r = fc == 0 ? z : fc == 1 ? -z : -1.0;
    const double s = fc == 0 ? -1.0 : fc == 1 ? z : -z;
    const double x = 0.5 * (-g.vx[0] * (r + s) + g.vx[1] * (1. + r) + g.vx[2] * (1. + s));
    const double y = 0.5 * (-g.vy[0] * (r + s) + g.vy[1] * (1. + r) + g.vy[2] * (1. + s));
    apply_bc<EQ, double>(d.bcs, tag, t, x, y, ge[6 + fc], ge[9 + fc], q, qb);
  }
  // its linear part at v
  __device__ __forceinline__ void hook_linear(const DgDev& d, int ke, int tag, int fc, double z, double t,
                                              const double* v, double* out) const {
    double zero[M], base[M];
#pragma unroll
    for (int f = 0; f < M; ++f) zero[f] = 0.0;
    hook(d, ke, tag, fc, z, t, zero, base);
    hook(d, ke, tag, fc, z, t, v, out);
#pragma unroll
    for (int f = 0; f < M; ++f) out[f] -= base[f];
  }
  // V q at block pb's two points of this lane
  __device__ __forceinline__ void to_points(const double* sV, int pb, const double* e, double (*q)[M]) const {
    double v[M][2];
#pragma unroll
    for (int k = 0; k < PK::KS; k += 2) {
      const double2 w = reinterpret_cast<const double2*>(sV)[(pb * ((PK::KS + 1) / 2) + k / 2) * 32 + lane];
      const int n0 = min(PK::node(k, lc), NP - 1), n1 = min(PK::node(k + 1, lc), NP - 1);
#pragma unroll
      for (int f = 0; f < M; ++f) {
        if (k == 0) dmma_8x8x4_first(v[f], e[n0 * M + f], w.x);
        else dmma_8x8x4(v[f], e[n0 * M + f], w.x);
      }
      if (k + 1 < PK::KS) {
#pragma unroll
        for (int f = 0; f < M; ++f) dmma_8x8x4(v[f], e[n1 * M + f], w.y);
      }
    }
#pragma unroll
    for (int f = 0; f < M; ++f) {
      q[0][f] = v[f][0];
      q[1][f] = v[f][1];
    }
  }
};

template <int EQ, int N>
__global__ void __launch_bounds__(32 * Deriv<EQ, N>::ADJ_WARPS, 1) k_adjoint64(DgDev d, AdjArgs a, const double* __restrict__ y) {
  using T = Deriv<EQ, N>;
  using PK = Pack64<N>;
  constexpr int M = T::M, NP = T::NP, NG = T::NG, NF = T::NF, KS = PK::KS;
  extern __shared__ __align__(16) double smem[];
  // operators: WT | Z, or E | V | DT | VT | ET
  double *sE = smem, *sV = sE + PK::E_SIZE, *sDT = sV + PK::V_SIZE, *sVT = sDT + PK::DT_SIZE, *sET = sVT + PK::VT_SIZE;
  double *sWT = smem, *sZ = sWT + PK::W_SIZE;
  auto stage = [&](double* dst, int off, int size) {
    for (int i = 2 * threadIdx.x; i < size; i += 2 * blockDim.x) cp_async16(dst + i, d.pack64 + off + i);
  };
  if constexpr (T::LIN) {
    stage(sWT, PK::WT_OFF, PK::W_SIZE);
    stage(sZ, PK::Z_OFF, PK::Q_SIZE);
  } else {
    stage(sE, PK::E_OFF, PK::E_SIZE);
    stage(sV, PK::V_OFF, PK::V_SIZE);
    stage(sDT, PK::DT_OFF, PK::DT_SIZE);
    stage(sVT, PK::VT_OFF, PK::VT_SIZE);
    stage(sET, PK::ET_OFF, PK::ET_SIZE);
  }
  Warp<EQ, N> W;
  W.init(d, smem, T::ADJ_OPS);
  allow_next();
  const int stride = gridDim.x * (blockDim.x >> 5), first = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
  cp_async_wait_all();
  __syncthreads();
  wait_previous();
  const int lane = W.lane, lr = W.lr, lc = W.lc;
  int err = 0;  // the float64 forward reports non-physical states
  const int ntiles = (d.K + 7) / 8;
  for (int tile = first; tile < ntiles; tile += stride) {
    const int ke = min(tile * 8 + lr, d.K - 1);
    double wv[PK::NBT][M][2];
#pragma unroll
    for (int b = 0; b < PK::NBT; ++b) load_block<M, PK>(a.wbar + (size_t)ke * NP * M, b, lc, wv[b]);
    W.load(d, tile, a.x, y);
    const double *ge = W.sG + kGeoStride * lr, *xe = W.sA + lr * T::ES, *ye = W.sB + lr * T::ES;
    const double rx = ge[0], ry = ge[1], sx = ge[2], sy = ge[3];
    Nodes<M, PK> acc;
    acc.zero();
    if constexpr (T::LIN) {
#pragma unroll
      for (int k = 0; k < KS; ++k) {
        double w[M], u[M], z[M];
#pragma unroll
        for (int f = 0; f < M; ++f) w[f] = wv[k / 2][f][k % 2];
        LinearFast64<EQ>::along_t(d.eqp, w, rx, ry, u);
        LinearFast64<EQ>::along_t(d.eqp, w, sx, sy, z);
        acc.add(sWT + k * PK::NS, lane, u, z);
      }
      // at the face nodes: sJ (y_own - y_partner) through the flux Jacobian
      W.faces_here();
#pragma unroll 1
      for (int qb = 0; qb < PK::QB; ++qb) {
        double A[2][M];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int p = min(qb * 8 + 2 * lc + j, PK::NFN - 1), fc = p / (N + 1);
          const double *om = ye + W.sFm[p] * M, *pm = W.sPB + lr * T::FS + p * M;
          const double nx = ge[6 + fc], ny = ge[9 + fc], hs = 0.5 * ge[12 + fc];
          const int2 cn = W.sC[lr * 3 + fc];
          double dv[M], t[M];
#pragma unroll
          for (int f = 0; f < M; ++f) dv[f] = hs * (cn.y < 0 ? om[f] : om[f] - pm[f]);
          LinearFast64<EQ>::along_t(d.eqp, dv, nx, ny, A[j]);
          LinearFast64<EQ>::dissipate(d.eqp, nx, ny, dv, t);
          if (cn.y < 0) {
            double bb[M], ab[M];
#pragma unroll
            for (int f = 0; f < M; ++f) bb[f] = A[j][f] - t[f];
            W.hook_linear(d, ke, -cn.x, fc, 0.0, a.t, bb, ab);
#pragma unroll
            for (int f = 0; f < M; ++f) A[j][f] += ab[f];
          }
#pragma unroll
          for (int f = 0; f < M; ++f) A[j][f] += t[f];
        }
        acc.add(sZ + (qb) * PK::NS, lane, A[0], A[1]);
      }
    } else {
      using X = EulerFast64<M>;
#pragma unroll 1
      for (int pb = 0; pb < PK::PB; ++pb) {
        double q[2][M], r[M][2], s[M][2], g[2][M];
        W.to_points(sV, pb, xe, q);
#pragma unroll
        for (int k = 0; k < KS; ++k) {
          const double2 op = reinterpret_cast<const double2*>(sDT)[(pb * KS + k) * 32 + lane];
#pragma unroll
          for (int f = 0; f < M; ++f) {
            if (k == 0) dmma_8x8x4_first(r[f], wv[0][f][0], op.x);
            else dmma_8x8x4(r[f], wv[k / 2][f][k % 2], op.x);
          }
#pragma unroll
          for (int f = 0; f < M; ++f) {
            if (k == 0) dmma_8x8x4_first(s[f], wv[0][f][0], op.y);
            else dmma_8x8x4(s[f], wv[k / 2][f][k % 2], op.y);
          }
        }
        double aR[2][M], aS[2][M];
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int f = 0; f < M; ++f) {
            aR[j][f] = r[f][j];
            aS[j][f] = s[f][j];
          }
        const typename X::Side s0 = X::side(d.eqp, q[0]), s1 = X::side(d.eqp, q[1]);
        if (s0.clean && s1.clean) {
          X::vol_t(d.eqp, s0, q[0], rx, ry, sx, sy, aR[0], aS[0], g[0]);
          X::vol_t(d.eqp, s1, q[1], rx, ry, sx, sy, aR[1], aS[1], g[1]);
        } else {
#pragma unroll
          for (int j = 0; j < 2; ++j) {
#pragma unroll
            for (int f = 0; f < M; ++f) g[j][f] = 0.0;
            EulerAdj<M>::dir(d.eqp, q[j], rx, ry, aR[j], g[j], &err);
            EulerAdj<M>::dir(d.eqp, q[j], sx, sy, aS[j], g[j], &err);
          }
        }
        acc.add(sVT + (pb) * PK::NS, lane, g[0], g[1]);
      }
      W.faces_here();
#pragma unroll 1
      for (int fb = 0; fb < PK::FB; ++fb) {
        const int p0 = min(fb * 8 + 2 * lc, NF - 2), fc = p0 / NG, g0 = p0 - fc * NG;
        const int2 cn = W.sC[lr * 3 + fc];
        const bool wall = cn.y < 0;
        double qM[2][M], qP[2][M], dv[2][M], A[2][M];
        const double2* se = reinterpret_cast<const double2*>(sE) + fb * (N + 1) * 4 + lc;
        const int face = lr * T::FS + fc * (N + 1) * M;
        const double hs = 0.5 * ge[12 + fc], nx = ge[6 + fc], ny = ge[9 + fc];
#pragma unroll
        for (int m = 0; m <= N; ++m) {
          const double2 w = se[m * 4];
          const int node = W.sFm[fc * (N + 1) + m] * M;
#pragma unroll
          for (int f = 0; f < M; ++f) {
            const double o = xe[node + f], p = W.sPA[face + m * M + f];
            const double u = wall ? ye[node + f] : ye[node + f] - W.sPB[face + m * M + f];
            qM[0][f] = m == 0 ? w.x * o : fma(w.x, o, qM[0][f]);
            qM[1][f] = m == 0 ? w.y * o : fma(w.y, o, qM[1][f]);
            qP[0][f] = m == 0 ? w.x * p : fma(w.x, p, qP[0][f]);
            qP[1][f] = m == 0 ? w.y * p : fma(w.y, p, qP[1][f]);
            dv[0][f] = m == 0 ? w.x * u : fma(w.x, u, dv[0][f]);
            dv[1][f] = m == 0 ? w.y * u : fma(w.y, u, dv[1][f]);
          }
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) {
#pragma unroll
          for (int f = 0; f < M; ++f) dv[j][f] *= hs;
          if (wall) W.hook(d, ke, -cn.x, fc, W.sGz[g0 + j], a.t, qM[j], qP[j]);
        }
        const typename X::Side a0 = X::side(d.eqp, qM[0]), b0 = X::side(d.eqp, qP[0]);
        const typename X::Side a1 = X::side(d.eqp, qM[1]), b1 = X::side(d.eqp, qP[1]);
        double bb[2][M];
        if (a0.clean && b0.clean && a1.clean && b1.clean) {
          X::lf2_t(d.eqp, a0, b0, qM[0], qP[0], nx, ny, dv[0], wall, A[0], bb[0]);
          X::lf2_t(d.eqp, a1, b1, qM[1], qP[1], nx, ny, dv[1], wall, A[1], bb[1]);
        } else {
#pragma unroll
          for (int j = 0; j < 2; ++j) EulerAdj<M>::lf2_t(d.eqp, nx, ny, qM[j], qP[j], dv[j], A[j], bb[j], wall, &err);
        }
        if (wall) {
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            double ab[M];
            W.hook_linear(d, ke, -cn.x, fc, W.sGz[g0 + j], a.t, bb[j], ab);
#pragma unroll
            for (int f = 0; f < M; ++f) A[j][f] += ab[f];
          }
        }
        acc.add(sET + (fb) * PK::NS, lane, A[0], A[1]);
      }
    }
    acc.finish();
    if (tile * 8 + lr < d.K) {
      const size_t off = (size_t)ke * NP * M;
#pragma unroll
      for (int b = 0; b < PK::NBT; ++b) {
        double o[M][2];
        acc.get(b, lc, o);
#pragma unroll
        for (int f = 0; f < M; ++f)
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            o[f][j] *= a.beta;
            if (a.alpha != 0.0) o[f][j] += a.alpha * wv[b][f][j];
          }
        if (a.z) {
          double z[M][2];
          load_block<M, PK>(a.z + off, b, lc, z);
#pragma unroll
          for (int f = 0; f < M; ++f)
#pragma unroll
            for (int j = 0; j < 2; ++j) o[f][j] += a.gamma * z[f][j];
        }
        store_block<M, PK>(a.out + off, b, lc, o);
      }
    }
  }
  (void)err;
}

template <int EQ, int N>
__global__ void __launch_bounds__(32 * Deriv<EQ, N>::TAN_WARPS, 1) k_tangent64(DgDev d, TanArgs a) {
  using T = Deriv<EQ, N>;
  using PK = Pack64<N>;
  constexpr int M = T::M, NP = T::NP, NG = T::NG, NF = T::NF, KS = PK::KS;
  extern __shared__ __align__(16) double smem[];
  for (int i = 2 * threadIdx.x; i < T::TAN_OPS; i += 2 * blockDim.x)
    cp_async16(smem + i, d.pack64 + (T::LIN ? PK::Q_OFF : PK::E_OFF) + i);
  Warp<EQ, N> W;
  W.init(d, smem, T::TAN_OPS);
  allow_next();
  const int stride = gridDim.x * (blockDim.x >> 5), first = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
  cp_async_wait_all();
  __syncthreads();
  wait_previous();
  const int lane = W.lane, lr = W.lr, lc = W.lc;
  // reported: a non-physical state at a cubature point and a NaN in the result
  // (at the face points the forward stage reports them)
  int err = 0, face_err = 0;
  const int ntiles = (d.K + 7) / 8;
  for (int tile = first; tile < ntiles; tile += stride) {
    const int ke = min(tile * 8 + lr, d.K - 1);
    W.load(d, tile, a.x, a.dx);
    const double *ge = W.sG + kGeoStride * lr, *xe = W.sA + lr * T::ES, *de = W.sB + lr * T::ES;
    const double rx = ge[0], ry = ge[1], sx = ge[2], sy = ge[3], miJ = -0.5 * ge[5];
    Nodes<M, PK> acc;
    acc.zero();
    if constexpr (T::LIN) {
      const double *sQ = smem, *sW = smem + PK::Q_SIZE;
#pragma unroll
      for (int k = 0; k < KS; ++k) {
        const int node = min(PK::node(k, lc), NP - 1);  // past the last node the operator is zero
        double q[M], R[M], S[M];
#pragma unroll
        for (int f = 0; f < M; ++f) q[f] = de[node * M + f];
        LinearFast64<EQ>::along(d.eqp, q, rx, ry, R);
        LinearFast64<EQ>::along(d.eqp, q, sx, sy, S);
        acc.add(sW + k * PK::NS, lane, R, S);
      }
      W.faces_here();
#pragma unroll 1
      for (int qb = 0; qb < PK::QB; ++qb) {
        double A[2][M];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int p = min(qb * 8 + 2 * lc + j, PK::NFN - 1), fc = p / (N + 1);
          const double *om = de + W.sFm[p] * M, *pm = W.sPB + lr * T::FS + p * M;
          double qM[M], qP[M];
#pragma unroll
          for (int f = 0; f < M; ++f) {
            qM[f] = om[f];
            qP[f] = pm[f];
          }
          const int2 cn = W.sC[lr * 3 + fc];
          if (cn.y < 0) W.hook_linear(d, ke, -cn.x, fc, 0.0, a.t, qM, qP);
          LinearFast64<EQ>::face2(d.eqp, ge[6 + fc], ge[9 + fc], miJ * ge[12 + fc], qM, qP, A[j]);
        }
        acc.add(sQ + (qb) * PK::NS, lane, A[0], A[1]);
      }
    } else {
      using X = EulerFast64<M>;
      const double *sE = smem, *sL = smem + PK::L_OFF, *sV = smem + PK::V_OFF, *sD = smem + PK::D_OFF;
#pragma unroll 1
      for (int pb = 0; pb < PK::PB; ++pb) {
        double q[2][M], v[2][M], R[2][M], S[2][M];
        W.to_points(sV, pb, xe, q);
        W.to_points(sV, pb, de, v);
        const typename X::Side s0 = X::side(d.eqp, q[0]), s1 = X::side(d.eqp, q[1]);
        if (s0.clean && s1.clean) {
          const typename X::Rate r0 = X::rate(d.eqp, s0, v[0]), r1 = X::rate(d.eqp, s1, v[1]);
          X::along_d(s0, r0, q[0], v[0], rx, ry, R[0]);
          X::along_d(s1, r1, q[1], v[1], rx, ry, R[1]);
          X::along_d(s0, r0, q[0], v[0], sx, sy, S[0]);
          X::along_d(s1, r1, q[1], v[1], sx, sy, S[1]);
        } else {
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            Dual<1> qc[M], F[M], G[M];
#pragma unroll
            for (int f = 0; f < M; ++f) {
              qc[f].v = q[j][f];
              qc[f].d[0] = v[j][f];
            }
            Eq<EQ>::flux2(d.eqp, qc, F, G, &err);
#pragma unroll
            for (int f = 0; f < M; ++f) {
              R[j][f] = rx * F[f].d[0] + ry * G[f].d[0];
              S[j][f] = sx * F[f].d[0] + sy * G[f].d[0];
            }
          }
        }
        acc.add(sD + (pb * 2) * PK::NS, lane, R[0], R[1]);
        acc.add(sD + (pb * 2 + 1) * PK::NS, lane, S[0], S[1]);
      }
      W.faces_here();
#pragma unroll 1
      for (int fb = 0; fb < PK::FB; ++fb) {
        const int p0 = min(fb * 8 + 2 * lc, NF - 2), fc = p0 / NG, g0 = p0 - fc * NG;
        const int2 cn = W.sC[lr * 3 + fc];
        double qM[2][M], qP[2][M], dM[2][M], dP[2][M], A[2][M];
        const double2* se = reinterpret_cast<const double2*>(sE) + fb * (N + 1) * 4 + lc;
        const int face = lr * T::FS + fc * (N + 1) * M;
        const double w = miJ * ge[12 + fc], nx = ge[6 + fc], ny = ge[9 + fc];
#pragma unroll
        for (int m = 0; m <= N; ++m) {
          const double2 e = se[m * 4];
          const int node = W.sFm[fc * (N + 1) + m] * M;
#pragma unroll
          for (int f = 0; f < M; ++f) {
            const double o = xe[node + f], p = W.sPA[face + m * M + f], u = de[node + f], v = W.sPB[face + m * M + f];
            qM[0][f] = m == 0 ? e.x * o : fma(e.x, o, qM[0][f]);
            qM[1][f] = m == 0 ? e.y * o : fma(e.y, o, qM[1][f]);
            qP[0][f] = m == 0 ? e.x * p : fma(e.x, p, qP[0][f]);
            qP[1][f] = m == 0 ? e.y * p : fma(e.y, p, qP[1][f]);
            dM[0][f] = m == 0 ? e.x * u : fma(e.x, u, dM[0][f]);
            dM[1][f] = m == 0 ? e.y * u : fma(e.y, u, dM[1][f]);
            dP[0][f] = m == 0 ? e.x * v : fma(e.x, v, dP[0][f]);
            dP[1][f] = m == 0 ? e.y * v : fma(e.y, v, dP[1][f]);
          }
        }
        if (cn.y < 0) {
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            W.hook(d, ke, -cn.x, fc, W.sGz[g0 + j], a.t, qM[j], qP[j]);
            W.hook_linear(d, ke, -cn.x, fc, W.sGz[g0 + j], a.t, dM[j], dP[j]);
          }
        }
        const typename X::Side a0 = X::side(d.eqp, qM[0]), b0 = X::side(d.eqp, qP[0]);
        const typename X::Side a1 = X::side(d.eqp, qM[1]), b1 = X::side(d.eqp, qP[1]);
        if (a0.clean && b0.clean && a1.clean && b1.clean) {
          X::lf2_d(d.eqp, a0, b0, qM[0], qP[0], dM[0], dP[0], w * nx, w * ny, w, A[0]);
          X::lf2_d(d.eqp, a1, b1, qM[1], qP[1], dM[1], dP[1], w * nx, w * ny, w, A[1]);
        } else {
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            Dual<1> ma[M], pa[M], nf[M];
#pragma unroll
            for (int f = 0; f < M; ++f) {
              ma[f].v = qM[j][f];
              ma[f].d[0] = dM[j][f];
              pa[f].v = qP[j][f];
              pa[f].d[0] = dP[j][f];
            }
            Eq<EQ>::lf(d.eqp, Dual<1>(nx), Dual<1>(ny), ma, pa, nf, &face_err);
#pragma unroll
            for (int f = 0; f < M; ++f) A[j][f] = 2.0 * w * nf[f].d[0];
          }
        }
        acc.add(sL + (fb) * PK::NS, lane, A[0], A[1]);
      }
    }
    // the stage update's tangent
    acc.finish();
    if (tile * 8 + lr < d.K) {
      const size_t off = (size_t)ke * NP * M;
      const double c_r = a.mode == MODE_STAGE ? a.dt / 4.0 : a.dt / 5.0;
      int top = 0;  // as in k_stage64: above infinity's, a NaN
#pragma unroll
      for (int b = 0; b < PK::NBT; ++b) {
        double o[M][2];
        acc.get(b, lc, o);
#pragma unroll
        for (int f = 0; f < M; ++f) {
          top = max(top, __double2hiint(o[f][0]) & 0x7fffffff);
          top = max(top, __double2hiint(o[f][1]) & 0x7fffffff);
        }
        if (a.mode != MODE_RHS) {
          double x[M][2];
          load_block<M, PK>(de, b, lc, x);
          if (a.mode == MODE_STAGE) {
#pragma unroll
            for (int f = 0; f < M; ++f)
#pragma unroll
              for (int j = 0; j < 2; ++j) o[f][j] = x[f][j] + c_r * o[f][j];
          } else {
            double u[M][2];
            load_block<M, PK>(a.du0 + off, b, lc, u);
#pragma unroll
            for (int f = 0; f < M; ++f)
#pragma unroll
              for (int j = 0; j < 2; ++j) o[f][j] = (4.0 / 5.0) * x[f][j] + c_r * o[f][j] + (1.0 / 5.0) * u[f][j];
          }
        }
        store_block<M, PK>(a.dout + off, b, lc, o);
      }
      if (top > 0x7ff00000) err |= ERRB_NAN;
    }
  }
  (void)face_err;
  if (err) atomicOr(&d.st->err, err);
}

template <class Kern>
cudaError_t allow_smem(Kern k, size_t bytes, unsigned& configured) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (configured & (1u << (dev & 31))) return cudaSuccess;
  const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess) configured |= 1u << (dev & 31);
  return e;
}

// one block per SM with as many warps as its share of the tiles needs
void shape(int K, int wmax, int* grid, int* warps) {
  const int tiles = (K + 7) / 8, sms = device_sms();
  *grid = tiles < sms ? tiles : sms;
  *warps = (tiles + *grid - 1) / *grid;
  if (*warps > wmax) *warps = wmax;
}

template <int EQ, int N>
cudaError_t adjoint_t(const DgDev& d, const AdjArgs& a, cudaStream_t s) {
  using T = Deriv<EQ, N>;
  static unsigned configured = 0;
  cudaError_t e = allow_smem(k_adjoint64<EQ, N>, T::bytes(T::ADJ_OPS, T::ADJ_WARPS), configured);
  if (e != cudaSuccess) return e;
  e = launch_kernel(k_adj_y<T::M, N>, (d.K + 31) / 32, 128, 0, s, false, d, a.wbar, a.sbar);
  if (e != cudaSuccess) return e;
  int grid, warps;
  shape(d.K, T::ADJ_WARPS, &grid, &warps);
  return launch_kernel(k_adjoint64<EQ, N>, grid, 32 * warps, T::bytes(T::ADJ_OPS, warps), s, true, d, a, a.sbar);
}

template <int EQ, int N>
cudaError_t tangent_t(const DgDev& d, const TanArgs& a, cudaStream_t s) {
  using T = Deriv<EQ, N>;
  static unsigned configured = 0;
  const cudaError_t e = allow_smem(k_tangent64<EQ, N>, T::bytes(T::TAN_OPS, T::TAN_WARPS), configured);
  if (e != cudaSuccess) return e;
  int grid, warps;
  shape(d.K, T::TAN_WARPS, &grid, &warps);
  return launch_kernel(k_tangent64<EQ, N>, grid, 32 * warps, T::bytes(T::TAN_OPS, warps), s, false, d, a);
}

template <int EQ>
cudaError_t adjoint_n(const DgDev& d, const AdjArgs& a, cudaStream_t s) {
  switch (d.N) {
    case 2: return adjoint_t<EQ, 2>(d, a, s);
    case 3: return adjoint_t<EQ, 3>(d, a, s);
    case 4: return adjoint_t<EQ, 4>(d, a, s);
    case 5: return adjoint_t<EQ, 5>(d, a, s);
    default: return cudaErrorInvalidValue;
  }
}
template <int EQ>
cudaError_t tangent_n(const DgDev& d, const TanArgs& a, cudaStream_t s) {
  switch (d.N) {
    case 2: return tangent_t<EQ, 2>(d, a, s);
    case 3: return tangent_t<EQ, 3>(d, a, s);
    case 4: return tangent_t<EQ, 4>(d, a, s);
    case 5: return tangent_t<EQ, 5>(d, a, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace

cudaError_t launch_adjoint64(int eq, const DgDev& d, const AdjArgs& a, cudaStream_t s) {
  switch (eq) {
    case EQ_ADVECTION: return adjoint_n<EQ_ADVECTION>(d, a, s);
    case EQ_EULER: return adjoint_n<EQ_EULER>(d, a, s);
    case EQ_MAXWELL: return adjoint_n<EQ_MAXWELL>(d, a, s);
    case EQ_EULER2D: return adjoint_n<EQ_EULER2D>(d, a, s);
    case EQ_MAXWELL_TM: return adjoint_n<EQ_MAXWELL_TM>(d, a, s);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_tangent64(int eq, const DgDev& d, const TanArgs& a, cudaStream_t s) {
  switch (eq) {
    case EQ_ADVECTION: return tangent_n<EQ_ADVECTION>(d, a, s);
    case EQ_EULER: return tangent_n<EQ_EULER>(d, a, s);
    case EQ_MAXWELL: return tangent_n<EQ_MAXWELL>(d, a, s);
    case EQ_EULER2D: return tangent_n<EQ_EULER2D>(d, a, s);
    case EQ_MAXWELL_TM: return tangent_n<EQ_MAXWELL_TM>(d, a, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace apollo
