// The fused float64 stage: the volume and surface terms of a tile of elements
// and the SSP stage update in one pass, one tile of eight elements per warp.
//
// Fragment chain.  A warp's GEMM rows are its eight elements and every field
// has accumulators of its own, so a lane of mma.m8n8k4 holds, for element
// lane/4, all fields of the points (or nodes) 2 (lane%4) and 2 (lane%4) + 1 of
// a block of eight: the pointwise flux needs no exchange between lanes, its
// result is already laid out as the next contraction's A operand (the k index
// of a step is permuted to those points, and the operator's fragments are
// stored in that order), and the stage update finds the node values in the
// lane that holds the node's accumulator.  Between the contractions nothing
// goes through shared memory and no block barrier is needed; one operator
// fragment serves the M fields.
//
// Linear equations (constant-coefficient flux) form R = rx F + ry G and
// S = sx F + sy G at the nodes and contract with Dr V and Ds V: the flux
// commutes with the interpolation to the cubature points, so the sum is the
// same to round-off with 2 NP^2 instead of 3 NC NP multiply-adds per field.
//
// Faces.  The trace on a face depends on the N + 1 nodes on that face only,
// so a neighbour contributes those nodes (read from its state, or from the
// ghost slot of a cut face), and both sides' traces are short contractions
// with the one-dimensional interpolation E [NG][N+1].  Every element evaluates
// its own faces, as Apollo does (wxnodaldg2dmethod.cc:389-472); no face buffer
// makes a round trip through memory.
//
// What bounds it.  The float64 pipe: mma.m8n8k4 and DFMA share 64 multiply-adds
// per clock and SM.
#include <cuda_runtime.h>
#include <stdint.h>

#include "dg_device.cuh"
#include "dg_dmma.cuh"
#include "dg_flux64.cuh"
#include "dg_stage64.h"

namespace apollo {

namespace {

template <int EQ> constexpr bool kLinearEq = EQ == EQ_ADVECTION || EQ == EQ_MAXWELL || EQ == EQ_MAXWELL_TM;

// Sizes of the chain for one equation and order (doubles unless said).
template <int EQ, int N> struct Chain {
  static constexpr int M = Eq<EQ>::M;
  static constexpr int NP = Sizes<N>::NP, NC = Sizes<N>::NC, NG = Sizes<N>::NG, NF = Sizes<N>::NF;
  static constexpr bool LIN = kLinearEq<EQ>;
  using P = Pack64<N>;
  static constexpr int KS = P::KS, NB = P::NB, PB = P::PB, FB = P::FB, EK = P::EK;
  static constexpr int OPS = P::E_SIZE + P::L_SIZE + (LIN ? P::W_SIZE : P::V_SIZE + P::D_SIZE);
  static constexpr int TAB = 2 * NG;                 // gz, gw
  static constexpr int TABI = 3 * (N + 1);           // face node table (ints)
  static constexpr int SHARED = round_up(OPS + TAB + (TABI + 1) / 2, 2);
  // per warp: states [8][NP M], neighbour face nodes [24][N+1][M], geometry
  // [8][16], connectivity [24] int2
  static constexpr int X = round_up(8 * NP * M, 2), PN = round_up(24 * (N + 1) * M, 2), G = 8 * 16, C = 24;
  static constexpr int WARP = X + PN + G + C;
  static constexpr size_t bytes(int warps) { return sizeof(double) * (size_t)(SHARED + warps * WARP); }
  // warps per block (one block per SM): what the registers allow
  static constexpr int fit(int w) { return bytes(w) <= 227 * 1024 ? w : fit(w - 1); }
  static constexpr int WMAX = fit(LIN ? (M == 8 ? 8 : 16) : (N >= 5 ? 8 : 12));
};

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// n consecutive doubles, 16-byte accesses when ALIGNED (both counts even)
template <int n, bool ALIGNED>
__device__ __forceinline__ void load_run(const double* __restrict__ p, double* v) {
  if constexpr (ALIGNED && n % 2 == 0) {
#pragma unroll
    for (int i = 0; i < n; i += 2) {
      const double2 t = *reinterpret_cast<const double2*>(p + i);
      v[i] = t.x;
      v[i + 1] = t.y;
    }
  } else {
#pragma unroll
    for (int i = 0; i < n; ++i) v[i] = p[i];
  }
}
template <int n, bool ALIGNED>
__device__ __forceinline__ void store_run(double* __restrict__ p, const double* v) {
  if constexpr (ALIGNED && n % 2 == 0) {
#pragma unroll
    for (int i = 0; i < n; i += 2) *reinterpret_cast<double2*>(p + i) = make_double2(v[i], v[i + 1]);
  } else {
#pragma unroll
    for (int i = 0; i < n; ++i) p[i] = v[i];
  }
}

// One SSPRK stage (or right-hand side).  Reads the neighbours of x: x and out
// must not overlap.  `list` (nlist entries) names the elements of this launch;
// nullptr: all of them.
template <int EQ, int N>
__global__ void __launch_bounds__(32 * Chain<EQ, N>::WMAX, 1)
    k_stage64(DgDev d, StageArgs a, const int* __restrict__ list, int nlist) {
  using T = Chain<EQ, N>;
  using PK = Pack64<N>;
  using P = Eq<EQ>;
  constexpr int M = T::M, NP = T::NP, NG = T::NG, NF = T::NF;
  constexpr int KS = T::KS, NB = T::NB, PB = T::PB, FB = T::FB, EK = T::EK;
  constexpr bool EVEN = (NP * M) % 2 == 0;  // every element's state starts on a 16-byte boundary
  extern __shared__ __align__(16) double smem[];
  // operator fragments: E | L | (V | D) or W
  double* sE = smem;
  double* sL = sE + PK::E_SIZE;
  double* sV = sL + PK::L_SIZE;
  double* sGz = smem + T::OPS;
  double* sGw = sGz + NG;
  int* sFm = (int*)(sGw + NG);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, lr = lane >> 2, lc = lane & 3;
  double* sX = smem + T::SHARED + warp * T::WARP;
  double* sP = sX + T::X;
  double* sG = sP + T::PN;
  int2* sC = (int2*)(sG + T::G);
  {
    const double* src = d.pack64;
    constexpr int head = PK::E_SIZE + PK::L_SIZE;
    const double* tail = src + (T::LIN ? PK::W_OFF : PK::V_OFF);
    for (int i = 2 * tid; i < head; i += 2 * blockDim.x) cp_async16(sE + i, src + i);
    for (int i = 2 * tid; i < T::OPS - head; i += 2 * blockDim.x) cp_async16(sV + i, tail + i);
    for (int i = tid; i < NG; i += blockDim.x) {
      sGz[i] = d.gz[i];
      sGw[i] = d.gw[i];
    }
    for (int i = tid; i < 3 * (N + 1); i += blockDim.x) sFm[i] = PK::face_node(i / (N + 1), i % (N + 1));
    cp_async_wait_all();
  }
  // the last stage of a step (and a lone right-hand side) reduces the wave
  // speeds; an earlier stage clears the word instead
  const bool want_lam = a.mode != MODE_STAGE;
  if (a.mode == MODE_STAGE && a.reset_lambda && blockIdx.x == 0)
    for (int i = tid; i < d.ninst; i += blockDim.x) d.st[i].lam_bits = 0ull;
  __syncthreads();
  int err = 0;
  LamAcc lam_acc;
  const int n = list ? nlist : d.K;
  const int ntiles = (n + 7) / 8;
  const int stride = gridDim.x * (blockDim.x >> 5);
  for (int tile = warp * gridDim.x + blockIdx.x; tile < ntiles; tile += stride) {
    // rows past the end repeat the last element (their results are not stored)
    auto elem = [&](int r) {
      const int i = min(tile * 8 + r, n - 1);
      return list ? list[i] : i;
    };
    const bool row_ok = tile * 8 + lr < n;
    const int ke = elem(lr);
    __syncwarp();
    if (lane < 24) sC[lane] = *reinterpret_cast<const int2*>(d.conn + (size_t)elem(lane / 3) * 6 + 2 * (lane % 3));
    __syncwarp();
    // states
    if (list == nullptr && tile * 8 + 8 <= n) {
      const double* src = a.x + (size_t)tile * 8 * NP * M;
#pragma unroll 4
      for (int i = lane; i < 4 * NP * M; i += 32) cp_async16(sX + 2 * i, src + 2 * i);
    } else {
      for (int i = lane; i < 8 * NP * M; i += 32) {
        const int e = i / (NP * M);
        cp_async8(sX + i, a.x + (size_t)elem(e) * NP * M + (i - e * NP * M));
      }
    }
    // geometry: rx, ry, sx, sy, J, 1/J, nx[3], ny[3], sJ[3]
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int i = lane + 32 * u, e = i >> 3, q = i & 7;
      cp_async16(sG + 16 * e + 2 * q, reinterpret_cast<const double*>(d.geo + elem(e)) + 2 * q);
    }
    // the neighbours' nodes on the shared faces, in this side's node order (a
    // boundary or cut face stands in its own nodes; the ghost state or the
    // remote trace replaces what they interpolate to)
    {
      constexpr int CH = M % 2 == 0 ? 2 : 1, CN = M / CH, PER = (N + 1) * CN;  // doubles per copy, copies per node, face
#pragma unroll 4
      for (int i = lane; i < 24 * PER; i += 32) {
        const int p = i / PER, r = i - p * PER, m = r / CN, c = (r - m * CN) * CH;
        const int2 cn = sC[p];
        const double* src;
        if (cn.y < 0 || cn.x >= d.K) src = a.x + ((size_t)elem(p / 3) * NP + sFm[(p % 3) * (N + 1) + m]) * M;
        else src = a.x + ((size_t)cn.x * NP + sFm[cn.y * (N + 1) + N - m]) * M;
        if constexpr (CH == 2) cp_async16(sP + (p * (N + 1) + m) * M + c, src + c);
        else cp_async8(sP + (p * (N + 1) + m) * M + c, src + c);
      }
    }
    cp_async_wait_all();
    __syncwarp();
    const double* xe = sX + lr * NP * M;
    const double* ge = sG + 16 * lr;
    double acc[NB][M][2];
#pragma unroll
    for (int b = 0; b < NB; ++b)
#pragma unroll
      for (int f = 0; f < M; ++f) acc[b][f][0] = acc[b][f][1] = 0.0;

    // ---- volume term
    const double rx = ge[0], ry = ge[1], sx = ge[2], sy = ge[3];
    if constexpr (T::LIN) {
#pragma unroll
      for (int k = 0; k < KS; ++k) {
        const int node = PK::node(k, lc);
        double q[M], R[M], S[M];
#pragma unroll
        for (int f = 0; f < M; ++f) q[f] = node < NP ? xe[node * M + f] : 0.0;
        volume_flux<EQ>(d.eqp, q, rx, ry, sx, sy, R, S, &err);
#pragma unroll
        for (int b = 0; b < NB; ++b) {
          const double2 w = reinterpret_cast<const double2*>(sV)[(k * NB + b) * 32 + lane];
#pragma unroll
          for (int f = 0; f < M; ++f) dmma_8x8x4(acc[b][f], R[f], w.x);
#pragma unroll
          for (int f = 0; f < M; ++f) dmma_8x8x4(acc[b][f], S[f], w.y);
        }
      }
    } else {
      const double* sD = sV + PK::V_SIZE;
      double q[KS][M];
#pragma unroll
      for (int k = 0; k < KS; ++k) {
        const int node = PK::node(k, lc);
#pragma unroll
        for (int f = 0; f < M; ++f) q[k][f] = node < NP ? xe[node * M + f] : 0.0;
      }
#pragma unroll 1
      for (int pb = 0; pb < PB; ++pb) {
        // the eight cubature points of the block, two per lane
        double v[M][2];
#pragma unroll
        for (int f = 0; f < M; ++f) v[f][0] = v[f][1] = 0.0;
#pragma unroll
        for (int k = 0; k < KS; k += 2) {
          const double2 w = reinterpret_cast<const double2*>(sV)[(pb * ((KS + 1) / 2) + k / 2) * 32 + lane];
#pragma unroll
          for (int f = 0; f < M; ++f) dmma_8x8x4(v[f], q[k][f], w.x);
          if (k + 1 < KS) {
#pragma unroll
            for (int f = 0; f < M; ++f) dmma_8x8x4(v[f], q[k + 1][f], w.y);
          }
        }
        double R[2][M], S[2][M];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          double qc[M];
#pragma unroll
          for (int f = 0; f < M; ++f) qc[f] = v[f][j];
          volume_flux<EQ>(d.eqp, qc, rx, ry, sx, sy, R[j], S[j], &err);
        }
#pragma unroll
        for (int b = 0; b < NB; ++b) {
          const double2 wr = reinterpret_cast<const double2*>(sD)[((pb * 2 + 0) * NB + b) * 32 + lane];
          const double2 ws = reinterpret_cast<const double2*>(sD)[((pb * 2 + 1) * NB + b) * 32 + lane];
#pragma unroll
          for (int f = 0; f < M; ++f) dmma_8x8x4(acc[b][f], R[0][f], wr.x);
#pragma unroll
          for (int f = 0; f < M; ++f) dmma_8x8x4(acc[b][f], R[1][f], wr.y);
#pragma unroll
          for (int f = 0; f < M; ++f) dmma_8x8x4(acc[b][f], S[0][f], ws.x);
#pragma unroll
          for (int f = 0; f < M; ++f) dmma_8x8x4(acc[b][f], S[1][f], ws.y);
        }
      }
    }
    const int inst = inst_of(d, ke);
    // sources at the cubature points: VS S into the volume term
    // (wxcubature2d.cc:297-325)
    if (d.src.n > 0) {
      const ElemGeo& g = d.geo[ke];
      const double t = a.time_from_state ? d.st[inst].t + d.st[inst].dt * a.frac : a.t_arg;
      unsigned fields = 0;
      for (int i = 0; i < d.src.n; ++i) fields |= 1u << d.src.out[i];
#pragma unroll 1
      for (int pb = 0; pb < PB; ++pb) {
        double s[2][M];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int c = min(pb * 8 + 2 * lc + j, T::NC - 1);  // a point past the last has a zero column
          const double r = d.cub_r[c], z = d.cub_s[c];
          const double x = 0.5 * (-g.vx[0] * (r + z) + g.vx[1] * (1. + r) + g.vx[2] * (1. + z));
          const double y = 0.5 * (-g.vy[0] * (r + z) + g.vy[1] * (1. + r) + g.vy[2] * (1. + z));
#pragma unroll
          for (int f = 0; f < M; ++f) s[j][f] = 0.0;
          source_terms<M>(d.src, t, x, y, s[j]);
        }
#pragma unroll
        for (int b = 0; b < NB; ++b) {
          const double2 w = __ldg(reinterpret_cast<const double2*>(d.pack64 + PK::S_OFF) + (pb * NB + b) * 32 + lane);
#pragma unroll
          for (int f = 0; f < M; ++f)
            if (fields & (1u << f)) {
              dmma_8x8x4(acc[b][f], s[0][f], w.x);
              dmma_8x8x4(acc[b][f], s[1][f], w.y);
            }
        }
      }
    }

    // ---- surface term
    const double miJ = -ge[5];
    const double* se = sE + lane;
#pragma unroll 1
    for (int fb = 0; fb < FB; ++fb) {
      double vm[M][2], vp[M][2];
#pragma unroll
      for (int f = 0; f < M; ++f) vm[f][0] = vm[f][1] = vp[f][0] = vp[f][1] = 0.0;
      const int f_hi = min(8 * fb + 7, NF - 1) / NG;
#pragma unroll 1
      for (int fc = 8 * fb / NG; fc <= f_hi; ++fc) {
#pragma unroll
        for (int k = 0; k < EK; ++k, se += 32) {
          const int m = 4 * k + lc;
          const bool in = m <= N;
          const double w = *se;
          const double* om = xe + sFm[fc * (N + 1) + (in ? m : 0)] * M;
          const double* pm = sP + ((lr * 3 + fc) * (N + 1) + (in ? m : 0)) * M;
#pragma unroll
          for (int f = 0; f < M; ++f) dmma_8x8x4(vm[f], in ? om[f] : 0.0, w);
#pragma unroll
          for (int f = 0; f < M; ++f) dmma_8x8x4(vp[f], in ? pm[f] : 0.0, w);
        }
      }
      // two face points per lane, on one face (NG is even); points past the
      // last repeat it (their lift columns are zero)
      const int p0 = min(fb * 8 + 2 * lc, NF - 2);
      const int fc = p0 / NG, g0 = p0 - fc * NG;
      const double nx = ge[6 + fc], ny = ge[9 + fc], ws = miJ * ge[12 + fc];
      const int2 cn = sC[lr * 3 + fc];
      double A[2][M];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        double qM[M], qP[M], nf[M];
#pragma unroll
        for (int f = 0; f < M; ++f) {
          qM[f] = vm[f][j];
          qP[f] = vp[f][j];
        }
        if (cn.y < 0) {
          // Gauss point coordinates on the face (wxcubature2d.cc:118-124)
          const ElemGeo& g = d.geo[ke];
          const double t = a.time_from_state ? d.st[inst].t + d.st[inst].dt * a.frac : a.t_arg;
          const double z = sGz[g0 + j];
          const double r = fc == 0 ? z : fc == 1 ? -z : -1.0;
          const double s = fc == 0 ? -1.0 : fc == 1 ? z : -z;
          const double x = 0.5 * (-g.vx[0] * (r + s) + g.vx[1] * (1. + r) + g.vx[2] * (1. + s));
          const double y = 0.5 * (-g.vy[0] * (r + s) + g.vy[1] * (1. + r) + g.vy[2] * (1. + s));
          apply_bc<EQ, double>(d.bcs, -cn.x, t, x, y, nx, ny, qM, qP);
        } else if (cn.x >= d.K) {
          // a cut face: the peer's trace, in its own point order
          const double* tp = d.trace + ((size_t)cn.x * NF + cn.y * NG + (NG - 1 - g0 - j)) * M;
#pragma unroll
          for (int f = 0; f < M; ++f) qP[f] = tp[f];
        }
        const double lam = face_flux<EQ>(d.eqp, nx, ny, qM, qP, nf, &err);
        if (want_lam) lam_acc.add(d.st, inst, fabs(lam));
        const double w = ws * sGw[g0 + j];
#pragma unroll
        for (int f = 0; f < M; ++f) A[j][f] = nf[f] * w;
      }
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        const double2 w = reinterpret_cast<const double2*>(sL)[(fb * NB + b) * 32 + lane];
#pragma unroll
        for (int f = 0; f < M; ++f) dmma_8x8x4(acc[b][f], A[0][f], w.x);
#pragma unroll
        for (int f = 0; f < M; ++f) dmma_8x8x4(acc[b][f], A[1][f], w.y);
      }
    }

    // ---- stage update, in the lanes that hold the nodes
    const double dt = a.time_from_state ? d.st[inst].dt : a.dt_arg;
    const double c_stage = dt / 4.0;  // dt/(s-1), s = 5
    const double c_al = 4.0 / 5.0, c_be = dt / 5.0, c_ga = 1.0 / 5.0;
    if (row_ok) {
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        constexpr int PAIR = 2 * M;
        if (PK::paired(b)) {
          // nodes n0, n0 + 1: 2 M consecutive values
          const int n0 = b * 8 + 2 * lc;
          if (n0 >= NP) continue;
          const bool both = n0 + 1 < NP;
          double r[PAIR], o[PAIR], xv[PAIR], uv[PAIR];
#pragma unroll
          for (int f = 0; f < M; ++f) {
            r[f] = acc[b][f][0];
            r[M + f] = acc[b][f][1];
          }
#pragma unroll
          for (int f = 0; f < PAIR; ++f) {
            const bool use = f < M || both;
            if (use && r[f] != r[f]) err |= ERRB_NAN;
            xv[f] = use ? xe[n0 * M + f] : 0.0;
            uv[f] = 0.0;
          }
          const size_t off = ((size_t)ke * NP + n0) * M;
          if (a.mode == MODE_FINAL) {
            if (both) load_run<PAIR, EVEN>(a.u0 + off, uv);
            else load_run<M, EVEN>(a.u0 + off, uv);
          }
#pragma unroll
          for (int f = 0; f < PAIR; ++f) {
            if (a.mode == MODE_RHS) o[f] = r[f];
            else if (a.mode == MODE_STAGE) o[f] = xv[f] + c_stage * r[f];
            else o[f] = c_al * xv[f] + c_be * r[f] + c_ga * uv[f];
          }
          if (both) store_run<PAIR, EVEN>(a.out + off, o);
          else store_run<M, EVEN>(a.out + off, o);
        } else {
          const int n0 = b * 8 + lc;
          if (n0 >= NP) continue;
          const size_t off = ((size_t)ke * NP + n0) * M;
#pragma unroll
          for (int f = 0; f < M; ++f) {
            const double r = acc[b][f][0], xv = xe[n0 * M + f];
            if (r != r) err |= ERRB_NAN;
            double o;
            if (a.mode == MODE_RHS) o = r;
            else if (a.mode == MODE_STAGE) o = xv + c_stage * r;
            else o = c_al * xv + c_be * r + c_ga * a.u0[off + f];
            a.out[off + f] = o;
          }
        }
      }
    }
  }
  if (want_lam) lam_acc.flush_warp(d.st);
  if (err) atomicOr(&d.st->err, err);
}

// Traces of the cut faces blocks[0, n) (face 3 k + f of the state x) into dst
// [n][NG][M], a warp per eight faces: the contraction a neighbour's own stage
// would form them with (its node order, its k-steps), so the ranks of a
// partitioned mesh compute what one handle on the whole mesh computes.
template <int M, int N>
__global__ void __launch_bounds__(128) k_cut_traces(const double* __restrict__ x, const double* __restrict__ pack,
                                                    const int* __restrict__ blocks, int n, double* __restrict__ dst) {
  using PK = Pack64<N>;
  constexpr int NP = PK::NP, NG = PK::NG;
  const int lane = threadIdx.x & 31, lr = lane >> 2, lc = lane & 3;
  const int row = (blockIdx.x * 4 + (threadIdx.x >> 5)) * 8 + lr;
  const int id = blocks[min(row, n - 1)];
  const double* xe = x + (size_t)(id / 3) * NP * M;
  double q[PK::EK][M];
#pragma unroll
  for (int k = 0; k < PK::EK; ++k) {
    const int m = 4 * k + lc;
#pragma unroll
    for (int f = 0; f < M; ++f) q[k][f] = m <= N ? xe[PK::face_node(id % 3, N - m) * M + f] : 0.0;
  }
#pragma unroll
  for (int tb = 0; tb < PK::TB; ++tb) {
    double v[M][2];
#pragma unroll
    for (int f = 0; f < M; ++f) v[f][0] = v[f][1] = 0.0;
#pragma unroll
    for (int k = 0; k < PK::EK; ++k) {
      const double w = pack[PK::T_OFF + (tb * PK::EK + k) * 32 + lane];
#pragma unroll
      for (int f = 0; f < M; ++f) dmma_8x8x4(v[f], q[k][f], w);
    }
    if (row >= n) continue;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int g = 8 * tb + 2 * lc + j;  // the neighbour's point
      if (g >= NG) continue;
#pragma unroll
      for (int f = 0; f < M; ++f) dst[((size_t)row * NG + (NG - 1 - g)) * M + f] = v[f][j];
    }
  }
}

template <int EQ>
cudaError_t cut_traces_n(const DgDev& d, const double* x, const int* blocks, int n, double* dst, cudaStream_t s) {
  constexpr int M = Eq<EQ>::M;
  const unsigned g = (unsigned)((n + 31) / 32);
  switch (d.N) {
    case 2: k_cut_traces<M, 2><<<g, 128, 0, s>>>(x, d.pack64, blocks, n, dst); break;
    case 3: k_cut_traces<M, 3><<<g, 128, 0, s>>>(x, d.pack64, blocks, n, dst); break;
    case 4: k_cut_traces<M, 4><<<g, 128, 0, s>>>(x, d.pack64, blocks, n, dst); break;
    case 5: k_cut_traces<M, 5><<<g, 128, 0, s>>>(x, d.pack64, blocks, n, dst); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

template <int EQ, int N>
cudaError_t launch_t(const DgDev& d, const StageArgs& a, const int* list, int nlist, cudaStream_t s) {
  using T = Chain<EQ, N>;
  static unsigned configured = 0;  // bit per device
  int dev = 0;
  cudaGetDevice(&dev);
  if (!(configured & (1u << (dev & 31)))) {
    cudaError_t e = cudaFuncSetAttribute(k_stage64<EQ, N>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)T::bytes(T::WMAX));
    if (e != cudaSuccess) return e;
    configured |= 1u << (dev & 31);
  }
  const int n = list ? nlist : d.K;
  if (n <= 0) return cudaSuccess;
  int sms = device_sms();
  if (d.grid_div > 1) sms = (sms + d.grid_div - 1) / d.grid_div;
  // one block per SM with as many warps as its share of the tiles needs (a
  // warp without a tile would only hold registers): the smallest meshes run
  // one tile per warp on as many SMs as there are tiles
  const int tiles = (n + 7) / 8, grid = tiles < sms ? tiles : sms;
  int warps = (tiles + grid - 1) / grid;
  if (warps > T::WMAX) warps = T::WMAX;
  k_stage64<EQ, N><<<grid, 32 * warps, T::bytes(warps), s>>>(d, a, list, nlist);
  return cudaGetLastError();
}

template <int EQ>
cudaError_t dispatch_n(const DgDev& d, const StageArgs& a, const int* list, int nlist, cudaStream_t s) {
  switch (d.N) {
    case 2: return launch_t<EQ, 2>(d, a, list, nlist, s);
    case 3: return launch_t<EQ, 3>(d, a, list, nlist, s);
    case 4: return launch_t<EQ, 4>(d, a, list, nlist, s);
    case 5: return launch_t<EQ, 5>(d, a, list, nlist, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace

cudaError_t launch_stage64(int eq, const DgDev& d, const StageArgs& a, const int* list, int nlist, cudaStream_t s) {
  switch (eq) {
    case EQ_ADVECTION: return dispatch_n<EQ_ADVECTION>(d, a, list, nlist, s);
    case EQ_EULER: return dispatch_n<EQ_EULER>(d, a, list, nlist, s);
    case EQ_MAXWELL: return dispatch_n<EQ_MAXWELL>(d, a, list, nlist, s);
    case EQ_EULER2D: return dispatch_n<EQ_EULER2D>(d, a, list, nlist, s);
    case EQ_MAXWELL_TM: return dispatch_n<EQ_MAXWELL_TM>(d, a, list, nlist, s);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_cut_traces(int eq, const DgDev& d, const double* x, const int* blocks, int n, double* dst,
                              cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  switch (eq) {
    case EQ_ADVECTION: return cut_traces_n<EQ_ADVECTION>(d, x, blocks, n, dst, s);
    case EQ_EULER: return cut_traces_n<EQ_EULER>(d, x, blocks, n, dst, s);
    case EQ_MAXWELL: return cut_traces_n<EQ_MAXWELL>(d, x, blocks, n, dst, s);
    case EQ_EULER2D: return cut_traces_n<EQ_EULER2D>(d, x, blocks, n, dst, s);
    case EQ_MAXWELL_TM: return cut_traces_n<EQ_MAXWELL_TM>(d, x, blocks, n, dst, s);
    default: return cudaErrorInvalidValue;
  }
}

// warps of one wave of k_stage64 (the launch-bound limit of form 2)
int stage64_wave_tiles(int eq, int N, int sms) {
  const int w = (eq == EQ_EULER || eq == EQ_EULER2D) ? (N >= 5 ? 8 : 12) : eq == EQ_MAXWELL ? 8 : 16;
  return sms * w;
}

}  // namespace apollo
