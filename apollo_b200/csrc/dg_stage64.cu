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
// ghost slot of a cut face), and both sides' traces are short sums with the
// one-dimensional interpolation E [NG][N+1].  The linear equations evaluate
// the numerical flux at those nodes (normal, boundary state and dissipation
// are constant along a straight face, so it too commutes with E) and lift from
// there.  Every element evaluates
// its own faces, as Apollo does (wxnodaldg2dmethod.cc:389-472); no face buffer
// makes a round trip through memory.
//
// What bounds it.  The float64 pipe: mma.m8n8k4 and DFMA share 64 multiply-adds
// per clock and SM (measured: either alone 63.9, the two in turn 86-93 % of
// that).  Euler N = 4 fills 69 % of it (K = 79,202: DMMA 48 %, DFMA 20 %), the
// rest is the latency of the pointwise flux; DRAM is at 6 %.  The linear
// equations' smaller contractions leave it at 58 % with the shared-memory pipe
// at 48 %.  A right-hand side, before (volume, face and LIFT kernels) and now:
// Euler 4 fields, K = 130,050, N = 2..5: 168, 259, 355, 572 us and 87, 132, 195,
// 329 us; Maxwell TM N = 5, K = 522,242: 1,796 and 300 us; 8 fields N = 5,
// K = 32,258: 333 and 71 us.
#include <cuda_runtime.h>
#include <stdint.h>

#include "dg_chain64.cuh"
#include "dg_device.cuh"
#include "dg_dmma.cuh"
#include "dg_flux64.cuh"
#include "dg_stage64.h"

namespace apollo {

namespace {

// Sizes of the chain for one equation and order (doubles unless said).
template <int EQ, int N, int KIND> struct Chain {
  static constexpr int M = Eq<EQ>::M;
  static constexpr int NP = Sizes<N>::NP, NC = Sizes<N>::NC, NG = Sizes<N>::NG, NF = Sizes<N>::NF;
  static constexpr bool LIN = kLinearEq<EQ>;
  using P = Pack64<N>;
  // operators in shared memory: E | L | V | D, or Q | W
  static constexpr int OPS_OFF = LIN ? P::Q_OFF : P::E_OFF, OPS = LIN ? P::S_OFF - P::Q_OFF : P::Q_OFF;
  static constexpr int TAB = NG;                     // gz
  static constexpr int TABI = 3 * (N + 1);           // face node table (ints)
  static constexpr int SHARED = round_up(OPS + TAB + (TABI + 1) / 2, 2);
  // per warp: states [8][ES] and geometry [8][18], double buffered where that
  // costs no resident warp (the next tile's arrive while this one computes),
  // neighbour face nodes [8][FS] (a row's three faces of N + 1 nodes), connectivity
  // [24] int2 and where the face nodes come from [24] int2
  static constexpr int ES = elem_stride(NP * M, M), FS = face_stride(3 * (N + 1) * M, M);
  static constexpr int X = 8 * ES, G = 8 * kGeoStride, PN = 8 * FS, C = 48;
  // (8 fields would lose warps to it; Euler up to order 4 gains more from
  // sixteen warps with one buffer than from twelve with two: K = 130,050, N = 4
  // 202 -> 195 us; at order 5 the registers allow eight warps)
  static constexpr int XB = (LIN && M != 8) || (!LIN && N >= 5) ? 2 : 1;
  // results leave by bulk copies where a row is long enough to pay for one:
  // K = 130,050: Euler N = 4 (480 bytes a row) 209 -> 204 us, Maxwell TM N = 5
  // (one copy of 4,032) 105 -> 95; Euler N = 2 (192 bytes) 89 -> 93
  static constexpr bool BULK = NP * M >= 30;
  static constexpr int WARP = XB * (X + G) + PN + C;
  static constexpr size_t bytes(int warps) { return sizeof(double) * (size_t)(SHARED + warps * WARP); }
  // Warps per block (one block per SM): what registers and shared memory allow.
  // Sixteen have 128 registers a lane, and the Euler kernels then spill 130 to
  // 670 bytes; eight spill nothing.  The spills cost less than the missing warps
  // on large meshes, more on small ones, and the longest bodies (HLL and Roe, 5
  // fields, orders 3 and 4) gain from eight at every size.  A right-hand side, K =
  // 2,048, 16,200, 50,562, with eight and with sixteen: Lax-Friedrichs N = 4, 4
  // fields 25, 44, 93 and 26, 42, 88 us, 5 fields 27, 52, 116 and 29, 50, 112; HLL
  // N = 3, 4 fields 26, 39, 76 and 27, 39, 74, 5 fields 24, 40, 84 and 29, 41, 87.
  static constexpr int fit(int w) { return bytes(w) <= 227 * 1024 ? w : fit(w - 1); }
  static constexpr bool LONG = M == 5 && N >= 3 && (KIND == NF_HLL || KIND == NF_ROE);
  static constexpr int WMAX = fit(LIN ? (M == 8 ? 8 : 16) : (N >= 5 || LONG ? 8 : 16));
};

// One SSPRK stage (or right-hand side).  Reads the neighbours of x: x and out
// must not overlap.  `list` (nlist entries) names the elements of this launch;
// nullptr: all of them.  KIND: the Euler numerical flux (a kernel of its own, so
// that the others' code takes no registers from it).
template <int EQ, int N, int KIND>
__global__ void __launch_bounds__(32 * Chain<EQ, N, KIND>::WMAX, 1)
    k_stage64(DgDev d, StageArgs a, const int* __restrict__ list, int nlist) {
  using T = Chain<EQ, N, KIND>;
  using PK = Pack64<N>;
  using P = Eq<EQ>;
  constexpr int M = T::M, NP = T::NP, NG = T::NG, NF = T::NF;
  constexpr int KS = PK::KS, PB = PK::PB, FB = PK::FB, NFN = PK::NFN;
  extern __shared__ __align__(16) double smem[];
  double* sOps = smem;
  double* sGz = smem + T::OPS;
  int* sFm = (int*)(sGz + NG);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, lr = lane >> 2, lc = lane & 3;
  double* sX0 = smem + T::SHARED + warp * T::WARP;  // XB x (states, geometry)
  double* sP = sX0 + T::XB * (T::X + T::G);
  int2 *sC = (int2*)(sP + T::PN), *sS = sC + 24;
  for (int i = 2 * tid; i < T::OPS; i += 2 * blockDim.x) cp_async16(sOps + i, d.pack64 + T::OPS_OFF + i);
  for (int i = tid; i < NG; i += blockDim.x) sGz[i] = d.gz[i];
  for (int i = tid; i < NFN; i += blockDim.x) sFm[i] = PK::face_node(i / (N + 1), i % (N + 1));
  allow_next();
  int err = 0;
  LamAcc lam_acc;
  const int n = list ? nlist : d.K;
  const int ntiles = (n + 7) / 8;
  const int stride = gridDim.x * (blockDim.x >> 5);
  // element of row r of a tile; rows past the end repeat the last element
  // (their results are not stored)
  auto elem = [&](int tile, int r) {
    const int i = min(tile * 8 + r, n - 1);
    return list ? list[i] : i;
  };
  auto load_conn = [&](int tile) {
    int2 c = make_int2(0, -1);
    if (lane < 24) c = *reinterpret_cast<const int2*>(d.conn + (size_t)elem(tile, lane / 3) * 6 + 2 * (lane % 3));
    return c;
  };
  // a tile's states and geometry (rx, ry, sx, sy, J, 1/J, nx[3], ny[3], sJ[3])
  auto load_tile = [&](int tile, double* X) {
    if (list == nullptr) {
      copy_tile<NP * M, T::ES>(X, a.x, tile, n, lane);
    } else {
      for (int i = lane; i < 8 * NP * M; i += 32) {
        const int e = i / (NP * M);
        cp_async8(X + e * T::ES + (i - e * NP * M), a.x + (size_t)elem(tile, e) * NP * M + (i - e * NP * M));
      }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int i = lane + 32 * u, e = i >> 3, q = i & 7;
      cp_async16(X + T::X + kGeoStride * e + 2 * q, reinterpret_cast<const double*>(d.geo + elem(tile, e)) + 2 * q);
    }
  };
  int tile = warp * gridDim.x + blockIdx.x;
  int2 conn_next = make_int2(0, -1);
  if (tile < ntiles) {
    conn_next = load_conn(tile);
  }
  wait_previous();
  // the last stage of a step (and a lone right-hand side) reduces the wave
  // speeds; an earlier stage clears the word instead
  const bool want_lam = a.mode != MODE_STAGE;
  if (a.mode == MODE_STAGE && a.reset_lambda && blockIdx.x == 0)
    for (int i = tid; i < d.ninst; i += blockDim.x) d.st[i].lam_bits = 0ull;
  if (T::XB == 2 && tile < ntiles) load_tile(tile, sX0);
  cp_async_wait_all();
  __syncthreads();
  for (int it = 0; tile < ntiles; tile += stride, ++it) {
    double* sX = sX0 + (T::XB == 2 && (it & 1) ? T::X + T::G : 0);
    const bool row_ok = tile * 8 + lr < n;
    const int ke = elem(tile, lr);
    if (T::XB == 1) bulk_read_done();
    __syncwarp();  // the previous tile's reads are done
    if (T::XB == 1) load_tile(tile, sX);
    if (lane < 24) {
      sC[lane] = conn_next;
      sS[lane] = face_source(conn_next, elem(tile, lane / 3), lane % 3, d.K);
    }
    __syncwarp();
    // the neighbours' nodes on the shared faces, in this side's node order:
    // from the neighbour's state, or the ghost slot of a cut face (the peer's
    // order); a boundary face stands in its own nodes, and the ghost state
    // replaces what they give.  They arrive during the volume term.
#pragma unroll
    for (int fc = 0; fc < 3; ++fc) {
      const int2 s = sS[lr * 3 + fc];
      const int f = s.y & 3;
      const double* from = (s.y & 8) ? d.trace + ((size_t)s.x * NF + f * NG) * M : a.x + (size_t)s.x * NP * M;
#pragma unroll
      for (int k = 0; k < (N + 4) / 4; ++k) {
        const int m = 4 * k + lc;
        if (m > N) continue;
        const int mm = s.y & 4 ? N - m : m;
        cp_async_node<M>(sP + lr * T::FS + (fc * (N + 1) + m) * M, from + ((s.y & 8) ? mm : sFm[f * (N + 1) + mm]) * M);
      }
    }
    cp_async_commit();
    if (T::XB == 2) {
      cp_async_wait<1>();  // this tile's states (all but the neighbours' nodes)
    } else {
      cp_async_wait<0>();
    }
    if (T::XB == 2) bulk_read_done();  // the other buffer's results are on their way
    __syncwarp();
    if (tile + stride < ntiles) {
      conn_next = load_conn(tile + stride);
      if (T::XB == 2) load_tile(tile + stride, sX0 + ((it & 1) ? 0 : T::X + T::G));
    }
    cp_async_commit();
    double* xe = sX + lr * T::ES;
    const double* ge = sX + T::X + kGeoStride * lr;
    Nodes<M, PK> acc;
    acc.zero();

    // ---- volume term
    const double rx = ge[0], ry = ge[1], sx = ge[2], sy = ge[3];
    if constexpr (T::LIN) {
#pragma unroll
      for (int k = 0; k < KS; ++k) {
        const int node = min(PK::node(k, lc), NP - 1);  // past the last node the operator is zero
        double q[M], R[M], S[M];
#pragma unroll
        for (int f = 0; f < M; ++f) q[f] = xe[node * M + f];
        LinearFast64<EQ>::along(d.eqp, q, rx, ry, R);
        LinearFast64<EQ>::along(d.eqp, q, sx, sy, S);
        acc.add(sOps + PK::Q_SIZE + k * PK::NS, lane, R, S);
      }
    } else {
      const double *sV = sOps + PK::V_OFF, *sD = sOps + PK::D_OFF;
#pragma unroll 1
      for (int pb = 0; pb < PB; ++pb) {
        // the eight cubature points of the block, two per lane
        double v[M][2];
#pragma unroll
        for (int k = 0; k < KS; k += 2) {
          const double2 w = reinterpret_cast<const double2*>(sV)[(pb * ((KS + 1) / 2) + k / 2) * 32 + lane];
          double q[2][M];
#pragma unroll
          for (int j = 0; j < 2; ++j) shared_run<M>(xe + min(PK::node(k + j, lc), NP - 1) * M, q[j]);
#pragma unroll
          for (int f = 0; f < M; ++f) {
            if (k == 0) dmma_8x8x4_first(v[f], q[0][f], w.x);
            else dmma_8x8x4(v[f], q[0][f], w.x);
          }
          if (k + 1 < KS) {
#pragma unroll
            for (int f = 0; f < M; ++f) dmma_8x8x4(v[f], q[1][f], w.y);
          }
        }
        double qc[2][M], R[2][M], S[2][M];
#pragma unroll
        for (int f = 0; f < M; ++f) {
          qc[0][f] = v[f][0];
          qc[1][f] = v[f][1];
        }
        volume_flux_pair<EQ>(d.eqp, qc, rx, ry, sx, sy, R, S, &err);
        acc.add(sD + (2 * pb) * PK::NS, lane, R[0], R[1]);
        acc.add(sD + (2 * pb + 1) * PK::NS, lane, S[0], S[1]);
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
        acc.add(d.pack64 + PK::S_OFF + pb * PK::NS, lane, s[0], s[1], fields);
      }
    }

    // ---- surface term
    if (T::XB == 2) cp_async_wait<1>();  // all but the next tile's states
    __syncwarp();
    const double miJ = -0.5 * ge[5];  // the face fluxes come out twice
    // the ghost state of one point of boundary face fc at face coordinate z
    auto ghost_state = [&](int tag, int fc, double z, const double* q, double* qb) {
      const ElemGeo& g = d.geo[ke];
      const double t = a.time_from_state ? d.st[inst].t + d.st[inst].dt * a.frac : a.t_arg;
      // point coordinates on the face (wxcubature2d.cc:118-124)
      const double r = fc == 0 ? z : fc == 1 ? -z : -1.0;
      const double s = fc == 0 ? -1.0 : fc == 1 ? z : -z;
      const double x = 0.5 * (-g.vx[0] * (r + s) + g.vx[1] * (1. + r) + g.vx[2] * (1. + s));
      const double y = 0.5 * (-g.vy[0] * (r + s) + g.vy[1] * (1. + r) + g.vy[2] * (1. + s));
      apply_bc<EQ, double>(d.bcs, tag, t, x, y, ge[6 + fc], ge[9 + fc], q, qb);
    };
    if constexpr (T::LIN) {
      // the flux at the face nodes, two per lane (a node past the last repeats
      // it; its lift column is zero).  The linear equations' boundary states
      // read neither position nor time.
#pragma unroll 1
      for (int qb = 0; qb < PK::QB; ++qb) {
        double A[2][M];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int p = min(qb * 8 + 2 * lc + j, NFN - 1), fc = p / (N + 1);
          const double *om = xe + sFm[p] * M, *pm = sP + lr * T::FS + p * M;
          double qM[M], qP[M];
#pragma unroll
          for (int f = 0; f < M; ++f) {
            qM[f] = om[f];
            qP[f] = pm[f];
          }
          const int2 cn = sC[lr * 3 + fc];
          if (cn.y < 0) ghost_state(-cn.x, fc, 0.0, qM, qP);
          const double lam = LinearFast64<EQ>::face2(d.eqp, ge[6 + fc], ge[9 + fc], miJ * ge[12 + fc], qM, qP, A[j]);
          if (want_lam) lam_acc.add(d.st, inst, lam);
        }
        acc.add(sOps + qb * PK::NS, lane, A[0], A[1]);
      }
    } else {
      const double* sL = sOps + PK::L_OFF;
#pragma unroll 1
      for (int fb = 0; fb < FB; ++fb) {
        // two face points per lane, on one face (NG is even); a pair past the
        // last repeats it (its lift columns are zero)
        const int p0 = min(fb * 8 + 2 * lc, NF - 2);
        const int fc = p0 / NG, g0 = p0 - fc * NG;
        // both sides' traces from the face's nodes.  On the vector units: the
        // N + 1 terms fill only part of the tensor instruction's k-steps, and
        // both forms run at the float64 pipe's rate.
        double qM[2][M], qP[2][M], A[2][M], lam[2];
        const double2* se = reinterpret_cast<const double2*>(sOps) + fb * (N + 1) * 4 + lc;
        const double* pm = sP + lr * T::FS + fc * (N + 1) * M;
#pragma unroll
        for (int m = 0; m <= N; ++m) {
          const double2 w = se[m * 4];
          const double* om = xe + sFm[fc * (N + 1) + m] * M;
#pragma unroll
          for (int f = 0; f < M; ++f) {
            const double o = om[f], p = pm[m * M + f];
            qM[0][f] = m == 0 ? w.x * o : fma(w.x, o, qM[0][f]);
            qM[1][f] = m == 0 ? w.y * o : fma(w.y, o, qM[1][f]);
            qP[0][f] = m == 0 ? w.x * p : fma(w.x, p, qP[0][f]);
            qP[1][f] = m == 0 ? w.y * p : fma(w.y, p, qP[1][f]);
          }
        }
        const int2 cn = sC[lr * 3 + fc];
        if (cn.y < 0) {
#pragma unroll
          for (int j = 0; j < 2; ++j) ghost_state(-cn.x, fc, sGz[g0 + j], qM[j], qP[j]);
        }
        face_flux2_pair<EQ, KIND>(d.eqp, ge[6 + fc], ge[9 + fc], miJ * ge[12 + fc], qM, qP, A, lam, &err);
        if (want_lam) {
          lam_acc.add(d.st, inst, fabs(lam[0]));
          lam_acc.add(d.st, inst, fabs(lam[1]));
        }
        acc.add(sL + fb * PK::NS, lane, A[0], A[1]);
      }
    }

    // ---- stage update, in the lanes that hold the nodes
    const double dt = a.time_from_state ? d.st[inst].dt : a.dt_arg;
    const double c_r = a.mode == MODE_STAGE ? dt / 4.0 : dt / 5.0;  // dt/(s-1) and dt/s, s = 5
    // a full tile's results replace its states in shared memory and leave by
    // bulk copies; rows of a partial tile or of a list, and short rows, are
    // stored from here
    acc.finish();
    const bool whole = T::BULK && list == nullptr && tile * 8 + 8 <= n;
    if (whole) __syncwarp();  // the states have been read
    if (row_ok) {
      double* out = a.out + (size_t)ke * NP * M;
      const double* u0 = a.u0 + (size_t)ke * NP * M;
      int top = 0;  // the largest exponent and leading fraction: above infinity's, a NaN
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
          load_block<M, PK>(xe, b, lc, x);
          if (a.mode == MODE_STAGE) {
#pragma unroll
            for (int f = 0; f < M; ++f)
#pragma unroll
              for (int j = 0; j < 2; ++j) o[f][j] = x[f][j] + c_r * o[f][j];
          } else {
            double u[M][2];
            load_block<M, PK>(u0, b, lc, u);
#pragma unroll
            for (int f = 0; f < M; ++f)
#pragma unroll
              for (int j = 0; j < 2; ++j) o[f][j] = (4.0 / 5.0) * x[f][j] + c_r * o[f][j] + (1.0 / 5.0) * u[f][j];
          }
        }
        if (whole) store_block<M, PK>(xe, b, lc, o);
        else store_block<M, PK>(out, b, lc, o);
      }
      if (top > 0x7ff00000) err |= ERRB_NAN;
    }
    if (whole) bulk_store_tile<NP * M, T::ES>(a.out + (size_t)tile * 8 * NP * M, sX, lane);
  }
  bulk_all_done();
  if (want_lam) lam_acc.flush_warp(d.st);
  if (err) atomicOr(&d.st->err, err);
}

// The N + 1 nodes on each of the cut faces blocks[0, n) (face 3 k + f of the
// state x), in face order, into the first (N + 1) M values of its block of
// dst [n][NG M].
template <int M, int N>
__global__ void __launch_bounds__(128) k_cut_nodes(const double* __restrict__ x, const int* __restrict__ blocks, int n,
                                                   double* __restrict__ dst) {
  using PK = Pack64<N>;
  const int i = blockIdx.x * 128 + threadIdx.x;
  if (i >= n * (N + 1)) return;
  const int j = i / (N + 1), m = i - j * (N + 1), id = blocks[j];
  const double* src = x + ((size_t)(id / 3) * PK::NP + PK::face_node(id % 3, m)) * M;
#pragma unroll
  for (int f = 0; f < M; ++f) dst[((size_t)j * PK::NG + m) * M + f] = src[f];
}

template <int EQ>
cudaError_t cut_nodes_n(const DgDev& d, const double* x, const int* blocks, int n, double* dst, cudaStream_t s) {
  constexpr int M = Eq<EQ>::M;
  const unsigned g = (unsigned)((n * (d.N + 1) + 127) / 128);
  switch (d.N) {
    case 2: k_cut_nodes<M, 2><<<g, 128, 0, s>>>(x, blocks, n, dst); break;
    case 3: k_cut_nodes<M, 3><<<g, 128, 0, s>>>(x, blocks, n, dst); break;
    case 4: k_cut_nodes<M, 4><<<g, 128, 0, s>>>(x, blocks, n, dst); break;
    case 5: k_cut_nodes<M, 5><<<g, 128, 0, s>>>(x, blocks, n, dst); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

template <int EQ, int N, int KIND>
cudaError_t launch_t(const DgDev& d, const StageArgs& a, const int* list, int nlist, cudaStream_t s, int spare) {
  using T = Chain<EQ, N, KIND>;
  static unsigned configured = 0;  // bit per device
  int dev = 0;
  cudaGetDevice(&dev);
  if (!(configured & (1u << (dev & 31)))) {
    cudaError_t e = cudaFuncSetAttribute(k_stage64<EQ, N, KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)T::bytes(T::WMAX));
    if (e != cudaSuccess) return e;
    configured |= 1u << (dev & 31);
  }
  const int n = list ? nlist : d.K;
  if (n <= 0) return cudaSuccess;
  int sms = device_sms();
  if (d.grid_div > 1) sms = (sms + d.grid_div - 1) / d.grid_div;
  if (sms > spare) sms -= spare;
  // one block per SM with as many warps as its share of the tiles needs (a
  // warp without a tile would only hold registers): the smallest meshes run
  // one tile per warp on as many SMs as there are tiles
  const int tiles = (n + 7) / 8, grid = tiles < sms ? tiles : sms;
  int warps = (tiles + grid - 1) / grid;
  if (warps > T::WMAX) warps = T::WMAX;
  return launch_kernel(k_stage64<EQ, N, KIND>, grid, 32 * warps, T::bytes(warps), s, a.overlap != 0, d, a, list, nlist);
}

template <int EQ, int KIND>
cudaError_t dispatch_n(const DgDev& d, const StageArgs& a, const int* list, int nlist, cudaStream_t s, int spare) {
  switch (d.N) {
    case 2: return launch_t<EQ, 2, KIND>(d, a, list, nlist, s, spare);
    case 3: return launch_t<EQ, 3, KIND>(d, a, list, nlist, s, spare);
    case 4: return launch_t<EQ, 4, KIND>(d, a, list, nlist, s, spare);
    case 5: return launch_t<EQ, 5, KIND>(d, a, list, nlist, s, spare);
    default: return cudaErrorInvalidValue;
  }
}

template <int EQ>
cudaError_t dispatch_kind(const DgDev& d, const StageArgs& a, const int* list, int nlist, cudaStream_t s, int spare) {
  switch ((int)d.eqp.p[3]) {
    case NF_HLL: return dispatch_n<EQ, NF_HLL>(d, a, list, nlist, s, spare);
    case NF_ROE: return dispatch_n<EQ, NF_ROE>(d, a, list, nlist, s, spare);
    case NF_WAVE: return dispatch_n<EQ, NF_WAVE>(d, a, list, nlist, s, spare);
    default: return dispatch_n<EQ, NF_LF>(d, a, list, nlist, s, spare);
  }
}

}  // namespace

cudaError_t launch_stage64(int eq, const DgDev& d, const StageArgs& a, const int* list, int nlist, cudaStream_t s,
                           int spare) {
  switch (eq) {
    case EQ_ADVECTION: return dispatch_n<EQ_ADVECTION, NF_LF>(d, a, list, nlist, s, spare);
    case EQ_EULER: return dispatch_kind<EQ_EULER>(d, a, list, nlist, s, spare);
    case EQ_MAXWELL: return dispatch_n<EQ_MAXWELL, NF_LF>(d, a, list, nlist, s, spare);
    case EQ_EULER2D: return dispatch_kind<EQ_EULER2D>(d, a, list, nlist, s, spare);
    case EQ_MAXWELL_TM: return dispatch_n<EQ_MAXWELL_TM, NF_LF>(d, a, list, nlist, s, spare);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_cut_nodes(int eq, const DgDev& d, const double* x, const int* blocks, int n, double* dst,
                             cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  switch (eq) {
    case EQ_ADVECTION: return cut_nodes_n<EQ_ADVECTION>(d, x, blocks, n, dst, s);
    case EQ_EULER: return cut_nodes_n<EQ_EULER>(d, x, blocks, n, dst, s);
    case EQ_MAXWELL: return cut_nodes_n<EQ_MAXWELL>(d, x, blocks, n, dst, s);
    case EQ_EULER2D: return cut_nodes_n<EQ_EULER2D>(d, x, blocks, n, dst, s);
    case EQ_MAXWELL_TM: return cut_nodes_n<EQ_MAXWELL_TM>(d, x, blocks, n, dst, s);
    default: return cudaErrorInvalidValue;
  }
}

namespace {
template <int EQ, int KIND> int warps_n(int N) {
  switch (N) {
    case 2: return Chain<EQ, 2, KIND>::WMAX;
    case 3: return Chain<EQ, 3, KIND>::WMAX;
    case 4: return Chain<EQ, 4, KIND>::WMAX;
    case 5: return Chain<EQ, 5, KIND>::WMAX;
    default: return 0;
  }
}
template <int EQ> int warps_kind(int N, int kind) {
  return kind == NF_HLL    ? warps_n<EQ, NF_HLL>(N)
         : kind == NF_ROE  ? warps_n<EQ, NF_ROE>(N)
         : kind == NF_WAVE ? warps_n<EQ, NF_WAVE>(N)
                           : warps_n<EQ, NF_LF>(N);
}
}  // namespace

// tiles of one wave of k_stage64 (the limit of form 2)
int stage64_wave_tiles(int eq, const DgDev& d, int sms) {
  const int kind = (int)d.eqp.p[3];
  switch (eq) {
    case EQ_ADVECTION: return sms * warps_n<EQ_ADVECTION, NF_LF>(d.N);
    case EQ_EULER: return sms * warps_kind<EQ_EULER>(d.N, kind);
    case EQ_MAXWELL: return sms * warps_n<EQ_MAXWELL, NF_LF>(d.N);
    case EQ_EULER2D: return sms * warps_kind<EQ_EULER2D>(d.N, kind);
    case EQ_MAXWELL_TM: return sms * warps_n<EQ_MAXWELL_TM, NF_LF>(d.N);
    default: return 0;
  }
}

}  // namespace apollo
