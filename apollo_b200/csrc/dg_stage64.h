// Layout of the fused float64 stage's operator fragments (host and device):
// the B operands of its mma.m8n8k4 contractions in the order the lanes read
// them, built once per mesh by build_pack64 (dg_operators.cpp) and copied to
// shared memory by every block.
//
// Lane l holds B[k = l % 4][n = l / 4].  Nodes: k-step s holds the nodes
// 4 s + k; accumulator block b has node 8 b + 4 (n % 2) + n / 2 in column n, so
// a lane's two columns are its nodes of the k-steps 2 b and 2 b + 1 (four
// neighbouring lanes then hold four consecutive nodes: their shared-memory and
// global accesses are consecutive).  Points (cubature and face) come in blocks
// of eight with k-step j on the points 8 b + 2 k + j.
//   E  [FB][N+1][4][2 (j)]  interpolation along a face to the points 8 b + 2 c + j (lane column c)
//   L  [FB][NB][32][2 (j)]  surface lift with the Gauss weights
//   V  [PB][ceil(KS/2)][32][2 (k-step)]   nodes -> cubature points
//   D  [PB][2 (Dr, Ds)][NB][32][2 (j)]    weak derivatives
// linear equations:
//   Q  [QB][NB][32][2 (j)]  L E: surface lift from the 3 (N + 1) face nodes
//   W  [KS][NB][32][2 (Dr V, Ds V)]       weak derivatives from the nodes
// all:
//   S  [PB][NB][32][2 (j)]                sources
// adjoint (dg_deriv64.cu), the transposes:
//   DT [PB][KS][32][2 (Dr, Ds)]           nodes -> cubature points
//   VT [PB][NB][32][2 (j)]                cubature points -> nodes
//   ET [FB][NB][32][2 (j)]                face points -> nodes with the Gauss weights
//   Y  [KS][NB][32]                       V V^T (the lift is V V^T I^T)
//   WT [KS][NB][32][2]                    of Dr V and Ds V (linear equations)
//   Z  [QB][NB][32][2 (j)]                E^T diag(w) E per face, face nodes -> nodes (linear equations)
#pragma once

#include "dg_device.cuh"

namespace apollo {

template <int N> struct Pack64 {
  static constexpr int NP = Sizes<N>::NP, NC = Sizes<N>::NC, NG = Sizes<N>::NG, NF = Sizes<N>::NF;
  static constexpr int KS = (NP + 3) / 4, NB = (NP + 7) / 8, PB = (NC + 7) / 8, FB = (NF + 7) / 8, NFN = 3 * (N + 1),
                       QB = (NFN + 7) / 8;
  // node of k-step `k`, k index c (NP or above: none)
  APOLLO_HD static constexpr int node(int k, int c) { return 4 * k + c; }
  // node of column n of accumulator block b (-1: none)
  APOLLO_HD static constexpr int out_node(int b, int n) {
    const int v = 8 * b + 4 * (n % 2) + n / 2;
    return v < NP ? v : -1;
  }
  // node m (0..N) of face f in face order: the edges of the triangular node
  // numbering (row by row), from the face's first vertex to its second
  APOLLO_HD static constexpr int face_node(int f, int m) {
    return f == 0 ? m : f == 1 ? row(m) + N - m : row(N - m);
  }
  APOLLO_HD static constexpr int row(int j) { return j * (N + 1) - j * (j - 1) / 2; }  // first node of row j
  static constexpr int E_SIZE = FB * (N + 1) * 8;
  static constexpr int L_SIZE = FB * NB * 64;
  static constexpr int V_SIZE = PB * ((KS + 1) / 2) * 64;
  static constexpr int D_SIZE = PB * 2 * NB * 64;
  static constexpr int Q_SIZE = QB * NB * 64;
  static constexpr int W_SIZE = KS * NB * 64;
  static constexpr int S_SIZE = PB * NB * 64;
  static constexpr int E_OFF = 0, L_OFF = E_SIZE, V_OFF = L_OFF + L_SIZE, D_OFF = V_OFF + V_SIZE,
                       Q_OFF = D_OFF + D_SIZE, W_OFF = Q_OFF + Q_SIZE, S_OFF = W_OFF + W_SIZE;
  static constexpr int DT_SIZE = PB * KS * 64, VT_SIZE = PB * NB * 64, ET_SIZE = FB * NB * 64, Y_SIZE = KS * NB * 32;
  static constexpr int DT_OFF = S_OFF + S_SIZE, VT_OFF = DT_OFF + DT_SIZE, ET_OFF = VT_OFF + VT_SIZE,
                       Y_OFF = ET_OFF + ET_SIZE, WT_OFF = Y_OFF + Y_SIZE, Z_OFF = WT_OFF + W_SIZE,
                       SIZE = Z_OFF + Q_SIZE;
};

}  // namespace apollo
