// Layout of the operator fragments of the float64 fragment chains (host and
// device): the B operands of their mma.m8n8k4 contractions in the order the
// lanes read them, built once per mesh by build_pack64 (dg_operators.cpp) and
// copied to shared memory by every block.
//
// Lane l holds B[k = l % 4][n = l / 4].  Nodes: k-step s holds the nodes
// 4 s + k; accumulator block b has node 8 b + 4 (n % 2) + n / 2 in column n, so
// a lane's two columns are its nodes of the k-steps 2 b and 2 b + 1 (four
// neighbouring lanes then hold four consecutive nodes: their shared-memory and
// global accesses are consecutive).  One or two nodes past the last full block
// (TL; order 3 has two) would leave a block's columns mostly empty: they are
// summed per lane over the lane's k indices instead, and over the four lanes at
// the end.  Points (cubature and face) come in blocks of eight with k-step j on
// the points 8 b + 2 k + j.
//
// A "nodes" entry (NS doubles) holds [NB][32][2] for the blocks and [TL][4][2]
// for the rest, the last index two A operands: the point pair (j) or the pair
// (Dr, Ds) of one node k-step.
//   E  [FB][N+1][4][2 (j)]  interpolation along a face to the points 8 b + 2 c + j (lane column c)
//   L  [FB] nodes           surface lift with the Gauss weights
//   V  [PB][ceil(KS/2)][32][2 (k-step)]   nodes -> cubature points
//   D  [PB][2] nodes        weak derivatives Dr, Ds
// linear equations:
//   Q  [QB] nodes           L E: surface lift from the 3 (N + 1) face nodes
//   W  [KS] nodes           Dr V, Ds V: weak derivatives from the nodes
// all:
//   S  [PB] nodes           sources
// adjoint (dg_deriv64.cu), the transposes:
//   DT [PB][KS][32][2 (Dr, Ds)]           nodes -> cubature points
//   VT [PB] nodes           cubature points -> nodes
//   ET [FB] nodes           face points -> nodes with the Gauss weights
//   Y  [KS] nodes           V V^T in the first of the pair (the lift is V V^T I^T)
//   WT [KS] nodes           of Dr V and Ds V (linear equations)
//   Z  [QB] nodes           E^T diag(w) E per face, face nodes -> nodes (linear equations)
#pragma once

#include "dg_device.cuh"

namespace apollo {

template <int N> struct Pack64 {
  static constexpr int NP = Sizes<N>::NP, NC = Sizes<N>::NC, NG = Sizes<N>::NG, NF = Sizes<N>::NF;
  static constexpr int TL = NP % 8 == 1 || NP % 8 == 2 ? NP % 8 : 0;
  static constexpr int KS = (NP + 3) / 4, NB = (NP - TL + 7) / 8, NBT = NB + (TL > 0), PB = (NC + 7) / 8,
                       FB = (NF + 7) / 8, NFN = 3 * (N + 1), QB = (NFN + 7) / 8;
  static constexpr int NS = NB * 64 + TL * 8;
  // node of k-step `k`, k index c (NP or above: none)
  APOLLO_HD static constexpr int node(int k, int c) { return 4 * k + c; }
  // place of node n, k index c, operand j in a "nodes" entry
  APOLLO_HD static constexpr int place(int n, int c, int j) {
    return n < 8 * NB ? ((n / 8 * 32) + ((n % 4) * 2 + n % 8 / 4) * 4 + c) * 2 + j : NB * 64 + ((n - 8 * NB) * 4 + c) * 2 + j;
  }
  // node m (0..N) of face f in face order: the edges of the triangular node
  // numbering (row by row), from the face's first vertex to its second
  APOLLO_HD static constexpr int face_node(int f, int m) {
    return f == 0 ? m : f == 1 ? row(m) + N - m : row(N - m);
  }
  APOLLO_HD static constexpr int row(int j) { return j * (N + 1) - j * (j - 1) / 2; }  // first node of row j
  static constexpr int E_SIZE = FB * (N + 1) * 8, L_SIZE = FB * NS, V_SIZE = PB * ((KS + 1) / 2) * 64,
                       D_SIZE = PB * 2 * NS, Q_SIZE = QB * NS, W_SIZE = KS * NS, S_SIZE = PB * NS,
                       DT_SIZE = PB * KS * 64, VT_SIZE = PB * NS, ET_SIZE = FB * NS, Y_SIZE = KS * NS;
  static constexpr int E_OFF = 0, L_OFF = E_SIZE, V_OFF = L_OFF + L_SIZE, D_OFF = V_OFF + V_SIZE,
                       Q_OFF = D_OFF + D_SIZE, W_OFF = Q_OFF + Q_SIZE, S_OFF = W_OFF + W_SIZE,
                       DT_OFF = S_OFF + S_SIZE, VT_OFF = DT_OFF + DT_SIZE, ET_OFF = VT_OFF + VT_SIZE,
                       Y_OFF = ET_OFF + ET_SIZE, WT_OFF = Y_OFF + Y_SIZE, Z_OFF = WT_OFF + W_SIZE,
                       SIZE = Z_OFF + Q_SIZE;
};

}  // namespace apollo
