// Bin sums collected onto the spline nodes, as the two folds (fold.cu, digits.cu) read them.
//
// Node j of set s takes A = V0(bin j) + V2(bin j - 1) and B/dx = V1(bin j) + V3(bin j - 1),
// V = vr - i vi, summed over the pieces of each bin.
#pragma once

#include "dsht_internal.cuh"

namespace dsht {

// Sums per piece: partial[piece][2 k + (re | im)][m], T = double (FP64 sums) or float
// (tensor-core sums); the pieces of key = set nbins + bin are [piece_first[key], piece_first[key + 1]).
template <typename T>
struct PieceSums {
  const int* piece_first;
  const T* partial;
  int nbins;
};

// acc[si][A re, A im, B/dx re, B/dx im] of node j and column m for the sets 2 h + si.  The
// first piece of every key is read before any further ones, so 16 loads are in flight together
// (most bins are one piece).
template <typename T>
__device__ __forceinline__ void node_sums(const PieceSums<T>& src, int Nl, int Nx, int h, int j, int m,
                                          double (&acc)[2][4]) {
  int pa[2][2], pb[2][2];
#pragma unroll
  for (int si = 0; si < 2; ++si)
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      const bool ok = m < Nl && j < Nx && (b ? j >= 1 : j < src.nbins);
      const int key = (2 * h + si) * src.nbins + j - b;
      pa[si][b] = ok ? src.piece_first[key] : 0;
      pb[si][b] = ok ? src.piece_first[key + 1] : 0;
    }
#pragma unroll
  for (int si = 0; si < 2; ++si) {
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[si][c] = 0.0;
#pragma unroll
    for (int b = 0; b < 2; ++b)
      if (pa[si][b] < pb[si][b]) {
        const T* v = src.partial + (size_t)pa[si][b] * 8 * Nl + (size_t)(4 * b) * Nl + m;
        acc[si][0] += v[0];
        acc[si][1] -= v[(size_t)Nl];
        acc[si][2] += v[(size_t)2 * Nl];
        acc[si][3] -= v[(size_t)3 * Nl];
      }
  }
#pragma unroll
  for (int si = 0; si < 2; ++si)
#pragma unroll
    for (int b = 0; b < 2; ++b)
      for (int p = pa[si][b] + 1; p < pb[si][b]; ++p) {
        const T* v = src.partial + (size_t)p * 8 * Nl + (size_t)(4 * b) * Nl + m;
        acc[si][0] += v[0];
        acc[si][1] -= v[(size_t)Nl];
        acc[si][2] += v[(size_t)2 * Nl];
        acc[si][3] -= v[(size_t)3 * Nl];
      }
}

// Sums per node slot (NUFFT sums): node i of the live nodes (numbered in key order) has one slot
// i + 2 c for every CTA c that holds points of its two bins; slots[slot][A re, A im, B/dx re, B/dx im][m],
// already as V = vr - i vi.
struct NodeSlots {
  const int* piece_first;
  const int* piece_cta;
  const uint32_t* node_first;
  const double* slots;
  int nbins;
};

__device__ __forceinline__ void node_sums(const NodeSlots& src, int Nl, int Nx, int h, int j, int m,
                                          double (&acc)[2][4]) {
  // the pieces that feed the node: the right side of bin j - 1, then the left side of bin j
  int pa[2], pb[2], mid[2];
  uint32_t node[2];
#pragma unroll
  for (int si = 0; si < 2; ++si) {
    const bool in = m < Nl && j < Nx;
    const int key = (2 * h + si) * src.nbins + j;  // bin j (absent for the last node)
    mid[si] = in ? src.piece_first[key] : 0;
    pa[si] = in && j >= 1 ? src.piece_first[key - 1] : mid[si];
    pb[si] = in && j < src.nbins ? src.piece_first[key + 1] : mid[si];
    // left node of bin j if that has points, else the right node of bin j - 1
    node[si] = pb[si] > mid[si] ? src.node_first[key + 1] - 2 : (pa[si] < mid[si] ? src.node_first[key] - 1 : 0u);
  }
#pragma unroll
  for (int si = 0; si < 2; ++si) {
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[si][c] = 0.0;
    int cta = -1;
    for (int p = pa[si]; p < pb[si]; ++p) {
      const int c = src.piece_cta[p];
      if (c == cta) continue;
      cta = c;
      const double* v = src.slots + (size_t)(node[si] + 2 * c) * 4 * Nl + m;
      acc[si][0] += v[0];
      acc[si][1] += v[(size_t)Nl];
      acc[si][2] += v[(size_t)2 * Nl];
      acc[si][3] += v[(size_t)3 * Nl];
    }
  }
}

// Calls f with the source the workspace's bin sums were written to.
template <typename F>
void with_node_source(const Geometry& g, const Workspace& ws, F f) {
  if (ws.nu_grid)
    f(NodeSlots{ws.piece_first, ws.piece_cta, ws.node_first, ws.partial, g.nbins});
  else if (ws.partial_f32)
    f(PieceSums<float>{ws.piece_first, reinterpret_cast<const float*>(ws.partial), g.nbins});
  else
    f(PieceSums<double>{ws.piece_first, ws.partial, g.nbins});
}

}  // namespace dsht
