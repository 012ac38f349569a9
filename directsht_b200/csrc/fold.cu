// Fold the bin sums onto the spline nodes for the FP64 contraction (contract_fp64.cu).
//
// The contraction of the reference (sht/sht.py:274-277, sht/interp_funcs_py.py:59-60),
//   alm[lm] = sum_b Yv[lm,b] V0[b] + dx Yd[lm,b] V1[b] + Yv[lm,b+1] V2[b] + dx Yd[lm,b+1] V3[b],
// with V = vr - i vi, is linear in the table entries, so each node j collects
//   A[m,j] = V0[m,j] + V2[m,j-1],   B[m,j] = dx (V1[m,j] + V3[m,j-1]).
// The x < 0 half enters with (-1)^(l-m) (sht/sht.py:279); rows with l-m even use
// A+ + A-, odd rows A+ - A-, for the equatorial and the rotated polar sets.  B is stored as
// B' = B / (1 - x^2), what the contraction of the Y table alone needs.
//
// Output, in the order the m8n8k4 products read it:
//   fold[m][group of 8 nodes][parity][column n][q = 0..3][2]: nodes 8 g + 2 q, 2 q + 1 of column
//   n = 0..3: A (equatorial re, im, polar re, im), 4..7: B'.
// Nodes beyond Nx in the last group are zero.  The kernel also clears the alm rows that two
// items of the contraction add to, and notes which blocks of 16 nodes have points at all.
#include "dsht_internal.cuh"
#include "node_sums.cuh"

namespace dsht {
namespace {

constexpr int kFoldNodes = 16;  // nodes per block: warp = node, lane = m while the sums are read
constexpr int kFoldM = 32;
constexpr int kRowDoubles = kFoldNodes * 16 + 2;  // one m of the staging buffer, 16-byte pad

// A block covers 32 m x 16 nodes.  Sums are read with consecutive m in a warp (coalesced), go
// through shared memory, and leave as 2 KB runs of one m.  HBM / L2 bound: the sums read once,
// 128 bytes per (m, node) written.
template <typename Src>
__global__ void __launch_bounds__(32 * kFoldNodes)
fold_kernel(int Nl, int Nx, int nbins, int ngroups, double dx, const Src src, const uint32_t* __restrict__ offset,
            const FoldOut o) {
  extern __shared__ __align__(16) double stage[];  // [kFoldM][kRowDoubles]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int m0 = blockIdx.y * kFoldM, j0 = blockIdx.x * kFoldNodes;
  const int m = m0 + lane, j = j0 + warp;
  double* out = stage + lane * kRowDoubles + (warp >> 3) * 128 + ((warp & 7) >> 1) * 2 + (warp & 1);
  const double x = (double)j * dx;
  const double bf = j < Nx ? dx / (1.0 - x * x) : 0.0;  // (a padding node may lie at x = 1)
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    double acc[2][4];
    node_sums(src, Nl, Nx, h, j, m, acc);
#pragma unroll
    for (int par = 0; par < 2; ++par)
#pragma unroll
      for (int ri = 0; ri < 2; ++ri) {
        const double a = par ? acc[0][ri] - acc[1][ri] : acc[0][ri] + acc[1][ri];
        const double b = par ? acc[0][2 + ri] - acc[1][2 + ri] : acc[0][2 + ri] + acc[1][2 + ri];
        const int n = 2 * h + ri;
        out[par * 64 + n * 8] = a;
        out[par * 64 + (n + 4) * 8] = b * bf;
      }
  }
  if (blockIdx.y == 0) {
    const bool any = lane < kSets && j < Nx &&
                     offset[lane * nbins + min(j + 1, nbins)] != offset[lane * nbins + max(j - 1, 0)];
    const int live = __syncthreads_or(any);
    if (threadIdx.x == 0) o.live[blockIdx.x] = live != 0;
    if (threadIdx.x == 0 && blockIdx.x == 0) *o.next_item = 0;
  }
  // rows m + kContractRows b - 1 and + 0 of the alm take two atomic contributions
  if (blockIdx.x == 0 && m < Nl)
    for (int l = m + kContractRows * ((warp >> 1) + 1) - (warp & 1); l < Nl; l += kContractRows * kFoldNodes / 2) {
      const int64_t i = 2 * hp_index(l, m, Nl);
      o.equ[i] = o.equ[i + 1] = 0.0;
      o.pol[i] = o.pol[i + 1] = 0.0;
    }
  __syncthreads();
  const int g0 = 2 * blockIdx.x, ng = min(2, ngroups - g0);
  for (int r = warp; r < kFoldM && m0 + r < Nl; r += kFoldNodes) {
    const double2* s = reinterpret_cast<const double2*>(stage + r * kRowDoubles);
    double2* d = reinterpret_cast<double2*>(o.fold + (size_t)(m0 + r) * fold_stride(Nx) + (size_t)g0 * 128);
    for (int e = lane; e < ng * 64; e += 32) d[e] = s[e];
  }
}

}  // namespace

void launch_fold(const Geometry& g, const Workspace& ws, const FoldOut& out, cudaStream_t s) {
  const int ngroups = (g.Nx + 7) / 8;
  dim3 grid((g.Nx + kFoldNodes - 1) / kFoldNodes, (g.Nl + kFoldM - 1) / kFoldM);
  constexpr int kBytes = kFoldM * kRowDoubles * (int)sizeof(double);
  with_node_source(g, ws, [&](auto src) {
    auto kern = fold_kernel<decltype(src)>;
    allow_shared(kern);
    kern<<<grid, 32 * kFoldNodes, kBytes, s>>>(g.Nl, g.Nx, g.nbins, ngroups, g.dx, src, ws.offset, out);
  });
  count_launches(1);
}

}  // namespace dsht
