// Mode-coupling matrix of pseudo-Cl on the device: MaskDeconvolution.get_M
// (sht/mask_deconvolution.py:171-192),
//   M[l1][l2] = (2 l2 + 1)/(4 pi) sum_{l3 = |l1-l2|..l1+l2, l1+l2+l3 even} (2 l3 + 1) W[l3] w(l1,l2,l3)^2
// with w the Wigner 3j symbol (l1 l2 l3; 0 0 0) (sht/threej000.py:9-41).
//
// With g = (l1+l2+l3)/2 and q(n) = C(2n, n) / 4^n the closed form of the symbol is
//   w^2 = q(g-l1) q(g-l2) q(g-l3) / (q(g) (2g+1)),
// so with a = max(l1, l2), b = min, d = a - b, l3 = d + 2i, g = a + i the sum is
//   S(a, b) = sum_{i=0..b} G_d[i] q[b-i] r[a+i],  G_d[i] = q[i] q[d+i] (4i+2d+1) W[d+2i],
//   r[g] = 1 / (q[g] (2g+1)),
// symmetric in l1, l2.  One CTA per diagonal d builds q (a scan of the ratios (2n-1)/(2n)), r and
// G_d in shared memory; a thread takes the entries b of its diagonal: two operations and three
// shared-memory reads per term, Nl^3/6 terms in all, bound by the shared-memory pipe: 146 us at
// Nl = 1000.  (A walk over l3 by the ratio of consecutive symbols, with a division in every step of
// a dependent chain and both triangles computed, took 1513 us and lost three digits: 1.1e-12
// against 64 bits, now 8.4e-16.)  Above kMaxNl the arrays do not fit and that walk remains.
#include "dsht_internal.cuh"

namespace dsht {
namespace {

constexpr int kThreads = 256;
constexpr int kMaxNl = 5700;  // 5 Nl doubles of shared memory

__global__ void __launch_bounds__(kThreads)
mode_coupling_kernel(int Nl, const double* __restrict__ W, int nW, double* __restrict__ M) {
  extern __shared__ double sm[];
  __shared__ double wprod[kThreads / 32];
  const int K = 2 * Nl - 1;  // q, r for n = 0 .. 2 Nl - 2
  double* q = sm;
  double* r = q + K;
  double* G = r + K;
  const int d = blockIdx.x, nb = Nl - d;  // entries b = 0 .. nb - 1
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // q[n] = prod_{k=1..n} (2k-1)/(2k): runs of consecutive n per thread
  const int per = (K + kThreads - 1) / kThreads, n0 = threadIdx.x * per, n1 = min(n0 + per, K);
  double p = 1.0;
  for (int n = n0; n < n1; ++n)
    if (n) p *= (2.0 * n - 1.0) / (2.0 * n);
  double x = p;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x *= y;
  }
  if (lane == 31) wprod[warp] = x;
  const double before = __shfl_up_sync(0xffffffffu, x, 1);
  __syncthreads();
  double run = lane ? before : 1.0;
  for (int w = 0; w < warp; ++w) run *= wprod[w];
  for (int n = n0; n < n1; ++n) {
    if (n) run *= (2.0 * n - 1.0) / (2.0 * n);
    q[n] = run;
    r[n] = 1.0 / (run * (2.0 * n + 1.0));
  }
  __syncthreads();
  for (int i = threadIdx.x; i < nb; i += kThreads) {
    const int l3 = d + 2 * i;
    G[i] = l3 < nW ? q[i] * q[d + i] * ((2.0 * l3 + 1.0) * W[l3]) : 0.0;
  }
  __syncthreads();
  for (int b = threadIdx.x; b < nb; b += kThreads) {
    const int a = b + d;
    const double *qb = q + b, *ra = r + a;
    double s0 = 0.0, s1 = 0.0;
    int i = 0;
#pragma unroll 2
    for (; i + 1 <= b; i += 2) {
      s0 = fma(G[i], qb[-i] * ra[i], s0);
      s1 = fma(G[i + 1], qb[-i - 1] * ra[i + 1], s1);
    }
    if (i <= b) s0 = fma(G[i], qb[-i] * ra[i], s0);
    const double s = (s0 + s1) / (4.0 * M_PI);
    M[(size_t)a * Nl + b] = s * (2.0 * b + 1.0);
    M[(size_t)b * Nl + a] = s * (2.0 * a + 1.0);
  }
}

// Any Nl: one thread per (l1, l2) walks l3 upwards in steps of 2 with the ratio of w^2 between l3 + 2
// and l3, a rational function of (J = l1+l2+l3, l1, l2, l3), from the first value, at l3 = |l1 - l2|,
//   (2a-2b)! (2b)! / (2a+1)! x C(a, b)^2,
// by lgamma.
__global__ void mode_coupling_walk_kernel(int Nl, const double* __restrict__ W, int nW, double* __restrict__ M) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (int64_t)Nl * Nl) return;
  const int l1 = (int)(t / Nl), l2 = (int)(t % Nl);
  const int a = max(l1, l2), b = min(l1, l2);
  // l3 = a - b: J = 2a, g = a
  double w2 = exp(lgamma(2.0 * (a - b) + 1.0) + lgamma(2.0 * b + 1.0) - lgamma(2.0 * a + 2.0) +
                  2.0 * (lgamma(a + 1.0) - lgamma(a - b + 1.0) - lgamma(b + 1.0)));
  double s = 0.0;
  for (int l3 = a - b; l3 <= a + b; l3 += 2) {
    if (l3 < nW) s = fma((2.0 * l3 + 1.0) * W[l3], w2, s);
    if (l3 + 2 > a + b) break;
    const double J = (double)(l1 + l2 + l3), g = 0.5 * J;
    const double num = (J + 2 - 2 * l1) * (J + 1 - 2 * l1) * (J + 2 - 2 * l2) * (J + 1 - 2 * l2);
    const double den = (J - 2 * l3) * (J - 2 * l3 - 1) * (J + 3) * (J + 2);
    const double f = (g + 1) * (g - l3) / ((g + 1 - l1) * (g + 1 - l2));
    w2 *= num / den * f * f;
  }
  M[t] = s * (2.0 * l2 + 1.0) / (4.0 * M_PI);
}

}  // namespace
}  // namespace dsht

using namespace dsht;

extern "C" int dsht_mode_coupling(int Nl, const double* W, int nW, double* M, void* stream) {
  if (Nl < 1 || Nl > 46340 || nW < 0 || (nW > 0 && !W) || !M)
    return set_error(DSHT_ERR_INVALID, "invalid arguments (Nl=%d, nW=%d)", Nl, nW);
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (Nl <= kMaxNl) {
    const int bytes = 5 * Nl * (int)sizeof(double);
    DSHT_CUDA_OK(allow_shared(mode_coupling_kernel));
    mode_coupling_kernel<<<Nl, kThreads, bytes, s>>>(Nl, W, nW, M);
  } else {
    const int64_t n = (int64_t)Nl * Nl;
    mode_coupling_walk_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(Nl, W, nW, M);
  }
  count_launches(1);
  return launch_error("mode_coupling_kernel");
}
