// Rotation of the polar points' alm back to the original frame, added to the equatorial alm.
//
// The polar points were rotated by +90 deg about y (Euler ZYZ (0, 90, 0)); their alm a'
// map back with Wigner d^l(pi/2):  a_lm = sum_{m'=-l..l} d^l_{m'm}(pi/2) a'_lm'.  For a
// real field (a'_{l,-m'} = (-1)^m' conj a'_lm') this is
//   Re a_lm = d_{0m} Re a'_l0 + 2 sum_{m'>0, l+m+m' even} d_{m'm} Re a'_lm'
//   Im a_lm =                   2 sum_{m'>0, l+m+m' odd}  d_{m'm} Im a'_lm'
// This stands in for healpy's Rotator(rot=(0,90,0), eulertype='ZYZ', inv=True).rotate_alm
// called at sht/sht.py:138-139.  d_{k,m}(pi/2) is generated per output m by the downward
// three-term recursion in k of Trapani & Navaza (Acta Cryst. A62, 262, 2006),
//   b_k d_{k-1,m} = 2m d_{k,m} - b_(k+1) d_{k+1,m},  b_k = sqrt((l+k)(l-k+1)),
// from d_{l,m} = (-1)^(l-m) 2^-l sqrt(C(2l, l+m)); values below the double range are
// carried with a binary exponent.
//
// Scaling the rows by d_k = s_k e_k with b_k s_(k-1) = b_(k+1) s_(k+1) turns the recursion into
//   e_(k-1) = 2m al_k e_k - e_(k+1),  al_k = s_k / (b_k s_(k-1)),
// one product and one FMA per step instead of two products and an FMA, and one FMA instead of
// three operations in its dependent chain; s_k goes into the coefficients a'.  al, s and the start
// values depend on (l, k) alone: they are tables of the plan (28 bytes per entry, 15 MB at
// Nl = 1024), built once with compensated products, so a call has no square roots, divisions or
// products over k to form.
//
// One CTA per l (the largest first); each thread runs up to four output columns m of one parity,
// which share every shared-memory read; one to eight maps share the recursion.  FP64 pipe bound: 3
// operations per (l, m, m') for one map, (2 + maps) for several; at Nl = 1024 1.1e9 operations,
// 60 us at the measured 62 per clock and SM.  Measured: one map 129 us (square roots and the start
// column in every call, four operations: 232), eight maps 522 (827).
#include <type_traits>

#include "dsht_internal.cuh"

namespace dsht {
namespace {

constexpr int kRotThreads = 256;

// Row l of a table starts at l (l + 1) / 2; entry i stands for k = l - i.
__host__ __device__ __forceinline__ int64_t tri(int l) { return (int64_t)l * (l + 1) / 2; }

// A product of quotients num / den with its relative rounding error: (1 + err) p 2^e.
struct Product {
  double p = 1.0, err = 0.0;
  int e = 0;
  __device__ void times(const Product& o) {
    const double n = __dmul_rn(p, o.p);
    err += o.err + fma(p, o.p, -n) / n;
    p = n;
    e += o.e;
    if (p > 0x1p64) {
      p *= 0x1p-64;
      e += 64;
    }
  }
  __device__ void times(double num, double den) {
    Product o;
    o.p = __ddiv_rn(num, den);
    o.err = fma(-o.p, den, num) / num;
    times(o);
  }
  // square root of 2^(2x) times the product, as a number and a binary exponent (e is a multiple of 64)
  __device__ double root(int x, int* exponent) const {
    *exponent = x + e / 2;
    return sqrt(p) * (1.0 + 0.5 * err);
  }
};

constexpr int kTabThreads = 128;

// s_k and the start values of row l = blockIdx.x as running products.  Chain 0: start values
// d_{l,m} = (-1)^(l-m) 2^-l sqrt(prod_{k=m+1..l} (l+k)/(l-k+1)); chains 1, 2: s_k for k = l, l-2, ...
// and k = l-1, l-3, ... from s_l = s_(l-1) = 1.  Each thread multiplies a run of factors, a block
// scan links the runs.
__global__ void __launch_bounds__(kTabThreads)
rotation_table_kernel(double* __restrict__ sc, double* __restrict__ start, int* __restrict__ start_e) {
  __shared__ Product total[kTabThreads / 32];
  const int l = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t row = tri(l);
  for (int chain = 0; chain < 3; ++chain) {
    // entry j of the chain stands for k; `step` multiplies by the factor between it and the next
    const int n = chain == 0 ? l + 1 : chain == 1 ? l / 2 + 1 : (l + 1) / 2;
    auto k_of = [&](int j) { return chain == 0 ? l - j : l - (chain - 1) - 2 * j; };
    auto step = [&](Product& p, int j) {
      const int k = k_of(j);
      if (j + 1 >= n) return;
      if (chain == 0) p.times((double)(l + k), (double)(l - k + 1));
      // s_(k-2)^2 = s_k^2 b_k^2 / b_(k-1)^2
      else p.times((double)(l + k) * (double)(l - k + 1), (double)(l + k - 1) * (double)(l - k + 2));
    };
    const int per = (n + kTabThreads - 1) / kTabThreads;
    const int j0 = min((int)threadIdx.x * per, n), j1 = min(j0 + per, n);
    Product p;
    for (int j = j0; j < j1; ++j) step(p, j);
    Product x = p;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      Product y;
      y.p = __shfl_up_sync(0xffffffffu, x.p, o);
      y.err = __shfl_up_sync(0xffffffffu, x.err, o);
      y.e = __shfl_up_sync(0xffffffffu, x.e, o);
      if (lane >= o) x.times(y);
    }
    __syncthreads();
    if (lane == 31) total[warp] = x;
    Product run;
    run.p = __shfl_up_sync(0xffffffffu, x.p, 1);
    run.err = __shfl_up_sync(0xffffffffu, x.err, 1);
    run.e = __shfl_up_sync(0xffffffffu, x.e, 1);
    if (lane == 0) run = Product{};
    __syncthreads();
    for (int w = 0; w < warp; ++w) run.times(total[w]);
    for (int j = j0; j < j1; ++j) {
      int e;
      if (chain == 0) {
        const double v = run.root(-l, &e);
        start[row + j] = (j & 1) ? -v : v;
        start_e[row + j] = e;
      } else {
        sc[row + l - k_of(j)] = run.root(0, &e);
      }
      step(run, j);
    }
  }
}

__global__ void rotation_alpha_kernel(int Nl, const double* __restrict__ sc, double* __restrict__ al) {
  const int l = blockIdx.y, i = blockIdx.x * blockDim.x + threadIdx.x, k = l - i;
  if (i > l) return;
  const int64_t at = tri(l) + i;
  al[at] = k >= 1 ? sc[at] / (sqrt((double)(l + k) * (double)(l - k + 1)) * sc[at + 1]) : 0.0;
}

// Columns m = m0, m0 + blockDim, ... (C of them, one parity) of degree l: out[map] += R(rot[map]), or (kAdd) out = add + R(rot).
// al: [i], S: [map][i] the coefficients of this parity's alternating real and imaginary rows, both
// padded with zeros.
template <int kMaps, int C, bool kAdd>
__device__ __forceinline__ void rotate_columns(int Nl, int l, int m0, int map0, int nm, const RotMaps& maps,
                                               const double* al, const double* S, int stride,
                                               const double* __restrict__ start, const int* __restrict__ start_e) {
  double c[C], n[C], m2[C], s[C][kMaps][2];
  int E[C];
#pragma unroll
  for (int j = 0; j < C; ++j) {
    const int m = m0 + j * kRotThreads;
    const bool in = m <= l;
    c[j] = in ? start[tri(l) + l - m] : 0.0;
    E[j] = in ? start_e[tri(l) + l - m] : 0;
    n[j] = 0.0;
    m2[j] = 2.0 * m;
#pragma unroll
    for (int g = 0; g < kMaps; ++g) s[j][g][0] = s[j][g][1] = 0.0;
  }
  // two steps at a time, the next two's values loaded meanwhile (the arrays end in a spare group)
  double2 an = *reinterpret_cast<const double2*>(al), vn[kMaps];
#pragma unroll
  for (int g = 0; g < kMaps; ++g) vn[g] = *reinterpret_cast<const double2*>(S + g * stride);
  for (int i = 0; i <= l; i += 4) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const double2 a = an;
      double2 v[kMaps];
      an = *reinterpret_cast<const double2*>(al + i + 2 * h + 2);
#pragma unroll
      for (int g = 0; g < kMaps; ++g) {
        v[g] = vn[g];
        vn[g] = *reinterpret_cast<const double2*>(S + g * stride + i + 2 * h + 2);
      }
#pragma unroll
      for (int j = 0; j < C; ++j) {
#pragma unroll
        for (int g = 0; g < kMaps; ++g) s[j][g][0] = fma(c[j], v[g].x, s[j][g][0]);
        const double p = fma(m2[j] * a.x, c[j], -n[j]);
#pragma unroll
        for (int g = 0; g < kMaps; ++g) s[j][g][1] = fma(p, v[g].y, s[j][g][1]);
        n[j] = p;
        c[j] = fma(m2[j] * a.y, p, -c[j]);
      }
    }
    // the growth of four steps is bounded, so a check every four is safe (on the exponent bits)
#pragma unroll
    for (int j = 0; j < C; ++j)
      if ((__double2hiint(c[j]) & 0x7fffffff) > 0x4ff00000) {  // |c| >= 2^256
        c[j] *= 0x1p-256;
        n[j] *= 0x1p-256;
#pragma unroll
        for (int g = 0; g < kMaps; ++g) {
          s[j][g][0] *= 0x1p-256;
          s[j][g][1] *= 0x1p-256;
        }
        E[j] += 256;
      }
  }
#pragma unroll
  for (int j = 0; j < C; ++j) {
    const int m = m0 + j * kRotThreads;
    if (m > l) continue;
    const double f = (E[j] > -1074) ? ldexp(1.0, E[j]) : 0.0;
    const int64_t at = 2 * hp_index(l, m, Nl);
#pragma unroll
    for (int g = 0; g < kMaps; ++g) {
      if (g < nm && (!maps.flags[map0 + g] || (*maps.flags[map0 + g] & kFlagHasPolar))) {
        double* out = maps.out[map0 + g];
        const double re = ((m & 1) ? s[j][g][1] : s[j][g][0]) * f, im = ((m & 1) ? s[j][g][0] : s[j][g][1]) * f;
        if constexpr (kAdd) {
          const double* add = maps.add;
          out[at] = (add ? add[at] : 0.0) + re;
          out[at + 1] = (add ? add[at + 1] : 0.0) + im;
        } else {
          out[at] += re;
          out[at + 1] += im;
        }
      }
    }
  }
}

// Maps blockIdx.y kMaps + g of degree l = Nl - 1 - blockIdx.x; a map without polar points is skipped
// (its rotated alm are zero).  C: most columns per thread at a time.
template <int kMaps, int C, bool kAdd>
__global__ void __launch_bounds__(kRotThreads)
rotate_back_kernel(int Nl, int nmaps, const RotMaps maps, const double* __restrict__ al_t,
                   const double* __restrict__ sc_t, const double* __restrict__ start,
                   const int* __restrict__ start_e) {
  extern __shared__ __align__(16) double sm[];
  const int l = Nl - 1 - blockIdx.x;
  const int map0 = blockIdx.y * kMaps;
  const int nm = min(kMaps, nmaps - map0);
  bool any = false;
#pragma unroll
  for (int g = 0; g < kMaps; ++g)
    any |= g < nm && (!maps.flags[map0 + g] || (*maps.flags[map0 + g] & kFlagHasPolar));
  if (!any) return;
  const int pad = ((l + 4) & ~3) + 2;  // l + 1 entries up to a multiple of four, and a spare pair
  double* al = sm;
  double* S = sm + pad;  // [parity of m][map][pad]
  for (int i = threadIdx.x; i < pad; i += blockDim.x) {
    const int k = l - i;
    al[i] = k >= 0 ? al_t[tri(l) + i] : 0.0;
    const double sc = k >= 0 ? sc_t[tri(l) + i] : 0.0;
    const int64_t at = k >= 0 ? 2 * hp_index(l, k, Nl) : 0;
#pragma unroll
    for (int g = 0; g < kMaps; ++g) {
      const bool ok = k >= 0 && g < nm && (!maps.flags[map0 + g] || (*maps.flags[map0 + g] & kFlagHasPolar));
      double re = 0.0, im = 0.0;
      if (ok) {
        re = maps.rot[map0 + g][at] * (k >= 1 ? 2.0 * sc : sc);
        im = k >= 1 ? maps.rot[map0 + g][at + 1] * (2.0 * sc) : 0.0;
      }
      // l + m + k even goes to the real part: i even for even m
      S[g * pad + i] = (i & 1) ? im : re;
      S[(kMaps + g) * pad + i] = (i & 1) ? re : im;
    }
  }
  __syncthreads();
  // a warp takes every second column: one parity, so that its shared-memory reads are broadcasts
  const int lane = threadIdx.x & 31, par = (threadIdx.x >> 5) & 1;
  const double* Sp = S + par * kMaps * pad;
  for (int first = (threadIdx.x >> 6) * 64 + par; first <= l; first += C * kRotThreads) {
    const int m0 = first + 2 * lane;
    const int left = (l - first) / kRotThreads + 1;  // columns of the warp's first lane from here on
    auto run = [&](auto columns) {
      constexpr int n = decltype(columns)::value < C ? decltype(columns)::value : C;
      rotate_columns<kMaps, n, kAdd>(Nl, l, m0, map0, nm, maps, al, Sp, pad, start, start_e);
    };
    switch (min(left, C)) {
      case 1: run(std::integral_constant<int, 1>{}); break;
      case 2: run(std::integral_constant<int, 2>{}); break;
      case 3: run(std::integral_constant<int, 3>{}); break;
      default: run(std::integral_constant<int, C>{}); break;
    }
  }
}

template <int kMaps, int C, bool kAdd = false>
void rotate_launch(const Geometry& g, const RotMaps& maps, int nmaps, const RotTables& t, cudaStream_t s) {
  const size_t smem = sizeof(double) * (size_t)(((g.Nl + 3) & ~3) + 2) * (1 + 2 * kMaps);
  allow_shared(rotate_back_kernel<kMaps, C, kAdd>);
  dim3 grid(g.Nl, (nmaps + kMaps - 1) / kMaps);
  rotate_back_kernel<kMaps, C, kAdd><<<grid, kRotThreads, smem, s>>>(g.Nl, nmaps, maps, t.al, t.sc, t.start, t.start_e);
  count_launches(1);
}

}  // namespace

size_t rotation_table_bytes(int Nl) { return (size_t)tri(Nl) * (3 * sizeof(double) + sizeof(int)); }

RotTables rotation_tables(void* base, int Nl) {
  double* d = static_cast<double*>(base);
  const size_t n = (size_t)tri(Nl);
  return RotTables{d, d + n, d + 2 * n, reinterpret_cast<int*>(d + 3 * n)};
}

void launch_rotation_tables(const Geometry& g, const RotTables& t, cudaStream_t s) {
  rotation_table_kernel<<<g.Nl, kTabThreads, 0, s>>>(t.sc, t.start, t.start_e);
  rotation_alpha_kernel<<<dim3((g.Nl + 255) / 256, g.Nl), 256, 0, s>>>(g.Nl, t.sc, t.al);
  count_launches(2);
}

void launch_rotate_back(const Geometry& g, const RotMaps& maps, int nmaps, const RotTables& t, cudaStream_t s) {
  if (nmaps <= 0) return;
  // As many maps per CTA (4, 2, 1) as shared memory holds.  For eight maps at
  // Nl = 1024 four maps and three columns take 522 us, two columns 541, four columns 765 and eight
  // maps with two columns 694 (registers: fewer CTAs per SM).
  auto bytes = [&](int k) { return sizeof(double) * (size_t)(((g.Nl + 3) & ~3) + 2) * (1 + 2 * k); };
  const size_t lim = 227 * 1024;
  if (maps.sum) rotate_launch<1, 4, true>(g, maps, 1, t, s);
  else if (nmaps > 2 && bytes(4) <= lim) rotate_launch<4, 3>(g, maps, nmaps, t, s);
  else if (nmaps == 2 && bytes(2) <= lim) rotate_launch<2, 2>(g, maps, nmaps, t, s);
  else rotate_launch<1, 4>(g, maps, nmaps, t, s);
}

}  // namespace dsht
