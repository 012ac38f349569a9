// Per-bin sums by a type-1 non-uniform FFT, collected on the spline nodes (the FP64 level, and
// the MIXED level's default bin-sum method).
//
// The sums of the points of one (set, bin) key (sht/shared_interp_funcs.py:88-105),
//   v_k[m] = sum_p g_k(p) e^{i m phi_p},  g_k = w h_k(t) (sht/sht.py:239-240),  0 <= m < Nl,
// are needed only as the node sums A_j = v_0(bin j) + v_2(bin j-1), B_j/dx = v_1(bin j) + v_3(bin j-1),
// so the points of bins j - 1 and j are spread onto one pair of periodic grids per node, A the real
// part and B the imaginary part of one complex sequence of n cells, with the "exponential of
// semicircle" kernel (Barnett, Magland & af Klinteberg, SIAM J. Sci. Comput. 41 (2019) C479)
//   psi(x) = exp(beta (sqrt(1 - (2x/W)^2) - 1)),  |x| < W/2 cells.
// One complex FFT per node gives
//   V[m] = (sum_j G[j] e^{2 pi i m j / n}) / Psi(m),  Psi(m) = int psi(x) e^{-2 pi i m x/n} dx,
// and A and B come apart by the conjugate symmetry of a real sequence's transform.  (One
// transform pair per bin, as the sums are written, would take twice the FFTs and twice the
// partial sums.)
//
// Two accuracy classes.  FP64 level: W = 16, polynomials of degree 15, n = 8 or 4 times
// 2^ceil(log2 Nl) (oversampling 4 up to Nl = 256, 2 above); the truncation error is 2.4e-15 of
// the root-sum-square of g at oversampling 2 and below rounding at 4, where the direct sums' angle
// recurrences lose m 2^-54: 1.4e-14 at Nl = 512, 5.9e-15 at 256.  MIXED: W = 12, degree 11,
// oversampling 2, error about 5e-12 of sum |g|.
//
// Kernel values: psi at the W cells next to a point is one polynomial per cell in the point's
// fractional offset f, s = 2 f - 1 (Chebyshev interpolants, converted to monomials on the host).
// Cells i and W - 1 - i have the same even part and opposite odd parts, so two cells take one
// Horner recursion in s^2 each for the even and the odd half.  The coefficients are kernel
// parameters: every step is one DFMA with a uniform operand.
//
// One CTA takes a contiguous run of pieces (up to eight points per thread, of one key, in key order), equal
// shares of points + C0 x pieces, and walks its keys with the left and the right node's grids in
// shared memory: when the key advances, the left node is finished (FFT, extraction, one slot of
// node sums written), and the right node becomes the next left node.  Every point is read and
// its kernel values are formed once.  Nodes at the ends of a run are finished by both CTAs; the
// folds add the two slots.  (n = 8192 has room for one grid: there every key is spread twice,
// once for each node.)
//
// The spread.  A piece's points are first counting-sorted by grid cell (shared memory histogram and
// scan).  Each half warp takes an equal share of the sorted points, 16 at a time: one lane
// per point forms the kernel values and weights and stages them; then the half warp takes the points
// in turn, lane s owning the cells congruent s mod 16 of the point's window, with the four
// running sums of its current cell in registers: one kernel value and the point's weights from
// shared memory and four DFMA.  When the window moves past a lane's cell the lane adds its sums to
// the grids with plain loads and stores: cells the window has left belong to one half warp
// alone, as the points are sorted.  The last windows, which may overlap the neighbours', are
// added with atomics after a barrier.  (Fixed-point reductions of every value into shared
// memory -- 96 per point, 3 clocks per warp instruction on random banks -- took 0.51 of
// 0.96 ms at Nl = 1024, N = 1e7; a whole warp per point with half the lanes for each node took 18
// clocks of an SM per point against 11 now, by its instruction count.)
//
// MIXED class: the sums do not depend on the order of the adds.  The weights are scaled by a
// power of two such that the node's sum |w| is below 2^50, and the running sums start at
// 1.5 2^52: every FMA then rounds its product to an integer and all later adds are exact.  So a
// transform repeats bit for bit although the sort leaves the points of a bin in any order.  (A NaN
// or infinite weight makes every sum of its nodes NaN.)  FP64 class: plain FP64 sums.
//
// The in-place decimation-in-frequency FFT takes a first radix-8, -16 or -4 pass (the remainder of
// log2 n by three), radix-8 passes, and a last radix-8 pass that keeps its outputs: a thread takes
// the butterflies of k and -k, separates A and B and writes the sums.  Grid index i is stored at i
// with its low octal digit XORed by the next three digits, so that strides of 1, 8, 64 and 512
// all hit distinct 16-byte banks (padding would not leave room for the staging areas).
#include <cmath>
#include <mutex>
#include <vector>

#include "dsht_internal.cuh"

namespace dsht {

// Kernel-parameter copy of the per-cell polynomials: c[i][d], cell i = 0..W/2-1 of a point
// whose cell is c0 is (c0 - W/2 + 1 + i) and its offset x = f + W/2 - 1 - i, f = u - c0.
template <int W, int DEG>
struct EsPoly {
  double c[W / 2][DEG + 1];
};

namespace {

// Points of a piece: eight per thread (their cells stay in registers through the sort).
__host__ __device__ constexpr int nu_piece(int threads) { return 8 * threads; }

constexpr int kNuSlots = 16;  // cells of a point's window (W <= 16; the rest weigh zero)
constexpr int kStagePts = 32;  // points staged at a time per warp
// Bytes staged per point: kernel values, weights (of both nodes, or of one), first cell.
constexpr int point_stage(bool two) { return kNuSlots * 8 + (two ? 32 : 16) + 2; }

// Place of grid index i: linear over XOR, so places of indices with disjoint bits XOR together.
__host__ __device__ __forceinline__ int sw(int i) { return i ^ (((i >> 3) ^ (i >> 6) ^ (i >> 9)) & 7); }

__device__ __forceinline__ double2 cmul2(double2 a, double2 b) {
  return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}

// cos, sin of 2 pi e / 16 for a compile-time e (after unrolling).
__device__ __forceinline__ double cos16(int e) {
  constexpr double kCos1 = 0.92387953251128675613, kCos2 = 0.70710678118654752440, kCos3 = 0.38268343236508977173;
  switch (e & 15) {
    case 0: return 1.0;
    case 1: return kCos1;
    case 2: return kCos2;
    case 3: return kCos3;
    case 4: return 0.0;
    case 5: return -kCos3;
    case 6: return -kCos2;
    case 7: return -kCos1;
    case 8: return -1.0;
    case 9: return -kCos1;
    case 10: return -kCos2;
    case 11: return -kCos3;
    case 12: return 0.0;
    case 13: return kCos3;
    case 14: return kCos2;
    default: return kCos1;
  }
}
__device__ __forceinline__ double sin16(int e) { return cos16(e - 4); }

// v * e^{2 pi i e / R}; the quarter turns are exact swaps and sign changes.
template <int R>
__device__ __forceinline__ double2 rot(double2 v, int e) {
  const int e16 = (e * (16 / R)) & 15;
  if (e16 == 0) return v;
  if (e16 == 4) return make_double2(-v.y, v.x);
  if (e16 == 8) return make_double2(-v.x, -v.y);
  if (e16 == 12) return make_double2(v.y, -v.x);
  const double c = cos16(e16), s = sin16(e16);
  return make_double2(fma(v.x, c, -v.y * s), fma(v.x, s, v.y * c));
}

// In-register R-point DFT with the + sign, y_S = sum_r x_r e^{2 pi i r S / R}.  R = 8, 16
// split as 4 x (R/4): radix-4 over r = 4-blocks, twiddle, R/4-point DFTs; output S lands
// in register dreg<R>(S).
template <int R>
__device__ __forceinline__ constexpr int dreg(int S) {
  return R <= 4 ? S : (R / 4) * (S % 4) + S / 4;
}

__device__ __forceinline__ void dft4(double2& x0, double2& x1, double2& x2, double2& x3) {
  const double2 a0 = make_double2(x0.x + x2.x, x0.y + x2.y), a1 = make_double2(x0.x - x2.x, x0.y - x2.y);
  const double2 b0 = make_double2(x1.x + x3.x, x1.y + x3.y), b1 = make_double2(x1.x - x3.x, x1.y - x3.y);
  x0 = make_double2(a0.x + b0.x, a0.y + b0.y);
  x2 = make_double2(a0.x - b0.x, a0.y - b0.y);
  x1 = make_double2(a1.x - b1.y, a1.y + b1.x);  // a1 + i b1
  x3 = make_double2(a1.x + b1.y, a1.y - b1.x);  // a1 - i b1
}

template <int R>
__device__ __forceinline__ void dft(double2 (&x)[R]) {
  if constexpr (R == 4) {
    dft4(x[0], x[1], x[2], x[3]);
  } else {
    constexpr int R2 = R / 4;
    // radix 4 over the blocks of R2: element t + R2 r, output s goes to register t + R2 s
#pragma unroll
    for (int t = 0; t < R2; ++t) {
      dft4(x[t], x[t + R2], x[t + 2 * R2], x[t + 3 * R2]);
#pragma unroll
      for (int s = 1; s < 4; ++s) x[t + R2 * s] = rot<R>(x[t + R2 * s], t * s);
    }
    // R2-point DFTs of each s: registers R2 s .. R2 s + R2 - 1, output k' in register R2 s + k'
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      if constexpr (R2 == 2) {
        const double2 a = x[R2 * s], b = x[R2 * s + 1];
        x[R2 * s] = make_double2(a.x + b.x, a.y + b.y);
        x[R2 * s + 1] = make_double2(a.x - b.x, a.y - b.y);
      } else {
        dft4(x[R2 * s], x[R2 * s + 1], x[R2 * s + 2], x[R2 * s + 3]);
      }
    }
  }
}


// x[S] times e^{2 pi i S j / L} after a butterfly, w1 = e^{2 pi i j / L}: S = 4 h + l takes the
// product of powers 4 h and l (at most four roundings deep).
template <int R>
__device__ __forceinline__ void twiddle(double2 (&x)[R], double2 w1) {
  const double2 w2 = cmul2(w1, w1), w3 = cmul2(w2, w1), w4 = cmul2(w2, w2);
  double2 wh = w4;
#pragma unroll
  for (int S = 1; S < R; ++S) {
    const double2 wl = (S & 3) == 1 ? w1 : (S & 3) == 2 ? w2 : w3;
    if (S > 4 && (S & 3) == 0) wh = cmul2(wh, w4);
    x[dreg<R>(S)] = cmul2(x[dreg<R>(S)], S < 4 ? wl : (S & 3) == 0 ? wh : cmul2(wh, wl));
  }
}

// One decimation-in-frequency pass of radix R over span L: butterfly (b, j), base = b L + j,
// elements base + r L/R; outputs S times e^{2 pi i j S / L} back to base + S L/R.
// tw[i] = e^{2 pi i i / n}.  The bits of base and r L/R are disjoint.
template <int R>
__device__ __forceinline__ void fft_pass(double2* z, int logn, int logL, const double2* __restrict__ tw) {
  constexpr int logR = R == 4 ? 2 : R == 8 ? 3 : 4;
  const int logs = logL - logR;
  for (int q = threadIdx.x; q < 1 << (logn - logR); q += blockDim.x) {
    const int j = q & ((1 << logs) - 1);
    const int base = sw(((q >> logs) << logL) + j);
    double2 x[R];
#pragma unroll
    for (int r = 0; r < R; ++r) x[r] = z[base ^ sw(r << logs)];
    dft<R>(x);
    if (j) twiddle<R>(x, tw[j << (logn - logL)]);
#pragma unroll
    for (int S = 0; S < R; ++S) z[base ^ sw(S << logs)] = x[dreg<R>(S)];
  }
}

// log2 of the first pass's radix: 3 when logn is a multiple of three, else 4 (one bit over) or 2.
__host__ __device__ constexpr int first_radix(int logn) { return logn % 3 == 0 ? 3 : logn % 3 == 1 ? 4 : 2; }

// Entries of the twiddle table: index j n / L < n / R of every pass.
__host__ __device__ __forceinline__ int tw_count(int logn) { return 1 << (logn - (first_radix(logn) < 3 ? 2 : 3)); }

// Position of the last pass's first element for output k < n / 8 (the first pass's digit is the
// most significant; output k + S n / 8 comes out S places on).
__device__ __forceinline__ int fft_pos(int k, int logn) {
  int lg = logn - first_radix(logn);
  int pos = (k & ((1 << first_radix(logn)) - 1)) << lg;
  k >>= first_radix(logn);
  while (lg > 3) {
    lg -= 3;
    pos += (k & 7) << lg;
    k >>= 3;
  }
  return pos;
}

// The whole transform of grid z and its node sums V[m] = (A re, A im, B re, B im), m < Nl <= n/4,
// with V = vr - i vi; R1: the first pass's radix.  A = (Z[m] + conj Z[-m]) / 2, B = (Z[m] - conj Z[-m]) / 2i, over Psi(m) and times f.
template <int R1>
__device__ __forceinline__ void fft_node(double2* z, int logn, const double2* __restrict__ tw, int Nl, double f,
                                         const double* __restrict__ dinv, double* __restrict__ o) {
  fft_pass<R1>(z, logn, logn, tw);
  __syncthreads();
  for (int logL = logn - first_radix(logn); logL > 3; logL -= 3) {
    fft_pass<8>(z, logn, logL, tw);
    __syncthreads();
  }
  const int B = 1 << (logn - 3);
  auto put = [&](int m, double di, double2 u, double2 v) {  // u = Z[m], v = Z[-m]
    if (m >= Nl) return;
    o[m] = (u.x + v.x) * di;
    o[(size_t)Nl + m] = (v.y - u.y) * di;
    o[(size_t)2 * Nl + m] = (u.y + v.y) * di;
    o[(size_t)3 * Nl + m] = (u.x - v.x) * di;
  };
  f *= 0.5;
  // Outputs k + S B of butterfly k; -(k + S B) = (B - k) + (7 - S) B for k > 0: the lower half warp takes
  // k = i, the upper one k = B - i, and they exchange outputs 6 and 7.
  const int lane = threadIdx.x & 31, up = lane >> 4;
  for (int i0 = 16 * (int)(threadIdx.x >> 5); i0 <= B / 2; i0 += blockDim.x / 2) {
    const int i = min(i0 + (lane & 15), B / 2);
    const int k = up ? (B - i) & (B - 1) : i;
    double2 x[8];
    const int base = sw(fft_pos(k, logn));
#pragma unroll
    for (int r = 0; r < 8; ++r) x[r] = z[base ^ r];
    const double d0 = k < Nl ? f * dinv[k] : 0.0, d1 = k + B < Nl ? f * dinv[k + B] : 0.0;
    dft<8>(x);
    const double2 x0 = x[dreg<8>(0)], x1 = x[dreg<8>(1)], x6 = x[dreg<8>(6)], x7 = x[dreg<8>(7)];
    double2 v0, v1;
    v0.x = __shfl_xor_sync(0xffffffffu, x7.x, 16);
    v0.y = __shfl_xor_sync(0xffffffffu, x7.y, 16);
    v1.x = __shfl_xor_sync(0xffffffffu, x6.x, 16);
    v1.y = __shfl_xor_sync(0xffffffffu, x6.y, 16);
    if (i0 + (lane & 15) > B / 2 || (up && (i == 0 || i == B / 2))) continue;
    put(k, d0, x0, k ? v0 : x0);
    put(k + B, d1, x1, k ? v1 : x7);
  }
}

constexpr int kMeta = 64;  // descriptors of upcoming pieces kept in shared memory

// The FP64 class's kernel values carry this power of two: a grid's transform sums the several cells of
// every point, and weights near the largest double must not overflow there where their sums do not.
constexpr double kRange = 0x1p-8;

// Shared memory of a launch: the grids, the twiddles, the sorted points' indices, then the warps'
// staging areas, which the cell counters share.
template <int T, bool TWO>
struct NuLayout {
  int n;
  __host__ __device__ explicit NuLayout(int logn) : n(1 << logn) {}
  __host__ __device__ int tw_off() const { return 16 * n * (TWO ? 2 : 1); }
  // (two CTAs of n = 2048 leave no room for the twiddles: those read them through L1)
  __host__ __device__ static constexpr bool tw_smem(int logn) { return first_radix(logn) != 2; }
  __host__ __device__ int idx_off(int logn) const { return tw_off() + (tw_smem(logn) ? 16 * tw_count(logn) : 0); }
  __host__ __device__ int stage_off(int logn) const { return idx_off(logn) + 2 * nu_piece(T); }
  __host__ __device__ int bytes(int logn) const {
    const int st = T / 32 * kStagePts * point_stage(TWO), cnt = 2 * n;
    return stage_off(logn) + (st > cnt ? st : cnt);
  }
};

struct NuArgs {
  int Nl, logn, nbins;
  const double* pay;
  const int64_t* piece_start;
  const int* piece_len;
  const int* piece_key;
  const int* cta_first;        // [grid + 1] first piece of every CTA
  const uint32_t* node_first;  // [nkeys + 1] live nodes before a key (points.cu)
  const double* dinv;
  const double2* tw;
  double* slots;  // [slot][A re, A im, B/dx re, B/dx im][Nl]
  double* wsum;   // [piece] sum |w| with a rounding margin, or null
};

template <int W, int DEG, int T, bool TWO, int R1>
__global__ void __launch_bounds__(T, T == 512 ? 1 : 2)
nufft_nodes_kernel(const NuArgs a, const EsPoly<W, DEG> es) {
  static_assert(W % 2 == 0 && W <= kNuSlots && DEG % 2 == 1, "window and polynomial shape");
  constexpr bool kExact = W == 12;    // MIXED class: sums of integers, independent of the order
  constexpr int kPer = nu_piece(T) / T;  // points of a piece per thread
  constexpr int kWarps = T / 32;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ uint32_t wtot[kWarps];
  __shared__ double wred[kWarps];
  __shared__ uint4 meta[kMeta];  // piece: key, points, first point, right node's number
  const int logn = a.logn, n = 1 << logn, Nl = a.Nl;
  const NuLayout<T, TWO> lay(logn);
  double2* X = reinterpret_cast<double2*>(smem);             // grid of the left node
  double2* Y = TWO ? X + n : X;                              // grid of the right node
  double2* tw_copy = reinterpret_cast<double2*>(smem + lay.tw_off());
  const double2* tws = R1 == 4 ? a.tw : tw_copy;
  uint16_t* sorted = reinterpret_cast<uint16_t*>(smem + lay.idx_off(logn));
  uint32_t* cnt = reinterpret_cast<uint32_t*>(smem + lay.stage_off(logn));  // two 16-bit counters per word
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, slot = lane & 15, half = lane >> 4;
  // staging of the warp's 32 points, sixteen of each half warp: kernel values (value i of point q at
  // place (i + q) mod 16 of its row), weights, first cells
  double* ker = reinterpret_cast<double*>(smem + lay.stage_off(logn) + warp * (kStagePts * point_stage(TWO)));
  double2* gst = reinterpret_cast<double2*>(ker + kStagePts * kNuSlots);
  int16_t* cbs = reinterpret_cast<int16_t*>(gst + (TWO ? 2 : 1) * kStagePts);
  const int p0 = a.cta_first[blockIdx.x], p1 = a.cta_first[blockIdx.x + 1];
  if (p0 >= p1) return;
  if (R1 != 4)
    for (int i = tid; i < tw_count(logn); i += T) tw_copy[i] = a.tw[i];
  auto clear = [&](double2* g) {
    for (int i = tid; i < n; i += T) g[i] = make_double2(0.0, 0.0);
  };
  clear(X);
  if (TWO) clear(Y);

  // Descriptors: the ring holds pieces up to p0 + loaded - 1, at least 32 beyond the current one.
  int loaded = 0;
  auto load_meta = [&]() {  // 32 more
    const int p = p0 + loaded + tid;
    if (tid < kMeta / 2 && p < p1) {
      const int key = a.piece_key[p];
      meta[(loaded + tid) & (kMeta - 1)] =
          make_uint4((uint32_t)key, (uint32_t)a.piece_len[p], (uint32_t)a.piece_start[p], a.node_first[key + 1] - 1u);
    }
    loaded += kMeta / 2;
  };
  auto desc = [&](int p) -> uint4 { return meta[(p - p0) & (kMeta - 1)]; };
  auto key_at = [&](int p) -> int {
    return p - p0 < loaded ? (int)meta[(p - p0) & (kMeta - 1)].x : a.piece_key[p];
  };
  auto end_of_key = [&](int p) {
    const int key = key_at(p);
    int q = p + 1;
    while (q < p1 && key_at(q) == key) ++q;
    return q;
  };
  auto records = [&](int p, int* len) -> const double* {
    if (p - p0 < loaded) {
      const uint4 d = desc(p);
      *len = (int)d.y;
      return a.pay + (size_t)kRec * d.z;
    }
    *len = a.piece_len[p];
    return a.pay + (size_t)kRec * a.piece_start[p];
  };

  // This thread's share of sum |w| of piece p.
  auto weigh_part = [&](int p) {
    int len;
    const double* r = records(p, &len);
    double v[kPer], t = 0.0;
#pragma unroll
    for (int u = 0; u < kPer; ++u) v[u] = tid + u * T < len ? fabs(r[(size_t)kRec * (tid + u * T) + 2]) : 0.0;
#pragma unroll
    for (int u = 0; u < kPer; ++u) t += v[u];
    return t;
  };
  auto warp_sum = [&](double t) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) wred[warp] = t;
  };
  // after a barrier: sum |w| of piece p with a margin for its own rounding, to wsum as well
  auto piece_sum = [&](int p) {
    int len;
    records(p, &len);
    double t = 0.0;
#pragma unroll
    for (int i = 0; i < kWarps; ++i) t += wred[i];
    t *= 1.0 + (double)len * 0x1p-52;
    if (tid == 0 && a.wsum) a.wsum[p] = t;
    return t;
  };
  // the same for pieces [p, q), nothing overlapped
  auto weigh = [&](int p, int q) {
    double total = 0.0;
#pragma unroll 1
    for (int r = p; r < q; ++r) {
      const double t = weigh_part(r);
      __syncthreads();
      warp_sum(t);
      __syncthreads();
      total += piece_sum(r);
    }
    return total;
  };
  // scale 2^(50 - e) with v < 2^e (NaN for a sum that is not finite)
  auto fixed_scale = [&](double v) {
    int e = 0;
    if (v > 0.0) frexp(v, &e);
    return v < __longlong_as_double(0x7ff0000000000000ll) ? ldexp(1.0, 50 - max(e, -900))
                                                          : __longlong_as_double(0x7ff8000000000000ll);
  };

  double w_cur = 0.0, w_next = 0.0;  // sum |w| of this key and the next
  double sx = 1.0, sy = 1.0;         // scales of X and Y

  // Adds the points of piece p: to both grids (TWO; weights of the bin's left node to
  // X, times sx, of its right node to Y, times sy), or to X with the weights of one role.  weigh_p >= 0: a
  // piece whose sum |w| is formed on the way and added to w_next before sy is needed.
  auto spread = [&](int p, int role, int weigh_p, bool adjoins) {
    int len;
    const double* rec0 = records(p, &len);
    // ---- counting sort of the piece by cell -----------------------------------------------
    double ph[kPer], wpart = 0.0;
#pragma unroll
    for (int u = 0; u < kPer; ++u) ph[u] = tid + u * T < len ? rec0[(size_t)kRec * (tid + u * T)] : 0.0;
    if (kExact && weigh_p >= 0) wpart = weigh_part(weigh_p);
    __syncthreads();  // the staging areas are free
    for (int i = tid; i < n / 2; i += T) cnt[i] = 0;
    __syncthreads();
    uint32_t cr[kPer];  // cell << 16 | rank within the cell
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      if (tid + u * T < len) {
        const int c = (int)(ph[u] * (double)n) & (n - 1);  // (a NaN azimuth stays in bounds)
        const int sh = 16 * (c & 1);
        cr[u] = (uint32_t)c << 16 | ((atomicAdd(&cnt[c >> 1], 1u << sh) >> sh) & 0xffffu);
      }
    }
    __syncthreads();
    {  // exclusive scan of the counters, in place
      const int words = n / 2, per = (words + T - 1) / T;
      const int b = tid * per;
      uint32_t sum = 0;
      for (int i = b; i < min(b + per, words); ++i) sum += (cnt[i] & 0xffffu) + (cnt[i] >> 16);
      uint32_t x = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      if (lane == 31) wtot[warp] = x;
      if (kExact && weigh_p >= 0) warp_sum(wpart);
      __syncthreads();
      uint32_t run = x - sum + __reduce_add_sync(0xffffffffu, lane < warp ? wtot[lane] : 0u);
      for (int i = b; i < min(b + per, words); ++i) {
        const uint32_t v = cnt[i];
        cnt[i] = run | (run + (v & 0xffffu)) << 16;
        run += (v & 0xffffu) + (v >> 16);
      }
    }
    if (kExact && weigh_p >= 0) {
      w_next += piece_sum(weigh_p);
      sy = fixed_scale(adjoins ? w_cur + w_next : w_cur);
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      if (tid + u * T < len) {
        const int c = cr[u] >> 16;
        sorted[((cnt[c >> 1] >> (16 * (c & 1))) & 0xffffu) + (cr[u] & 0xffffu)] = (uint16_t)(tid + u * T);
      }
    }
    __syncthreads();
    // ---- spread: this half warp's share [b0, b1) of the sorted points ------------------------
    // (an empty share stays on one point with no weight; its window never moves)
    constexpr int kOff = W / 2 - 1;
    constexpr double kBias = kExact ? 6755399441055744.0 : 0.0;  // 1.5 2^52
    const int st = 2 * warp + half;
    const int b0 = (int)((int64_t)st * len / (2 * kWarps)), b1 = (int)((int64_t)(st + 1) * len / (2 * kWarps));
    const int last = max(min(b0, len - 1), b1 - 1);
    const int rounds = __reduce_max_sync(0xffffffffu, b1 - b0);
    // sums of this lane's cell in block blk of 16 cells and in the next block: left and right node
    const double2 zero = make_double2(kBias, kBias);
    double2 px = zero, py = zero, qx = zero, qy = zero;
    const double2* rp = reinterpret_cast<const double2*>(rec0 + (size_t)kRec * sorted[min(b0 + slot, last)]);
    double2 r0 = rp[0], r1 = rp[1];
    int blk = 0;
    auto add = [&](int block, double2 vx, double2 vy) {
      const int i = sw((16 * block + slot) & (n - 1));
      double2 v = X[i];
      v.x += vx.x - kBias;
      v.y += vx.y - kBias;
      X[i] = v;
      if (TWO) {
        v = Y[i];
        v.x += vy.x - kBias;
        v.y += vy.y - kBias;
        Y[i] = v;
      }
    };
    for (int base = 0; base < rounds; base += kStagePts / 2) {
      // this lane's point: offset in its cell (exact to the double-double azimuth), weights
      const double u = r0.x * (double)n;
      const int c = (int)u & (n - 1);
      const double s = 2.0 * ((u - (double)c) + r0.y * (double)n) - 1.0;
      double h[4];
      hermite(r1.y, b0 + base + slot < b1 ? r1.x : 0.0, h);
      if (kExact) {
        h[0] *= sx;
        h[1] *= sx;
        h[2] *= sy;
        h[3] *= sy;
      }
      if (base + kStagePts / 2 < rounds) {  // the next round's record
        rp = reinterpret_cast<const double2*>(rec0 + (size_t)kRec * sorted[min(b0 + base + kStagePts / 2 + slot, last)]);
        r0 = rp[0];
        r1 = rp[1];
      }
      __syncwarp();  // the staged points have been taken
      if (TWO) {
        gst[2 * lane] = make_double2(h[0], h[1]);
        gst[2 * lane + 1] = make_double2(h[2], h[3]);
      } else {
        gst[lane] = role ? make_double2(h[2], h[3]) : make_double2(h[0], h[1]);
      }
      cbs[lane] = (int16_t)(c - kOff);
      {
        const double s2 = s * s;
        double* kd = ker + lane * kNuSlots;
#pragma unroll
        for (int i = 0; i < W / 2; ++i) {
          double ev = es.c[i][DEG - 1], od = es.c[i][DEG];
#pragma unroll
          for (int d = DEG - 3; d >= 0; d -= 2) {
            ev = fma(ev, s2, es.c[i][d]);
            od = fma(od, s2, es.c[i][d + 1]);
          }
          kd[(i + lane) & (kNuSlots - 1)] = fma(od, s, ev);
          kd[(W - 1 - i + lane) & (kNuSlots - 1)] = fma(-od, s, ev);
        }
#pragma unroll
        for (int i = W; i < kNuSlots; ++i) kd[(i + lane) & (kNuSlots - 1)] = 0.0;
      }
      __syncwarp();
      const int np = min(kStagePts / 2, rounds - base);
      const int16_t* ch = cbs + 16 * half;
      if (base == 0) blk = ch[0] >> 4;
      // two points at a time, their loads issued before any sum is written back (beyond the last
      // point the staged ones repeat it with no weight)
#pragma unroll 1
      for (int q = 0; q < np; q += 2) {
        double k[2];
        double2 g0[2], g1[2];
        const int cc = *reinterpret_cast<const int*>(ch + q);
        const int cb[2] = {(int)(int16_t)cc, cc >> 16};
#pragma unroll
        for (int v = 0; v < 2; ++v) {
          const int pt = 16 * half + q + v;
          k[v] = ker[pt * kNuSlots + ((slot - cb[v] + q + v) & (kNuSlots - 1))];
          if (TWO) {
            g0[v] = gst[2 * pt];
            g1[v] = gst[2 * pt + 1];
          } else {
            g0[v] = gst[pt];
          }
        }
#pragma unroll
        for (int v = 0; v < 2; ++v) {
          if (cb[v] >> 4 != blk) {  // the window has left block blk
            add(blk, px, py);
            if (cb[v] >> 4 != blk + 1) {
              add(blk + 1, qx, qy);
              qx = qy = zero;
            }
            px = qx;
            py = qy;
            qx = qy = zero;
            blk = cb[v] >> 4;
          }
          if (slot >= (cb[v] & 15)) {
            px.x = fma(k[v], g0[v].x, px.x);
            px.y = fma(k[v], g0[v].y, px.y);
            if (TWO) {
              py.x = fma(k[v], g1[v].x, py.x);
              py.y = fma(k[v], g1[v].y, py.y);
            }
          } else {
            qx.x = fma(k[v], g0[v].x, qx.x);
            qx.y = fma(k[v], g0[v].y, qx.y);
            if (TWO) {
              qy.x = fma(k[v], g1[v].x, qy.x);
              qy.y = fma(k[v], g1[v].y, qy.y);
            }
          }
        }
      }
    }
    __syncthreads();
    // the last two blocks, which other half warps may share
    auto add_shared = [&](double2* d, double2 v) {
      if (v.x != kBias) atomicAdd(&d->x, v.x - kBias);
      if (v.y != kBias) atomicAdd(&d->y, v.y - kBias);
    };
    const int i0 = sw((16 * blk + slot) & (n - 1)), i1 = sw((16 * blk + 16 + slot) & (n - 1));
    add_shared(X + i0, px);
    add_shared(X + i1, qx);
    if (TWO) {
      add_shared(Y + i0, py);
      add_shared(Y + i1, qy);
    }
  };

  // Finishes a node: its sums to a slot, the grid cleared.
  auto emit = [&](double2* z, int64_t slot_out, double scale) {
    __syncthreads();
    fft_node<R1>(z, logn, tws, Nl, kExact ? 1.0 / scale : 1.0 / kRange, a.dinv, a.slots + (size_t)slot_out * 4 * Nl);
    __syncthreads();
    clear(z);
  };

  load_meta();
  load_meta();
  __syncthreads();
  int q = end_of_key(p0);
  if (kExact) {
    w_cur = weigh(p0, q);
    sx = fixed_scale(w_cur);
  }
  for (int p = p0; p < p1;) {
    if (p - p0 + kMeta / 2 >= loaded) {  // (the half that is overwritten lies before p)
      __syncthreads();
      load_meta();
      __syncthreads();
    }
    const int key = key_at(p);
    const bool more = q < p1;
    const int qn = more ? end_of_key(q) : q;
    const int next_key = more ? key_at(q) : 0;
    const bool next_adjoins = more && next_key == key + 1 && next_key % a.nbins != 0;
    // the key after the next: its records into L2 while this one is summed (warp 0)
    if (warp == 0 && qn < p1) {
      int len;
      const double* r = records(qn, &len);
      prefetch_l2(r, sizeof(double) * kRec * (size_t)len, lane, 32);
    }
    if (kExact) {  // sum |w| of the next key: its first piece during this key's first sort
      w_next = more ? weigh(q + 1, qn) : 0.0;
      if (!more) sy = fixed_scale(w_cur);
    }
    // nodes are numbered in key order; runs that share a node keep separate slots (2 per CTA)
    const int64_t right = (int64_t)(p - p0 < loaded ? desc(p).w : a.node_first[key + 1] - 1u) + 2 * (int64_t)blockIdx.x;
#pragma unroll 1
    for (int role = 0; role < 2; ++role) {
      if (!TWO || role == 0)
#pragma unroll 1
        for (int r = p; r < q; ++r) {
          spread(r, role, more && r == p && role == 0 ? q : -1, next_adjoins);
        }
      if (role == 0 || !next_adjoins) emit(TWO && role ? Y : X, right - 1 + role, role ? sy : sx);
    }
    if (TWO && next_adjoins) {
      double2* t = X;
      X = Y;
      Y = t;
    }
    sx = next_adjoins ? sy : fixed_scale(w_next);
    w_cur = w_next;
    p = q;
    q = qn;
  }
}

}  // namespace

// ---- host: kernel polynomials and the deconvolution factors ----------------------------

namespace {

// Window width, polynomial degree and shape parameter of the two accuracy classes.
struct EsShape {
  int W, deg;
  long double beta;
};
EsShape es_shape(int cls, int oversample4) {
  if (cls == kNuMixed) return {12, 11, 2.30L * 12};
  return {16, 15, oversample4 ? 2.70L * 16 : 2.30L * 16};
}

long double es_kernel(const EsShape& e, long double x) {
  const long double z = 2.0L * x / e.W;
  if (!(std::fabs(z) < 1.0L)) return 0.0L;
  return std::exp(e.beta * (std::sqrt(1.0L - z * z) - 1.0L));
}

constexpr long double kPiL = 3.14159265358979323846264338327950288L;

// Chebyshev interpolation of psi(f + W/2 - 1 - i) at deg + 1 nodes in s = 2f - 1, converted to
// monomial coefficients in s: out[i * (deg + 1) + d].
std::vector<double> make_es_poly(const EsShape& e) {
  const int np = e.deg + 1;
  std::vector<double> out((size_t)e.W * np);
  for (int i = 0; i < e.W; ++i) {
    std::vector<long double> y(np), a(np), c(np, 0.0L);
    for (int j = 0; j < np; ++j)
      y[j] = es_kernel(e, (std::cos(kPiL * (j + 0.5L) / np) + 1.0L) / 2.0L + e.W / 2 - 1 - i);
    for (int k = 0; k < np; ++k) {
      long double acc = 0.0L;
      for (int j = 0; j < np; ++j) acc += y[j] * std::cos(kPiL * k * (j + 0.5L) / np);
      a[k] = acc * (k == 0 ? 1.0L : 2.0L) / np;
    }
    // sum_k a_k T_k(s) in monomials: T_(k+1) = 2 s T_k - T_(k-1)
    std::vector<long double> tkm(np, 0.0L), tk(np, 0.0L), tkp(np, 0.0L);
    tkm[0] = 1.0L;  // T_0
    tk[1] = 1.0L;   // T_1
    for (int d = 0; d < np; ++d) c[d] = a[0] * tkm[d] + a[1] * tk[d];
    for (int k = 1; k + 1 < np; ++k) {
      for (int d = 0; d < np; ++d) tkp[d] = (d > 0 ? 2.0L * tk[d - 1] : 0.0L) - tkm[d];
      for (int d = 0; d < np; ++d) c[d] += a[k + 1] * tkp[d];
      tkm.swap(tk);
      tk.swap(tkp);
    }
    for (int d = 0; d < np; ++d) out[(size_t)i * np + d] = (double)c[d];
  }
  return out;
}

template <int W, int DEG>
EsPoly<W, DEG> half_poly(const EsShape& e, double scale) {
  const std::vector<double> c = make_es_poly(e);
  EsPoly<W, DEG> P;
  for (int i = 0; i < W / 2; ++i)
    for (int d = 0; d <= DEG; ++d) P.c[i][d] = scale * c[(size_t)i * (DEG + 1) + d];
  return P;
}

// Gauss-Legendre nodes and weights on [-1, 1] (Newton iteration on P_q from the
// Chebyshev-like initial guesses).
struct GaussLegendre {
  std::vector<long double> x, w;
  explicit GaussLegendre(int q) : x(q, 0.0L), w(q, 0.0L) {
    for (int i = 0; i < (q + 1) / 2; ++i) {
      long double z = std::cos(kPiL * (i + 0.75L) / (q + 0.5L)), dp = 0.0L;
      for (int it = 0; it < 100; ++it) {
        long double p0 = 1.0L, p1 = z;
        for (int k = 2; k <= q; ++k) {
          const long double p2 = ((2.0L * k - 1.0L) * z * p1 - (k - 1.0L) * p0) / k;
          p0 = p1;
          p1 = p2;
        }
        if (q == 1) p0 = 1.0L;
        dp = q * (z * p1 - p0) / (z * z - 1.0L);
        const long double dz = p1 / dp;
        z -= dz;
        if (std::fabs(dz) < 1e-19L) break;
      }
      x[i] = -z;
      x[q - 1 - i] = z;
      w[i] = w[q - 1 - i] = 2.0L / ((1.0L - z * z) * dp * dp);
    }
  }
};

int ceil_log2(int v) {
  int lg = 0;
  while ((1 << lg) < v) ++lg;
  return lg;
}

}  // namespace

// log2 of the grid cells: oversampling 2 of the 2 Nl frequencies -Nl < m < Nl, 4 for the FP64 class
// up to Nl = 256 (the grids are small there, and the direct sums it replaces are accurate to 2-6e-15);
// at least 128 cells.
int nufft_logn(int Nl, int cls) {
  const int lg = ceil_log2(Nl) + (cls == kNuFp64 && Nl <= 256 ? 3 : 2);
  return lg < 7 ? 7 : lg;
}

// 1 / Psi(m), m < Nl, and the twiddles e^{2 pi i i / n} of the FFT passes, for a plan.
void nufft_host_tables(int Nl, int cls, std::vector<double>& dinv, std::vector<double>& tw) {
  const int logn = nufft_logn(Nl, cls), n = 1 << logn;
  const EsShape e = es_shape(cls, cls == kNuFp64 && Nl <= 256);
  static const GaussLegendre nodes(120);  // the same for every plan (200 of 600 us at Nl = 1024)
  const std::vector<long double>&gx = nodes.x, &gw = nodes.w;
  // the integrand is even: 60 nodes; cos(m theta) by repeated rotation (error m ulps of long double)
  std::vector<long double> sum(Nl, 0.0L);
  for (size_t i = gx.size() / 2; i < gx.size(); ++i) {
    const long double wt = 2.0L * gw[i] * es_kernel(e, gx[i] * (e.W / 2.0L));
    const long double th = kPiL * e.W * gx[i] / n, ct = std::cos(th), st = std::sin(th);
    long double c = wt, s = 0.0L;
    for (int m = 0; m < Nl; ++m) {
      sum[m] += c;
      const long double cn = c * ct - s * st;
      s = s * ct + c * st;
      c = cn;
    }
  }
  dinv.assign(Nl, 0.0);
  for (int m = 0; m < Nl; ++m) dinv[m] = (double)(1.0L / (sum[m] * (e.W / 2.0L)));
  const int nt = tw_count(logn);
  tw.assign(2 * (size_t)nt, 0.0);
  for (int i = 0; i < nt; ++i) {
    tw[2 * i] = (double)std::cos(2.0L * kPiL * i / n);
    tw[2 * i + 1] = (double)std::sin(2.0L * kPiL * i / n);
  }
}

namespace {

// 512 threads and one CTA per SM from 4096 cells (two grids: 150 KB), else 256 and two.
int nufft_threads(int logn) { return logn >= 12 ? 512 : 256; }

template <int W, int DEG, int T, bool TWO, int R1>
int nufft_launch(const Workspace& ws, const NuArgs& a, const EsPoly<W, DEG>& es, cudaStream_t s) {
  auto kern = nufft_nodes_kernel<W, DEG, T, TWO, R1>;
  const int bytes = NuLayout<T, TWO>(a.logn).bytes(a.logn);
  const cudaError_t e = allow_shared(kern);
  if (e != cudaSuccess) return set_cuda_error(e, "nufft attributes", __FILE__, __LINE__);
  kern<<<(unsigned)ws.nu_grid, T, bytes, s>>>(a, es);
  count_launches(1);
  return DSHT_OK;
}

template <int W, int DEG>
int nufft_go(const Workspace& ws, const NuArgs& a, const EsPoly<W, DEG>& es, cudaStream_t s) {
  if (a.logn == 13) return nufft_launch<W, DEG, 512, false, 16>(ws, a, es, s);
  if (a.logn == 12) return nufft_launch<W, DEG, 512, true, 8>(ws, a, es, s);
  switch (first_radix(a.logn)) {
    case 2: return nufft_launch<W, DEG, 256, true, 4>(ws, a, es, s);
    case 3: return nufft_launch<W, DEG, 256, true, 8>(ws, a, es, s);
    default: return nufft_launch<W, DEG, 256, true, 16>(ws, a, es, s);
  }
}

}  // namespace

// Runs (CTAs) of a launch and the cost of a piece in points (its share of the sorts and FFTs) for
// the balance: measured 2.0e4 clocks of an SM per node and 11 per point at n = 4096.
int nufft_grid(int Nl, int cls) {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return nufft_threads(nufft_logn(Nl, cls)) == 512 ? sms : 2 * sms;
}
int nufft_piece(int Nl, int cls) { return nu_piece(nufft_threads(nufft_logn(Nl, cls))); }
int nufft_piece_cost(int Nl, int cls) { return (1 << nufft_logn(Nl, cls)) / 2; }

int launch_bin_sums_nufft(const Geometry& g, const Workspace& ws, const NufftTables& t, cudaStream_t s) {
  if (!t.dinv || nufft_logn(g.Nl, t.cls) > 13)
    return set_error(DSHT_ERR_INVALID, "NUFFT bin sums support Nl <= 2048 (Nl=%d)", g.Nl);
  NuArgs a{};
  a.Nl = g.Nl;
  a.logn = nufft_logn(g.Nl, t.cls);
  a.nbins = g.nbins;
  a.pay = ws.pay;
  a.piece_start = ws.piece_start;
  a.piece_len = ws.piece_len;
  a.piece_key = ws.piece_key;
  a.cta_first = ws.cta_first;
  a.node_first = ws.node_first;
  a.dinv = t.dinv;
  a.tw = reinterpret_cast<const double2*>(t.tw);
  a.slots = ws.partial;
  a.wsum = t.cls == kNuMixed ? ws.wsum : nullptr;
  if (t.cls == kNuMixed) {
    static const EsPoly<12, 11> P = half_poly<12, 11>(es_shape(kNuMixed, 0), 1.0);
    return nufft_go(ws, a, P, s);
  }
  static const EsPoly<16, 15> P2 = half_poly<16, 15>(es_shape(kNuFp64, 0), kRange);
  static const EsPoly<16, 15> P4 = half_poly<16, 15>(es_shape(kNuFp64, 1), kRange);
  return nufft_go(ws, a, g.Nl <= 256 ? P4 : P2, s);
}

}  // namespace dsht

extern "C" int dsht_test_nufft_tables(int Nl, int* logn, double* poly, double* dinv) {
  if (Nl < 1 || Nl > 2048 || !logn || !poly || !dinv)
    return dsht::set_error(DSHT_ERR_INVALID, "invalid arguments");
  *logn = dsht::nufft_logn(Nl, dsht::kNuMixed);
  const std::vector<double> P = dsht::make_es_poly(dsht::es_shape(dsht::kNuMixed, 0));
  std::copy(P.begin(), P.end(), poly);
  std::vector<double> dv, tw;
  dsht::nufft_host_tables(Nl, dsht::kNuMixed, dv, tw);
  for (int m = 0; m < Nl; ++m) dinv[m] = dv[m];
  return DSHT_OK;
}
