// FP64 contraction of the Ylm table with the folded node sums (the FP64 and
// DSHT_PREC_MIXED_F64_TABLES levels): FP64 matrix instructions fed by TMA.
//
//   alm[lm] = sum_j Y[lm,j] A[m,j] + dY[lm,j] B[m,j]            (sht/sht.py:266-279)
//
// for the equatorial and the rotated polar halves, A and B by the parity q of l - m.  Only the
// Y table is read: the rows of dY/dx follow from the two neighbour rows of Y,
//   (1 - x^2) dY[l] = (l+1) a_l Y[l-1] - l a_(l+1) Y[l+1],  a_l = sqrt((l^2 - m^2)/(4 l^2 - 1))
// (sht/legendre_py.py:115-116 with x Y[l] = a_(l+1) Y[l+1] + a_l Y[l-1]), so with B' = B/(1 - x^2)
//   alm[l] = Y[l] . A_q + (l+1) a_l Y[l-1] . B'_q - l a_(l+1) Y[l+1] . B'_q:
// row l is multiplied with the four columns A of its own parity and the four columns B' of the
// other one, and the latter products go to rows l - 1 and l + 1.  (The last row, l = Nl - 1, has
// no upper neighbour in the table; there x Y[l] . B'_q is formed instead.)  That is 8 bytes of
// table and 8 FMA per (l, m, node) where the two tables take 16 bytes and 8 FMA: at Nl = 1024,
// Nx = 2048 8.6 GB, 1.33 ms at the measured copy bandwidth, beside 0.47 ms of FP64 products.
// The products are m8n8k4 matrix instructions (63 FMA per clock and SM measured, DFMA 61): they
// take 8 x 4 and 4 x 8 operands for 256 FMA, while vector FMAs would pass every fold value
// through the shared-memory pipe once per warp and row pair and be bound by that pipe.
//
// Persistent CTAs claim work items (m, 128 consecutive rows l) from a global counter, in order: the
// largest columns first, so that the last items are small, and neighbour CTAs share a column's
// fold in L2 (a fixed assignment gave some CTAs full and others partial blocks: 248 instead of
// 220 us at Nl = 500, Nx = 1000).  Warp 0 (one thread) claims and issues, for
// every stage of 32 nodes that has points, the table boxes (16 nodes x 8 to 128 rows, one for each
// binary digit of the rows that the column has left, 128-byte swizzle) and one bulk copy per map of
// the fold.  (With boxes of 64 and 8 rows only, up to 16 issues a stage: 222 instead of 216 us at
// Nl = 500, 1412 instead of 1382 at Nl = 1024, Nx = 2048.)
// Warps 1-8 consume: parity (w & 1), two row tiles of eight rows of that parity each, so every
// fold fragment feeds two products.  The fold comes in fragment order (fold.cu): lane 4 n + k
// reads its column n and its two nodes as one 16-byte word.  Up to four maps share a pass: three
// take as long in the products as the table read, a fourth amortises what is not overlapped.
//
// Products for neighbour rows go through shared memory.  Across items (the last of 128 rows and
// the first of the next) both contributions are added with atomics onto zeros (the fold
// kernel clears those rows); 0 + a + b does not depend on the order.
//
// What bounds it: at Nl = 1024, Nx = 2048 the table (1364 us, 6.30 TB/s of the 6.45 measured); at
// smaller Nl what an item costs beyond its bytes (208 us at Nl = 500, Nx = 1000, where the bytes
// take 155; 64-row items: 318).  So the consumers take m and the row group from the claim instead of
// searching again, and form the square roots of an item before its first stage, while that is
// loading (216 and 1382 us with both after the last).  Finishing an item inside the next one's stage
// loop costs more in that loop than it hides (217, 1400); twice the accumulators change nothing.
#include <cudaTypedefs.h>

#include <algorithm>

#include "dsht_internal.cuh"
#include "tc_ptx.cuh"

namespace dsht {
namespace {

constexpr int kRows = kContractRows;      // rows per work item
constexpr int kStageNodes = 32;
constexpr int kConsumers = 8;             // warps 1..8
constexpr int kThreads = 32 * (1 + kConsumers);
constexpr int kItemRing = 16;  // claimed items in flight: the producer leads by at most kStages + 2
constexpr int kTab = kRows * kStageNodes * (int)sizeof(double);  // two halves of [128 rows][16 nodes]
constexpr int kFoldStage = kStageNodes * 16 * (int)sizeof(double);  // one map: 4 groups x 2 parities x 512 B

__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          tc::smem_addr(dst)),
      "l"(src), "r"(bytes), "r"(tc::smem_addr(bar))
      : "memory");
}

// 2D tiled TMA load of a table box (x = node, y = table row).
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* tm, int x, int y, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], "
      "[%4];" ::"r"(tc::smem_addr(dst)),
      "l"(reinterpret_cast<uint64_t>(tm)), "r"(x), "r"(y), "r"(tc::smem_addr(bar))
      : "memory");
}

// c += a b, m8n8k4 in FP64: lane 4 i + k holds a[i][k] and b[k][i], and c[i][2k], c[i][2k + 1].
__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

// Work items in m order: group g < ceil((Nl - m) / kRows) of column m.
__device__ __forceinline__ void item_of(int64_t item, int Nl, int* m_out, int* g_out) {
  // cumulative groups before m: G(m) = sum_{m' < m} ceil((Nl - m') / kRows); binary search.
  int lo = 0, hi = Nl;  // find largest m with G(m) <= item
  auto G = [&](int m) -> int64_t {
    // sum_{n = Nl-m+1}^{Nl} ceil(n / R) with n = Nl - m'
    auto S = [](int64_t n) -> int64_t {  // sum_{k=1}^{n} ceil(k / R)
      const int64_t q = n / kRows, r = n % kRows;
      return kRows * q * (q + 1) / 2 + r * (q + 1);
    };
    return S(Nl) - S(Nl - m);
  };
  while (hi - lo > 1) {
    const int mid = (lo + hi) / 2;
    if (G(mid) <= item) lo = mid;
    else hi = mid;
  }
  *m_out = lo;
  *g_out = (int)(item - G(lo));
}

template <int G>
struct StreamLayout {
  static constexpr int kStage = kTab + G * kFoldStage;
  static constexpr int kStages = G <= 2 ? 5 : 4;
  static constexpr int kExch = 2 * kRows * 2 * G * 2 * (int)sizeof(double);  // double-buffered B' products
  static constexpr int kBarOff = kStages * kStage + kExch;
  // barriers, abort flag and item ring, then one byte per stage of nodes, and the alignment slack
  static constexpr int kLiveOff = kBarOff + 384;
  static constexpr int bytes(int nstage) { return kLiveOff + (nstage + 15) / 16 * 16 + 1024; }
};

template <int G>
__global__ void __launch_bounds__(kThreads, 1)
contract_fp64_kernel(int Nl, int Nx, double dx, int64_t nitems, const __grid_constant__ TableMaps tm,
                     const FoldIn in, int nstage, unsigned* __restrict__ next_item, int stall) {
  using L = StreamLayout<G>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  constexpr int kStages = L::kStages;
  double2* exch = reinterpret_cast<double2*>(smem + kStages * L::kStage);  // [2][kRows][G][2]
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + L::kBarOff);
  uint64_t* empty = full + kStages;
  uint64_t* item_full = empty + kStages;  // [kItemRing] producer -> consumers
  uint64_t* ex_full = item_full + kItemRing;  // the consumers' exchange of B' products
  volatile int* abort_flag = reinterpret_cast<volatile int*>(ex_full + 1);
  int* item_ring = const_cast<int*>(abort_flag) + 1;  // [kItemRing] claimed item, -1 = none left
  uint8_t* live = smem + L::kLiveOff;  // [nstage] any point feeds a node of the stage
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) {
      tc::mbar_init(&full[s], 1);
      tc::mbar_init(&empty[s], kConsumers);
    }
    for (int r = 0; r < kItemRing; ++r) tc::mbar_init(&item_full[r], 1);
    tc::mbar_init(ex_full, kConsumers);
    *abort_flag = 0;
    tc::mbar_fence_init();
  }
  auto timed_out = [&]() {  // the alm of every map of the pass are invalid
    for (int k = 0; k < G; ++k) atomicOr(in.map[k].flags, kFlagTimeout);
  };
  auto fail = [&]() {
    *abort_flag = 1;
    timed_out();
  };
  bool some = false;
  for (int t = tid; t < nstage; t += blockDim.x) {
    uint8_t any = 0;
    for (int k = 0; k < G; ++k) {
      any |= in.map[k].live[2 * t];
      if (2 * t + 1 < (Nx + 15) / 16) any |= in.map[k].live[2 * t + 1];
    }
    live[t] = any;
    some |= any != 0;
  }
  // an item always has a stage (the ring bounds the producer's lead by its stages)
  if (!__syncthreads_or(some) && tid == 0) live[0] = 1;
  __syncthreads();

  if (warp == 0) {
    // ---- producer (one thread) --------------------------------------------------------
    if (lane == 0) {
      uint32_t n = 0;  // stages issued
      for (uint32_t j = 0; !*abort_flag; ++j) {
        int item = (int)atomicAdd(next_item, 1u);
        int m = 0, g = 0;
        if (item < nitems) item_of(item, Nl, &m, &g);
        else item = -1;
        item_ring[j % kItemRing] = item < 0 ? -1 : m << 8 | g;  // g < 16384 / kRows
        // releases the ring entry (stall, a test hook: block 0 never releases its first one, so the
        // consumers' bounded wait runs out)
        if (!(stall && blockIdx.x == 0 && j == 0)) tc::mbar_arrive(&item_full[j % kItemRing]);
        if (item < 0) break;
        const int l0 = m + g * kRows;
        const int row0 = (int)hp_index(l0, m, Nl);
        const int nrows = min(kRows, Nl - l0);
        const int nr8 = (nrows + 7) / 8 * 8;  // the column's rows left, one box per set bit
        for (int t = 0; t < nstage; ++t) {
          if (!live[t]) continue;
          const int s = n % kStages;
          const uint32_t use = n / kStages;
          if (use > 0 && !tc::mbar_wait(&empty[s], (use - 1) & 1, abort_flag)) {
            fail();
            break;
          }
          const int j0 = t * kStageNodes;
          uint8_t* st = smem + s * L::kStage;
          const uint32_t fold_bytes = (uint32_t)min(kFoldStage, (Nx - j0 + 7) / 8 * 1024);
          // boxes always transfer all their elements (zero fill out of range)
          tc::mbar_arrive_expect_tx(&full[s], (uint32_t)nr8 * 256u + (uint32_t)G * fold_bytes);
          for (int h = 0; h < 2; ++h) {
            uint8_t* dst = st + h * (kTab / 2);
            int r = 0;
#pragma unroll
            for (int b = kTableMaps - 1; b >= 0; --b)
              if (nr8 & (8 << b)) {
                tma_load_2d(dst + r * 128, &tm.box[b], j0 + 16 * h, row0 + r, &full[s]);
                r += 8 << b;
              }
          }
#pragma unroll
          for (int k = 0; k < G; ++k)
            bulk_g2s(st + kTab + k * kFoldStage, in.map[k].fold + (size_t)m * fold_stride(Nx) + (size_t)j0 * 16,
                     fold_bytes, &full[s]);
          ++n;
        }
      }
      // no copy may still be writing shared memory when the block leaves
      const uint32_t last = n < (uint32_t)kStages ? n : (uint32_t)kStages;
      for (uint32_t k = 0; k < last; ++k) {
        const uint32_t i = n - 1 - k;
        const long long t0 = clock64();
        while (!tc::mbar_try_wait_for(&full[i % kStages], (i / kStages) & 1, 10000u))
          if (clock64() - t0 > (1ll << 31)) {
            timed_out();
            break;
          }
      }
    }
    __syncwarp();
  } else {
    // ---- consumers: parity p, row tiles t = tq and tq + 4 (rows p + 16 t + 2 rho(i)) --------
    const int cw = warp - 1;
    const int p = cw & 1, tq = cw >> 1;
    const int i = lane >> 2, q = lane & 3;
    // the table rows of a quarter warp's two MMA rows differ in bit 2, so their swizzled 16-byte chunks
    // cover a whole 128-byte line
    const int rho = (i & 4) | ((i & 1) << 1) | ((i >> 1) & 1);
    int row[2];
    row[0] = p + 16 * tq + 2 * rho;
    row[1] = row[0] + 64;
    uint32_t n = 0, iter = 0;
    for (;; ++iter) {
      if (!tc::warp_wait(&item_full[iter % kItemRing], (iter / kItemRing) & 1, abort_flag)) {
        if (lane == 0) fail();
        break;
      }
      const int item = item_ring[iter % kItemRing];
      if (item < 0) break;
      const int m = item >> 8, l0 = m + (item & 255) * kRows;
      const int nrows = min(kRows, Nl - l0);
      const bool on0 = p + 16 * tq < nrows, on1 = p + 16 * tq + 64 < nrows;
      // the tile (0 or 1) that holds the column's last row, if this warp does: it also forms x B'
      const int rl = Nl - 1 - l0 - p;  // offset of row Nl - 1 from the warp's first row of parity
      const int lt = (l0 + nrows == Nl && (rl & 1) == 0 && ((rl >> 4) & 3) == tq) ? rl >> 6 : -1;
      // factors of the neighbour rows' products, while the item's first stages are on their way
      auto a_l = [&](int l) {  // a_l of this column
        return sqrt((double)(l - m) * (double)(l + m) / ((2.0 * l - 1.0) * (2.0 * l + 1.0)));
      };
      auto from_below = [&](int l) {  // factor of Y[l - 1] . B'
        return (l + 1 < Nl ? (double)(l + 1) : (double)(2 * l + 1)) * a_l(l);
      };
      double f1[2], f2[2];
#pragma unroll
      for (int a = 0; a < 2; ++a) {
        const int r = row[a], l = l0 + r;
        f1[a] = f2[a] = 0.0;
        if (r >= nrows) continue;
        if (q < 2) {  // of rows l - 1 and l + 1, added to row l
          if (l > m) f1[a] = from_below(l);
          if (l + 1 < Nl) f2[a] = -(double)l * a_l(l + 1);
        } else {  // of row l, added to a row of the item before or of the next
          if (r == 0 && l > m) f1[a] = -(double)(l - 1) * a_l(l);
          if (r == kRows - 1 && l + 1 < Nl) f2[a] = from_below(l + 1);
        }
      }
      double acc[2][G][2], accx[G][2];
#pragma unroll
      for (int k = 0; k < G; ++k) {
        acc[0][k][0] = acc[0][k][1] = acc[1][k][0] = acc[1][k][1] = 0.0;
        accx[k][0] = accx[k][1] = 0.0;
      }
      for (int t = 0; t < nstage; ++t) {
        if (!live[t]) continue;
        const int s = n % kStages;
        const uint32_t use = n / kStages;
        const bool ok = tc::warp_wait(&full[s], use & 1, abort_flag);
        if (!ok && lane == 0) fail();
        if (ok && on0) {
          const uint8_t* st = smem + s * L::kStage;
          const int ng = min(kStageNodes / 8, (Nx - t * kStageNodes + 7) / 8);
          auto group = [&](int g8) {
            // lanes n < 4: A of this parity, n >= 4: B' of the other
            const uint8_t* fg = st + kTab + g8 * 1024;
            double2 b[G];
#pragma unroll
            for (int k = 0; k < G; ++k)
              b[k] = *reinterpret_cast<const double2*>(fg + k * kFoldStage + (i < 4 ? p : p ^ 1) * 512 + lane * 16);
            const uint8_t* th = st + (g8 >> 1) * (kTab / 2);
            const int chunk = 4 * (g8 & 1) + q;
            const double2 y0 = *reinterpret_cast<const double2*>(th + row[0] * 128 + ((chunk ^ (row[0] & 7)) << 4));
            const double2 y1 = *reinterpret_cast<const double2*>(th + row[1] * 128 + ((chunk ^ (row[1] & 7)) << 4));
#pragma unroll
            for (int k = 0; k < G; ++k) dmma(acc[0][k], y0.x, b[k].x);
            if (on1) {
#pragma unroll
              for (int k = 0; k < G; ++k) dmma(acc[1][k], y1.x, b[k].x);
            }
#pragma unroll
            for (int k = 0; k < G; ++k) dmma(acc[0][k], y0.y, b[k].y);
            if (on1) {
#pragma unroll
              for (int k = 0; k < G; ++k) dmma(acc[1][k], y1.y, b[k].y);
            }
            if (lt >= 0) {  // columns n < 4: x B' of this parity
              const double jd = (double)(t * kStageNodes + 8 * g8 + 2 * q);  // this lane's first node
              const double2 y = lt ? y1 : y0;
#pragma unroll
              for (int k = 0; k < G; ++k) {
                const double2 c =
                    *reinterpret_cast<const double2*>(fg + k * kFoldStage + p * 512 + 256 + (lane & 15) * 16);
                dmma(accx[k], y.x, i < 4 ? jd * dx * c.x : 0.0);
                dmma(accx[k], y.y, i < 4 ? (jd + 1.0) * dx * c.y : 0.0);
              }
            }
          };
          if (ng == kStageNodes / 8) {
#pragma unroll
            for (int g8 = 0; g8 < kStageNodes / 8; ++g8) group(g8);
          } else {
            for (int g8 = 0; g8 < ng; ++g8) group(g8);
          }
        }
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&empty[s]);
        ++n;
      }
      // Results: lane (i, q) holds columns 2q, 2q + 1 of its row: q = 0, 1: A of the equatorial,
      // polar half, q = 2, 3: B' of them (for the neighbour rows); accx: x B' (q = 0, 1).
      double2* ex = exch + (iter & 1) * kRows * G * 2;
      if (q >= 2) {
#pragma unroll
        for (int a = 0; a < 2; ++a) {
          const int r = row[a], l = l0 + r;
          if (r >= nrows) continue;
#pragma unroll
          for (int k = 0; k < G; ++k) {
            const double2 v = make_double2(acc[a][k][0], acc[a][k][1]);
            ex[(r * G + k) * 2 + (q & 1)] = v;
            double* alm = (q & 1) ? in.map[k].pol : in.map[k].equ;
            if (r == 0 && l > m) {  // to the last row of the item before
              double* o = alm + 2 * hp_index(l - 1, m, Nl);
              atomicAdd(o, f1[a] * v.x);
              atomicAdd(o + 1, f1[a] * v.y);
            }
            if (r == kRows - 1 && l + 1 < Nl) {  // to the first row of the next item
              double* o = alm + 2 * hp_index(l + 1, m, Nl);
              atomicAdd(o, f2[a] * v.x);
              atomicAdd(o + 1, f2[a] * v.y);
            }
          }
        }
      }
      // every consumer warp has written (a bounded wait: a warp that gave up never arrives)
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(ex_full);
      if (!tc::warp_wait(ex_full, iter & 1, abort_flag)) {
        if (lane == 0) fail();
        break;
      }
      if (q < 2) {
#pragma unroll
        for (int a = 0; a < 2; ++a) {
          const int r = row[a], l = l0 + r;
          if (r >= nrows) continue;
          const bool shared = (r == 0 && l > m) || (r == kRows - 1 && l + 1 < Nl);  // two items add to the row
#pragma unroll
          for (int k = 0; k < G; ++k) {
            double vr = acc[a][k][0], vi = acc[a][k][1];
            if (r > 0) {
              const double2 e = ex[((r - 1) * G + k) * 2 + q];
              vr = fma(f1[a], e.x, vr);
              vi = fma(f1[a], e.y, vi);
            }
            if (r + 1 < nrows) {
              const double2 e = ex[((r + 1) * G + k) * 2 + q];
              vr = fma(f2[a], e.x, vr);
              vi = fma(f2[a], e.y, vi);
            }
            if (l + 1 == Nl) {
              vr = fma(-(double)l, accx[k][0], vr);
              vi = fma(-(double)l, accx[k][1], vi);
            }
            double* o = (q ? in.map[k].pol : in.map[k].equ) + 2 * hp_index(l, m, Nl);
            if (shared) {
              atomicAdd(o, vr);
              atomicAdd(o + 1, vi);
            } else {
              o[0] = vr;
              o[1] = vi;
            }
          }
        }
      }
    }
  }
  __syncthreads();
}

// 2D tensor map of an FP64 table (node x row), boxes of 16 nodes x box_rows, 128-byte swizzle.
int encode_table(CUtensorMap* tm, const void* base, const Geometry& g, int box_rows) {
  static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
  if (!encode) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess || !fn)
      return set_error(DSHT_ERR_CUDA, "cuTensorMapEncodeTiled is not available");
    encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
  }
  const cuuint64_t dims[2] = {(cuuint64_t)g.Nx, (cuuint64_t)g.Nlm};
  const cuuint64_t strides[1] = {(cuuint64_t)g.pitch * sizeof(double)};
  const cuuint32_t box[2] = {16u, (cuuint32_t)box_rows};
  const cuuint32_t estr[2] = {1, 1};
  CUresult r = encode(tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 2, const_cast<void*>(base), dims, strides, box, estr,
                      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return set_error(DSHT_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
  return DSHT_OK;
}

template <int G>
void launch_g(const Geometry& g, const TableMaps& tm, const FoldIn& in, unsigned* next_item, cudaStream_t s) {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int nstage = (g.Nx + kStageNodes - 1) / kStageNodes;
  int64_t nitems = 0;
  for (int m = 0; m < g.Nl; ++m) nitems += (g.Nl - m + kRows - 1) / kRows;
  const int64_t grid = nitems < sms ? nitems : sms;
  const int bytes = StreamLayout<G>::bytes(nstage);
  allow_shared(contract_fp64_kernel<G>);
  contract_fp64_kernel<G><<<(unsigned)grid, kThreads, bytes, s>>>(g.Nl, g.Nx, g.dx, nitems, tm, in, nstage,
                                                                  next_item, take_stall());
  count_launches(1);
}

}  // namespace

int make_table_tmaps(TableMaps* tm, const void* base, const Geometry& g) {
  for (int b = 0; b < kTableMaps; ++b)
    if (int rc = encode_table(&tm->box[b], base, g, 8 << b)) return rc;
  return DSHT_OK;
}

void launch_contract_fp64(const Geometry& g, const TableMaps& tm, const FoldIn& in, int nmaps, unsigned* next_item,
                          cudaStream_t s) {
  switch (nmaps) {
    case 1: launch_g<1>(g, tm, in, next_item, s); break;
    case 2: launch_g<2>(g, tm, in, next_item, s); break;
    case 3: launch_g<3>(g, tm, in, next_item, s); break;
    default: launch_g<4>(g, tm, in, next_item, s); break;
  }
}

}  // namespace dsht
