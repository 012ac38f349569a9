// Internal declarations shared by the DirectSHT B200 kernels.
//
// Data layout in HBM (Nlm = Nl(Nl+1)/2, rows in Healpy order m(2Nl-1-m)/2 + l):
//   tables   Yv, Yd      double [Nlm][pitch]       (sht/sht.py:50-56 layout, numpy path; Nx even up)
//   points   key         uint32 [N]                set*(Nx-1) + bin, or DSHT_KEY_DROP
//            sorted      double [N][4]             (cos phi, sin phi, w, t) by key; for the NUFFT sums
//                                                  (turns hi, lo, w, t)
//   pieces   <= 1 bin each, <= piece_max points    (key, start, len)
//   partial  double [piece][8][Nl]                 (k, re/im) bin sums for every m
//   fold     double [Nl][Nx/8][2 parity][8][8]     columns A, B' of eight nodes (fold.cu)
//   alm      double2 [Nlm]                         complex128, Healpy order
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stddef.h>

#include <vector>

#include "../../include/dsht.h"

#define DSHT_KEY_DROP 0xffffffffu

namespace dsht {

// Number of point sets: {equatorial, rotated polar} x {cos >= 0, cos < 0}.
constexpr int kSets = 4;
// Error-flag bits written by the point kernel.
constexpr unsigned kFlagThetaRange = 1u;   // basic_sht assertion (sht/sht.py:171-172)
constexpr unsigned kFlagPolarRange = 2u;   // rotated polar point still outside (-xmax, xmax)
constexpr unsigned kFlagHasPolar = 4u;     // at least one point went through the rotation
constexpr unsigned kFlagTimeout = 8u;      // a bounded wait in a tensor-core kernel gave up

struct Geometry {
  int Nl, Nx;
  int pitch;          // doubles from one FP64 table row to the next: Nx rounded up to even (TMA rows
                      // start on 16 bytes)
  double xmax;
  double dx;          // xmax / (Nx-1), the numpy grid step  (sht/sht.py:48)
  double acos_xmax;   // numpy arccos(xmax), arccos(-xmax) (sht/sht.py:171)
  double acos_mxmax;
  int64_t Nlm;
  int nbins;          // Nx - 1 right-open bins
  int nkeys;          // kSets * nbins
};

// Output pointers of one tensor-core contraction pass (contract_tc.cu): map k's equatorial
// alm to equ[k], its rotated-polar alm to pol[k] (2 Nlm doubles each); a wait that runs out is
// recorded in every map's flags[k].
constexpr int kTcMaxMaps = 8;
struct TcOut {
  double* equ[kTcMaxMaps];
  double* pol[kTcMaxMaps];
  unsigned* flags[kTcMaxMaps];
};

// One pass of the FP64 contraction: each map's fold, its equatorial and rotated polar alm.
constexpr int kFp64Maps = 4;
constexpr int kContractRows = 128;  // rows of one work item
// Tensor maps of the FP64 table Yv with boxes of 8, 16, 32, 64 and 128 rows.
constexpr int kTableMaps = 5;
struct alignas(64) TableMaps {
  CUtensorMap box[kTableMaps];
};
struct FoldOut {
  double* fold;   // fold.cu's layout
  uint8_t* live;  // [ceil(Nx/16)] any point feeds a node of the block of 16
  double* equ;    // equatorial alm, rotated polar alm
  double* pol;
  unsigned* flags;      // the map's flag word: a wait of the contraction that runs out is recorded there
  unsigned* next_item;  // the contraction's work counter (cleared by the fold)
};
struct FoldIn {
  FoldOut map[kFp64Maps];
};
// Doubles of one m of an FP64 fold: 16 per node, nodes in groups of eight.
__host__ __device__ inline size_t fold_stride(int Nx) { return (size_t)((Nx + 7) / 8) * 128; }

// Maps of one batched rotation: out[k] += R(rot[k]) when *flags[k] has polar points; or (sum) of a lone
// one: out[0] = add + R(rot[0]), add null for zeros, out[0] any of the others.
constexpr int kMaxRot = 8;
struct RotMaps {
  const double* rot[kMaxRot];
  double* out[kMaxRot];
  const unsigned* flags[kMaxRot];
  const double* add;
  bool sum;
};

// Flag words of finished transforms: *all |= *slot[k]; status[k] (if set) = *slot[k].
struct StatusOut {
  const unsigned* slot[kMaxRot];
  unsigned* status[kMaxRot];
};

// Workspace carve-up for one execute call.
struct Workspace {
  uint32_t* key;        // [N]
  double* pay;          // [N][4] sorted records (cos phi, sin phi, w, t)
  uint32_t* sidx;       // [N] input index of each sorted slot (multi-map transforms)
  uint32_t* piecemax;   // [pmax] largest |w h_k| of the piece's points (float bits; tensor-core sums)
  double* wsum;         // [pmax] sum of |w| of the piece's points (fold digit scales), or null
  uint32_t* count;      // [nkeys + 1]
  uint32_t* offset;     // [nkeys + 1]
  uint32_t* cursor;     // [nkeys] (of a single transform in the place of its fold, which is written later)
  int* piece_first;     // [nkeys + 1]  first piece of each key (exclusive scan)
  int* piece_key;       // [pmax]
  int64_t* piece_start; // [pmax]
  int* piece_len;       // [pmax]
  int* npieces;         // [1]
  int* piece_cta;       // [pmax] NUFFT sums: the CTA that takes each piece (the place of piecemax)
  int* cta_first;       // [nu_grid + 1] first piece of every CTA
  uint32_t* node_first; // [nkeys + 1] nodes with points before each key (those of its left node included)
  int nu_grid;          // CTAs of the NUFFT sums (0: the direct sums of this call leave sums per piece)
  int nu_piece_cost;    // cost of a piece in points, for their balance
  unsigned* flags;      // [1]
  double* partial;      // sums per piece [pmax][8][Nl], or per node slot [slot][4][Nl] (NUFFT)
  double* fold;         // FP64 folds of up to kFp64Maps maps (fold.cu); the tensor-core route's fold
                        // digits [Nl][2][4][4 tc_maps][Kp] (int8) share this region
  uint8_t* live;        // [fp64_maps][ceil(Nx/16)] blocks of nodes with points (FP64 folds)
  int fp64_maps;        // maps one FP64 contraction pass can hold
  int16_t* cexp;        // [tc_maps][2] fold column scale exponents (tensor-core route)
  unsigned long long* cmax;  // [tc_maps][2] largest node |w| sum per half (bits of a double)
  unsigned* tc_next;    // [1] work counter of the contractions
  int tc_maps;          // maps one tensor-core contraction pass can hold
  double* alm_pol;      // [Nlm][2] (x nmaps for multi-map transforms)
  int64_t npts;         // N, the stride of pay
  int partial_f32;      // partial sums stored as float (tensor-core path) instead of double
  int64_t pmax;
  int piece_max;
  unsigned* slot_flags; // [kMaxRot] flags of the transforms awaiting rotation (multi-transform calls)
  unsigned* all_flags;  // [1] OR of every finished transform's flags
  size_t bytes;
};

// Workspace of a call of ntrans transforms of up to N points on a plan.
size_t call_layout(const dsht_plan_s* p, int64_t N, int ntrans, bool multi, uint8_t* base, Workspace* ws);
// The fold of map k of an FP64 contraction pass and where its alm go.
FoldOut fold_slot(const Geometry& g, const Workspace& ws, int k, double* equ, double* pol, unsigned* flags);
// How a transform of N points runs on a plan: tensor-core bin sums (tc), tensor-core
// contraction of the digit tables (digits), else the FP64 table streamed by TMA.
struct Route {
  bool tc, digits;
};
Route plan_route(const dsht_plan_s* p, int64_t N);

// Lets a kernel take all the dynamic shared memory beside its static one, once per kernel and device.  (Set
// to a launch's own size before every launch, threads with plans of different sizes could come between
// the setting and the launch of one another, and the larger launch failed.)
cudaError_t allow_shared_memory(const void* kernel);
template <typename... Args>
cudaError_t allow_shared(void (*kernel)(Args...)) {
  return allow_shared_memory(reinterpret_cast<const void*>(kernel));
}

// Kernels launched by api.cu (each file owns its launch helpers).
void launch_tables(const Geometry& g, double* Yv, double* Yd, cudaStream_t s);
void launch_points(const Geometry& g, const double* theta, const double* phi, const void* w, int w_f32,
                   int64_t N, int mode, const Workspace& ws, cudaStream_t s);
void launch_gather(const Geometry& g, const void* w, int w_f32, int64_t N, const Workspace& ws, cudaStream_t s);
// Largest |w h_k| of every piece of the sorted records (needed by the tensor-core sums).
void launch_piece_maxima(const Workspace& ws, cudaStream_t s);
void launch_publish_flags(const StatusOut& st, int n, unsigned* all, cudaStream_t s);
void launch_bin_sums_fp64(const Geometry& g, const Workspace& ws, cudaStream_t s);
int launch_bin_sums_tc(const Geometry& g, const Workspace& ws, cudaStream_t s);
// NUFFT node sums (nufft.cu) in two accuracy classes: sums of every node with points, and (mixed
// class) the pieces' |w| sums.
constexpr int kNuMixed = 0, kNuFp64 = 1;
struct NufftTables {
  int cls;
  const double* dinv;  // [Nl] 1 / Psi(m); null when the plan has none
  const double* tw;    // twiddles
};
int nufft_logn(int Nl, int cls);
int nufft_grid(int Nl, int cls);
int nufft_piece(int Nl, int cls);       // most points of a piece
int nufft_piece_cost(int Nl, int cls);
void nufft_host_tables(int Nl, int cls, std::vector<double>& dinv, std::vector<double>& tw);
int launch_bin_sums_nufft(const Geometry& g, const Workspace& ws, const NufftTables& t, cudaStream_t s);
constexpr int kNufftMinPerKey = 512;  // AUTO bin sums: NUFFT from this many points per key on average
constexpr int kFp64MaxPerKey = 28;    // AUTO bin sums: FP64 direct sums below this many per key
int tc_inner_factor(int Nl);
// FP64 fold of the current map (fold.cu); clears the alm rows that two items of the contraction add to.
void launch_fold(const Geometry& g, const Workspace& ws, const FoldOut& out, cudaStream_t s);
// Digit tables and folds (digits.cu) and the tensor-core contraction (contract_tc.cu).
int digit_kp(int Nx);                   // bytes per digit row: 2 Nx rounded up to 64
constexpr int kTcMaxNx = 8192;          // S32 class sums stay below 2^31 for 2 Nx <= 16384
void launch_tables_cols(const Geometry& g, int m0, int m1, double* Yv, double* Yd, cudaStream_t s);
void launch_table_rowexp(const Geometry& g, int64_t row0, int64_t nrows, const double* Yv, const double* Yd,
                         int16_t* rexp, cudaStream_t s);
void launch_table_digits(const Geometry& g, int64_t row0, int64_t nrows, const double* Yv, const double* Yd,
                         const int16_t* rexp, uint8_t* dig, cudaStream_t s);
void launch_table_decode(const Geometry& g, int which, int64_t r0, int64_t n, const uint8_t* dig,
                         const int16_t* rexp, double* out, cudaStream_t s);
void launch_fold_scale(const Geometry& g, const Workspace& ws, unsigned long long* cmax, cudaStream_t s);
void launch_fold_digits(const Geometry& g, const Workspace& ws, const unsigned long long* cmax, int16_t* cexp,
                        int map, int ncols,
                        uint8_t* fdig, cudaStream_t s);
int make_table_digit_tmap(CUtensorMap* tm, const uint8_t* dig, int Nx, int64_t Nlm);
std::vector<uint32_t> tc_items(int Nl);
int launch_contract_tc(const Geometry& g, const CUtensorMap& tmA, const uint32_t* items, int nitems,
                       const int16_t* rexp, const uint8_t* fdig, int fdig_cols, const int16_t* cexp, int nmaps,
                       const TcOut& out, unsigned* next_item, cudaStream_t s);
// Test hook (dsht_test_stall_next_contraction): whether this launch, of either contraction, is to leave one
// wait unsatisfied.
bool take_stall();

// FP64 contraction of the Y table (contract_fp64.cu) for nmaps <= kFp64Maps folds.
void launch_contract_fp64(const Geometry& g, const TableMaps& tm, const FoldIn& in, int nmaps, unsigned* next_item,
                          cudaStream_t s);
// 2D tensor maps of an FP64 table (node x row), boxes of 16 nodes x 8 to 128 rows.
int make_table_tmaps(TableMaps* tm, const void* base, const Geometry& g);
// An FP64 table in the JAX path's layout out[m][l - m][j] (Nl x Nl x Nx doubles, zeros
// where l >= Nl) on the device.
void launch_table_mlayout(const Geometry& g, const double* t64, double* out, cudaStream_t s);
// Tables of the rotation (rotate.cu): recursion coefficients, row scales and start values of every
// (l, k), Nl (Nl + 1) / 2 entries each.
struct RotTables {
  double* al;
  double* sc;
  double* start;
  int* start_e;
};
size_t rotation_table_bytes(int Nl);
RotTables rotation_tables(void* base, int Nl);
void launch_rotation_tables(const Geometry& g, const RotTables& t, cudaStream_t s);
// alm out[k] += R(rot[k]) for k < nmaps <= kMaxRot (a map without polar points is left as it is; flags
// null: rotate anyway), or the sum of a lone map.
void launch_rotate_back(const Geometry& g, const RotMaps& maps, int nmaps, const RotTables& t, cudaStream_t s);

// Hint: bring [p, p + bytes) into L2 (cp.async.bulk.prefetch.L2, 16-byte aligned chunks of at
// most 32 KB; the unaligned ends are left out).  lane, nlanes: the calling threads share the
// chunks.  A prefetch only warms the cache: it reads nothing into registers and cannot fault
// on the addresses of a live buffer.
__device__ __forceinline__ void prefetch_l2(const void* p, size_t bytes, int lane, int nlanes) {
  const uintptr_t a = reinterpret_cast<uintptr_t>(p);
  const uintptr_t a0 = (a + 15) & ~uintptr_t(15);
  if (bytes <= a0 - a) return;
  const size_t n = (bytes - (a0 - a)) & ~size_t(15);
  for (size_t off = (size_t)lane * 32768; off < n; off += (size_t)nlanes * 32768) {
    const size_t sz = n - off < 32768 ? n - off : 32768;
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a0 + off), "r"((unsigned)sz) : "memory");
  }
}

// Hermite weights w * {(2t+1)(1-t)^2, t(1-t)^2, t^2(3-2t), t^2(t-1)} of one point, in the
// rounding order of sht/sht.py:239-240.
__device__ __forceinline__ void hermite(double t, double wi, double* out4) {
  const double omt = __dadd_rn(1.0, -t);
  const double omt2 = __dmul_rn(omt, omt);
  const double t2 = __dmul_rn(t, t);
  out4[0] = __dmul_rn(wi, __dmul_rn(__dadd_rn(__dmul_rn(2.0, t), 1.0), omt2));
  out4[1] = __dmul_rn(wi, __dmul_rn(t, omt2));
  out4[2] = __dmul_rn(wi, __dmul_rn(t2, __dadd_rn(3.0, -__dmul_rn(2.0, t))));
  out4[3] = __dmul_rn(wi, __dmul_rn(t2, __dadd_rn(t, -1.0)));
}

// The sorted record of a point: (cos phi, sin phi, w, t), 32 bytes.
constexpr int kRec = 4;

// Healpy index of (l, m).
__host__ __device__ inline int64_t hp_index(int l, int m, int Nl) {
  return ((int64_t)m * (2 * Nl - 1 - m)) / 2 + l;
}

}  // namespace dsht

// A plan: geometry, its FP64 tables, and buffers it owns (see api.cu).
#include <mutex>
struct dsht_plan_s {
  dsht::Geometry g;
  int device = 0;
  double* Yv = nullptr;  // FP64 tables (null in a compact plan)
  void* rot_tab = nullptr;  // tables of the rotation (rotate.cu)
  double* Yd = nullptr;
  dsht::TableMaps tmY;
  // Digit tables of the tensor-core contraction (digits.cu): 4 planes [Nlm][Kp] int8 in
  // rows grouped by parity, row exponents, the work items and the TMA map of the planes.
  uint8_t* dig = nullptr;
  int16_t* rexp = nullptr;
  uint32_t* tc_items = nullptr;
  int tc_nitems = 0;
  alignas(64) CUtensorMap tmDig;
  bool tmdig = false;
  // Plan-owned buffers, grown on demand (used when the caller passes no workspace and by
  // the host-pointer entry points).
  void* ws = nullptr;
  size_t ws_bytes = 0;
  double* in = nullptr;  // [3][N] device copies of host inputs
  int64_t in_n = 0;
  double* alm = nullptr;  // [2 Nlm]
  unsigned* h_flags = nullptr;  // pinned
  int precision = DSHT_PREC_FP64;
  // NUFFT sums (nufft.cu) of the two accuracy classes: 1/Psi(m) [Nl], then the twiddles (complex),
  // built for Nl <= 2048 at the first precision level that uses the class.
  double* nu_tab[2] = {nullptr, nullptr};
  int tune_bin_sums = DSHT_BIN_SUMS_AUTO;
  int tune_piece_max = 0;      // points per bin piece (0: chosen from N and the method)
  int tune_maps_per_pass = 0;  // maps per multi-map contraction pass (0: the most that fit)
  // Stage timers: one event per stage boundary of a call, in stream order; the interval
  // from mark k to mark k+1 belongs to stage ev_stage[k] (-1: no stage).  Summed per stage
  // into prof_ms when the call has synchronised.
  static constexpr int kProfMarks = 4096;
  bool prof = false;
  cudaEvent_t* ev = nullptr;  // [kProfMarks], created by dsht_profile_enable
  int8_t ev_stage[kProfMarks] = {};
  int ev_n = 0;
  double prof_ms[DSHT_STAGE_COUNT] = {};
  int64_t prof_calls = 0;
  std::mutex mu;
};

namespace dsht {
Geometry make_geometry(int Nl, int Nx, double xmax);
// Enqueue the whole transform on `s` (flags are left in ws.flags; no synchronisation).
int run_pipeline(dsht_plan_s* p, const double* theta, const double* phi, const double* w, int64_t N, int mode,
                 double* alm, const Workspace& ws, cudaStream_t s);
// The stages after the sort: bin sums, fold, contraction, rotation.
int run_after_sort(dsht_plan_s* p, int64_t N, int mode, double* alm, const Workspace& ws, cudaStream_t s,
                   bool marks);
// One transform of a multi-transform call.  same_points: the points are those of the
// previous item (its sort is reused and only the weights are gathered again).
struct Item {
  const double* theta;
  const double* phi;
  const void* w;
  int w_f32;
  int64_t N;
  double* alm;
  bool same_points;
  unsigned* status;  // device word that receives the item's flags, or null
};
// Runs the items in order; every finished item's flags are OR-ed into ws.all_flags.
int run_items(dsht_plan_s* p, const Item* items, int n, int mode, const Workspace& ws, cudaStream_t s);
// After the stream has been synchronised: fold the stage events into the plan's totals.
void collect_profile(dsht_plan_s* p);
// Stage boundary on stream s when profiling: what follows belongs to `stage` (-1: none).
void prof_mark(dsht_plan_s* p, int stage, cudaStream_t s);
// Map device flag bits to a DSHT status code (and set the error message).
int flags_to_status(unsigned f, int mode);
}  // namespace dsht

#define DSHT_CUDA_OK(expr)                                   \
  do {                                                       \
    cudaError_t _e = (expr);                                 \
    if (_e != cudaSuccess) return dsht::set_cuda_error(_e, #expr, __FILE__, __LINE__); \
  } while (0)

namespace dsht {
int set_error(int code, const char* fmt, ...);
// Adds n to the process-wide count of kernels this library launched.
void count_launches(int n);
int set_cuda_error(cudaError_t e, const char* what, const char* file, int line);
// First kernel-launch error since the last call (recorded by count_launches), as a status.
int launch_error(const char* where);
}  // namespace dsht
