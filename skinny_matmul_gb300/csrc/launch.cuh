// launch.cuh -- host-side planning and launch of the CUDA-core TSMTTSM / TSMM kernels.
//
// The reference fixes (M, N) at compile time and picks one variant per binary
// (Makefile:11-20, versions.hpp:48-177, tsmm/fix_blend.cuh:7-29).  Here (M, N) are runtime
// values: the plan picks a register tile (TM x TN) per thread from a small set of compiled
// shapes, a row-tile size for the shared-memory ring, the ring depth and a persistent grid of
// one wave.  An autotuned grid size (blocks per SM) may override the default.
#pragma once
#include <algorithm>
#include <atomic>
#include <cmath>
#include <string>

#include "skinny.h"
#include "tsmm.cuh"
#include "tsmm_tile.cuh"
#include "tsmttsm.cuh"
#include "tsmttsm_rows.cuh"

namespace skinny {

struct DeviceInfo {
  int id = 0;
  int sms = 0;
  int smem_optin = 0;
  uint32_t wait_polls = kWaitPolls;  // poll limit of the CUDA-core TSMTTSM's bounded waits
};

// Per-(handle, stream) workspace: CTA partials + ticket counter for the in-launch reduction.
struct Workspace {
  void* partials = nullptr;
  size_t bytes = 0;
  unsigned* counter = nullptr;
};

// Implemented in api.cu: grow the workspace to `bytes` (synchronises `stream` before freeing
// the old buffer) and make sure the ticket counter exists and is zero.
skinny_status workspace_ensure(Workspace& ws, size_t bytes, cudaStream_t stream);
void set_error(const std::string& msg);
// Counts every kernel launch of the library (skinny_kernel_launches()).
void count_launch();

// Launch options chosen by the caller (autotuner / request loop).  0 = default.
struct LaunchOpts {
  int blocks_per_sm = 0;
  int rows_per_tile = 0;
  int method = -1;  // for SKINNY_ACC_AUTO: the method the autotuner measured fastest (-1: none)
};

inline int pow2ceil(int64_t v) {
  int p = 1;
  while (p < v && p < (1 << 30)) p <<= 1;
  return p;
}
inline int64_t round_up(int64_t v, int64_t m) { return (v + m - 1) / m * m; }

// The dynamic shared-memory attribute a kernel has been given, per device (the attribute is set
// per device: cudaFuncSetAttribute acts on the current one).  Zero-initialised as a static.
constexpr int kMaxDevices = 64;
struct SmemAttr {
  std::atomic<int> bytes[kMaxDevices];
};

// Raises `kernel`'s dynamic shared-memory limit on the current device to at least `bytes`;
// records only a successful call.  Returns false if the attribute could not be set.
template <typename K>
inline bool ensure_smem_attr(K kernel, int bytes, SmemAttr& done) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
    cudaGetLastError();
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess;
  }
  std::atomic<int>& d = done.bytes[dev];
  if (d.load(std::memory_order_relaxed) >= bytes) return true;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) {
    cudaGetLastError();
    set_error("cudaFuncSetAttribute(MaxDynamicSharedMemorySize) failed");
    return false;
  }
  int cur = d.load();
  while (cur < bytes && !d.compare_exchange_weak(cur, bytes)) {
  }
  return true;
}

// ----------------------------------------------------------------------------------- TSMTTSM
template <typename T, typename Acc, int TM, int TN, bool VEC>
skinny_status tsmttsm_launch_tile(const TsmttsmArgs<T>& a, dim3 grid, int smem, cudaStream_t st) {
  static SmemAttr attr;
  auto kern = tsmttsm_kernel<T, Acc, TM, TN, VEC>;
  ensure_smem_attr(kern, smem, attr);
  kern<<<grid, TSMTTSM_THREADS, smem, st>>>(a);
  count_launch();
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_error(std::string("tsmttsm launch: ") + cudaGetErrorString(e));
    return SKINNY_DEVICE_ERROR;
  }
  return SKINNY_OK;
}

// Register-tile entries (accumulators) a thread of the ring kernel may hold: 64 FP64-sized ones,
// 32 of 16 bytes, 8 of 32 bytes (complex double-double)
template <typename Acc>
constexpr int tile_cap() {
  return sizeof(Acc) >= 32 ? 8 : (int)(128 / (sizeof(Acc) / 4) < 64 ? 128 / (sizeof(Acc) / 4) : 64);
}
struct TsmttsmPlan {
  int tm, tn, rows, stages, grid, groups, smem, bulk, vec;
  int64_t ntiles, lda_s, ldb_s;
  int entries;  // of a CTA's partial: its cells' register tiles
  // workspace bytes of a grid of nb CTAs (fewer than planned: less)
  template <typename Acc>
  size_t partials(int nb) const {
    return (groups > 1 ? (size_t)nb * groups * TSMTTSM_THREADS * tm * tn : (size_t)finish_entries<Acc>(nb, entries)) *
           sizeof(Acc);
  }
};

template <typename T, typename Acc>
skinny_status tsmttsm_dispatch(const TsmttsmPlan& pl, const TsmttsmArgs<T>& a, cudaStream_t st) {
  const dim3 grid(pl.grid, pl.groups);
#define SK_TILE(X, Y)                                                                             \
  if constexpr (X * Y <= tile_cap<Acc>())                                                         \
    if (pl.tm == X && pl.tn == Y) {                                                               \
      if constexpr (std::is_same<T, float>::value && std::is_same<Acc, float>::value && X * Y > 1) \
        if (pl.vec) return tsmttsm_launch_tile<T, Acc, X, Y, true>(a, grid, pl.smem, st);         \
      return tsmttsm_launch_tile<T, Acc, X, Y, false>(a, grid, pl.smem, st);                      \
    }
  SK_TILE(1, 1) SK_TILE(1, 2) SK_TILE(1, 4) SK_TILE(1, 8)
  SK_TILE(2, 1) SK_TILE(2, 2) SK_TILE(2, 4) SK_TILE(2, 8)
  SK_TILE(4, 1) SK_TILE(4, 2) SK_TILE(4, 4) SK_TILE(4, 8)
  SK_TILE(8, 1) SK_TILE(8, 2) SK_TILE(8, 4) SK_TILE(8, 8)
#undef SK_TILE
  set_error("tsmttsm: no compiled register tile");
  return SKINNY_UNSUPPORTED;
}

// FP32 storage summed in FP64 (the double-double method of float and complex float)
template <typename T, typename Acc>
constexpr bool widens() {
  return sizeof(Acc) == 2 * sizeof(T) && !std::is_same<Acc, dd>::value && !std::is_same<Acc, zdd>::value;
}

// Clocks one SM takes for `rows` rows with TM x TN cells, and for its reduction (model).  FP64-pipe
// types: a warp instruction holds the pipe of its SM partition (one of 4) for ~68 clocks, so the
// time is the busiest partition's warps times the tile, padding included, and reducing the CTA
// costs about 1.5 more tiles per thread.  FP32: 128 FMAs per clock and SM against shared-memory
// wavefronts (one per 16-byte vector load of a warp, two counted), with HBM below both.
template <typename T, typename Acc>
double tsmttsm_tile_cost(int64_t M, int64_t N, int tm, int tn, int64_t cells, bool vec, double rows, double row_bytes) {
  const int RS = (int)(TSMTTSM_THREADS / cells);
  const int warps = (int)((cells * RS + 31) / 32), busiest = (warps + 3) / 4;
  const int t = tm * tn;
  if (!fp32_sums<Acc>()) {
    const double macs = std::is_same<Acc, zdd>::value ? 32 : std::is_same<Acc, dd>::value ? 8 : sizeof(Acc) / 4;
    const double adds = std::is_same<Acc, zdd>::value ? 40 : std::is_same<Acc, dd>::value ? 20 : sizeof(Acc) / 8;
    const double ops = t * macs * (sizeof(Acc) == 8 ? 0.5 : 1.0);
    if constexpr (widens<T, Acc>()) {
      // FP32 values are widened on the FP64 pipe too: 1 x 1 cells spend two thirds of it on that.  Large cells
      // have many row slices, whose passes over a CTA's rows are counted whole.
      const int ctas = rows < 256.0 ? 1 : tsmttsm_ctas<Acc>(t);
      const double passes = std::ceil(rows / ctas / RS), widen = (double)(sizeof(T) / 4) * (tm + tn);
      return 68.0 * busiest * ctas * ((ops + widen) * passes + 1.5 * adds * t);
    }
    return 68.0 * busiest * (ops * rows / RS + 1.5 * adds * t);
  }
  const double flops = std::is_same<Acc, float>::value ? 1 : 4;
  const double fma = busiest * t * flops;
  const double lds = warps * (vec ? 2.0 * ((tm + 3) / 4 + (tn + 3) / 4) : 1.5 * (tm + tn));
  const double step = std::max(fma, lds) + 0.3 * std::min(fma, lds) + 4.0 * busiest;
  return std::max(step / RS, row_bytes / 44.0) * rows + t * 8.0 * busiest;
}

// Whole rows of both operands, leading dimension and all, are bulk copied: they start on 16 bytes (a tile holds a
// multiple of 16 rows) and carry little besides the columns that count
inline bool bulk_rows(int64_t M, int64_t N, const void* A, int64_t lda, const void* B, int64_t ldb, bool gram) {
  return (uintptr_t)A % 16 == 0 && lda <= 2 * M + 16 && (gram || ((uintptr_t)B % 16 == 0 && ldb <= 2 * N + 16));
}

template <typename T, typename Acc>
skinny_status tsmttsm_plan(const DeviceInfo& dev, int64_t M, int64_t N, int64_t K, const void* A,
                           int64_t lda, const void* B, int64_t ldb, bool gram, const LaunchOpts& o,
                           TsmttsmPlan& pl) {
  const int cap = tile_cap<Acc>();
  const int64_t s = sizeof(T);
  const bool whole = bulk_rows(M, N, A, lda, B, ldb, gram);
  // shared row strides: ld when bulk-copied, dense (M / N) when loaded by threads
  const int64_t row_bytes_bulk = (lda + (gram ? 0 : ldb)) * s;
  const int64_t row_bytes_dense = (M + (gram ? 0 : N)) * s;
  const int64_t rb = whole ? row_bytes_bulk : row_bytes_dense;
  const int64_t las = whole ? lda : M, lbs = gram ? las : (whole ? ldb : N);
  pl.vec = std::is_same<T, float>::value && las % 4 == 0 && lbs % 4 == 0;

  // the tile: the cheapest one whose cells fit one group of threads; beyond, the largest
  const double sm_rows = (double)K / (dev.sms > 0 ? dev.sms : 1);
  double best = -1.0;
  pl.tm = pl.tn = 0;
  const int pm = std::min(pow2ceil(M), 8), pn = std::min(pow2ceil(N), 8);
  for (int tm = 1; tm <= pm; tm *= 2)
    for (int tn = 1; tn <= pn; tn *= 2) {
      if (tm * tn > cap || (gram && tm != tn)) continue;
      if (sizeof(Acc) == 8 && tm * tn > 16 && !widens<T, Acc>()) continue;
      const int64_t gm = (M + tm - 1) / tm, gn = (N + tn - 1) / tn;
      const int64_t cells = gram ? gm * (gm + 1) / 2 : gm * gn;
      if (cells > TSMTTSM_THREADS) continue;
      const double c = tsmttsm_tile_cost<T, Acc>(M, N, tm, tn, cells, pl.vec != 0, sm_rows, (double)rb);
      if (best < 0.0 || c < best) {
        best = c;
        pl.tm = tm;
        pl.tn = tn;
      }
    }
  if (best < 0.0) {
    pl.tm = pm;
    pl.tn = pn;
    while (pl.tm * pl.tn > cap) (pl.tm >= pl.tn ? pl.tm : pl.tn) /= 2;
  }
  const int tm = pl.tm, tn = pl.tn;
  const int64_t gm = (M + tm - 1) / tm, gn = (N + tn - 1) / tn;
  const int64_t Gall = gram && tm == tn ? gm * (gm + 1) / 2 : gm * gn;
  const int64_t groups = (Gall + TSMTTSM_THREADS - 1) / TSMTTSM_THREADS;
  if (groups > 64) {  // one ticket counter per group in the 256-byte counter block
    set_error("tsmttsm: M, N too large for the CUDA-core kernel");
    return SKINNY_UNSUPPORTED;
  }
  const int64_t G = Gall < TSMTTSM_THREADS ? Gall : TSMTTSM_THREADS;
  const int RS = (int)(TSMTTSM_THREADS / G);
  // as many CTAs as stay resident once an SM has rows enough to repay their reductions
  int bps = o.blocks_per_sm;
  if (bps <= 0) {
    bps = tsmttsm_ctas<Acc>(tm * tn);
    if (sm_rows < 256.0) bps = 1;
  }
  const int64_t ctas = (int64_t)std::max(dev.sms, 1) * bps;
  int rows = o.rows_per_tile;
  if (rows <= 0) {
    // FP64-pipe types: 16 KB.  FP32: a third of the CTA's shared memory, for a tile of 16 KB is
    // only a few rows per thread and the hand-offs show (13 x 7, 3.4e6 rows: 102 us; 69 with 32 KB)
    // and widened types 32 KB, for the choice of rows below
    const int64_t most = fp32_sums<Acc>() ? (int64_t)208 * 1024 / bps / 3 - 256 : widens<T, Acc>() ? 32768 : 16384;
    rows = (int)std::max<int64_t>(16, std::min<int64_t>(1024, most / rb / 16 * 16));
    // the same whole number of tiles for every CTA (rows are handed out in 16s), at least two
    // each where K allows, so that copies and sums overlap
    const int64_t per_cta = std::max<int64_t>((K + ctas - 1) / ctas, 1);
    const int64_t n = std::max<int64_t>((per_cta + rows - 1) / rows, per_cta >= 64 ? 2 : 1);
    const int most_rows = (int)std::min<int64_t>(rows, round_up((per_cta + 1) / (per_cta >= 64 ? 2 : 1), 16));
    rows = (int)std::min<int64_t>(rows, round_up((per_cta + n - 1) / n, 16));
    // widened types take the largest tiles, so the most row slices: of the rows that fit, the ones with the
    // fewest passes of the slices over the tiles of the CTA with most, a hand-off counting a quarter
    // (144 rows for 128 slices are two passes, the second nearly empty: complex FP32 7 x 7, 2^20 rows:
    // 749 us, 585 with 128 rows; FP64 and FP32 lose as much as they gain by it, up to 10 %)
    if (widens<T, Acc>()) {
      int64_t fewest = -1;
      for (int r = most_rows; r >= 16; r -= 16) {
        const int64_t tiles = ((K + r - 1) / r + ctas - 1) / ctas, passes = tiles * (4 * ((r + RS - 1) / RS) + 1);
        if (fewest < 0 || passes < fewest) {
          fewest = passes;
          rows = r;
        }
      }
    }
  }
  rows = (int)round_up(rows < RS ? RS : rows, 16);
  const int64_t stage_a = round_up(rows * las * s, 128);
  const int64_t stage_b = gram ? 0 : round_up(rows * lbs * s, 128);
  const int64_t stage = stage_a + stage_b;
  const bool bulk = whole && stage <= 65536 && K > rows;
  const int64_t budget = (int64_t)dev.smem_optin - SMEM_HEADER - 1024;
  int stages = (int)std::min<int64_t>(TSMTTSM_MAX_STAGES, (208 * 1024 / bps) / std::max<int64_t>(stage, 1));
  if (stages < 2) stages = 2;
  if (stages * stage > budget) stages = (int)(budget / stage);
  if (stages < 1) {
    set_error("tsmttsm: row tile does not fit in shared memory");
    return SKINNY_UNSUPPORTED;
  }
  pl.rows = rows;
  pl.stages = stages;
  pl.bulk = bulk;
  pl.lda_s = bulk ? lda : M;
  pl.ldb_s = gram ? pl.lda_s : (bulk ? ldb : N);
  if (!bulk) pl.vec = std::is_same<T, float>::value && pl.lda_s % 4 == 0 && pl.ldb_s % 4 == 0;
  pl.ntiles = (K + rows - 1) / rows;
  const int64_t E = G * tm * tn;
  // shared memory of the reduction: full groups of cells have one row slice, a last group with fewer
  // cells as many as fit the threads, whose sums need the more room (double-double Gram 89: 104 cells
  // behind a group of 256, 123 008 bytes where the ring takes 91 520)
  const int64_t Glast = Gall - (groups - 1) * TSMTTSM_THREADS;
  const int64_t red = std::max(tsmttsm_red_entries((int)G, tm * tn), tsmttsm_red_entries((int)Glast, tm * tn)) *
                      (int64_t)sizeof(Acc);
  pl.smem = (int)(SMEM_HEADER + std::max(stages * stage + SMEM_SLACK, red));
  int64_t grid = ctas;
  if (grid > pl.ntiles) grid = pl.ntiles;
  if (grid < 1) grid = 1;
  pl.grid = (int)grid;
  pl.groups = (int)groups;
  pl.entries = (int)E;
  return SKINNY_OK;
}

// ----------------------------------------------------------------- TSMTTSM, narrow products
// Register-tile entries a thread of the row-streaming kernel may hold: 64 for FP32 and complex FP32 storage
// (8 x 8; complex FP32 summed in FP64: 16), 16 for FP64 (8 x 8 on the ring kernel: 11.1 us against 14.6 at 2^14 rows, the same at
// 2^20; 7 x 7 116 us against 143 at 1.2e6 rows), 16 for other 16-byte accumulators (complex FP64, double-double), 4 for
// 32-byte ones (complex double-double).
template <typename T, typename Acc>
constexpr int rows_cap() {
  return fp32_sums<Acc>() || (widens<T, Acc>() && sizeof(Acc) == 8) ? 64 : (sizeof(Acc) <= 16 ? 16 : 4);
}

// The row-streaming kernel takes a product when both padded widths are <= 8 and their tile fits
// rows_cap; an autotuned row-tile size asks for the ring kernel instead.  Tiles above 16 entries
//   * go to it where the ring could not be filled by bulk copies (columns out of a wide block, 2^20 rows, L2 flushed,
//     ring / rows: FP32 6 x 6 76/52 us, in double-double, from 2^16 rows on, 226/187, 8 x 8 282/183);
//   * else FP32-pipe tiles stay with it below 2^20 rows (8 x 8 FP32: 5.1 us against 7.6 at 2^14 rows, 10.8
//     against 12.3 at 2^18, the same at 2^20; 70 against 55 at 2^22: 64 sums a thread leave few loads in flight),
//     32 entries below 3 * 2^19 (5 x 3 FP32, 2^20 rows: 16.8 against 19.7; the same at 2^21);
//   * and FP32 summed in FP64 goes to the ring (6 x 6, 2^14 rows: 11.9 us against 15.1; 2^20: 171 against 178), but
//     for long Gram products of 7 or 8 columns, one 8 x 8 cell there too (8 x 8, 2^18 rows: 80 against 69).
template <typename T, typename Acc>
bool rows_eligible(int64_t M, int64_t N, int64_t K, const void* A, int64_t lda, const void* B, int64_t ldb, bool gram,
                   const LaunchOpts& o) {
  if (o.rows_per_tile > 0 || M < 1 || N < 1 || M > 8 || N > 8) return false;
  int tm = pow2ceil(M), tn = pow2ceil(N);
  if (gram) tm = tn = std::max(tm, tn);
  if (tm * tn > rows_cap<T, Acc>()) return false;
  if (tm * tn <= 16) return true;
  const bool whole = bulk_rows(M, N, A, lda, B, ldb, gram);
  if (widens<T, Acc>()) return whole ? gram && M >= 7 && K >= (1 << 17) : K >= (1 << 16);
  return !whole || K < (tm * tn <= 32 ? 3 << 19 : 1 << 20);
}

template <typename T, typename Acc, int TM, int TN>
skinny_status tsmttsm_rows_launch(RowsArgs<T>& a, const DeviceInfo& dev, Workspace& ws, int bps_opt,
                                  cudaStream_t st) {
  if constexpr (TM * TN > rows_cap<T, Acc>()) {
    set_error("tsmttsm: register tile too large for the accumulator type");
    return SKINNY_UNSUPPORTED;
  } else {
    constexpr int U = TM * TN <= 2 ? 4 : (TM * TN <= 8 ? 2 : 1);
    auto kern = tsmttsm_rows_kernel<T, Acc, TM, TN, U>;
    int occ = 1;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, ROWS_THREADS, 0);
    if (occ < 1) occ = 1;
    if (bps_opt > 0 && bps_opt < occ) occ = bps_opt;
    // FP64-pipe types: at least 4 rows per thread, or reducing the extra CTAs costs more than they
    // save (FP64 4 x 4, 2^18 rows: 21.7 us with full occupancy, 16.0 with 2 CTAs per SM)
    if (!fp32_sums<Acc>() && bps_opt <= 0) {
      const int64_t most = (a.K + (int64_t)dev.sms * ROWS_THREADS * 4 - 1) / ((int64_t)dev.sms * ROWS_THREADS * 4);
      if (most < occ) occ = (int)std::max<int64_t>(most, 1);
    }
    const int64_t per_cta = (int64_t)ROWS_THREADS * U;
    int64_t grid = std::min<int64_t>((int64_t)dev.sms * occ, (a.K + per_cta - 1) / per_cta);
    if (grid < 1) grid = 1;
    skinny_status s = workspace_ensure(ws, (size_t)finish_entries<Acc>((int)grid, TM * TN) * sizeof(Acc), st);
    if (s != SKINNY_OK) return s;
    a.partials = ws.partials;
    a.counter = ws.counter;
    kern<<<(int)grid, ROWS_THREADS, 0, st>>>(a);
    count_launch();
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
      set_error(std::string("tsmttsm launch: ") + cudaGetErrorString(e));
      return SKINNY_DEVICE_ERROR;
    }
    return SKINNY_OK;
  }
}

template <typename T, typename Acc>
skinny_status tsmttsm_rows_run(const DeviceInfo& dev, Workspace& ws, cudaStream_t st, int64_t M, int64_t N,
                               int64_t K, const T* A, int64_t lda, T alpha, const T* B, int64_t ldb, T beta,
                               bool beta_zero, T* C, int64_t ldc, bool gram, const LaunchOpts& o) {
  int tm = pow2ceil(M), tn = pow2ceil(N);
  if (gram) tm = tn = std::max(tm, tn);
  RowsArgs<T> a;
  a.A = A;
  a.B = B;
  a.C = C;
  a.K = K;
  a.lda = lda;
  a.ldb = ldb;
  a.ldc = ldc;
  a.M = (int)M;
  a.N = (int)N;
  a.alpha = alpha;
  a.beta = beta;
  a.beta_zero = beta_zero;
  a.gram = gram;
  // 16-byte pairs: FP64, an aligned base, an even leading dimension covering the padded width
  const bool f64 = std::is_same<T, double>::value;
  a.vec_a = f64 && tm >= 2 && (uintptr_t)A % 16 == 0 && lda % 2 == 0 && lda >= tm;
  a.vec_b = f64 && tn >= 2 && (uintptr_t)B % 16 == 0 && ldb % 2 == 0 && ldb >= tn;
  a.partials = nullptr;
  a.counter = nullptr;
  const int b = o.blocks_per_sm;
#define SK_ROWS(X, Y) \
  if (tm == X && tn == Y) return tsmttsm_rows_launch<T, Acc, X, Y>(a, dev, ws, b, st);
  SK_ROWS(1, 1) SK_ROWS(1, 2) SK_ROWS(1, 4) SK_ROWS(1, 8)
  SK_ROWS(2, 1) SK_ROWS(2, 2) SK_ROWS(2, 4) SK_ROWS(2, 8)
  SK_ROWS(4, 1) SK_ROWS(4, 2) SK_ROWS(4, 4) SK_ROWS(4, 8)
  SK_ROWS(8, 1) SK_ROWS(8, 2) SK_ROWS(8, 4) SK_ROWS(8, 8)
#undef SK_ROWS
  set_error("tsmttsm: no compiled row tile");
  return SKINNY_UNSUPPORTED;
}

// Workspace asked for up to 64 x 64, whatever the tile and the rows: what the cells, padded by at most 7 columns
// either way, take with all CTAs that any tile may have per SM.  It only grows with M and N, so that a smaller product
// captured after a larger one on its stream allocates nothing (complex FP64 43 x 45 takes 1.7 times the entries of
// 48 x 48, whose tiles fit).
template <typename Acc>
size_t tsmttsm_workspace(const DeviceInfo& dev, int64_t M, int64_t N) {
  if (M > 64 || N > 64) return 0;
  const int64_t ctas = (int64_t)std::max(dev.sms, 1) * tsmttsm_ctas<Acc>(1) + FINISH_MAX_GROUPS;
  return (size_t)(ctas * round_up(M, 8) * round_up(N, 8)) * sizeof(Acc);
}

template <typename T, typename Acc>
skinny_status tsmttsm_run(const DeviceInfo& dev, Workspace& ws, int* err, cudaStream_t st,
                          int64_t M, int64_t N, int64_t K, const T* A, int64_t lda, T alpha,
                          const T* B, int64_t ldb, T beta, bool beta_zero, T* C, int64_t ldc,
                          const LaunchOpts& o) {
  const bool gram = (A == B) && (lda == ldb) && (M == N);
  if (rows_eligible<T, Acc>(M, N, K, A, lda, B, ldb, gram, o))
    return tsmttsm_rows_run<T, Acc>(dev, ws, st, M, N, K, A, lda, alpha, B, ldb, beta, beta_zero, C, ldc, gram, o);
  TsmttsmPlan pl;
  skinny_status s = tsmttsm_plan<T, Acc>(dev, M, N, K, A, lda, B, ldb, gram, o, pl);
  if (s != SKINNY_OK) return s;
  s = workspace_ensure(ws, std::max(pl.partials<Acc>(pl.grid), tsmttsm_workspace<Acc>(dev, M, N)), st);
  if (s != SKINNY_OK) return s;
  TsmttsmArgs<T> a;
  a.A = A;
  a.B = B;
  a.C = C;
  a.K = K;
  a.lda = lda;
  a.ldb = ldb;
  a.ldc = ldc;
  a.lda_s = pl.lda_s;
  a.ldb_s = pl.ldb_s;
  a.M = (int)M;
  a.N = (int)N;
  a.alpha = alpha;
  a.beta = beta;
  a.beta_zero = beta_zero;
  a.gram = gram;
  a.bulk = pl.bulk;
  a.rows = pl.rows;
  a.stages = pl.stages;
  a.ntiles = pl.ntiles;
  const int64_t sz = sizeof(T);
  a.bytes_a = (uint32_t)round_up(pl.rows * pl.lda_s * sz, 128);
  a.bytes_b = gram ? 0u : (uint32_t)round_up(pl.rows * pl.ldb_s * sz, 128);
  a.partials = ws.partials;
  a.counter = ws.counter;
  a.err = err;
  a.polls = dev.wait_polls;
  return tsmttsm_dispatch<T, Acc>(pl, a, st);
}

// -------------------------------------------------------------------------------------- TSMM
template <typename T, typename Acc, int TN, int U>
skinny_status tsmm_launch_tile(const TsmmArgs<T>& a, int bps, int sms, int smem, cudaStream_t st) {
  static SmemAttr attr;
  auto kern = tsmm_kernel<T, Acc, TN, U>;
  ensure_smem_attr(kern, smem, attr);
  int occ = 1;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, TSMM_THREADS, smem);
  if (occ < 1) occ = 1;
  if (bps > 0 && bps < occ) occ = bps;
  const int RS = TSMM_THREADS / a.gn * U;
  int64_t need = (a.K + RS - 1) / RS;
  int64_t grid = (int64_t)sms * occ;
  if (grid > need) grid = need;
  if (grid < 1) grid = 1;
  kern<<<(int)grid, TSMM_THREADS, smem, st>>>(a);
  count_launch();
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_error(std::string("tsmm launch: ") + cudaGetErrorString(e));
    return SKINNY_DEVICE_ERROR;
  }
  return SKINNY_OK;
}

template <typename T, int R>
skinny_status tsmm_tile_launch(const TsmmTileArgs<T>& a, int bps, int sms, int smem, cudaStream_t st) {
  static SmemAttr attr;
  auto kern = tsmm_tile_kernel<T, R>;
  if (!ensure_smem_attr(kern, smem, attr)) return SKINNY_DEVICE_ERROR;
  int occ = smem <= 112 * 1024 ? 2 : 1;  // what the registers and the shared memory of an SM hold
  if (bps > 0 && bps < occ) occ = bps;
  const int64_t rows = TSMM_THREADS / a.t.gn * R;
  const int64_t grid = std::max<int64_t>(1, std::min<int64_t>((int64_t)sms * occ, (a.t.K + rows - 1) / rows));
  kern<<<(int)grid, TSMM_THREADS, smem, st>>>(a);
  count_launch();
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_error(std::string("tsmm launch: ") + cudaGetErrorString(e));
    return SKINNY_DEVICE_ERROR;
  }
  return SKINNY_OK;
}

// Whether tsmm_kernel, whose threads walk a row each, is the better one for float and complex float (us, walking /
// tiled, 2^20 rows, L2 flushed):
//   * at most 16 bytes in and out, which it streams at 0.75 of HBM rate;
//   * few columns out of rows that share cache lines (at most 128 bytes apart) and cannot be copied 16 bytes at a
//     time: FP32 9 x 2 12.5/18.6, 16 x 1 in rows of 17 21/28.5, 24 x 3 the same; complex 9 x 1 in rows of 10 1.1x;
//   * complex FP32 up to 6 x 2 also out of wide blocks (4 x 2, beta, 2^18 rows: 1.5x);
//   * complex FP32, 5 to 9 outputs that do not fill the cells, from 2^17 packed rows that are not aligned: from 16 columns
//     in on (33 x 9, 2^18 rows, L2 warm: 39/47; 17 x 5 1.2x; but 17 x 8 0.95x, 20 x 12 0.7x, 33 x 9 at 2^14 rows 0.8x),
//     with beta and an odd number of outputs from 7 on (9 x 5 39.5/45; without 35/38).
template <typename T>
bool tsmm_walks(int M, int N, int np, int64_t K, int64_t lda, bool vec_a, bool beta) {
  if (M * (int)sizeof(T) <= 16 && N * (int)sizeof(T) <= 16) return true;
  const bool lines = lda * (int64_t)sizeof(T) <= 128;
  if (sizeof(T) == 4) return lines && (vec_a ? N <= (beta ? 2 : 1) && M <= 8 : N <= 3 || (N == 4 && M > 8));
  if ((N <= 2 && M <= 6) || (lines && N <= 3 && M <= (vec_a ? 4 : 9))) return true;
  return K >= (1 << 17) && !vec_a && lda <= M + 8 && N >= 5 && N <= 9 && np > N && M >= (beta && N % 2 ? 7 : 16);
}

// The tiled kernel for float and complex float; false: the shape is left to tsmm_kernel (the rule above, more than
// 128 outputs, or a tile that does not fit).  Rows per thread: 8 where the FMA pipe is near (more than 16
// columns of output), 4 otherwise, fewer while a CTA's ring is above 110 KB (two CTAs per SM) or SMs would go
// without rows.
template <typename T>
bool tsmm_tile_run(const DeviceInfo& dev, cudaStream_t st, const TsmmArgs<T>& t, const LaunchOpts& o, skinny_status& s) {
  constexpr int V = 16 / (int)sizeof(T);
  const int M = t.M, N = t.N;
  TsmmTileArgs<T> a;
  a.t = t;
  a.t.gn = pow2ceil((N + V - 1) / V);
  a.t.np = a.t.gn * V;
  if (a.t.gn > 32) return false;
  const int chunks = (M + V - 1) / V;
  a.stride = (chunks % 2 ? chunks : chunks + 1) * V;
  a.vec_a = M % V == 0 && t.lda % V == 0 && (uintptr_t)t.A % 16 == 0;
  a.vec_c = t.ldc % V == 0 && (uintptr_t)t.C % 16 == 0;
  if (tsmm_walks<T>(M, N, a.t.np, t.K, t.lda, a.vec_a != 0, !t.beta_zero && !t.fold)) return false;
  const int64_t bs = (int64_t)M * a.t.np * sizeof(T);
  const int RP = TSMM_THREADS / a.t.gn;
  auto smem = [&](int R) { return bs + (int64_t)TSMM_TILE_STAGES * RP * R * a.stride * sizeof(T); };
  int R = N * (int)sizeof(T) > 64 ? 8 : 4;
  while (R > 1 && (smem(R) > 110 * 1024 || (t.K + RP * R - 1) / (RP * R) < 2 * dev.sms)) R /= 2;
  if (smem(R) > dev.smem_optin - 1024) return false;
  const int sm = (int)smem(R), b = o.blocks_per_sm;
  s = R == 8   ? tsmm_tile_launch<T, 8>(a, b, dev.sms, sm, st)
      : R == 4 ? tsmm_tile_launch<T, 4>(a, b, dev.sms, sm, st)
      : R == 2 ? tsmm_tile_launch<T, 2>(a, b, dev.sms, sm, st)
               : tsmm_tile_launch<T, 1>(a, b, dev.sms, sm, st);
  return true;
}

template <typename T, typename Acc>
skinny_status tsmm_run(const DeviceInfo& dev, cudaStream_t st, int64_t M, int64_t N, int64_t K,
                       const T* A, int64_t lda, T alpha, const T* B, int64_t ldb, T beta,
                       bool beta_zero, T* C, int64_t ldc, const LaunchOpts& o) {
  const int cap = sizeof(Acc) <= 8 ? 8 : (sizeof(Acc) <= 16 ? 4 : 2);
  int tn = pow2ceil(N) < cap ? pow2ceil(N) : cap;
  int gn = pow2ceil((N + tn - 1) / tn);
  if (gn > 32) {
    set_error("tsmm: N too large");
    return SKINNY_UNSUPPORTED;
  }
  const int np = gn * tn;
  const int64_t smem = (int64_t)M * np * sizeof(T);
  if (smem > dev.smem_optin) {
    set_error("tsmm: B does not fit in shared memory");
    return SKINNY_UNSUPPORTED;
  }
  TsmmArgs<T> a;
  a.A = A;
  a.B = B;
  a.C = C;
  a.K = K;
  a.lda = lda;
  a.ldb = ldb;
  a.ldc = ldc;
  a.M = (int)M;
  a.N = (int)N;
  a.alpha = alpha;
  a.beta = beta;
  a.beta_zero = beta_zero;
  // in place with M == N: C = A (alpha B + beta I), folded while B is staged
  a.fold = (const void*)A == (const void*)C && lda == ldc && M == N && !beta_zero && sizeof(Acc) == sizeof(T);
  a.gn = gn;
  a.np = np;
  if constexpr (std::is_same<T, Acc>::value && (std::is_same<T, float>::value || std::is_same<T, c32>::value)) {
    skinny_status s;
    if (tsmm_tile_run<T>(dev, st, a, o, s)) return s;
  }
  const int sm = (int)(smem < 16 ? 16 : smem);
  // narrow rows (M <= 4, a few outputs per thread): 4 rows per thread and step
  // (32-byte accumulators: one row per thread and step)
  const bool multi = M <= 4 && tn <= 4 && sizeof(Acc) <= 16;
  switch (tn) {
    case 1:
      if constexpr (sizeof(Acc) <= 16)
        if (multi) return tsmm_launch_tile<T, Acc, 1, 4>(a, o.blocks_per_sm, dev.sms, sm, st);
      return tsmm_launch_tile<T, Acc, 1, 1>(a, o.blocks_per_sm, dev.sms, sm, st);
    case 2:
      if constexpr (sizeof(Acc) <= 16)
        if (multi) return tsmm_launch_tile<T, Acc, 2, 4>(a, o.blocks_per_sm, dev.sms, sm, st);
      return tsmm_launch_tile<T, Acc, 2, 1>(a, o.blocks_per_sm, dev.sms, sm, st);
    case 4:
      if constexpr (sizeof(Acc) <= 16) {
        return multi ? tsmm_launch_tile<T, Acc, 4, 4>(a, o.blocks_per_sm, dev.sms, sm, st)
                     : tsmm_launch_tile<T, Acc, 4, 1>(a, o.blocks_per_sm, dev.sms, sm, st);
      }
      break;
    default:
      if constexpr (sizeof(Acc) <= 8) return tsmm_launch_tile<T, Acc, 8, 1>(a, o.blocks_per_sm, dev.sms, sm, st);
  }
  set_error("tsmm: no compiled column tile");
  return SKINNY_UNSUPPORTED;
}

// Explicit instantiation of both launchers for a (storage, accumulator) pair (EXT empty: the
// inst_*.cu units, one pair or two each, so that the build compiles them in parallel) or its
// extern declaration (EXT extern: the units that call them).
#define SKINNY_LAUNCHERS(EXT, T, ACC)                                                                         \
  EXT template skinny_status tsmttsm_run<T, ACC>(const DeviceInfo&, Workspace&, int*, cudaStream_t, int64_t, \
                                                 int64_t, int64_t, const T*, int64_t, T, const T*, int64_t, T, \
                                                 bool, T*, int64_t, const LaunchOpts&);                      \
  EXT template skinny_status tsmm_run<T, ACC>(const DeviceInfo&, cudaStream_t, int64_t, int64_t, int64_t,     \
                                              const T*, int64_t, T, const T*, int64_t, T, bool, T*, int64_t,   \
                                              const LaunchOpts&);

}  // namespace skinny
