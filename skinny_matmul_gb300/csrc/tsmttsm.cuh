// tsmttsm.cuh -- TSMTTSM on CUDA cores: C(MxN) = alpha * A^T B + beta * C.
//
// Replaces the reference's GENV{3,3X,5,6,7,8}/SPECSMALL blockProductKernel + deviceReduce pairs
// (tsmttsm/genv5.cuh:9-114, genv7.cuh:10-154, specsmall.cuh:10-125).  Same layouts:
//   A: K x M row-major (A[k*lda+m]), B: K x N row-major (B[k*ldb+n]), C[n*ldc+m].
//
// Design (one persistent launch, no second reduce kernel):
//   * The K rows are cut into tiles of R rows; each CTA owns a contiguous run of tiles.
//   * Full tiles stream global -> shared with 1-D TMA bulk copies (cp.async.bulk) into a ring of
//     `stages` buffers.  After each tile, warp 0 refills the buffer of the tile before it, once
//     every warp has released it (mbarriers, bounded waits, no trap); the warps run at their own
//     pace, there is no CTA barrier while streaming.  The last tile of the matrix (which may be short, and whose last row
//     may end the allocation) and unaligned operands use plain coalesced loads instead.
//   * A thread owns a TM x TN register tile of C (a cell) for every RS-th row of a tile.  The cells
//     of all row slices fill the 256 threads; the tile is picked by launch.cuh from the
//     time the rows and the reduction take on the pipe that bounds the type: FP64 sums want few
//     padded entries and small tiles (every accumulator costs an addition on the FP64 pipe when
//     the CTA reduces), FP32 wants 4 x 4 to 8 x 8 tiles read as 16-byte vectors.
//   * Columns beyond M or N of an edge cell are read from whatever follows in shared memory and
//     only feed entries that are never written, so the inner loop has no bounds checks.
//   * Gram mode (A == B, lda == ldb, M == N) copies only A (reference SELF mode, genv7.cuh:139) and
//     computes only the cells on and below the diagonal; the others are mirrored when C is written.
//   * Partials are reduced within the CTA (halving warp shuffles, a shared-memory tree over the
//     row slices) and across CTAs on one or two levels by ticket (reduce.cuh).  The result is
//     deterministic and the tickets are reset to 0 for the next launch.
#pragma once
#include <type_traits>

#include "common.cuh"
#include "reduce.cuh"

namespace skinny {

template <typename T>
struct TsmttsmArgs {
  const T* A;
  const T* B;
  T* C;
  int64_t K, lda, ldb, ldc;
  int64_t lda_s, ldb_s;  // row strides of the shared tiles (= lda/ldb when bulk, else M/N)
  int M, N;
  T alpha, beta;
  int beta_zero, gram, bulk;
  int rows;    // rows per tile (multiple of 16)
  int stages;  // ring depth
  int64_t ntiles;
  uint32_t bytes_a, bytes_b;  // shared bytes per stage for A and B (multiples of 128)
  void* partials;
  unsigned* counter;
  int* err;
  uint32_t polls;  // poll limit of the bounded waits on the copy ring
};

constexpr int TSMTTSM_THREADS = 256;
constexpr int SMEM_HEADER = 128;  // mbarriers live here: 8 full, 8 empty
constexpr int TSMTTSM_MAX_STAGES = 8;
// Shared bytes behind the ring that an edge cell of the last row may read (at most 7 entries)
constexpr int SMEM_SLACK = 256;

// Sums on the FP32 pipe (all other types: on the FP64 pipe)
template <typename Acc>
constexpr bool fp32_sums() {
  return std::is_same<Acc, float>::value || std::is_same<Acc, c32>::value || std::is_same<Acc, c32h>::value;
}
// CTAs per SM the registers are laid out for.  FP32 tiles stream at HBM rate and need several
// CTAs' copies in flight; FP64 and complex FP64 need more than 2 warps per scheduler to cover the
// loads between their sums (16 x 16 FP64, 2^19 rows: 265 us with one CTA, 237 with two; the pipe's
// bound is 225).  Double-double sums are long enough for one CTA, and its reduction is half as
// long (16 x 16 Gram, 2^18 rows: 549 us against 578).
template <typename Acc>
constexpr int tsmttsm_ctas(int te) {
  return std::is_same<Acc, dd>::value || std::is_same<Acc, zdd>::value ? 1
         : te * (int)sizeof(Acc) <= 64 && fp32_sums<Acc>()             ? 3
         : te * (int)sizeof(Acc) <= 256                                ? 2
                                                                       : 1;
}

// The W columns of a cell: x < 4 at 4 c + x, x >= 4 in a second band 4 g further (g cells side by
// side), so that the 16-byte loads of neighbouring cells are neighbours too (8 consecutive columns
// per cell would be a 2-way bank conflict).  W < 4: W c + x.
template <int W>
__host__ __device__ __forceinline__ int cell_col(int c, int g, int x) {
  if constexpr (W <= 4) {
    return W * c + x;
  } else {
    return 4 * c + (x & 3) + (x >= 4 ? 4 * g : 0);
  }
}
// The values of a cell's columns in one row (p: the row's first column of the cell, band: 4 g); VEC:
// FP32 columns as 8- or 16-byte loads
template <typename T, int W, bool VEC>
__device__ __forceinline__ void cell_slice(const T* p, int band, T (&v)[W]) {
  if constexpr (VEC && W % 4 == 0) {
#pragma unroll
    for (int x = 0; x < W; x += 4) {
      const float4 f = *reinterpret_cast<const float4*>(p + (x ? band : 0));
      v[x] = f.x;
      v[x + 1] = f.y;
      v[x + 2] = f.z;
      v[x + 3] = f.w;
    }
  } else if constexpr (VEC && W == 2) {
    const float2 f = *reinterpret_cast<const float2*>(p);
    v[0] = f.x;
    v[1] = f.y;
  } else {
#pragma unroll
    for (int x = 0; x < W; x++) v[x] = p[x >= 4 ? band + x - 4 : x];
  }
}

// How many sums of each entry of G cells (TE entries each) a CTA joins in shared memory: one per warp
// where the lanes of a warp hold a power of two of cells, else one per row slice
__host__ __device__ __forceinline__ int tsmttsm_slots(int G) {
  return G < 32 && (G & (G - 1)) == 0 ? TSMTTSM_THREADS / 32 : TSMTTSM_THREADS / G;
}
// Accumulators of shared memory behind the ring barriers that reducing those cells takes: the slots,
// where there are several, and one per thread for the cross-CTA sum
__host__ __device__ __forceinline__ int64_t tsmttsm_red_entries(int G, int TE) {
  const int64_t slots = tsmttsm_slots(G), e = slots > 1 ? slots * G * TE : 0;
  return e > TSMTTSM_THREADS ? e : TSMTTSM_THREADS;
}

// Cell c of the lower triangle of a square cell grid, row by row: (i, j), j <= i
__host__ __device__ __forceinline__ void tri_cell(int c, int& i, int& j) {
  i = (int)((sqrtf(8.0f * (float)c + 1.0f) - 1.0f) * 0.5f);
  while (i * (i + 1) / 2 > c) i--;
  while ((i + 1) * (i + 2) / 2 <= c) i++;
  j = c - i * (i + 1) / 2;
}

template <typename T, typename Acc, int TM, int TN, bool VEC>
__global__ void __launch_bounds__(TSMTTSM_THREADS, tsmttsm_ctas<Acc>(TM * TN)) tsmttsm_kernel(const TsmttsmArgs<T> p) {
  typedef Ops<T, Acc> O;
  constexpr int NT = TSMTTSM_THREADS, NW = NT / 32, TE = TM * TN;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ int s_flag;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem);
  uint64_t* empty = full + TSMTTSM_MAX_STAGES;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int M = p.M, N = p.N;
  const int gm = ceil_div(M, TM), gn = ceil_div(N, TN);
  const bool tri = TM == TN && p.gram;
  // Cells (TM x TN blocks of C) are split into groups of <= NT along gridDim.y; every group
  // streams all rows and owns a disjoint set of C entries.
  const int cbase = blockIdx.y * NT;
  const int G = min(NT, (tri ? gm * (gm + 1) / 2 : gm * gn) - cbase);  // cells of this group per row slice
  const int RS = NT / G;                                                // row slices
  const int cell = tid % G, rs = tid / G;
  const bool active = rs < RS;
  auto cell_at = [&](int c, int& ci, int& cj) {
    if (tri) {
      tri_cell(c, ci, cj);
    } else {
      ci = c % gm;
      cj = c / gm;
    }
  };
  int ci, cj;
  cell_at(cbase + cell, ci, cj);

  const int64_t t_begin = p.ntiles * blockIdx.x / gridDim.x;
  const int64_t t_end = p.ntiles * (blockIdx.x + 1) / gridDim.x;
  const int nt = (int)(t_end - t_begin);
  const int lda_s = (int)p.lda_s, ldb_s = (int)(p.gram ? p.lda_s : p.ldb_s);
  const uint32_t stage_bytes = p.bytes_a + p.bytes_b;

  auto stage_a = [&](int s) { return reinterpret_cast<T*>(smem + SMEM_HEADER + (size_t)s * stage_bytes); };
  auto stage_b = [&](int s) {
    return p.gram ? stage_a(s) : reinterpret_cast<T*>(smem + SMEM_HEADER + (size_t)s * stage_bytes + p.bytes_a);
  };
  // A tile is bulk-loadable if its byte range ends before the last row starts: all but the last
  // tile of the matrix, which is the last of its CTA.
  const int nbulk = !p.bulk ? 0 : (t_end * (int64_t)p.rows < p.K ? nt : nt - 1);
  auto issue = [&](int i, int s) {
    const int64_t r0 = (t_begin + i) * p.rows;
    const uint32_t ba = (uint32_t)(p.rows * p.lda * (int64_t)sizeof(T));
    const uint32_t bb = p.gram ? 0u : (uint32_t)(p.rows * p.ldb * (int64_t)sizeof(T));
    mbar_arrive_expect_tx(&full[s], ba + bb);
    bulk_g2s(stage_a(s), p.A + r0 * p.lda, ba, &full[s]);
    if (!p.gram) bulk_g2s(stage_b(s), p.B + r0 * p.ldb, bb, &full[s]);
  };

  int issued = 0;  // bulk tiles issued (thread 0)
  if (tid == 0) {
    for (int s = 0; s < p.stages; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], NW);
    }
    fence_mbar_init();
    for (; issued < nbulk && issued < p.stages; issued++) issue(issued, issued);
  }
  __syncthreads();

  Acc acc[TE];
#pragma unroll
  for (int i = 0; i < TE; i++) acc[i] = O::zero();

  // A wait that gives up is recorded in *err and skips the work that is left, not the barriers:
  // every warp reaches the reduction's first barrier, where the CTA ends.
  bool bail = false;
  int s = 0, sp = 0;              // stage of tile i and of tile i - 1
  uint32_t phase = 0, phase_p = 0;  // and how often (mod 2) the ring has gone round
  const int stages = p.stages;
  // rows at a time; one for tiles of more than 256 bytes, whose few passes a tile (16 rows, 5 slices) end in half a
  // step otherwise (complex FP64 40 x 40, 2^16 rows: 915 us with two, 810; double-double 1940 and 1768)
  constexpr int UNROLL = TE <= 16 && sizeof(T) == 4 ? 4 : TE * (int)sizeof(Acc) > 256 ? 1 : 2;
  for (int i = 0; i < nt; i++) {
    const int64_t r0 = (t_begin + i) * p.rows;
    const int rows = (int)((p.K - r0) < p.rows ? (p.K - r0) : p.rows);
    T* As = stage_a(s);
    T* Bs = stage_b(s);
    if (i < nbulk) {
      if (!bail) {
        const bool ok = mbar_wait_bounded(&full[s], phase, p.err, p.polls);
        bail = !__all_sync(0xffffffffu, ok);
      }
    } else {
      // plain coalesced loads of columns [0, M) / [0, N) of `rows` rows
      __syncthreads();  // every warp is done with the stage
      for (int e = tid; e < rows * M; e += NT) {
        int r = e / M, m = e - r * M;
        As[r * lda_s + m] = p.A[(r0 + r) * p.lda + m];
      }
      if (!p.gram)
        for (int e = tid; e < rows * N; e += NT) {
          int r = e / N, n = e - r * N;
          Bs[r * ldb_s + n] = p.B[(r0 + r) * p.ldb + n];
        }
      __syncthreads();
    }
    if (active && !bail) {
      const T* ar = As + rs * lda_s + cell_col<TM>(ci, gm, 0);
      const T* br = Bs + rs * ldb_s + cell_col<TN>(cj, gn, 0);
      const int sa = RS * lda_s, sb = RS * ldb_s;
#pragma unroll UNROLL
      for (int r = rs; r < rows; r += RS, ar += sa, br += sb) {
        T a[TM], b[TN];
        cell_slice<T, TM, VEC>(ar, 4 * gm, a);
        cell_slice<T, TN, VEC>(br, 4 * gn, b);
#pragma unroll
        for (int x = 0; x < TM; x++)
#pragma unroll
          for (int y = 0; y < TN; y++) acc[x * TN + y] = O::mac(acc[x * TN + y], a[x], b[y]);
      }
    }
    if (i < nbulk) {
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[s]);
      if (warp == 0 && i > 0 && i - 1 + stages < nbulk) {  // refill the buffer of the tile before
        bool ok = true;
        if (lane == 0 && !bail) {
          ok = mbar_wait_bounded(&empty[sp], phase_p, p.err, p.polls);
          if (ok) {
            issue(issued, sp);
            issued++;
          }
        }
        bail = bail || !__all_sync(0xffffffffu, ok);
      }
    }
    sp = s;
    phase_p = phase;
    if (++s == stages) {
      s = 0;
      phase ^= 1u;
    }
  }
  // copies still in flight after a wait gave up land before the CTA ends (default bound)
  if (tid == 0 && bail)
    for (int j = max(0, issued - p.stages); j < issued; j++)
      mbar_wait_bounded(&full[j % p.stages], (uint32_t)((j / p.stages) & 1), nullptr);
  if (__syncthreads_or(bail)) {
    // a warp other than 0 may have given up alone: its CTA's copies have landed all the same,
    // warp 0 has waited for every one of them
    return;
  }

  // ---- CTA reduction: lanes of one cell, then the row slices ------------------------------------
  // Entry i of cell c is at i * G + c, so that neighbouring threads touch neighbouring words.
  const int E = G * TE;  // entries of this group
  Acc* part = reinterpret_cast<Acc*>(p.partials) + (size_t)blockIdx.y * gridDim.x * NT * TE;
  Acc* mine = part + (size_t)blockIdx.x * E;
  Acc* red = reinterpret_cast<Acc*>(smem + SMEM_HEADER);
  const int nslots = tsmttsm_slots(G);
  int base = 0, n = TE, slot = rs;
  bool owner = active;
  if (G < 32 && (G & (G - 1)) == 0) {  // every warp is active
    slot = warp;
    warp_halve<O, Acc, TE>(acc, G, lane, base, n, owner);
  }
  if (owner) {
    Acc* dst = (nslots > 1 ? red + slot * E : mine) + base * G + cell;
#pragma unroll
    for (int i = 0; i < TE; i++)
      if (i < n) dst[i * G] = acc[i];
  }
  if (nslots > 1) {
    __syncthreads();
    slot_tree<O, Acc, NT>(red, nslots, E);
    for (int e = tid; e < E; e += NT) mine[e] = red[e];
  }

  // ---- across CTAs, and the epilogue -------------------------------------------------------------
  finish_partials<O, Acc, NT>(part, p.counter + blockIdx.y, E, gridDim.y == 1, red, &s_flag, [&](int e, Acc s) {
    const int c = e % G, k = e / G;
    int i, j;
    cell_at(cbase + c, i, j);
    const int m = cell_col<TM>(i, gm, k / TN), n = cell_col<TN>(j, gn, k % TN);
    if (m >= M || n >= N) return;
    T* cp = p.C + (int64_t)n * p.ldc + m;
    *cp = O::finish(s, p.alpha, p.beta, p.beta_zero != 0, cp);
    if (tri && i != j) {
      cp = p.C + (int64_t)m * p.ldc + n;
      *cp = O::finish(gram_mirror<T, Acc>(s), p.alpha, p.beta, p.beta_zero != 0, cp);
    }
  });
}

}  // namespace skinny
