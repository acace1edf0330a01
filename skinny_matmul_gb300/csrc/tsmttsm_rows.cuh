// tsmttsm_rows.cuh -- TSMTTSM on CUDA cores for narrow products (padded M x N up to 16 entries, or
// up to 8 x 8 for FP32 and complex FP32 storage): C(MxN) = alpha * A^T B + beta * C.
//
// Replaces, for these widths, the reference's GENV3X / SPECSMALL blockProductKernel +
// deviceReduce pairs (tsmttsm/genv3x.cuh:29-81, specsmall.cuh:28-90), which on GB300 stream
// narrow products faster than the tiled ring kernel (tsmttsm.cuh) because every warp reads
// global memory directly and many warps per SM keep loads in flight.  Same layouts:
//   A: K x M row-major (A[k*lda+m]), B: K x N row-major (B[k*ldb+n]), C[n*ldc+m].
//
// Design (one launch, no separate reduction kernel):
//   * A thread owns whole rows: U rows per step, NT rows apart (consecutive threads read
//     consecutive rows, so every load instruction of a warp is one coalesced run), and keeps the
//     full TM x TN register tile of partial sums; FP64 rows are read as 16-byte pairs where the
//     leading dimensions allow it.  Gram mode (A == B) reads A only.
//   * Rows are spread grid-stride over a grid of several CTAs per SM; no shared-memory staging,
//     no barriers in the streaming loop.
//   * Reduction (reduce.cuh): halving warp shuffles, the warps of a CTA in a shared-memory tree,
//     one partial per CTA in the workspace, summed by ticket on one or two levels by the last CTAs,
//     which apply alpha / beta.  The result is deterministic; the tickets are reset for the next
//     launch.
#pragma once
#include <type_traits>

#include "common.cuh"
#include "reduce.cuh"
#include "tsmttsm.cuh"

namespace skinny {

constexpr int ROWS_THREADS = 256;

template <typename T>
struct RowsArgs {
  const T* A;
  const T* B;
  T* C;
  int64_t K, lda, ldb, ldc;
  int M, N;
  T alpha, beta;
  int beta_zero, gram;
  int vec_a, vec_b;  // FP64 rows read as 16-byte pairs (aligned base, even ld >= the padded width)
  void* partials;
  unsigned* counter;
};

template <typename V>
__host__ __device__ __forceinline__ V read_only(const V* p) {
#ifdef __CUDA_ARCH__
  return __ldg(p);
#else
  return *p;
#endif
}

// W values of one row (zero beyond n or for a row past the end); nothing but those n is read, for the last
// row may end the allocation
template <typename T, int W>
__host__ __device__ __forceinline__ void row_vals(const T* __restrict__ row, int n, bool ok, bool vec, T (&v)[W]) {
  if constexpr (std::is_same<T, double>::value && W >= 2) {
    if (vec) {
#pragma unroll
      for (int x = 0; x < W; x += 2) {
        double2 d = make_double2(0.0, 0.0);
        if (ok && x + 1 < n)
          d = read_only(reinterpret_cast<const double2*>(row + x));
        else if (ok && x < n)
          d.x = read_only(row + x);
        v[x] = d.x;
        v[x + 1] = d.y;
      }
      return;
    }
  }
#pragma unroll
  for (int x = 0; x < W; x++) {
    if (ok && x < n)
      v[x] = row[x];
    else
      v[x] = T{};
  }
}

template <typename T, typename Acc, int TM, int TN, int U>
__global__ void __launch_bounds__(ROWS_THREADS) tsmttsm_rows_kernel(const RowsArgs<T> p) {
  typedef Ops<T, Acc> O;
  constexpr int NT = ROWS_THREADS, NW = NT / 32, TMN = TM * TN;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int M = p.M, N = p.N;
  const bool gram = p.gram != 0;

  Acc acc[TMN];
#pragma unroll
  for (int i = 0; i < TMN; i++) acc[i] = O::zero();

  const int64_t stride = (int64_t)gridDim.x * NT * U;
  for (int64_t base = (int64_t)blockIdx.x * NT * U + tid; base < p.K; base += stride) {
    T a[U][TM], b[U][TN];
#pragma unroll
    for (int j = 0; j < U; j++) {
      const int64_t r = base + (int64_t)j * NT;
      const bool ok = r < p.K;
      row_vals<T, TM>(p.A + (ok ? r : 0) * p.lda, M, ok, p.vec_a != 0, a[j]);
      if (!gram) row_vals<T, TN>(p.B + (ok ? r : 0) * p.ldb, N, ok, p.vec_b != 0, b[j]);
    }
#pragma unroll
    for (int j = 0; j < U; j++)
#pragma unroll
      for (int x = 0; x < TM; x++)
#pragma unroll
        for (int y = 0; y < TN; y++) {
          T bv;
          if constexpr (TN <= TM) {
            bv = gram ? a[j][y] : b[j][y];
          } else {
            bv = b[j][y];  // Gram mode is never planned with TN > TM
          }
          acc[x * TN + y] = O::mac(acc[x * TN + y], a[j][x], bv);
        }
  }

  // ---- CTA reduction: halving shuffles, the warps in a tree, then the CTAs --------------------
  __shared__ Acc wsum[NW * TMN];
  __shared__ Acc slices[NT];
  __shared__ int s_flag;
  int e0 = 0, ne = TMN;
  bool owner = true;
  warp_halve<O, Acc, TMN>(acc, 1, lane, e0, ne, owner);
  if (owner) {
#pragma unroll
    for (int i = 0; i < (TMN + 31) / 32; i++) wsum[warp * TMN + e0 + i] = acc[i];
  }
  __syncthreads();
  slot_tree<O, Acc, NT>(wsum, NW, TMN);
  Acc* part = reinterpret_cast<Acc*>(p.partials);
  if (tid < TMN) part[(size_t)blockIdx.x * TMN + tid] = wsum[tid];
  finish_partials<O, Acc, NT>(part, p.counter, TMN, true, slices, &s_flag, [&](int e, Acc s) {
    const int m = e / TN, n = e % TN;
    if (m >= M || n >= N) return;
    T* c = p.C + (int64_t)n * p.ldc + m;
    *c = O::finish(s, p.alpha, p.beta, p.beta_zero != 0, c);
  });
}

}  // namespace skinny
