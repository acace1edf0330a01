// tsmm_tile.cuh -- TSMM on the FP32 pipe (float, complex float): C(KxN) = alpha A(KxM) B(MxN) + beta C,
// C may be A.
//
// Replaces the row-per-thread tsmm_kernel (tsmm.cuh) for these types but where that is faster (tsmm_walks in
// launch.cuh: few outputs of rows that share cache lines).
// There every thread walked a row of A in global memory, one element per load, all lanes of a row
// loading the same words: L1 wavefronts bounded it at a sixth of HBM rate (20 x 12 out of a block 32
// wide, 1e6 rows: 108 us; here 37).  Same layouts: A[r*lda+m], B[n*ldb+m], C[r*ldc+n].
//
// Design:
//   * Rows stream in tiles through a ring of shared-memory buffers filled by cp.async (16 bytes where
//     rows allow it, single elements otherwise); the row stride in shared memory is an odd multiple of
//     16 bytes, so that the 8 rows of a 16-byte load phase lie in different banks.
//   * A thread owns R rows (a tile pass apart) and 16 bytes of output columns; the cells of a row are
//     consecutive lanes.  Per 16 bytes of A it reads R vectors of A and one of B per column m, for
//     R * V * V products (V = 4 floats or 2 complex).  R = 8 keeps wide products on the FMA pipe's
//     side of shared memory; short calls take smaller R, so that all SMs have a tile.
//   * Sums run over m in ascending order, one FMA chain per output, as in tsmm.cuh and group.cu, so
//     all three give the same bits.
//   * In place: a tile is wholly in shared memory before the CTA writes any of its rows, and nobody
//     else reads or writes them.  Old C values are read by the thread that overwrites them.
#pragma once
#include "common.cuh"
#include "tsmm.cuh"

namespace skinny {

constexpr int TSMM_TILE_STAGES = 3;

template <typename T>
struct TsmmTileArgs {
  TsmmArgs<T> t;
  int stride;  // row stride of a shared tile, elements (16 bytes times an odd number)
  int vec_a;   // rows copied 16 bytes at a time
  int vec_c;   // 16-byte loads and stores of C
};

template <int B>
__device__ __forceinline__ void tile_copy(void* dst, const void* src) {
  if constexpr (B == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_u32(dst)), "l"(src), "n"(B) : "memory");
}

template <typename T, int R>
__global__ void __launch_bounds__(TSMM_THREADS, 2) tsmm_tile_kernel(const TsmmTileArgs<T> q) {
  typedef Ops<T, T> O;
  constexpr int NT = TSMM_THREADS, V = 16 / (int)sizeof(T), S = TSMM_TILE_STAGES;
  union Vec {
    uint4 w;
    T v[V];
    __device__ Vec() {}
  };
  const TsmmArgs<T>& p = q.t;
  extern __shared__ __align__(128) unsigned char smem[];
  T* Bs = reinterpret_cast<T*>(smem);
  const int M = p.M, N = p.N, np = p.np, gn = p.gn, stride = q.stride;
  const int RP = NT / gn, TR = RP * R;  // rows per pass and per tile
  T* ring = Bs + M * np;
  const int tid = threadIdx.x;
  const int64_t ntiles = (p.K + TR - 1) / TR;
  const int nt = (int)((ntiles - blockIdx.x + gridDim.x - 1) / gridDim.x);

  // chunks of a row and where this thread starts among them (advanced without divisions)
  const int cpr = q.vec_a ? M / V : M, r0 = tid / cpr, c0 = tid % cpr, rstep = NT / cpr, cstep = NT % cpr;
  auto issue = [&](int i) {
    if (i < nt) {
      const int64_t base = ((int64_t)blockIdx.x + (int64_t)i * gridDim.x) * TR;
      const int rows = (int)min((int64_t)TR, p.K - base);
      T* dst = ring + (i % S) * (TR * stride);
      const T* src = p.A + base * p.lda;
      int r = r0, c = c0;
      if (q.vec_a) {
        while (r < rows) {
          tile_copy<16>(dst + r * stride + c * V, src + (int64_t)r * p.lda + c * V);
          r += rstep;
          c += cstep;
          if (c >= cpr) {
            c -= cpr;
            r++;
          }
        }
      } else {
        while (r < rows) {
          tile_copy<(int)sizeof(T)>(dst + r * stride + c, src + (int64_t)r * p.lda + c);
          r += rstep;
          c += cstep;
          if (c >= cpr) {
            c -= cpr;
            r++;
          }
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int i = 0; i < S - 1; i++) issue(i);

  const bool fold = p.fold != 0;
  for (int n = tid >> 5; n < np; n += NT / 32)
    for (int m = tid & 31; m < M; m += 32) {
      const T b = n < N ? p.B[(int64_t)n * p.ldb + m] : tzero<T>();
      Bs[m * np + n] = (fold && n < N) ? fold_entry(p.alpha, b, p.beta, m == n) : b;
    }

  const int cell = tid % gn, rg = tid / gn, n0 = cell * V;
  const bool alpha_one = fold || O::is_one(p.alpha), bz = fold || p.beta_zero != 0;
  const bool whole = n0 + V <= N && q.vec_c;
  for (int i = 0; i < nt; i++) {
    asm volatile("cp.async.wait_group %0;" ::"n"(S - 2) : "memory");
    __syncthreads();  // tile i is in; everyone is done with tile i - 1, whose buffer is refilled
    issue(i + S - 1);
    const int64_t base = ((int64_t)blockIdx.x + (int64_t)i * gridDim.x) * TR + rg;
    const T* as = ring + (i % S) * (TR * stride) + rg * stride;

    Vec cv[R];
    if (!bz) {  // old values of C, on their way while the sums run
#pragma unroll
      for (int j = 0; j < R; j++) {
        const T* c = p.C + (base + j * RP) * p.ldc + n0;
        if (base + j * RP >= p.K) continue;
        if (whole) {
          cv[j].w = *reinterpret_cast<const uint4*>(c);
        } else {
#pragma unroll
          for (int u = 0; u < V; u++)
            if (n0 + u < N) cv[j].v[u] = c[u];
        }
      }
    }
    T acc[R][V];
#pragma unroll
    for (int j = 0; j < R; j++)
#pragma unroll
      for (int u = 0; u < V; u++) acc[j][u] = O::zero();
    int m = 0;
    const T* b = Bs + n0;
#pragma unroll 1
    for (; m + V <= M; m += V) {
      Vec a[R];
#pragma unroll
      for (int j = 0; j < R; j++) a[j].w = *reinterpret_cast<const uint4*>(as + j * RP * stride + m);
#pragma unroll
      for (int x = 0; x < V; x++, b += np) {
        Vec bv;
        bv.w = *reinterpret_cast<const uint4*>(b);
#pragma unroll
        for (int j = 0; j < R; j++)
#pragma unroll
          for (int u = 0; u < V; u++) acc[j][u] = O::mac(acc[j][u], a[j].v[x], bv.v[u]);
      }
    }
    for (; m < M; m++, b += np) {
      Vec bv;
      bv.w = *reinterpret_cast<const uint4*>(b);
#pragma unroll
      for (int j = 0; j < R; j++) {
        const T a = as[j * RP * stride + m];
#pragma unroll
        for (int u = 0; u < V; u++) acc[j][u] = O::mac(acc[j][u], a, bv.v[u]);
      }
    }
#pragma unroll
    for (int j = 0; j < R; j++) {
      if (base + j * RP >= p.K) continue;
      T* c = p.C + (base + j * RP) * p.ldc + n0;
      Vec o;
#pragma unroll
      for (int u = 0; u < V; u++)
        o.v[u] = alpha_one ? O::finish1(acc[j][u], p.beta, bz, &cv[j].v[u])
                           : O::finish(acc[j][u], p.alpha, p.beta, bz, &cv[j].v[u]);
      if (whole) {
        *reinterpret_cast<uint4*>(c) = o.w;
      } else {
#pragma unroll
        for (int u = 0; u < V; u++)
          if (n0 + u < N) c[u] = o.v[u];
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

}  // namespace skinny
