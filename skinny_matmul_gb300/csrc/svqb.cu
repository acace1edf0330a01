// svqb.cu -- SVQB orthogonalisation entirely on the device.
//
// Follows svqb/svqb.cu:72-130 of the reference step by step, but keeps every step on the GPU
// (the reference copies S to the host and calls MAGMA's dsyevd there, svqb.cu:95-120):
//   1. S = X^T X                      TSMTTSM in Gram mode, method chosen by the caller
//   2. d_i = 1/sqrt(S_ii) if |S_ii| > 1e-15 else 0;  S <- D S D        (svqb.cu:99-110)
//   3. S = U L U^T                    cyclic Jacobi (parallel round-robin order: the M/2 rotations
//                                     of a round at once) in FP32, refined in FP64 by products of
//                                     M x M matrices, finished by FP64 Jacobi sweeps where pairs are
//                                     left; eigenvalues ascending as dsyevd returns them
//   4. T = D U diag(1/sqrt(max(1e-15, l)))  stored as TSMM's B (B[n*M+m])  (svqb.cu:115-119)
//   5. X <- X T                       in-place TSMM                      (svqb.cu:124-129)
//   6. optional ||Q^T Q - I||_F with a double-double Gram                (svqb.cu:184-211)
// Eigenvector signs are fixed so that the largest-magnitude entry of each is positive.
#include <cuda_runtime.h>

#include <cstring>
#include <string>

#include "api_internal.h"

namespace skinny {

constexpr int SVQB_MAX_M = 64;
constexpr int SVQB_THREADS = 256;
constexpr int EIG_THREADS = 544;  // 17 warps, one for each distance (0 .. 16) between pairs
constexpr int EIG_SWEEPS32 = 12;  // FP32 sweeps at most
constexpr size_t EIG_LOG = (size_t)EIG_SWEEPS32 * (SVQB_MAX_M - 1) * 32;  // rotations they can have
// Leading dimension of the shared M x M arrays: even, so that the lanes of a warp, which walk rows
// and columns up or down together, step by an odd number of banks.
constexpr int EIG_LD = 66;
constexpr int EIG_SIZE = 8192;  // entries from one buffer of the matrix to the other (a power of two)
static_assert(EIG_SIZE >= SVQB_MAX_M * EIG_LD, "a buffer holds the matrix");
// Smallest M that goes through the FP32 stage: its launches take ~90 us together at M = 8, a whole
// FP64 Jacobi 45 us at M = 4, 75 at M = 6, ~110 at M = 8 and several ms at M = 64
constexpr int EIG_MIXED_MIN = 8;
// A pair of eigenvectors is refined to first order when its rotation is below this
constexpr double EIG_SMALL = 1.0 / 1024.0;
// and when the eigenvalues differ by more than this: far below the rounding level of a matrix of unit
// diagonal, far above the smallest FP32 number with a finite reciprocal (2^-128), which null vectors of
// dependent columns, whose eigenvalues are 1e-33 to 1e-50 apart, are not
constexpr double EIG_GAP = 0x1p-100;

// Round-robin order in slots: pair l of a round is slots l and 32 + l.  From one round to the next the
// players move one pair on, p to the pair below, q to the pair above, with player n - 1 fixed in slot
// 0, pair 1's p turning into pair 0's q and the last pair's q into its p; after n - 1 rounds everybody
// is back.  Rows and columns are kept in slot order, so every thread reads and writes the same
// addresses in every round.
__device__ __forceinline__ int slot_of(int player, int n) {
  return player == n - 1 ? 0 : player == 0 ? 32 : player < n / 2 ? player : 32 + n - 1 - player;
}
__device__ __forceinline__ int next_slot(int slot, int np) {
  if (slot >= 32) return slot - 32 == np - 1 && np > 1 ? np - 1 : slot - 32 == 0 && np == 1 ? 32 : slot + 1;
  return slot == 0 ? 0 : slot == 1 ? 32 : slot - 1;
}
__device__ __forceinline__ float rsqrt_approx(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Cyclic Jacobi (n players, n - 1 rounds a sweep, n / 2 rotations a round) on the matrix in A, which changes
// between two buffers (cur: the one that holds it).  FP64: V <- V J (columns in slot order).  FP32: the rotations
// of round i go to log[32 i ..] (cosine, sine per pair; log points to this lane's), for eig_replay_kernel.
//
// A round is one pass: the pairs (k, l) of pairs cut the matrix into 2 x 2 blocks, each is rotated
// from both sides by one lane and written, with its mirror image, into the other buffer.  The last
// warp forms the rotations while the others' loads are under way.
// FP32 rounds are bound by the latency of that chain: 710 clocks at M = 64 (with the players'
// addresses worked out anew in each round 1200; with the next round's rotations formed from the last
// warp's own copy of the rotated entries, one barrier less but a longer chain, 870).
// FP64 rounds are bound by the pipe (1.89 operations per clock).  The tangent is taken in FP32 and
// refined by one FP64 Newton step, the cosine normalised by two, so the rotation is orthogonal to
// rounding.  A round without a pair that matters costs its moves only (~0.4 us instead of ~5 at
// M = 64): behind the refinement only the pairs that it could not separate are left.
//
// Rotation of a pair with diagonal app, aqq and coupling apq: cos 2x = |d| / hypot(d, b) with
// d = aqq - app, b = 2 apq, then cos x and sin x; tan x = sin 2x / (2 cos^2 x).
template <typename R>
__device__ __forceinline__ void rotation(R app, R aqq, R apq, R& c, R& s) {
  const float d = (float)(aqq - app), b = 2.0f * (float)apq;
  const float h = rsqrt_approx(fmaf(d, d, b * b));
  const float u = fmaf(0.5f * fabsf(d), h, 0.5f), w = copysignf(0.5f, d) * b * h;
  const bool ok = fmaxf(fabsf(d), fabsf(b)) > 1.0e-18f;
  if constexpr (sizeof(R) == 4) {
    const float x = rsqrt_approx(u);
    c = ok ? u * x : 1.0f;
    s = ok ? w * x : 0.0f;
  } else {
    double t = ok ? (double)__fdividef(w, u) : 0.0;
    if (ok) {  // apq (1 - t^2) = (aqq - app) t: one Newton step, its slope in FP32
      const double e = fma(-t, fma(apq, t, aqq - app), apq);
      t = fma(e, (double)__fdividef(1.0f, fmaf(b, (float)t, d)), t);
    }
    const double y = fma(t, t, 1.0);
    double x = (double)rsqrt_approx((float)y);
    x = x * fma(-0.5 * y * x, x, 1.5);
    x = x * fma(-0.5 * y * x, x, 1.5);
    c = x;
    s = t * x;
  }
}

template <typename R>
__device__ int jacobi_sweeps(R* A, int& cur, R* V, R* cs, R* red, int M, int n, R tol, int max_sweeps, float2* log) {
  constexpr int NW = EIG_THREADS / 32, LD = EIG_LD, H = 32 * LD, ROT = NW - 1;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int np = n / 2;
  // this lane's block: pair `lane` and the pair `warp` further, the half distance only once each
  int k = lane + warp;
  if (k >= np) k -= np;
  const bool mine = lane < np && 2 * warp <= np && !(2 * warp == np && lane >= warp);
  if (!mine) k = 0;
  const bool mirror = mine && warp > 0, blocks = sizeof(R) == 4 || 2 * warp <= np;
  const int rd = k * LD + lane;
  const int cp = next_slot(lane, np), cq = next_slot(32 + lane, np), rp = next_slot(k, np), rq = next_slot(32 + k, np);
  const int w00 = rp * LD + cp, w01 = rp * LD + cq, w10 = rq * LD + cp, w11 = rq * LD + cq;
  const int m00 = cp * LD + rp, m01 = cq * LD + rp, m10 = cp * LD + rq, m11 = cq * LD + rq;
  R prev_off = 0;
  int sweeps = 0;
  bool extra = false;
  for (; sweeps < max_sweeps; sweeps++) {
    // converged when the off-diagonal mass is at the rounding level of the matrix, or when it is
    // small and a sweep no longer reduces it (rounding noise).  FP64: where an entry still couples
    // two small eigenvalues (above 1e-13 of their geometric mean), one more sweep follows.
    // Warp 0 sums and decides.
    R off = 0, dia = 0;
    bool coupled = false;
    for (int i = warp; i < n; i += NW)
      for (int j = lane; j < n; j += 32) {
        const int si = i < np ? i : 32 + i - np, sj = j < np ? j : 32 + j - np;
        const R a = A[cur + si * LD + sj], q = a * a;
        if (i != j)
          off += q;
        else
          dia += q;
        if constexpr (sizeof(R) == 8)
          if (i < j) coupled |= q > 1.0e-26 * fabs(A[cur + si * (LD + 1)] * A[cur + sj * (LD + 1)]);
      }
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) off += __shfl_xor_sync(0xffffffffu, off, o);
    // a warp has one or more whole rows: their diagonal entries are in as many lanes
    for (int o = 16; o >= 1; o >>= 1) dia += __shfl_xor_sync(0xffffffffu, dia, o);
    if (lane == 0) {
      red[2 * warp] = off;
      red[2 * warp + 1] = dia;
    }
    coupled = __syncthreads_or(coupled);
    if (warp == 0) {
      off = lane < NW ? red[2 * lane] : 0;
      dia = lane < NW ? red[2 * lane + 1] : 0;
#pragma unroll
      for (int o = 16; o >= 1; o >>= 1) {
        off += __shfl_xor_sync(0xffffffffu, off, o);
        dia += __shfl_xor_sync(0xffffffffu, dia, o);
      }
      const R near = sizeof(R) == 4 ? (R)1.0e-10 : (R)1.0e-20, all = off + dia;
      const bool met =
          off <= tol * all || (sweeps > 0 && off <= near * all && off >= (R)0.25 * prev_off);
      prev_off = off;
      if (lane == 0) red[2 * NW] = met ? 1 : 0;
    }
    __syncthreads();
    if (red[2 * NW] != 0 || M == 1) {
      if (!coupled || extra || M == 1) break;
      extra = true;
    }

#pragma unroll 1
    for (int r = 0; r < n - 1; r++) {
      const R* a = A + cur + rd;
      R b00 = 0, b01 = 0, b10 = 0, b11 = 0;
      if (blocks) b00 = a[0], b01 = a[32], b10 = a[H], b11 = a[H + 32];
      if (warp == ROT) {
        const R* g = A + cur + (lane < np ? lane * (LD + 1) : 0);
        R c = 1, s = 0;
        if constexpr (sizeof(R) == 8) {
          // pairs coupled by less than 1e-14 of their geometric mean are left alone; a round of such
          // pairs only moves entries on
          const R app = g[0], aqq = g[H + 32], apq = g[32];
          const bool turn = lane < np && apq * apq > 1.0e-28 * fabs(app * aqq);
          if (turn) rotation<R>(app, aqq, apq, c, s);
          if (lane == 0) cs[64] = 0;
          __syncwarp();
          if (turn) cs[64] = 1;
        } else {
          if (lane < np) rotation<R>(g[0], g[H + 32], g[32], c, s);
        }
        cs[2 * lane] = c;
        cs[2 * lane + 1] = s;
        if constexpr (sizeof(R) == 4) {
          *log = make_float2((float)c, (float)s);
          log += 32;
        }
      }
      __syncthreads();
      const R c = cs[2 * lane], s = cs[2 * lane + 1], ck = cs[2 * k], sk = cs[2 * k + 1];
      const bool turns = sizeof(R) == 4 || cs[64] != 0;
      if (blocks) {
        R* o = A + (cur ^ EIG_SIZE);
        R v00 = b00, v01 = b01, v10 = b10, v11 = b11;
        if (turns) {
          const R u00 = c * b00 - s * b01, u01 = s * b00 + c * b01;
          const R u10 = c * b10 - s * b11, u11 = s * b10 + c * b11;
          v00 = ck * u00 - sk * u10, v10 = sk * u00 + ck * u10;
          v01 = ck * u01 - sk * u11, v11 = sk * u01 + ck * u11;
        }
        if (mine) {
          o[w00] = v00;
          o[w01] = v01;
          o[w10] = mirror ? v10 : v01;
          o[w11] = v11;
        }
        if (mirror) {
          o[m00] = v00;
          o[m01] = v01;
          o[m10] = v10;
          o[m11] = v11;
        }
      }
      if constexpr (sizeof(R) == 8) {
        for (int i = warp; i < M; i += NW) {
          const R vp = V[i * LD + lane], vq = V[i * LD + 32 + lane];
          __syncwarp();
          if (lane < np) {
            V[i * LD + cp] = turns ? c * vp - s * vq : vp;
            V[i * LD + cq] = turns ? s * vp + c * vq : vq;
          }
        }
      }
      __syncthreads();
      cur ^= EIG_SIZE;
    }
  }
  return sweeps;
}

template <typename R>
__host__ __device__ constexpr size_t eig_smem() {
  return (2 * EIG_SIZE + (sizeof(R) == 4 ? 0 : SVQB_MAX_M * EIG_LD) + 66 + 2 * (EIG_THREADS / 32) + 1) * sizeof(R);
}

// First stage: d_i = 1 / sqrt(S_ii) (0 where |S_ii| <= 1e-15), A <- D S D in FP64, and a Jacobi of it in
// FP32, whose rotations are logged; *rounds: how many rounds.
__global__ void __launch_bounds__(EIG_THREADS) svqb_jacobi32_kernel(const double* __restrict__ S, int M,
                                                                             double* __restrict__ d,
                                                                             double* __restrict__ A, float2* __restrict__ log,
                                                                             int* __restrict__ rounds) {
  extern __shared__ __align__(16) float shf[];
  __shared__ double ds[SVQB_MAX_M];
  constexpr int NT = EIG_THREADS;
  float* cs = shf + 2 * EIG_SIZE;
  const int tid = threadIdx.x, n = (M + 1) & ~1;
  for (int i = tid; i < M; i += NT) {
    const double sii = S[i * M + i];
    ds[i] = fabs(sii) > 1.0e-15 ? 1.0 / sqrt(sii) : 0.0;
    d[i] = ds[i];
  }
  __syncthreads();
  for (int e = tid; e < n * n; e += NT) {
    const int i = e / n, j = e - i * n;
    double a = 0.0;
    if (i < M && j < M) {
      a = S[i * M + j] * ds[i] * ds[j];
      A[i * M + j] = a;
    }
    shf[slot_of(i, n) * EIG_LD + slot_of(j, n)] = (float)a;
  }
  __syncthreads();
  int cur = 0;
  const int sweeps = jacobi_sweeps<float>(shf, cur, nullptr, cs, cs + 66, M, n, (float)(M * M) * 3.6e-15f,
                                          EIG_SWEEPS32, log + (tid & 31));
  if (tid == 0) *rounds = sweeps * (n - 1);
}

// X <- the product of the logged rotations: one warp per row of X = I J J' ..., lane l holding the row's
// entries of pair l, which move on by shuffles as the slots do.
constexpr int REPLAY_THREADS = 64;
__global__ void __launch_bounds__(REPLAY_THREADS) eig_replay_kernel(const float2* __restrict__ log,
                                                                    const int* __restrict__ rounds, int M,
                                                                    double* __restrict__ X) {
  const int lane = threadIdx.x & 31, row = (blockIdx.x * REPLAY_THREADS + threadIdx.x) >> 5;
  if (row >= M) return;
  const int n = (M + 1) & ~1, np = n / 2, R = *rounds;
  // the players of slots l and 32 + l before the first round
  const int p = lane == 0 ? n - 1 : lane, q = lane == 0 ? 0 : n - 1 - lane;
  float vp = lane < np && p == row ? 1.0f : 0.0f, vq = lane < np && q == row ? 1.0f : 0.0f;
  constexpr int U = 8;  // rounds read ahead
  float2 w[U];
#pragma unroll
  for (int u = 0; u < U; u++) w[u] = u < R ? log[u * 32 + lane] : make_float2(1.0f, 0.0f);
  for (int r0 = 0; r0 < R; r0 += U) {
    float2 x[U];
#pragma unroll
    for (int u = 0; u < U; u++) x[u] = r0 + U + u < R ? log[(r0 + U + u) * 32 + lane] : make_float2(1.0f, 0.0f);
#pragma unroll
    for (int u = 0; u < U; u++)
      if (r0 + u < R) {
        const float a = w[u].x * vp - w[u].y * vq, b = w[u].y * vp + w[u].x * vq;
        const float dn = __shfl_down_sync(0xffffffffu, a, 1), up = __shfl_up_sync(0xffffffffu, b, 1);
        vp = lane == 0 ? a : lane == np - 1 ? b : dn;
        vq = lane == 0 ? (np > 1 ? dn : b) : up;
      }
#pragma unroll
    for (int u = 0; u < U; u++) w[u] = x[u];
  }
  // after whole sweeps the players are back where they started
  if (lane < np) {
    if (p < M) X[row * M + p] = (double)vp;
    if (q < M) X[row * M + q] = (double)vq;
  }
}

// 4 x 8 block of a product of M x M matrices: sum_k L(i, k) R(k, j); a warp takes an eighth of k for
// all 32 entries, a tree joins them; the results end in out[0 .. 32) (row-major within the block).
// EXACT: error-free products and sums (two-product by FMA, two-sum), so the result is the rounded
// exact sum but for ~2^-100; ten operations a term on the FP64 pipe, hence blocks small enough to
// spread over the GPU (8 x 8 blocks, a quarter of k per thread: 17 us instead of 8).
constexpr int EIG_BI = 4, EIG_BJ = 8;
template <bool EXACT, typename LF, typename RF>
__device__ __forceinline__ void eig_block(int M, LF left, RF right, double* out) {
  constexpr int NE = EIG_BI * EIG_BJ, NS = SVQB_THREADS / NE, LS = SVQB_MAX_M + 1, RS = EIG_BJ + 1;
  __shared__ double ls[EIG_BI * LS], rs[SVQB_MAX_M * RS], hi[NS][NE], lo[NS][NE];
  const int tid = threadIdx.x, o = tid % NE, w = tid / NE;
  for (int e = tid; e < EIG_BI * M; e += SVQB_THREADS) ls[(e % EIG_BI) * LS + e / EIG_BI] = left(e % EIG_BI, e / EIG_BI);
  for (int e = tid; e < EIG_BJ * M; e += SVQB_THREADS) rs[(e / EIG_BJ) * RS + e % EIG_BJ] = right(e / EIG_BJ, e % EIG_BJ);
  __syncthreads();
  const double *l = ls + (o / EIG_BJ) * LS, *r = rs + o % EIG_BJ;
  dd s = {0.0, 0.0};
  for (int k = w; k < M; k += NS) {
    const double a = l[k], b = r[k * RS];
    if constexpr (EXACT) {
      const double q = __dmul_rn(a, b), e = __fma_rn(a, b, -q);
      const dd t = dd_gen2sum(s.s, q);
      s = {t.s, __dadd_rn(s.t, __dadd_rn(t.t, e))};
    } else {
      s.s = fma(a, b, s.s);
    }
  }
  if constexpr (EXACT) s = dd_fast2sum(s.s, s.t);
  for (int h = NS / 2; h >= 1; h /= 2) {
    if (w >= h && w < 2 * h) {
      hi[w][o] = s.s;
      lo[w][o] = s.t;
    }
    __syncthreads();
    if (w < h) {
      if constexpr (EXACT)
        s = dd_accu(s, {hi[w + h][o], lo[w + h][o]});
      else
        s.s += hi[w + h][o];
    }
  }
  if (w == 0) out[o] = EXACT ? __dadd_rn(s.s, s.t) : s.s;
  __syncthreads();
}

// P <- A X
template <bool EXACT>
__global__ void __launch_bounds__(SVQB_THREADS) eig_ax_kernel(const double* __restrict__ A, const double* __restrict__ X,
                                                              int M, double* __restrict__ P) {
  __shared__ double out[EIG_BI * EIG_BJ];
  const int i0 = blockIdx.y * EIG_BI, j0 = blockIdx.x * EIG_BJ;
  eig_block<EXACT>(
      M, [&](int i, int k) { return i0 + i < M ? A[(i0 + i) * M + k] : 0.0; },
      [&](int k, int j) { return j0 + j < M ? X[k * M + j0 + j] : 0.0; }, out);
  const int i = i0 + threadIdx.x / EIG_BJ, j = j0 + threadIdx.x % EIG_BJ;
  if (threadIdx.x < EIG_BI * EIG_BJ && i < M && j < M) P[i * M + j] = out[threadIdx.x];
}

// S <- X^T P (z = 0) and G <- X^T X (z = 1): blocks on and above the diagonal, mirrored, so both are
// symmetric to the bit.
template <bool EXACT>
__global__ void __launch_bounds__(SVQB_THREADS) eig_xtp_kernel(const double* __restrict__ X, const double* __restrict__ P,
                                                               int M, double* __restrict__ S, double* __restrict__ G) {
  __shared__ double out[EIG_BI * EIG_BJ];
  const int i0 = blockIdx.y * EIG_BI, j0 = blockIdx.x * EIG_BJ;
  if (i0 >= j0 + EIG_BJ) return;  // wholly below the diagonal
  const double* R = blockIdx.z == 0 ? P : X;
  double* D = blockIdx.z == 0 ? S : G;
  if (!D) return;
  eig_block<EXACT>(
      M, [&](int i, int k) { return i0 + i < M ? X[k * M + i0 + i] : 0.0; },
      [&](int k, int j) { return j0 + j < M ? R[k * M + j0 + j] : 0.0; }, out);
  const int i = i0 + threadIdx.x / EIG_BJ, j = j0 + threadIdx.x % EIG_BJ;
  if (threadIdx.x < EIG_BI * EIG_BJ && i < M && j < M && i <= j) {
    D[i * M + j] = out[threadIdx.x];
    D[j * M + i] = out[threadIdx.x];
  }
}

// X' <- X (I + E).  refine: the first-order correction of approximate eigenvectors X of A, with
// S = X^T A X, G = X^T X and l_j = S_jj / G_jj: E_ij = (S_ij - l_j G_ij) / (l_j - l_i) where that is
// small (it also takes the non-orthogonality out), half the non-orthogonality elsewhere (pairs
// closer than their coupling are left to the Jacobi sweeps) -- T. Ogita, K. Aishima, "Iterative
// refinement for symmetric eigenvalue decomposition", Japan J. Indust. Appl. Math. 35 (2018), with a
// pairwise instead of a global threshold.  Without refine: E = (I - G) / 2, a Newton step towards
// orthonormal columns.
__global__ void __launch_bounds__(SVQB_THREADS) eig_update_kernel(const double* __restrict__ X, const double* __restrict__ S,
                                                                  const double* __restrict__ G, int M, int refine,
                                                                  double* __restrict__ Y) {
  __shared__ double out[EIG_BI * EIG_BJ], lam[SVQB_MAX_M];
  const int i0 = blockIdx.y * EIG_BI, j0 = blockIdx.x * EIG_BJ;
  if (refine && threadIdx.x < M) lam[threadIdx.x] = S[threadIdx.x * (M + 1)] * (2.0 - G[threadIdx.x * (M + 1)]);
  __syncthreads();
  eig_block<false>(
      M, [&](int i, int k) { return i0 + i < M ? X[(i0 + i) * M + k] : 0.0; },
      [&](int k, int j) {
        j += j0;
        if (j >= M) return 0.0;
        const double g = G[k * M + j];
        if (k == j) return 0.5 * (1.0 - g);
        if (refine) {
          const double s = S[k * M + j], gap = lam[j] - lam[k];
          const double num = s - lam[j] * g, lim = EIG_SMALL * fabs(gap);
          if (fabs(num) <= lim && fabs(s - lam[k] * g) <= lim && fabs(gap) > EIG_GAP) return num * (double)(1.0f / (float)gap);
        }
        return -0.5 * g;
      },
      out);
  const int i = i0 + threadIdx.x / EIG_BJ, j = j0 + threadIdx.x % EIG_BJ;
  if (threadIdx.x < EIG_BI * EIG_BJ && i < M && j < M) Y[i * M + j] = X[i * M + j] + out[threadIdx.x];
}

// Last stage: FP64 Jacobi on A (M x M; scaled here by D from S when `scale`), starting from the
// eigenvector approximation X (I when null), until the off-diagonal mass is at the rounding level
// ((M u)^2 of the whole; after the refinement usually no sweep is left), then T (B layout of TSMM)
// and the sweep count.
__global__ void __launch_bounds__(EIG_THREADS) svqb_eig_kernel(const double* __restrict__ A, const double* __restrict__ X,
                                                               const double* __restrict__ dg, int M, int scale,
                                                               double* __restrict__ T, int* info, int max_sweeps) {
  extern __shared__ __align__(16) double sh[];
  __shared__ double d[SVQB_MAX_M];
  __shared__ int order[SVQB_MAX_M];
  double* V = sh + 2 * EIG_SIZE;
  double* cs = V + SVQB_MAX_M * EIG_LD;
  const int tid = threadIdx.x, n = (M + 1) & ~1;
  constexpr int LD = EIG_LD;
  for (int i = tid; i < M; i += EIG_THREADS) {
    if (scale) {
      const double sii = A[i * M + i];
      d[i] = fabs(sii) > 1.0e-15 ? 1.0 / sqrt(sii) : 0.0;
    } else {
      d[i] = dg[i];
    }
  }
  __syncthreads();
  for (int e = tid; e < n * n; e += EIG_THREADS) {
    const int i = e / n, j = e - i * n;
    const bool in = i < M && j < M;
    const int sj = slot_of(j, n);
    sh[slot_of(i, n) * LD + sj] = !in ? 0.0 : scale ? A[i * M + j] * d[i] * d[j] : A[i * M + j];
    V[i * LD + sj] = !in ? 0.0 : X ? X[i * M + j] : (i == j ? 1.0 : 0.0);
  }
  __syncthreads();
  int cur = 0;
  const int sweeps = jacobi_sweeps<double>(sh, cur, V, cs, cs + 66, M, n, (double)M * M * 1.23e-32, max_sweeps, nullptr);

  const double* A0 = sh + cur;

  // ascending eigenvalues: rank of each diagonal entry (ties broken by index; NaN ranks as infinity, so
  // that the ranks are a permutation whatever the block holds)
  auto eigenvalue = [&](int i) { return fmin(A0[slot_of(i, n) * (LD + 1)], HUGE_VAL); };
  bool nan = false;
  for (int i = tid / 8; i < (M + 3) / 4 * 4; i += EIG_THREADS / 8) {  // whole warps, 8 lanes per entry
    const double li = i < M ? eigenvalue(i) : 0.0;
    nan |= i < M && isnan(A0[slot_of(i, n) * (LD + 1)]);
    int rank = 0;
    for (int j = tid % 8; j < M; j += 8) {
      const double lj = eigenvalue(j);
      rank += (lj < li) || (lj == li && j < i);
    }
#pragma unroll
    for (int o = 4; o >= 1; o >>= 1) rank += __shfl_xor_sync(0xffffffffu, rank, o);
    if (i < M && tid % 8 == 0) order[rank] = i;
  }
  // NaN or infinity in the block (and so on the Gram's diagonal): T is NaN throughout, as rotations by
  // NaN would make it; M == 1 has none
  nan = __syncthreads_or(nan && M > 1);
  // T[col*M + m] = V[m][src] * d[m] / sqrt(max(1e-15, l_src)), sign: largest |V[.][src]| positive
  // (8 lanes per column; equal magnitudes: the first)
  for (int col = tid / 8; col < (M + 3) / 4 * 4; col += EIG_THREADS / 8) {  // whole warps
    const int src = slot_of(order[min(col, M - 1)], n), sub = tid % 8;
    double big = -1.0, sg = 1.0;
    int at = SVQB_MAX_M;
    for (int m = sub; m < M; m += 8) {
      const double v = V[m * LD + src];
      if (fabs(v) > big) {
        big = fabs(v);
        sg = v < 0.0 ? -1.0 : 1.0;
        at = m;
      }
    }
#pragma unroll
    for (int o = 4; o >= 1; o >>= 1) {
      const double b2 = __shfl_xor_sync(0xffffffffu, big, o), s2 = __shfl_xor_sync(0xffffffffu, sg, o);
      const int a2 = __shfl_xor_sync(0xffffffffu, at, o);
      if (b2 > big || (b2 == big && a2 < at)) {
        big = b2;
        sg = s2;
        at = a2;
      }
    }
    const double f = nan ? HUGE_VAL - HUGE_VAL : sg / sqrt(fmax(1.0e-15, A0[src * LD + src]));
    if (col < M)
      for (int m = sub; m < M; m += 8) T[col * M + m] = V[m * LD + src] * d[m] * f;
  }
  if (tid == 0 && info) *info = sweeps;
}

// ||S - I||_F for an M x M matrix
__global__ void __launch_bounds__(SVQB_THREADS) svqb_orth_kernel(const double* __restrict__ S, int M, double* out) {
  __shared__ double red[SVQB_THREADS];
  double acc = 0.0;
  for (int e = threadIdx.x; e < M * M; e += SVQB_THREADS) {
    const int i = e / M, j = e % M;
    const double v = (i == j ? 1.0 : 0.0) - S[e];
    acc += v * v;
  }
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int s = SVQB_THREADS / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = sqrt(red[0]);
}

// Cholesky S = R^T R (R upper, positive diagonal) of the Gram matrix and T = R^-1 in TSMM's B
// layout (B[n*M + m] = Rinv[m][n]), so that X <- X T gives Q = X R^-1.  *info = 0, or j + 1 when
// the pivot of column j is not positive (the Gram is not numerically positive definite).
__global__ void __launch_bounds__(SVQB_THREADS) cholqr_kernel(const double* __restrict__ S, int M,
                                                              double* __restrict__ T, int* info) {
  extern __shared__ __align__(16) double sh[];
  const int LD = M + 1;
  double* A = sh;         // M x LD: the trailing matrix, then R in the upper triangle
  double* Y = A + M * LD;  // M x LD: R^-1
  __shared__ int bad;
  const int tid = threadIdx.x;
  for (int e = tid; e < M * M; e += SVQB_THREADS) A[(e / M) * LD + e % M] = S[e];
  if (tid == 0) bad = 0;
  __syncthreads();
  for (int j = 0; j < M; j++) {
    const double piv = A[j * LD + j];
    if (!(piv > 0.0)) {  // uniform: every thread reads the same pivot
      if (tid == 0) bad = j + 1;
      break;
    }
    const double r = sqrt(piv);
    __syncthreads();
    for (int i = j + 1 + tid; i < M; i += SVQB_THREADS) A[j * LD + i] /= r;  // row j of R
    if (tid == 0) A[j * LD + j] = r;
    __syncthreads();
    // trailing update A[i][l] -= R[j][i] R[j][l] for j < i <= l
    const int w = M - j - 1;
    for (int e = tid; e < w * w; e += SVQB_THREADS) {
      const int i = j + 1 + e / w, l = j + 1 + e % w;
      if (l >= i) A[i * LD + l] -= A[j * LD + i] * A[j * LD + l];
    }
    __syncthreads();
  }
  __syncthreads();
  if (bad) {
    if (tid == 0) *info = bad;
    return;
  }
  // R^-1 column by column (back substitution), one thread per column
  for (int c = tid; c < M; c += SVQB_THREADS) {
    for (int i = M - 1; i >= 0; i--) {
      double v = (i == c) ? 1.0 : 0.0;
      for (int k = i + 1; k <= c; k++) v -= A[i * LD + k] * Y[k * LD + c];
      Y[i * LD + c] = i > c ? 0.0 : v / A[i * LD + i];
    }
  }
  __syncthreads();
  for (int e = tid; e < M * M; e += SVQB_THREADS) {
    const int n = e / M, m = e % M;
    T[e] = Y[m * LD + n];
  }
  if (tid == 0) *info = 0;
}

// Scratch of SVQB and CholQR on a stream: S, T, S2, A, X, Y, P, R, G (M x M each), d, the error word
// and counts (8 doubles), the log of FP32 rotations
static skinny_status svqb_scratch(skinny_handle h, cudaStream_t st, double*& out) {
  void*& buf = h->svqb_ws[st];
  if (!buf) {
    if (cudaMalloc(&buf, (9 * (size_t)SVQB_MAX_M * SVQB_MAX_M + SVQB_MAX_M + 8 + EIG_LOG) * sizeof(double)) != cudaSuccess) {
      cudaGetLastError();
      buf = nullptr;
      set_error("svqb / cholqr: cudaMalloc failed");
      return SKINNY_NO_MEM;
    }
    h->extra_allocs.push_back(buf);
  }
  out = static_cast<double*>(buf);
  return SKINNY_OK;
}

// T from the Gram matrix S: eigenvectors to FP32 accuracy, two steps of refinement and two Newton
// steps towards orthonormality in FP64 (products of M x M matrices, spread over the GPU), then FP64
// Jacobi sweeps for what is left.  The matrix the sweeps start from, X^T A X, is formed with exact
// products and sums: rounding it would move the smallest eigenvalues by u times the largest.  M = 64 with a
// well-conditioned block: 5.4 ms -> 0.28 ms (157 us of it the FP32 Jacobi, 29 the last kernel); condition 1e8,
// where FP64 sweeps are left: 11.4 -> 4.8 ms.  ||Q^T Q - I|| falls with it (M = 64: 4.9e-14 -> 1.5e-14; condition
// 100: 2e-12 -> 5e-13).
static skinny_status svqb_transform(const double* S, int M, double* T, double* ws, double* d, int* info,
                                    cudaStream_t st) {
  static SmemAttr attr32, attr64;
  if (!ensure_smem_attr(svqb_jacobi32_kernel, (int)eig_smem<float>(), attr32) ||
      !ensure_smem_attr(svqb_eig_kernel, (int)eig_smem<double>(), attr64))
    return SKINNY_DEVICE_ERROR;
  const size_t MM = (size_t)SVQB_MAX_M * SVQB_MAX_M;
  double *A = ws, *X = A + MM, *Y = X + MM, *P = Y + MM, *R = P + MM, *G = R + MM;
  if (M >= EIG_MIXED_MIN) {
    const dim3 one((M + EIG_BJ - 1) / EIG_BJ, (M + EIG_BI - 1) / EIG_BI, 1), two(one.x, one.y, 2);
    float2* log = reinterpret_cast<float2*>(d + SVQB_MAX_M + 8);
    svqb_jacobi32_kernel<<<1, EIG_THREADS, eig_smem<float>(), st>>>(S, M, d, A, log, info);
    eig_replay_kernel<<<(M * 32 + REPLAY_THREADS - 1) / REPLAY_THREADS, REPLAY_THREADS, 0, st>>>(log, info, M, X);
    count_launch();
    count_launch();
    for (int it = 0; it < 4; it++) {
      const int refine = it < 2;
      if (refine) {
        eig_ax_kernel<false><<<one, SVQB_THREADS, 0, st>>>(A, X, M, P);
        count_launch();
      }
      eig_xtp_kernel<false><<<two, SVQB_THREADS, 0, st>>>(X, P, M, refine ? R : nullptr, G);
      eig_update_kernel<<<one, SVQB_THREADS, 0, st>>>(X, R, G, M, refine, Y);
      count_launch();
      count_launch();
      double* t = X;
      X = Y;
      Y = t;
    }
    eig_ax_kernel<true><<<one, SVQB_THREADS, 0, st>>>(A, X, M, P);
    eig_xtp_kernel<true><<<one, SVQB_THREADS, 0, st>>>(X, P, M, R, nullptr);
    count_launch();
    count_launch();
    svqb_eig_kernel<<<1, EIG_THREADS, eig_smem<double>(), st>>>(R, X, d, M, 0, T, info, 30);
  } else {
    svqb_eig_kernel<<<1, EIG_THREADS, eig_smem<double>(), st>>>(S, nullptr, nullptr, M, 1, T, info, 30);
  }
  count_launch();
  if (cudaGetLastError() != cudaSuccess) {
    set_error("svqb: eigensolver launch failed");
    return SKINNY_DEVICE_ERROR;
  }
  return SKINNY_OK;
}

}  // namespace skinny

using namespace skinny;

extern "C" skinny_status skinny_svqb(skinny_handle h, skinny_acc gram_acc, int64_t K, int64_t M,
                                     double* X, int64_t ldx, double* orth_err_out, void* stream) {
  set_error("");
  if (!h) {
    set_error("null handle");
    return SKINNY_BAD_ARG;
  }
  if (M < 1 || K < 0 || ldx < M || (K > 0 && !X)) {
    set_error("svqb: bad sizes or null X");
    return SKINNY_BAD_ARG;
  }
  if (M > SVQB_MAX_M) {
    set_error("svqb: M > 64 not provided");
    return SKINNY_UNSUPPORTED;
  }
  DevGuard g(h->dev.id);
  cudaStream_t st = (cudaStream_t)stream;
  std::lock_guard<std::mutex> lk(h->mu);
  double* S = nullptr;
  skinny_status s = svqb_scratch(h, st, S);
  if (s != SKINNY_OK) return s;
  double* T = S + SVQB_MAX_M * SVQB_MAX_M;
  double* S2 = T + SVQB_MAX_M * SVQB_MAX_M;
  double* ws = S2 + SVQB_MAX_M * SVQB_MAX_M;
  double* d = ws + 6 * SVQB_MAX_M * SVQB_MAX_M;
  double* errd = d + SVQB_MAX_M;
  int* info = reinterpret_cast<int*>(errd + 1);
  const double one = 1.0, zero = 0.0;
  LaunchOpts o{};
  s = dispatch_product(h, false, SKINNY_R64, gram_acc, M, M, K, X, ldx, &one, X, ldx,
                                     &zero, S, M, st, o);
  if (s == SKINNY_UNSUPPORTED && gram_acc == SKINNY_ACC_SPLIT)  // split not provided at this M
    s = dispatch_product(h, false, SKINNY_R64, SKINNY_ACC_NATIVE, M, M, K, X, ldx, &one, X, ldx, &zero, S,
                         M, st, o);
  if (s != SKINNY_OK) return s;
  s = svqb_transform(S, (int)M, T, ws, d, info, st);
  if (s != SKINNY_OK) return s;
  s = dispatch_product(h, true, SKINNY_R64, SKINNY_ACC_AUTO, M, M, K, X, ldx, &one, T, M, &zero, X,
                       ldx, st, o);
  if (s != SKINNY_OK) return s;
  if (orth_err_out) {
    s = dispatch_product(h, false, SKINNY_R64, SKINNY_ACC_DD, M, M, K, X, ldx, &one, X, ldx, &zero, S2,
                         M, st, o);
    if (s != SKINNY_OK) return s;
    svqb_orth_kernel<<<1, SVQB_THREADS, 0, st>>>(S2, (int)M, errd);
    count_launch();
    double v = -1.0;
    if (cudaMemcpyAsync(&v, errd, sizeof(double), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess) {
      cudaGetLastError();
      set_error("svqb: reading the orthogonality error failed");
      return SKINNY_DEVICE_ERROR;
    }
    *orth_err_out = v;
  }
  return SKINNY_OK;
}

// CholQR (passes = 1) / CholQR2 (passes = 2): Gram, Cholesky and in-place TSMM with R^-1 per pass.
// No counterpart in the reference (whose orthogonalisation is SVQB, svqb/svqb.cu:72-130); it
// reuses the same Gram and in-place TSMM.  SKINNY_BAD_ARG when a Gram is not numerically positive
// definite (X is then left as the previous pass made it).
extern "C" skinny_status skinny_cholqr(skinny_handle h, skinny_acc gram_acc, int64_t K, int64_t M, double* X,
                                       int64_t ldx, int passes, double* orth_err_out, void* stream) {
  set_error("");
  if (!h) {
    set_error("null handle");
    return SKINNY_BAD_ARG;
  }
  if (M < 1 || K < 0 || ldx < M || (K > 0 && !X) || passes < 1 || passes > 4) {
    set_error("cholqr: bad sizes, null X or passes outside 1..4");
    return SKINNY_BAD_ARG;
  }
  if (M > SVQB_MAX_M) {
    set_error("cholqr: M > 64 not provided");
    return SKINNY_UNSUPPORTED;
  }
  DevGuard g(h->dev.id);
  cudaStream_t st = (cudaStream_t)stream;
  std::lock_guard<std::mutex> lk(h->mu);
  double* S = nullptr;
  if (skinny_status e = svqb_scratch(h, st, S); e != SKINNY_OK) return e;
  double* T = S + SVQB_MAX_M * SVQB_MAX_M;
  double* S2 = T + SVQB_MAX_M * SVQB_MAX_M;
  double* errd = S2 + SVQB_MAX_M * SVQB_MAX_M;
  int* info = reinterpret_cast<int*>(errd + 1);
  const double one = 1.0, zero = 0.0;
  LaunchOpts o{};
  const size_t smem = (size_t)2 * M * (M + 1) * sizeof(double);
  static SmemAttr attr;
  ensure_smem_attr(cholqr_kernel, (int)smem, attr);
  for (int pass = 0; pass < passes; pass++) {
    skinny_status s = dispatch_product(h, false, SKINNY_R64, gram_acc, M, M, K, X, ldx, &one, X, ldx, &zero, S, M,
                                       st, o);
    if (s == SKINNY_UNSUPPORTED && gram_acc == SKINNY_ACC_SPLIT)
      s = dispatch_product(h, false, SKINNY_R64, SKINNY_ACC_NATIVE, M, M, K, X, ldx, &one, X, ldx, &zero, S, M, st, o);
    if (s != SKINNY_OK) return s;
    cholqr_kernel<<<1, SVQB_THREADS, smem, st>>>(S, (int)M, T, info);
    count_launch();
    int hinfo = 0;
    if (cudaGetLastError() != cudaSuccess ||
        cudaMemcpyAsync(&hinfo, info, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess) {
      cudaGetLastError();
      set_error("cholqr: Cholesky launch failed");
      return SKINNY_DEVICE_ERROR;
    }
    if (hinfo != 0) {
      set_error("cholqr: Gram matrix not positive definite at column " + std::to_string(hinfo - 1));
      return SKINNY_BAD_ARG;
    }
    s = dispatch_product(h, true, SKINNY_R64, SKINNY_ACC_AUTO, M, M, K, X, ldx, &one, T, M, &zero, X, ldx, st, o);
    if (s != SKINNY_OK) return s;
  }
  if (orth_err_out) {
    skinny_status s = dispatch_product(h, false, SKINNY_R64, SKINNY_ACC_DD, M, M, K, X, ldx, &one, X, ldx, &zero,
                                       S2, M, st, o);
    if (s != SKINNY_OK) return s;
    svqb_orth_kernel<<<1, SVQB_THREADS, 0, st>>>(S2, (int)M, errd);
    count_launch();
    double v = -1.0;
    if (cudaMemcpyAsync(&v, errd, sizeof(double), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess) {
      cudaGetLastError();
      set_error("cholqr: reading the orthogonality error failed");
      return SKINNY_DEVICE_ERROR;
    }
    *orth_err_out = v;
  }
  return SKINNY_OK;
}
