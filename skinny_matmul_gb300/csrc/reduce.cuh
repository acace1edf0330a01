// reduce.cuh -- deterministic reductions shared by the CUDA-core TSMTTSM kernels.
//
// What bounds them: GB300's FP64 pipe does 1.89 additions per clock and SM, so for FP64, complex
// FP64 and double-double sums the additions themselves are the cost, not the shuffles or loads.
// A butterfly over 32 lanes of a 64-entry register tile is 320 additions per thread (~23 us for a
// CTA of 256 threads); 152 CTA partials of a 16 x 16 double-double product summed by one CTA took
// ~200 us.  So the warp reduction halves the entries a lane keeps at every stage (63 additions for
// the same tile, and the same sums in the same order), slot sums are trees over all threads, and
// many or long partials are summed on two levels, the first spread over the GPU.
#pragma once
#include <type_traits>

#include "common.cuh"

namespace skinny {

// Sums acc over the lanes that differ in the bits >= `low` of the lane index (low a power of two,
// <= 32): at each stage a lane keeps one half of its entries and hands the other half to its
// partner, until one entry is left, which is then exchanged as it is.  On return acc[0 .. n)
// holds entries base .. base + n - 1 (n = max(1, W / (32 / low))); `owner` is false in the lanes
// that hold a copy of another lane's entry.  The sums are those of a butterfly, bit for bit.
template <typename O, typename Acc, int W, int BIT = 16>
__device__ __forceinline__ void warp_halve(Acc* acc, int low, int lane, int& base, int& n, bool& owner) {
  if constexpr (BIT >= 1) {
    if (BIT < low) return;
    const bool up = (lane & BIT) != 0;
    if constexpr (W >= 2) {
      constexpr int H = W / 2;
#pragma unroll
      for (int i = 0; i < H; i++) {
        const Acc lo = acc[i], hi = acc[i + H];
        const Acc keep = up ? hi : lo, send = up ? lo : hi;
        acc[i] = O::add(keep, O::shfl_xor(send, BIT));
      }
      base += up ? H : 0;
      n = H;
      warp_halve<O, Acc, H, BIT / 2>(acc, low, lane, base, n, owner);
    } else {
      acc[0] = O::add(acc[0], O::shfl_xor(acc[0], BIT));
      owner = owner && !up;
      warp_halve<O, Acc, 1, BIT / 2>(acc, low, lane, base, n, owner);
    }
  }
}

// sm[0 .. E) <- sum over n slots of E entries each (slot s at sm + s * E); all NT threads of the
// block call it, after a barrier behind the writes; ends with a barrier.
template <typename O, typename Acc, int NT>
__device__ __forceinline__ void slot_tree(Acc* sm, int n, int E) {
  while (n > 1) {
    const int half = (n + 1) / 2;
    for (int i = threadIdx.x; i < (n - half) * E; i += NT) sm[i] = O::add(sm[i], sm[i + half * E]);
    __syncthreads();
    n = half;
  }
}

// out(e, sum over cnt partials of E entries each, partial b at src + b * E).  The partials were
// written by other CTAs (L2-coherent loads).  Few entries: the threads share the range of partials
// and a tree joins them (sm: NT entries).  Many: 16 bytes of entries per thread and step, eight
// partials in flight (a 64 x 64 FP32 sum of 12 partials: 3 us; with four single loads, 12 us).  Few partials of 4096 or
// more FP64 entries are better summed one entry a thread, four partials in flight (128 x 128, 4 partials: 144 us
// the call, 126; FP32 100 x 100 in FP64, 12 on each level: 284 and 266; but 152 of them 1004 and 1112; complex FP32 64 x 64
// with 12 on each level 101 and 129).
template <typename O, typename Acc, int NT, typename Out>
__device__ __forceinline__ void sum_partials(const Acc* src, int cnt, int E, Acc* sm, Out out) {
  const int tid = threadIdx.x;
  constexpr int V = sizeof(Acc) < 16 ? 16 / (int)sizeof(Acc) : 1;
  if constexpr (V > 1) {
    if (E >= NT && E % V == 0 && (!std::is_same<Acc, double>::value || E < 4096 || cnt > 32)) {
      union Pack {
        uint4 w;
        Acc v[V];
        __device__ Pack() {}
      };
      for (int e = tid * V; e < E; e += NT * V) {
        Acc s[V];
#pragma unroll
        for (int k = 0; k < V; k++) s[k] = O::zero();
        for (int b = 0; b < cnt; b += 8) {
          Pack q[8];
#pragma unroll
          for (int u = 0; u < 8; u++)
            if (b + u < cnt) q[u].w = __ldcg(reinterpret_cast<const uint4*>(src + (size_t)(b + u) * E + e));
#pragma unroll
          for (int u = 0; u < 8; u++)
            if (b + u < cnt) {
#pragma unroll
              for (int k = 0; k < V; k++) s[k] = O::add(s[k], q[u].v[k]);
            }
        }
#pragma unroll
        for (int k = 0; k < V; k++) out(e + k, s[k]);
      }
      return;
    }
  }
  auto run = [&](int e, int b, int step) {
    Acc s = O::zero();
    for (; b < cnt; b += 4 * step) {
      Acc v[4];
#pragma unroll
      for (int u = 0; u < 4; u++)
        if (b + u * step < cnt) v[u] = ldcg(&src[(size_t)(b + u * step) * E + e]);
#pragma unroll
      for (int u = 0; u < 4; u++)
        if (b + u * step < cnt) s = O::add(s, v[u]);
    }
    return s;
  };
  if (2 * E > NT) {
    for (int e = tid; e < E; e += NT) out(e, run(e, 0, 1));
    return;
  }
  const int P = min(cnt, NT / E);
  const int e = tid % E, j = tid / E;
  if (j < P) sm[tid] = run(e, j, P);
  __syncthreads();
  slot_tree<O, Acc, NT>(sm, P, E);
  if (tid < E) out(tid, sm[tid]);
}

// Groups of the first level for nb CTA partials of E entries of Acc; 0: one level.  A second level
// costs a ticket and a round trip through L2 (~2 us).  One CTA summing everything needs nb * E /
// 1024 rounds of loads (~0.35 us each: a 16 x 16 FP32 sum of 147 partials took 13 us) and nb * E
// additions at 1.89 per clock on the FP64 pipe (double-double: 20 operations each); the lines lie
// where that passes about 2 us.
constexpr int FINISH_MAX_GROUPS = 32;
template <typename Acc>
__host__ __device__ inline int finish_groups(int nb, int E) {
  const int64_t line = std::is_same<Acc, dd>::value || std::is_same<Acc, zdd>::value ? 512 : sizeof(Acc) > 8 ? 4096 : 8192;
  if (nb < 8 || (int64_t)nb * E <= line) return 0;
  int g = 4;
  while (g * g < nb && g < FINISH_MAX_GROUPS) g++;
  return g;
}
// Accumulators a launch of nb CTAs needs in the workspace (CTA partials, then group sums)
template <typename Acc>
__host__ __device__ inline int64_t finish_entries(int nb, int E) {
  return ((int64_t)nb + finish_groups<Acc>(nb, E)) * E;
}

// Cross-CTA sum in one launch: called by every thread of a CTA that has written its partial to
// part[blockIdx.x * E ..].  The last CTA to take the ticket (of its group, then of the groups) sums;
// nobody waits.  The order of the sums is fixed, so the result is deterministic; tickets
// (counter[0], counter[1 ..]) are back at 0 for the next launch.  sm: NT accumulators, s_flag: one
// shared int.
template <typename O, typename Acc, int NT, typename Out>
__device__ __forceinline__ void finish_partials(Acc* part, unsigned* counter, int E, bool two_levels, Acc* sm,
                                                int* s_flag, Out out) {
  const int tid = threadIdx.x, nb = gridDim.x;
  const int ng = two_levels ? finish_groups<Acc>(nb, E) : 0;
  if (nb == 1) {
    __syncthreads();
    for (int e = tid; e < E; e += NT) out(e, part[e]);
    return;
  }
  const int g = ng ? (int)((int64_t)blockIdx.x * ng / nb) : 0;
  const int b0 = ng ? (g * nb + ng - 1) / ng : 0, b1 = ng ? ((g + 1) * nb + ng - 1) / ng : nb;
  __threadfence();
  __syncthreads();
  if (tid == 0) *s_flag = atomicAdd(counter + (ng ? 1 + g : 0), 1u) == (unsigned)(b1 - b0 - 1);
  __syncthreads();
  if (!*s_flag) return;
  __threadfence();
  if (ng) {
    Acc* sums = part + (size_t)nb * E;
    sum_partials<O, Acc, NT>(part + (size_t)b0 * E, b1 - b0, E, sm, [&](int e, Acc v) { sums[(size_t)g * E + e] = v; });
    __threadfence();
    __syncthreads();
    if (tid == 0) {
      counter[1 + g] = 0u;
      *s_flag = atomicAdd(counter, 1u) == (unsigned)(ng - 1);
    }
    __syncthreads();
    if (!*s_flag) return;
    __threadfence();
    sum_partials<O, Acc, NT>(sums, ng, E, sm, out);
  } else {
    sum_partials<O, Acc, NT>(part, nb, E, sm, out);
  }
  if (tid == 0) counter[0] = 0u;
}

}  // namespace skinny
