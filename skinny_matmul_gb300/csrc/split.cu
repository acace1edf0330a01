// split.cu -- FP64 TSMTTSM in split precision on tcgen05 tensor cores for M, N <= 16 (no
// counterpart in the reference, whose FP64 kernels are CUDA-core DFMA loops, e.g.
// tsmttsm/genv5.cuh:28-89).  Wider products go to split_wide.cu.
//
// Why: GB300 executes 595 G FP64 FMA/s but 2.25 P FP16 / BF16 tensor flop/s.  A CUDA-core FP64
// TSMTTSM is FP64-bound for every M = N >= 2.  Here each FP64 product is computed exactly from
// 8-bit pieces on the tensor cores, and FP64 arithmetic is used only a few times per 1024 rows.
//
// Scheme (Ozaki-style error-free splitting, written for this kernel):
//   * Per column m of A (and n of B) a shared exponent E holds for an epoch: each element x is a
//     62-bit fixed-point integer F = |x| * 2^(1084 - E) written as 8 balanced base-256 digits
//     d_1..d_8 (d_1 most significant): x = sign * sum_i d_i 2^(8(8-i)) 2^(E-1084).  Digits are
//     exact in FP16 (byte permutes, digits.cuh).  When a round of rows holds an element above
//     2^E's range, that column's E is raised with HEAD bits of headroom and a new period starts.
//   * Digit planes are stacked along the MMA dimensions: A rows (i-1)*MP + m, B rows
//     (j-1)*NP + n, so one tcgen05.mma (M = 128, N = 8*NP, K = 16, FP16 x FP16 -> FP32 in TMEM)
//     forms every digit-pair product d_i(a) d_j(b) for 16 rows of K.
//   * |d_i d_j| <= 2^14, so over a period of <= 1024 rows every partial sum is an integer of
//     magnitude <= 2^24: the FP32 accumulation in TMEM is exact.  Two accumulator sets alternate
//     between periods, so the drain of one period runs while the MMAs of the next proceed.
//   * Drain: TMEM -> int32, added per digit pair (i, j) in registers over up to 15 periods of the same
//     exponents (8 * 15 * 2^24 < 2^31); then a few columns of C at a time pass through shared memory
//     and one thread forms the level sums S_L = sum_{i+j=L} D_ij (L = 2..9) of a cell;
//     V = sum_L S_L 2^(8(16-L)) is assembled from two int64 words and added to an FP64
//     accumulator per C entry with weight 2^(EA+EB-2168).  Levels L >= 10 are dropped: their
//     weight is below 2^-56 of the leading level (2^-52 with the headroom).
//   * Warp roles, hand-offs through mbarriers (no CTA-wide barrier while streaming):
//       warps 0-15 slicers: per round of rr rows (rr * (M + N) / 8 units of one column and 8 rows,
//                  at most one per thread) read the FP64 values from the stage ring (or from
//                  global memory where rows are not 16-byte aligned), check them against the
//                  column exponents (one named barrier per round; two more only when a period
//                  starts), slice them into a digit stage;
//       warps 16-19 drain: one TMEM lane quadrant each;
//       warp 20    producer: whole rounds of rows by 1-D TMA bulk copies into the FP64 ring;
//       warp 21    MMA issuer: rr/16 MMAs per round into the period's accumulator set.
//     Bound: at 8 x 8 a round of 256 rows takes ~3500 clocks.  Of these the ALU pipe needs ~1100 for
//     the digits, the tensor pipe 640 and shared memory 1800, but the phases of a round (read, vote on
//     the exponents, slice) follow one another in all warps at once.  With 8 slicer warps of two units
//     a thread it was ~5400, and the drain sorted every period by level with shuffles and atomics
//     (8000 clocks a period, of which the last one's was not hidden).  Measured f64 8 x 8: K = 2^20
//     90 -> 64 us, K = 2^14 16.7 -> 14.8; 16 x 16, K = 2^20: 166 -> 118; Gram 16: 111 -> 72.
//     The roles that wait most of the time (drain, producer, MMA) sleep between polls, so that
//     their polling leaves issue slots to the slicers.  Every wait is bounded; a wait that runs
//     out sets the error word, every role stops at its next wait, and the CTA writes no C.
//   * Cross-CTA finish in two levels: CTA partials in FP64; the last CTA of each group of 16
//     (ticket) sums its group in CTA order, the last group sums the group sums in group order
//     and applies alpha/beta (deterministic).
//   * Infinities and NaN have no fixed-point form: a column that holds one gets the exponent NONFINITE, whose
//     power of two is NaN, and so are the entries of C that it enters.

#include <cstring>

#include "api_internal.h"
#include "digits.cuh"

namespace skinny {

namespace split {

constexpr int PERIOD = 1024;   // rows accumulated exactly in TMEM (|sum| <= 1024 * 2^14)
constexpr int MAXSUM = 15;     // periods summed before the levels are (8 pairs * 15 * 2^24 < 2^31)
constexpr int DIGITS = 8;
constexpr int NSLICE = 16;     // slicer warps 0-15
constexpr int NDRAIN = 4;      // drain warps 16-19 (one TMEM lane quadrant each)
constexpr int WPROD = NSLICE + NDRAIN, WMMA = WPROD + 1;
// six warpgroups (the last one: producer, MMA issuer, two idle warps) launched with 80 registers a
// thread, of which the last group gives back 40 and the slicers 8 for the drain warps' 152
constexpr int THREADS = (WMMA + 3) * 32;
constexpr int SLICERS = NSLICE * 32;
constexpr int HEAD = 2;        // exponent headroom granted when a column's exponent is raised
constexpr int EMAX = 2046;     // largest exponent field of a finite number, and of a column of such
constexpr int NONFINITE = 6000;  // exponent of a column with an infinity or NaN: out of the range of any sum
constexpr int MAXST = 4;       // FP64 stages (at most)
constexpr int MAXDST = 3;      // digit stages (at most)
constexpr int DPAD = 128 * 16; // slack after an A digit buffer: the MMA reads 128 rows per k-octet
constexpr int HDR = 2048;      // barriers, TMEM slot, round and period records, exponents
// columns of B whose digit pairs the drain sorts by level at a time, and the stride of their rows: 4
// where that leaves the stages as they are, else 2 (8 x 8 at 2^14 rows 14.6 us and 16.4)
template <int NCB>
struct SortBuf {
  static constexpr int NC = NCB, STRIDE = NCB == 4 ? 128 + 8 : 128, BYTES = DIGITS * NCB * STRIDE * 4;
};
constexpr int CBYTES = 256 * 8;          // FP64 accumulators of the C entries
constexpr int STATIC_RESERVE = 1024;     // the kernel's static shared memory
constexpr uint32_t SLEEP_DRAIN = 256;    // ns between polls of the drain warps (a period is ~8 rounds)
constexpr uint32_t SLEEP_PRODUCER = 64;  // ns between polls of the producer warp
constexpr uint32_t SLEEP_MMA = 32;       // ns between polls of the MMA thread
constexpr int GROUP = 16;                // CTAs per first-level group of the cross-CTA finish
constexpr int MAXGROUPS = 16;            // groups at most (grid <= 256); counter[MAXGROUPS] is the last level's

struct Args {
  const void* A;  // FP64, or FP32 with in_f32 (widened exactly when read)
  const void* B;
  void* C;        // FP64, or FP32 with out_f32
  int64_t K, lda, ldb, ldc;
  int M, N, MP, NP;  // padded widths (powers of two); NP = MP in Gram mode
  double alpha, beta;
  int beta_zero, gram, bulk;
  int stages, dstages;   // FP64 stages, digit stages
  int rr;                // rows per round (a multiple of 128, <= PERIOD)
  int64_t nrounds;
  uint32_t stage_bytes;  // FP64 stage: rr rows of A (tile_a bytes), then rr rows of B
  uint32_t tile_a;
  int nmma;              // MMA N (multiple of 16, >= 16)
  int tmem_cols;         // two accumulator sets of nmma columns
  uint32_t lbo_a, lbo_b; // bytes between k-octets of the A / B digit buffers
  int sort_bytes;        // SortBuf<2> or <4>
  uint32_t dig_a, dig_b; // bytes of one A / B digit buffer (A includes DPAD)
  double* partials;
  unsigned* counter;
  int* err;
  int out_f32;
};

__device__ __forceinline__ uint64_t make_desc(uint32_t saddr, uint32_t lbo) {
  uint64_t d = (uint64_t)((saddr & 0x3FFFF) >> 4);
  d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;  // K-direction core-matrix stride
  d |= (uint64_t)((128 >> 4) & 0x3FFF) << 32;  // 8-row-group stride
  d |= (uint64_t)1 << 46;                      // descriptor version
  return d;                                    // no swizzle
}

__device__ __forceinline__ void mma_f16(uint32_t tmem, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
      "l"(da), "l"(db), "r"(idesc), "r"(acc));
}
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

template <int X>
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[X]);
template <>
__device__ __forceinline__ void tmem_ld<1>(uint32_t taddr, uint32_t (&r)[1]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(r[0]) : "r"(taddr));
}
template <>
__device__ __forceinline__ void tmem_ld<2>(uint32_t taddr, uint32_t (&r)[2]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0,%1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(taddr));
}
template <>
__device__ __forceinline__ void tmem_ld<4>(uint32_t taddr, uint32_t (&r)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr));
}
template <>
__device__ __forceinline__ void tmem_ld<8>(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// exponent field used for the shared exponent: 0 for zero, 1 for subnormals
__device__ __forceinline__ uint32_t exp_field(double x) {
  uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
  uint32_t ef = (hi >> 20) & 0x7FF;
  bool nz = ((hi & 0x7FFFFFFFu) | lo) != 0;
  return nz ? (ef ? ef : 1u) : 0u;
}

__device__ __forceinline__ double pow2i(int e) {  // 2^e from -1022 to 1023, 2^-1022 below, NaN above (only NONFINITE gets there)
  e = min(max(e, -1022), 1024);
  return __hiloint2double((e + 1023) << 20, e > 1023);
}

// Slice one unit: 8 consecutive rows of column c into the octet `buf` of a digit buffer
// (rows (i-1)*CP + c), relative to exponent E (FAST: E > EMIN_FAST).  FP16 digits formed from the bytes of G with byte
// permutes and one HFMA2 per digit pair (digits.cuh), stored as they are formed.
template <bool FAST>
__device__ __forceinline__ void slice_unit(const double (&v)[8], uint32_t E, int c, int CP, unsigned char* buf) {
  uint32_t gw[2][8];
  SignPair sg[4];  // row pairs (0,1), (2,3), (4,5), (6,7) of the octet
#pragma unroll
  for (int q = 0; q < 8; q++) g_words<FAST>(v[q], E, gw[0][q], gw[1][q]);
#pragma unroll
  for (int q = 0; q < 4; q++) sg[q] = sign_pair(v[2 * q], v[2 * q + 1]);
#pragma unroll
  for (int i = 0; i < DIGITS; i += 2) {
    uint32_t d0[4], d1[4];
#pragma unroll
    for (int q = 0; q < 4; q++) digit_pairs2(gw[i / 4][2 * q], gw[i / 4][2 * q + 1], i & 2, sg[q], d0[q], d1[q]);
    const int r0 = i * CP + c, r1 = r0 + CP;
    *reinterpret_cast<uint4*>(buf + (r0 >> 3) * 128 + (r0 & 7) * 16) = make_uint4(d0[0], d0[1], d0[2], d0[3]);
    *reinterpret_cast<uint4*>(buf + (r1 >> 3) * 128 + (r1 & 7) * 16) = make_uint4(d1[0], d1[1], d1[2], d1[3]);
  }
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// named barriers over one role's threads; return 1 on every thread if pred holds on any
__device__ __forceinline__ int slicers_any(int pred) {
  int r;
  asm volatile(
      "{\n .reg .pred p, q;\n setp.ne.s32 p, %1, 0;\n bar.red.or.pred q, 1, %2, p;\n selp.s32 %0, 1, 0, q;\n}\n"
      : "=r"(r)
      : "r"(pred), "n"(SLICERS)
      : "memory");
  return r;
}
__device__ __forceinline__ int drainers_any(int pred) {
  int r;
  asm volatile(
      "{\n .reg .pred p, q;\n setp.ne.s32 p, %1, 0;\n bar.red.or.pred q, 2, 128, p;\n selp.s32 %0, 1, 0, q;\n}\n"
      : "=r"(r)
      : "r"(pred)
      : "memory");
  return r;
}
__device__ __forceinline__ void drainers_sync() { asm volatile("bar.sync 2, 128;" ::: "memory"); }

// bounded wait that also gives up as soon as another thread of the CTA has given up; sleep_ns
// between polls for the roles that wait most of the time
__device__ __forceinline__ bool wait_ab(uint64_t* bar, uint32_t parity, volatile int* ab, int* err,
                                        uint32_t sleep_ns = 0) {
  for (uint32_t i = 0; i < kWaitPolls; i++) {
    if (mbar_try_wait(bar, parity)) return true;
    if (*ab) return false;
    if (sleep_ns) __nanosleep(sleep_ns);
  }
  *ab = 1;
  if (err) atomicExch(err, SKINNY_DEVERR_TIMEOUT);
  return false;
}

template <int NP, typename TI>
__global__ void __launch_bounds__(THREADS, 1) split_tsmttsm_kernel(const Args p) {
  constexpr int BN = NP < 8 ? NP : 8;  // B columns per drain block
  constexpr int NB = NP / BN;          // drain blocks
  extern __shared__ __align__(1024) unsigned char smem[];
  uint64_t* full = reinterpret_cast<uint64_t*>(smem);           // [MAXST] FP64 stage landed
  uint64_t* empty = full + MAXST;                                // [MAXST] FP64 stage consumed
  uint64_t* dfull = reinterpret_cast<uint64_t*>(smem + 64);      // [MAXDST] digit stage written
  uint64_t* dempty = reinterpret_cast<uint64_t*>(smem + 96);     // [MAXDST] its MMAs completed
  uint64_t* pdone = reinterpret_cast<uint64_t*>(smem + 128);     // [2] a period's MMAs completed
  uint64_t* pfin = reinterpret_cast<uint64_t*>(smem + 144);      // [2] a period's record published
  uint64_t* drained = reinterpret_cast<uint64_t*>(smem + 160);   // [2] a set's drain finished
  uint64_t* bar_fin = reinterpret_cast<uint64_t*>(smem + 176);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(smem + 192);
  volatile int* abort_f = reinterpret_cast<volatile int*>(smem + 196);
  volatile int* rinfo = reinterpret_cast<volatile int*>(smem + 208);  // [MAXDST] period | first << 30
  volatile int* plast = reinterpret_cast<volatile int*>(smem + 224);  // [2] the period is the last
  volatile int* pchg = reinterpret_cast<volatile int*>(smem + 232);  // [2] the period's exponents are new
  int* Ecur = reinterpret_cast<int*>(smem + 256);                      // [32] A columns, then B
  int* pe = reinterpret_cast<int*>(smem + 384);                        // [2][32] a period's exponents
  int* ae = reinterpret_cast<int*>(smem + 640);                        // [32] exponents of the drain's sums
  int* D = reinterpret_cast<int*>(smem + HDR);                         // SortBuf: [8 * NC][STRIDE]
  double* cacc = reinterpret_cast<double*>(smem + HDR + p.sort_bytes);
  unsigned char* ring = smem + HDR + p.sort_bytes + CBYTES;
  unsigned char* dig = ring + (size_t)p.stages * p.stage_bytes;  // 1024-aligned by the host
  auto digA = [&](int d) { return dig + (size_t)d * (p.dig_a + p.dig_b); };
  auto digB = [&](int d) { return p.gram ? digA(d) : digA(d) + p.dig_a; };

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int M = p.M, N = p.N, MP = p.MP;
  const int chunk = blockIdx.x, nchunks = gridDim.x;
  const int64_t t_begin = p.nrounds * chunk / nchunks;
  const int64_t t_end = p.nrounds * (chunk + 1) / nchunks;
  const int nt = (int)(t_end - t_begin);
  const int DST = p.dstages;
  // a round is bulk-copied when its rows end before the last row of the operand starts
  auto is_bulk = [&](int64_t t) { return p.bulk && (t + 1) * (int64_t)p.rr < p.K; };

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)),
                 "r"(p.tmem_cols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    for (int s = 0; s < p.stages; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], NSLICE);
    }
    for (int d = 0; d < DST; d++) {
      mbar_init(&dfull[d], NSLICE);
      mbar_init(&dempty[d], 1);
    }
    for (int i = 0; i < 2; i++) {
      mbar_init(&pdone[i], 1);
      mbar_init(&pfin[i], 1);
      mbar_init(&drained[i], NDRAIN);
    }
    mbar_init(bar_fin, 1);
    *abort_f = 0;
    fence_mbar_init();
  }
  if (tid < 32) Ecur[tid] = 0;
  for (int e = tid; e < CBYTES / 8; e += THREADS) cacc[e] = 0.0;
  // padding rows of the digit stages stay zero: clear every stage once
  for (uint32_t o = tid * 16; o < (uint32_t)DST * (p.dig_a + p.dig_b); o += THREADS * 16)
    *reinterpret_cast<uint4*>(dig + o) = make_uint4(0, 0, 0, 0);
  fence_proxy_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tslot;

  if (warp >= WPROD) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
    if (warp == WPROD) {
      // ---- producer: whole rounds of rows of A and B into the FP64 stage ring ----------------------
      int issued = 0;
      for (int t = 0; t < nt; t++) {
        const int s = t % p.stages, use = t / p.stages;
        if (use > 0) {
          int ok = 0;
          if (lane == 0) ok = wait_ab(&empty[s], (uint32_t)((use - 1) & 1), abort_f, p.err, SLEEP_PRODUCER);
          if (!__shfl_sync(0xffffffffu, ok, 0)) break;
        }
        if (lane == 0) {
          const int64_t tt = t_begin + t;
          if (is_bulk(tt)) {
            const int64_t r0 = tt * p.rr;
            constexpr uint32_t ES = sizeof(TI);
            const uint32_t ba = (uint32_t)(p.rr * p.lda * ES), bb = p.gram ? 0u : (uint32_t)(p.rr * p.ldb * ES);
            unsigned char* st = ring + (size_t)s * p.stage_bytes;
            mbar_arrive_expect_tx(&full[s], ba + bb);
            bulk_g2s(st, static_cast<const TI*>(p.A) + r0 * p.lda, ba, &full[s]);
            if (!p.gram) bulk_g2s(st + p.tile_a, static_cast<const TI*>(p.B) + r0 * p.ldb, bb, &full[s]);
          } else {
            mbar_arrive(&full[s]);  // no copy: the slicers read this round from global memory
          }
        }
        issued = t + 1;
      }
      // copies in flight land before the CTA ends
      if (lane == 0)
        for (int t = max(0, issued - p.stages); t < issued; t++)
          mbar_wait_bounded(&full[t % p.stages], (uint32_t)((t / p.stages) & 1), nullptr);
    } else if (warp == WMMA) {
      // ---- MMA issuer -------------------------------------------------------------------------------
      if (lane == 0) {
        // idesc: D f32, A/B f16, K-major both, N = nmma, M = 128
        const uint32_t idesc = (1u << 4) | ((uint32_t)(p.nmma >> 3) << 17) | ((128u >> 4) << 24);
        const uint32_t lbb = p.gram ? p.lbo_a : p.lbo_b;
        int pcur = -1, issued = 0;
        bool ok = true;
        for (int t = 0; t < nt; t++) {
          const int d = t % DST;
          if (!wait_ab(&dfull[d], (uint32_t)((t / DST) & 1), abort_f, p.err, SLEEP_MMA)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const int info = rinfo[d];
          const int pp = info & 0x3FFFFFFF;
          const bool first = (info >> 30) & 1;
          if (first) {
            if (pp >= 1) {  // the previous period is complete once its MMAs finish
              mma_commit(&pdone[(pp - 1) & 1]);
              plast[(pp - 1) & 1] = 0;
              mbar_arrive(&pfin[(pp - 1) & 1]);
            }
            if (pp >= 2) {  // this period's accumulator set was drained (period pp - 2)
              if (!wait_ab(&drained[pp & 1], (uint32_t)(((pp - 2) >> 1) & 1), abort_f, p.err, SLEEP_MMA)) {
                ok = false;
                break;
              }
              tc_fence_after();
            }
          }
          const uint32_t a0 = smem_u32(digA(d)), b0 = smem_u32(digB(d));
          const uint32_t dcol = tmem + (uint32_t)((pp & 1) * p.nmma);
          const int ksteps = p.rr / 16;
          uint64_t da = make_desc(a0, p.lbo_a), db = make_desc(b0, lbb);
          for (int ks = 0; ks < ksteps; ks++) {
            mma_f16(dcol, da, db, idesc, (first && ks == 0) ? 0u : 1u);
            da += (2 * p.lbo_a) >> 4;  // the next two k-octets
            db += (2 * lbb) >> 4;
          }
          mma_commit(&dempty[d]);
          pcur = pp;
          issued++;
        }
        if (ok && pcur >= 0) {
          mma_commit(&pdone[pcur & 1]);
          plast[pcur & 1] = 1;
          mbar_arrive(&pfin[pcur & 1]);
        }
        if (issued) {  // every MMA has finished before the TMEM is released
          mma_commit(bar_fin);
          mbar_wait_bounded(bar_fin, 0, nullptr);
        }
      }
    }
  } else if (warp >= NSLICE) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 152;");
    // ---- drain: a period's TMEM set -> level sums -> FP64 accumulators ---------------------------
    const int q = warp - NSLICE;        // TMEM lane quadrant
    const int dtid = tid - SLICERS;     // 0..127
    const int r = 32 * q + lane;        // TMEM lane = A digit row
    const bool qvalid = 32 * q < DIGITS * MP;  // quadrants without a digit row have nothing to drain
    // Sums of the digit pairs (i0, j) of this lane's row over the periods since the exponents last
    // changed (MAXSUM at most): one conversion and one addition per value and period
    int acc[DIGITS * NP];
#pragma unroll
    for (int x = 0; x < DIGITS * NP; x++) acc[x] = 0;
    int cnt = 0;
    bool done = nt == 0;  // K = 0: no rounds, no periods
    for (int pp = 0;; pp++) {
      const int set = pp & 1;
      bool chg = false, last = false;
      if (!done) {
        const uint32_t par = (uint32_t)((pp >> 1) & 1);
        // one lane per warp polls (sleeping in between); the warp follows
        int ok = 1;
        if (lane == 0) {
          ok = wait_ab(&pfin[set], par, abort_f, p.err, SLEEP_DRAIN);
          if (ok) ok = wait_ab(&pdone[set], par, abort_f, p.err, SLEEP_DRAIN);
        }
        ok = __shfl_sync(0xffffffffu, ok, 0);
        if (drainers_any(!ok)) break;
        tc_fence_after();
        last = plast[set] != 0;
        chg = pchg[set] != 0;
      }
      if (cnt && (done || chg || cnt == MAXSUM)) {  // levels -> FP64 accumulators
        // a few columns n at a time through shared memory; a thread then forms the eight level sums of a cell
        auto sort = [&](auto buf) {
          constexpr int NC = NP < decltype(buf)::NC ? NP : decltype(buf)::NC, STRIDE = decltype(buf)::STRIDE;
#pragma unroll
          for (int n0 = 0; n0 < NP; n0 += NC) {
            if (qvalid) {
#pragma unroll
              for (int j = 0; j < DIGITS; j++)
#pragma unroll
                for (int x = 0; x < NC; x++) D[(j * NC + x) * STRIDE + r] = acc[j * NP + n0 + x];
            }
            drainers_sync();
            for (int e = dtid; e < M * min(NC, N - n0); e += NDRAIN * 32) {
              const int mm = e % M, x = e / M;
              const int* Dc = D + x * STRIDE + mm;
              long long sv[8];
#pragma unroll
              for (int t = 0; t < DIGITS; t++) {
                int sum = 0;  // |sum| <= 8 * MAXSUM * 2^24
#pragma unroll
                for (int i = 0; i <= t; i++) sum += Dc[(t - i) * NC * STRIDE + i * MP];
                sv[t] = sum;
              }
              const long long vhi = (sv[0] << 24) + (sv[1] << 16) + (sv[2] << 8) + sv[3];
              const long long vlo = (sv[4] << 24) + (sv[5] << 16) + (sv[6] << 8) + sv[7];
              const int ea = ae[mm], eb = ae[(p.gram ? 0 : 16) + n0 + x];
              const double v = fma((double)vlo, 0x1p-32, (double)vhi);  // in units of 2^(EA+EB-2080)
              double& ca = cacc[(n0 + x) * M + mm];
              // (one factor where it is in range, so that a small one of the two does not round v)
              const int es = ea + eb - 2080;
              ca = (unsigned)(es + 1022) <= 2045u ? fma(v, pow2i(es), ca)
                                                  : fma(v * pow2i(ea - 1040), pow2i(eb - 1040), ca);
            }
            drainers_sync();
          }
        };
        if (p.sort_bytes == SortBuf<4>::BYTES)
          sort(SortBuf<4>{});
        else
          sort(SortBuf<2>{});
#pragma unroll
        for (int x = 0; x < DIGITS * NP; x++) acc[x] = 0;
        cnt = 0;
      }
      if (done) break;
      if (cnt == 0) {
        drainers_sync();  // ae has been read
        if (dtid < 32) ae[dtid] = pe[set * 32 + dtid];
      }
      if (qvalid) {
#pragma unroll
        for (int b = 0; b < DIGITS * NB; b++) {
          uint32_t tmp[BN];
          tmem_ld<BN>(tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(set * p.nmma + b * BN), tmp);
          tmem_wait_ld();
          // exact (|sum| <= 2^24)
#pragma unroll
          for (int x = 0; x < BN; x++) acc[b * BN + x] += __float2int_rn(__uint_as_float(tmp[x]));
        }
      }
      cnt++;
      done = last;
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&drained[set]);
    }
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
    // ---- slicers: one unit = one column and 8 rows per thread; A units first, then B units -------
    const int NUA = (p.rr / 8) * MP;
    const int NU = NUA + (p.gram ? 0 : (p.rr / 8) * NP);  // <= SLICERS (host guarantees)
    const bool isB = tid >= NUA;
    const int uv = isB ? tid - NUA : tid, CP = isB ? NP : MP;
    const int col = uv % CP, oct = uv / CP;
    const bool uval = tid < NU && col < (isB ? N : M);
    const int64_t ld = isB ? p.ldb : p.lda;
    const TI* gsrc = static_cast<const TI*>(isB ? p.B : p.A);
    const uint32_t lbo = isB ? p.lbo_b : p.lbo_a;
    // The 8 rows of an octet o are visited in the order q ^ (o & 7), the same for A and B (a
    // permutation of k inside a k-octet leaves the MMA's sum unchanged): lanes of a half-warp
    // holding different octets then read different banks of the FP64 stage.
    const int g = oct & 7;
    int Ereg = 0;
    bool slow = true;  // warp-uniform: a column of this warp may hold subnormal numbers in its range
    int pp = -1, period_rows = 0, s = -1, d = -1, elast = -1;
    uint32_t sph = 1, dph = 1;
    for (int t = 0; t < nt; t++) {
      if (++s == p.stages) s = 0;
      if (s == 0) sph ^= 1u;
      if (++d == DST) d = 0;
      if (d == 0) dph ^= 1u;
      const int64_t tt = t_begin + t;
      bool ok = mbar_wait_warp(&full[s], sph, abort_f);
      double v[8];
      if (is_bulk(tt)) {  // shared-memory stage
        const TI* src = reinterpret_cast<const TI*>(ring + (size_t)s * p.stage_bytes + (isB ? p.tile_a : 0)) +
                        (oct * 8) * (int)ld + col;
#pragma unroll
        for (int q2 = 0; q2 < 8; q2++) v[q2] = uval ? (double)src[(q2 ^ g) * (int)ld] : 0.0;
      } else {  // global memory (rows not 16-byte aligned, or the last round)
        const int64_t r0 = tt * p.rr;
        const int rows = (int)((p.K - r0) < p.rr ? (p.K - r0) : p.rr);
#pragma unroll
        for (int q2 = 0; q2 < 8; q2++) {
          const int rr = oct * 8 + (q2 ^ g);
          v[q2] = (uval && rr < rows) ? (double)gsrc[(r0 + rr) * ld + col] : 0.0;
        }
      }
      // largest exponent field of the unit (1 if only subnormals, 0 if all zero): the largest
      // high word without its sign bit gives the field; an OR of the magnitudes tells zero
      uint32_t hmax = 0u, nz = 0u;
#pragma unroll
      for (int q2 = 0; q2 < 8; q2++) {
        const uint32_t h = (uint32_t)__double2hiint(v[q2]) & 0x7FFFFFFFu;
        hmax = max(hmax, h);
        nz |= h | (uint32_t)__double2loint(v[q2]);
      }
      uint32_t eu = hmax >> 20;
      if (eu == 0u && nz != 0u) eu = 1u;
      const bool exceed = uval && (int)eu > Ereg;
      const bool newp = pp < 0 || period_rows + p.rr > PERIOD || exceed;
      bool first = false;
      if (slicers_any(!ok || newp)) {
        if (slicers_any(!ok)) {
          *abort_f = 1;
          if (lane == 0) atomicExch(p.err, SKINNY_DEVERR_TIMEOUT);
          break;
        }
        // a new period: raise the exponents of the columns that met larger elements
        if (exceed) atomicMax(&Ecur[(isB ? 16 : 0) + col], (int)eu > EMAX ? NONFINITE : min((int)eu + HEAD, EMAX));
        pp++;
        bool ok2 = true;  // the period's exponent slot and accumulator set held period pp - 2
        if (pp >= 2) ok2 = wait_ab(&drained[pp & 1], (uint32_t)(((pp - 2) >> 1) & 1), abort_f, p.err);
        if (slicers_any(!ok2)) break;  // also orders the atomics before the reads below
        if (warp == 0) {
          const int e = Ecur[lane];
          pe[(pp & 1) * 32 + lane] = e;
          const int chg = __any_sync(0xffffffffu, e != elast);
          if (lane == 0) pchg[pp & 1] = chg;
          elast = e;
        }
        if (uval) Ereg = Ecur[(isB ? 16 : 0) + col];
        slow = __any_sync(0xffffffffu, uval && Ereg <= EMIN_FAST);
        period_rows = 0;
        first = true;
      }
      // the FP64 stage is consumed: the values are in registers
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[s]);
      // the digit stage is free once the MMAs of round t - DST completed
      if (t >= DST) ok = mbar_wait_warp(&dempty[d], dph ^ 1u, abort_f);
      if (__all_sync(0xffffffffu, ok)) {
        if (uval) {
          unsigned char* buf = (isB ? digB(d) : digA(d)) + oct * lbo;
          if (slow)
            slice_unit<false>(v, (uint32_t)Ereg, col, CP, buf);
          else
            slice_unit<true>(v, (uint32_t)Ereg, col, CP, buf);
        }
        if (tid == 0) rinfo[d] = pp | (first ? (1 << 30) : 0);
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&dfull[d]);
      } else {
        *abort_f = 1;
        if (lane == 0) atomicExch(p.err, SKINNY_DEVERR_TIMEOUT);
      }
      period_rows += p.rr;
    }
  }

  tc_fence_before();
  __syncthreads();
  // back to the registers of the launch (a warpgroup's warps have met since the first change)
  if (warp >= NSLICE && warp < WPROD)
    asm volatile("setmaxnreg.dec.sync.aligned.u32 80;");
  else
    asm volatile("setmaxnreg.inc.sync.aligned.u32 80;");
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(p.tmem_cols));
  if (*abort_f) return;  // timeout recorded in the error word; no partial, no ticket

  // ---- cross-CTA finish, two levels: the last CTA of each group of GROUP CTAs sums the group's
  // partials in CTA order, the last group to finish sums the group sums in group order and applies
  // alpha and beta (deterministic; each level is one round of independent loads) -----------------
  const int MN = M * N;
  if (tid < MN) p.partials[(size_t)chunk * MN + tid] = cacc[tid];
  __threadfence();
  __syncthreads();
  __shared__ int s_last;
  const int ngroups = (nchunks + GROUP - 1) / GROUP, grp = chunk / GROUP;
  const int gsize = min(GROUP, nchunks - grp * GROUP);
  if (tid == 0) s_last = (atomicAdd(p.counter + grp, 1u) == (unsigned)(gsize - 1));
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  double* Gs = p.partials + (size_t)nchunks * MN;  // [group][MN]
  for (int e = tid; e < MN; e += THREADS) {
    double v[GROUP];
#pragma unroll
    for (int i = 0; i < GROUP; i++) v[i] = i < gsize ? __ldcg(&p.partials[(size_t)(grp * GROUP + i) * MN + e]) : 0.0;
    double sum = 0.0;
#pragma unroll
    for (int i = 0; i < GROUP; i++) sum += v[i];
    Gs[(size_t)grp * MN + e] = sum;
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) {
    p.counter[grp] = 0u;
    s_last = (atomicAdd(p.counter + MAXGROUPS, 1u) == (unsigned)(ngroups - 1));
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  if (tid < MN) {
    double v[MAXGROUPS];
#pragma unroll
    for (int i = 0; i < MAXGROUPS; i++) v[i] = i < ngroups ? __ldcg(&Gs[(size_t)i * MN + tid]) : 0.0;
    double sum = 0.0;
#pragma unroll
    for (int i = 0; i < MAXGROUPS; i++) sum += v[i];
    const int mm = tid % M, nn = tid / M;
    const int64_t ci = (int64_t)nn * p.ldc + mm;
    if (p.out_f32) {  // the one rounding of an FP32 result
      float* c = static_cast<float*>(p.C) + ci;
      *c = (float)(p.beta_zero ? p.alpha * sum : (double)(*c) * p.beta + sum * p.alpha);
    } else {
      double* c = static_cast<double*>(p.C) + ci;
      *c = p.beta_zero ? p.alpha * sum : (*c) * p.beta + sum * p.alpha;
    }
  }
  if (tid == 0) p.counter[MAXGROUPS] = 0u;
}

template <int NP, typename TI>
static skinny_status launch(const Args& a, int grid, int smem, cudaStream_t st) {
  static SmemAttr attr;
  auto kern = split_tsmttsm_kernel<NP, TI>;
  ensure_smem_attr(kern, smem, attr);
  kern<<<grid, THREADS, smem, st>>>(a);
  count_launch();
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_error(std::string("split tsmttsm launch: ") + cudaGetErrorString(e));
    return SKINNY_DEVICE_ERROR;
  }
  return SKINNY_OK;
}

}  // namespace split

skinny_status split_product(skinny_handle h, bool tsmm, int64_t M, int64_t N, int64_t K,
                            const double* A, int64_t lda, const void* alpha, const double* B,
                            int64_t ldb, const void* beta, double* C, int64_t ldc,
                            cudaStream_t st, bool autoselect) {
  if (tsmm) return split_tsmm(h, false, M, N, K, A, lda, alpha, B, ldb, beta, C, ldc, st, autoselect);
  return split_tsmttsm_t(h, false, false, M, N, K, A, lda, alpha, B, ldb, beta, C, ldc, st, autoselect);
}

skinny_status split_tsmttsm_t(skinny_handle h, bool in_f32, bool out_f32, int64_t M, int64_t N, int64_t K,
                              const void* A, int64_t lda, const void* alpha, const void* B, int64_t ldb,
                              const void* beta, void* C, int64_t ldc, cudaStream_t st, bool autoselect) {
  using namespace split;
  const int64_t es = in_f32 ? 4 : 8;
  if (M > 128 || N > 128) {
    set_error("split precision TSMTTSM: M, N <= 128");
    return SKINNY_UNSUPPORTED;
  }
  // auto selection (measured on GB300, us, CUDA-core FP64 kernel / this one):
  //   * both widths at least 4 and M N >= 32.  Rows of 2^20: 4x8 71/56, 6x6 75/60, 8x8 120/64, 4x16
  //     128/94, 4x32 244/179, 4x64 489/306; but 4x4 41/40, 16x2 73/87, 2x64 290/308.
  //   * K M N >= 2^22, or 3 * 2^22 with a width below 8: the kernels' fixed costs differ by 5 to 10 us.  At
  //     2^22: 8x8 17.2/15.3, 16x16 20.5/16.5, 32x8 21.8/19.1, 32x32 27.7/28.4; at 2^21 12.4/13.4, 15.9/16.4,
  //     16.5/18.1 and (24x24) 24.2/22.4.  4x16 at 2^22 17.9/18.8, 4x32 at 2^23 27.1/28.3.
  //   * the wide kernel's blocks of 64 x 64 filled by a quarter of a 32 x 32 or 4 x 64 at least (128
  //     cells where the stages fold, else 256 a block).  With a width below 8 it does not win over bulk copies of
  //     the CUDA-core kernel where its own are row by row (2^18 rows, 4x32 72/60, with an odd leading dimension
  //     72/114; 4x64 141/97 and 141/196; out of a wide block, where neither has any, 4x32 114/115, 6x32 141/117).
  // The autotuner can override per shape.
  const bool wide = M > 16 || N > 16;
  const int64_t sym_w = (A == B && lda == ldb && M == N) ? 1 : 0;
  const int64_t bm = (M + 63) / 64, bn = (N + 63) / 64;
  const int64_t nblk_w = sym_w ? bm * (bm + 1) / 2 : bm * bn;
  const int64_t per_blk = (M <= 32 && N <= 32) ? 128 : 256;
  const bool widths_win = M >= 4 && N >= 4 && M * N >= 32;
  const bool dense_w = lda == M && ldb == N && (uintptr_t)A % 16 == 0 && (uintptr_t)B % 16 == 0;
  const int64_t work_min = (M >= 8 && N >= 8) ? (int64_t)1 << 22 : (int64_t)3 << 22;
  const bool shape_wins = widths_win && !(wide && M * N < per_blk * nblk_w) &&
                          !(wide && (M < 8 || N < 8) && !dense_w && bulk_rows(M, N, A, lda, B, ldb, sym_w != 0));
  if (autoselect && (K < 4096 || K * M * N < work_min || !shape_wins)) {
    if (wide && shape_wins) split_wide_reserve(h, M, N, K, sym_w != 0, st);  // for more rows
    set_error("split precision: not selected automatically for this shape");
    return SKINNY_UNSUPPORTED;
  }
  // M or N > 16: the wide kernel (64 x 64 blocks, FP16 digit planes, level accumulators)
  if (wide) return split_wide_t(h, in_f32, out_f32, M, N, K, A, lda, alpha, B, ldb, beta, C, ldc, st);
  Args a;
  a.A = A;
  a.B = B;
  a.C = C;
  a.K = K;
  a.lda = lda;
  a.ldb = ldb;
  a.ldc = ldc;
  a.M = (int)M;
  a.N = (int)N;
  if (out_f32) {  // FP32 scalars widened (exactly)
    float af, bf;
    std::memcpy(&af, alpha, 4);
    std::memcpy(&bf, beta, 4);
    a.alpha = af;
    a.beta = bf;
  } else {
    std::memcpy(&a.alpha, alpha, 8);
    std::memcpy(&a.beta, beta, 8);
  }
  a.out_f32 = out_f32;
  a.beta_zero = a.beta == 0.0;
  a.gram = (A == B) && (lda == ldb) && (M == N);
  const int NP = pow2ceil(a.gram ? M : N);
  a.MP = a.gram ? NP : pow2ceil(M);
  a.NP = NP;
  // rows per round: 128 * R with R the largest power of two whose slicing units (one column and
  // 8 rows each) fit one per slicer thread and whose FP64 and digit stages fit in shared memory
  // (at least two of each; bulk copies of whole rounds where aligned dense rows fit, else the
  // slicers read global memory).  A round's fixed costs -- the slicers' barrier, the hand-offs,
  // the MMA commit -- then spread over as many rows as possible.
  const int cols = a.MP + (a.gram ? 0 : NP);
  a.nmma = std::max(16, 8 * NP);
  a.tmem_cols = std::max(32, 2 * a.nmma);
  a.lbo_a = (uint32_t)(8 * a.MP * 16);
  a.lbo_b = (uint32_t)(a.nmma * 16);
  // a round starts at a multiple of 128 rows, so its bytes start 16-byte aligned with the operand
  const bool aligned = ((uintptr_t)A % 16 == 0) && (a.gram || (uintptr_t)B % 16 == 0);
  const bool dense = lda <= 2 * M + 16 && (a.gram || ldb <= 2 * N + 16);
  const int64_t fixed = HDR + SortBuf<2>::BYTES + CBYTES + STATIC_RESERVE;
  int64_t dstage = 0;
  a.stages = 0;
  for (int R = PERIOD / 128; R >= 1 && a.stages == 0; R /= 2) {
    if (R * 16 * cols > SLICERS) continue;
    a.rr = 128 * R;
    const int64_t octs = a.rr / 8;
    a.dig_a = (uint32_t)round_up(octs * a.lbo_a + DPAD, 1024);
    a.dig_b = a.gram ? 0u : (uint32_t)round_up(octs * a.lbo_b, 1024);
    a.tile_a = (uint32_t)round_up((int64_t)a.rr * lda * es, 128);
    const int64_t tile_b = a.gram ? 0 : round_up((int64_t)a.rr * ldb * es, 128);
    dstage = (int64_t)a.dig_a + a.dig_b;
    for (int bulk = (aligned && dense && K > a.rr) ? 1 : 0; bulk >= 0 && a.stages == 0; bulk--) {
      a.bulk = bulk;
      a.stage_bytes = bulk ? (uint32_t)round_up(a.tile_a + tile_b, 1024) : 1024u;
      for (int dst = MAXDST; dst >= 2 && a.stages == 0; dst--)
        for (int nst = MAXST; nst >= 2; nst--)
          if (fixed + (int64_t)nst * a.stage_bytes + (int64_t)dst * dstage <= h->dev.smem_optin) {
            a.stages = nst;
            a.dstages = dst;
            break;
          }
    }
  }
  if (a.stages == 0) {
    set_error("split precision: stages do not fit in shared memory");
    return SKINNY_UNSUPPORTED;
  }
  a.nrounds = (K + a.rr - 1) / a.rr;
  int64_t smem2 = fixed + (int64_t)a.stages * a.stage_bytes + (int64_t)a.dstages * dstage;
  a.sort_bytes = SortBuf<2>::BYTES;
  if (smem2 + SortBuf<4>::BYTES - SortBuf<2>::BYTES <= h->dev.smem_optin) {
    a.sort_bytes = SortBuf<4>::BYTES;
    smem2 += SortBuf<4>::BYTES - SortBuf<2>::BYTES;
  }
  smem2 -= STATIC_RESERVE;
  const int64_t grid = std::max<int64_t>(1, std::min<int64_t>({a.nrounds, h->dev.sms, (int64_t)GROUP * MAXGROUPS}));
  Workspace& ws = h->ws[st];
  // CTA partials, then the group sums
  skinny_status s = workspace_ensure(ws, ((size_t)grid + MAXGROUPS) * M * N * 8, st);
  if (s != SKINNY_OK) return s;
  a.partials = (double*)ws.partials;
  a.counter = ws.counter;
  a.err = h->err;
  if (!in_f32) {
    switch (NP) {
      case 1: return launch<1, double>(a, (int)grid, (int)smem2, st);
      case 2: return launch<2, double>(a, (int)grid, (int)smem2, st);
      case 4: return launch<4, double>(a, (int)grid, (int)smem2, st);
      case 8: return launch<8, double>(a, (int)grid, (int)smem2, st);
      case 16: return launch<16, double>(a, (int)grid, (int)smem2, st);
    }
  } else {
    switch (NP) {
      case 1: return launch<1, float>(a, (int)grid, (int)smem2, st);
      case 2: return launch<2, float>(a, (int)grid, (int)smem2, st);
      case 4: return launch<4, float>(a, (int)grid, (int)smem2, st);
      case 8: return launch<8, float>(a, (int)grid, (int)smem2, st);
      case 16: return launch<16, float>(a, (int)grid, (int)smem2, st);
    }
  }
  set_error("split precision: unsupported N");
  return SKINNY_UNSUPPORTED;
}

}  // namespace skinny
