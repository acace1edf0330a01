// split_wide.cu -- FP64 TSMTTSM in split precision for widths 17..128 on tcgen05 tensor cores
// (no counterpart in the reference, whose FP64 TSMTTSM kernels are CUDA-core DFMA loops, e.g.
// tsmttsm/genv5.cuh:28-89; the product and its alpha/beta semantics are those of
// tsmttsm/genv5.cuh:92-98 with the cross-block sum done inside the launch).
//
// From M = N = 32 on, a CUDA-core FP64 TSMTTSM is bound by the FP64 pipe (1.2 TFLOP/s on GB300).
// Here each C block of 64 x 64 is formed from 8-bit digit products on the tensor cores, exactly,
// with every element sliced once.
//
// Scheme:
//   * Per column of A (and of B) a shared exponent E holds for an epoch: an element x is
//     x = sign * F * 2^(E - 1084) with F < 2^62 a fixed-point integer, and F is written as 8
//     balanced base-256 digits d_1..d_8 (d_1 in [-64, 64], the others in [-128, 127]), to each of
//     which the sign of x is applied (digits.cuh).
//     When a column meets an element larger than 2^E allows, E is raised (with 4 bits of
//     headroom) and a new epoch starts for the whole CTA (drained words do not mix exponents).
//   * Digits are exact in FP16.  For a stage of 16 rows the digits are laid out as FP16 planes
//     (K-major, no swizzle): A' holds 12 planes of 64 rows in the order
//     [0, 1, 5 | 0, 2, 6 | 0, 3, 7 | 0, 4, 8] (0 = a zero plane, p = digit p of the 64 columns),
//     so the 128-row window [A_i ; A_{i+4}] is contiguous for i = -3..4; B' holds the planes
//     [0, 1, 2, ..., 8], so the 128-row window [B_j ; B_{j+1}] is contiguous for j = 0..7.
//   * A tcgen05.mma (M = 128, K = 16, FP16 x FP16 -> FP32 in TMEM) of window i of A' and
//     planes j, j + 1 of B' forms four 64 x 64 quadrants at digit levels (i + j, i + j + 1) in TMEM
//     lanes 0..63 and (i + j + 4, i + j + 5) in lanes 64..127.  Two accumulators of 128 columns
//     collect all 36 digit pairs with level i + j <= 9:
//        key 2:  i = -3..2, j = 2 - i   -> levels 2, 3 (lanes 0-63) and 6, 7 (lanes 64-127)
//        key 4:  i = -3..4, j = 4 - i   -> levels 4, 5 and 8, 9
//     For i <= 2 the two keys' planes 2 - i .. 5 - i are adjacent, so one MMA with N = 256 serves
//     both and reads the window of A' once: 8 MMAs per 16 rows (14 with N = 128, each with its own
//     read of both operands, 12 KB against 16 per window: 64 x 64, K = 2^20, 428 -> 415 us; the
//     operand reads, not the products, bound them).  Each pair is counted once.  Levels >= 10
//     are dropped (weight below 2^-56 of the leading level).
//   * A cell of an accumulator sums at most 8 digit products per row (|d d| <= 2^14), so over a
//     period of 128 rows every partial sum is an integer of magnitude < 2^24 and the FP32
//     accumulation is exact.  The two accumulators take 256 TMEM columns; two sets alternate
//     between periods, so the drain of one period runs while the MMAs of the next one proceed.
//   * Drain: TMEM -> int32 -> per C cell one int64 word per lane half (levels 2..5 packed with
//     shifts 24, 16, 8, 0 on lanes 0..63; levels 6..9 on lanes 64..127), summed over the periods
//     of an epoch in registers.  FP64 arithmetic happens only when an epoch ends: the int64 words
//     are converted, scaled by 2^(EA + EB - 2080) (levels 2..5) or 2^(EA + EB - 2112) (6..9) and
//     added to the CTA's FP64 partials.
//   * Warp roles (28 warps): 0-15 slice (8 columns of A or B each, 4 rows per thread; Gram: 4 columns of
//     A, 2 rows), 16-23 drain, 24 fetches rows of A and B into a ring of stages (1-D TMA bulk copies of
//     dense rows; other rows by cp.async, warps 26 and 27 helping), 25 issues the MMAs and opens and
//     closes the periods.  No two slicer warps wait for each other: a column's rows all lie with one
//     warp, which raises its exponent by itself, leaves (stage, exponent before, since) for the drain
//     warps and marks the stage for the MMA warp.  Every wait is bounded; a wait that runs
//     out sets the error word and the CTA finishes without waiting further and writes no C.
//   * Bound: a stage of 16 x (64 + 64) values takes ~1650 clocks.  The MMAs alone take ~1400 (900 of
//     products; operands from shared memory), slicing alone ~1400 (~25 instructions a value, two
//     thirds of the issue slots), and a TMA copy of the same rows would take ~700.  With 8 warps that
//     sliced and drained by turns and voted on the exponents of each stage it was 3600: each step of a
//     stage (two mbarriers, the vote, the drain) was waited out by all of them.
//     Measured, K rows: f64 64 x 64, K = 2^20, 794 -> 389 us;
//     32 x 32, K = 2^22, 1252 -> 686; 48 x 24, K = 2^20, 714 -> 325; Gram 64, K = 2^20, 738 -> 364;
//     rows of 80 (64 x 64, K = 2^20) 776 -> 583; f32 64 x 64, K = 2^18, 308 -> 146.
//   * Blocks of 64 x 64 (M or N > 64) run in the same launch, as do the row chunks of every
//     block; the last CTA of a block (ticket) sums the chunks' partials in chunk order and
//     applies alpha and beta.  Gram (A = B) computes the upper blocks only and mirrors them.
//   * Folded stages (M, N <= 32): a stage holds 32 rows; rows 0..15 fill plane rows 0..31 and
//     rows 16..31 fill plane rows 32..63 (column c of row 16 + r is plane row 32 + c).  The
//     diagonal quadrants of the 64 x 64 accumulators then hold the sums over the two row halves
//     (the off-diagonal quadrants pair different rows and are not read), so a 32-wide product
//     uses every slicer and every MMA column, and the halves are added at the end.
//   * Infinities and NaN have no fixed-point form: a column that holds one gets the exponent NONFINITE, whose
//     power of two is NaN, and so are the entries of C that it enters.
#include <atomic>
#include <cstring>

#include "api_internal.h"
#include "digits.cuh"

namespace skinny {

namespace splitw {

constexpr int ROWS = 16;     // K rows per stage (one MMA K-step)
constexpr int PSTAGES = 8;   // stages per accumulation period (128 rows: exact FP32 sums)
constexpr int DSLOTS = 3;    // digit slots
constexpr int MAXR = 8;      // FP64 stages (at most)
constexpr int HEAD = 4;      // exponent headroom granted when a column's exponent is raised
constexpr uint32_t EMAX = 2046;  // largest exponent field of a finite number, and of a column of such
constexpr int NONFINITE = 6000;  // exponent of a column with an infinity or NaN: out of the range of any sum
constexpr int SW = 16;       // slicer warps: 0-15
constexpr int DW = 8;        // drain warps: 16-23
constexpr int WPROD = SW + DW, WMMA = WPROD + 1;  // producer warps: WPROD and, for rows copied one by one, two more
// seven warpgroups (the last one: producers and MMA issuer) launched with 72 registers a
// thread, of which the slicers give back 8 and the last group 32 for the drain warps' 104
constexpr int THREADS = 32 * (SW + DW + 4);
constexpr int W = 64;        // block width
constexpr uint32_t LBO_A = 12 * 64 * 16;  // bytes between the two k-octets of A'
constexpr uint32_t LBO_B = 9 * 64 * 16;
constexpr uint32_t SLOT_A = 2 * LBO_A;
constexpr uint32_t SLOT = SLOT_A + 2 * LBO_B;  // 43008
constexpr uint32_t RAW_OP = ROWS * W * 8;      // one operand of an FP64 stage
constexpr int HDR = 4096;
constexpr int MAX_EPOCH_PERIODS = 1 << 14;     // int64 words hold 2^15 periods of < 2^48.1
constexpr int GROUP = 16;                      // chunks per first-level group of the finish (<= 15 groups)

struct Args {
  const void* A;  // FP64, or FP32 (widened exactly when read); the stage ring keeps the type
  const void* B;
  void* C;        // FP64, or FP32 with out_f32
  int64_t K, lda, ldb, ldc;
  int M, N;
  double alpha, beta;
  int beta_zero;
  int nblk, bm, sym;  // 64 x 64 blocks; sym: A == B, upper blocks only
  int bulk;           // rows start and end on 16-byte boundaries
  int abase16, bbase16;  // A / B start on a 16-byte boundary (dense stages by one bulk copy)
  int rstages;
  uint32_t raw_stage;  // bytes per FP64 stage
  int64_t nstages;     // ceil(K / rows per stage)
  double* partials;    // [nblk][nchunks][2][4096], then [nblk][15][4096] group sums
  unsigned* counter;   // tickets: [nblk][16] (15 groups + the block)
  int* err;
  int out_f32;
};

// A' plane slot of digit plane p (p <= 0: zero planes), for the chain order above
__host__ __device__ constexpr int slot_a(int p) { return 3 * ((p + 3) & 3) + ((p + 3) >> 2); }

__device__ __forceinline__ uint64_t desc(uint32_t saddr, uint32_t lbo) {
  uint64_t d = (uint64_t)((saddr & 0x3FFFF) >> 4);
  d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;  // k-octet stride
  d |= (uint64_t)(128 >> 4) << 32;              // 8-row-group stride
  d |= (uint64_t)1 << 46;
  return d;
}
// one lane of a converged warp, the same one every time
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n .reg .pred e;\n elect.sync _|e, 0xffffffff;\n selp.u32 %0, 1, 0, e;\n}\n" : "=r"(p));
  return p != 0;
}
// (descriptors as their lower words: the upper ones are constants)
__device__ __forceinline__ void mma_f16(uint32_t tmem, uint32_t da, uint32_t db, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n .reg .b64 a, b;\n setp.ne.b32 p, %4, 0;\n"
      " mov.b64 a, {%1, %5};\n mov.b64 b, {%2, %5};\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, p;\n}\n" ::"r"(tmem),
      "r"(da), "r"(db), "r"(idesc), "r"(acc), "n"((128 >> 4) | (1 << 14)));
}
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void tc_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// bytes a bulk copy will complete on the barrier, without an arrival
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
// arrive on the mbarrier once every cp.async of this thread so far has landed
__device__ __forceinline__ void cp_async_arrive(uint64_t* bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tmem_ld4(uint32_t taddr, uint32_t (&r)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// bounded wait that also gives up as soon as another thread of the CTA has given up; the producer
// and MMA warps sleep between polls so that their polling leaves issue slots to the slicers
__device__ __forceinline__ bool wait_ab(uint64_t* bar, uint32_t parity, volatile int* ab, int* err,
                                        uint32_t sleep_ns = 0) {
  for (uint32_t i = 0; i < (1u << 22); i++) {
    if (mbar_try_wait(bar, parity)) return true;
    if (*ab) return false;
    if (sleep_ns) __nanosleep(sleep_ns);
  }
  *ab = 1;
  if (err) atomicExch(err, SKINNY_DEVERR_TIMEOUT);
  return false;
}

// G (digits.cuh) of an element from its bits (FP32: hi) and sh = E - exponent field >= 0, for E > 64
// (FP32: 64 above the offset of its exponents), where zeros and subnormal numbers shift out entirely
// and need no case of their own
template <typename TI>
__device__ __forceinline__ uint64_t fixed_fast(uint32_t hi, uint32_t lo, uint32_t sh) {
  uint32_t H, L;
  if constexpr (sizeof(TI) == 8) {
    H = __funnelshift_l(lo, (hi & 0xFFFFFu) | 0x100000u, 9);
    L = lo << 9;
  } else {
    H = ((hi & 0x7FFFFFu) | 0x800000u) << 6;
    L = 0;
  }
  uint64_t F;
  asm("shr.u64 %0, %1, %2;" : "=l"(F) : "l"(((uint64_t)H << 32) | L), "r"(sh));  // 0 from 64 on
  return F + 0x8080808080808080ull;
}
// exponent field of x's magnitude (subnormal numbers: 1), 0 for zero; of the FP64 value for FP32
__device__ __forceinline__ uint32_t exp_field(double x) {
  const uint32_t mh = (uint32_t)__double2hiint(x) & 0x7FFFFFFFu;
  const uint32_t e = mh >> 20;
  return e == 0 && (mh | (uint32_t)__double2loint(x)) ? 1u : e;
}

__device__ __forceinline__ double pow2i(int e) {  // 2^e from -1022 to 1023, 2^-1022 below, NaN above (only NONFINITE gets there)
  e = min(max(e, -1022), 1024);
  return __hiloint2double((e + 1023) << 20, e > 1023);
}

// GR: how Gram blocks occur (0: none, A and B differ; 1: the only block; 2: among others), so that the
// two ways of slicing are compiled together only where a launch has both
template <typename TI, bool FOLD, int GR>
__global__ void __launch_bounds__(THREADS, 1) split_wide_kernel(const Args p) {
  constexpr uint32_t ES = sizeof(TI);
  extern __shared__ __align__(1024) unsigned char smem[];
  uint64_t* raw_full = reinterpret_cast<uint64_t*>(smem);  // [MAXR]
  uint64_t* raw_empty = raw_full + MAXR;                   // [MAXR]
  uint64_t* dfull = raw_full + 2 * MAXR;                   // [DSLOTS]
  uint64_t* dempty = dfull + 4;                            // [DSLOTS]
  uint64_t* tfull = dempty + 4;                            // [2]: a TMEM set holds a finished period
  uint64_t* tempty = tfull + 2;                            // [2]: and has been drained
  uint64_t* bar_fin = tempty + 2;
  uint32_t* tslot = reinterpret_cast<uint32_t*>(smem + 512);
  volatile int* abort_f = reinterpret_cast<volatile int*>(smem + 516);
  volatile int* nperiods = reinterpret_cast<volatile int*>(smem + 520);  // number of periods, once known
  volatile int* vflag = reinterpret_cast<volatile int*>(smem + 544);  // [4]: stage + 1 where an exponent is raised
  volatile int* mstart = reinterpret_cast<volatile int*>(smem + 576);  // [2]: first stage of a TMEM set's period,
  volatile int* mend = mstart + 2;                                     // [2]: the stage after its last,
  volatile int* mepoch = mstart + 4;                                   // [2]: its epoch
  volatile int* dprog = reinterpret_cast<volatile int*>(smem + 640);  // [DW]: periods up to here have their exponents
  // [128] exponents of A's and B's columns: (stage of the last raise, before, since)
  volatile uint64_t* rec = reinterpret_cast<volatile uint64_t*>(smem + 1024);
  unsigned char* dig = smem + HDR;
  unsigned char* raw = dig + DSLOTS * SLOT;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int blk = blockIdx.x % p.nblk, chunk = blockIdx.x / p.nblk, nchunks = gridDim.x / p.nblk;
  int bi, bj;
  if (p.sym) {  // upper triangle, column by column: (0,0), (0,1), (1,1), ...
    int b = blk;
    bj = 0;
    while (b > bj) {
      b -= bj + 1;
      bj++;
    }
    bi = b;
  } else {
    bi = blk % p.bm;
    bj = blk / p.bm;
  }
  const int Mb = min(W, p.M - W * bi), Nb = min(W, p.N - W * bj);
  const TI* Ab = static_cast<const TI*>(p.A) + W * bi;
  const TI* Bb = static_cast<const TI*>(p.sym ? p.A : p.B) + W * bj;
  const int64_t ldb = p.sym ? p.lda : p.ldb;
  const bool gram = GR == 0 ? false : GR == 1 ? true : p.sym && bi == bj;
  const int64_t s_begin = p.nstages * chunk / nchunks, s_end = p.nstages * (chunk + 1) / nchunks;
  const int nst = (int)(s_end - s_begin);
  const int R = p.rstages;
  // row strides (doubles) of the FP64 stages: dense operands land as one block of rows
  // dense operands (ld == block width, 16-byte aligned start): a stage's rows are one contiguous run
  const bool dense_a = p.abase16 && p.lda == Mb, dense_b = (p.sym ? p.abase16 : p.bbase16) && ldb == Nb;
  // rows per stage; row stride of the stage's rows that are copied one by one (a folded stage
  // holds 32 rows of at most 32 values in the same 16 x 64 space)
  const int SR = FOLD ? 2 * ROWS : ROWS, rw = FOLD ? W / 2 : W;
  const int rsa = dense_a ? Mb : rw, rsb = dense_b ? Nb : rw;

  const bool allbulk = p.bulk && dense_a && (gram || dense_b);  // one bulk copy per operand and stage

  // slicer warps with a column: 8 columns of A or B each (Gram: 4 of A)
  const int nslice = (FOLD ? 2 : 1) * (gram ? (Mb + 3) / 4 : (Mb + 7) / 8 + (Nb + 7) / 8);

  if (tid < 128) rec[tid] = 0;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tslot)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    for (int s = 0; s < R; s++) {
      mbar_init(&raw_full[s], allbulk ? 1 : 96);
      mbar_init(&raw_empty[s], nslice);
    }
    for (int s = 0; s < DSLOTS; s++) {
      mbar_init(&dfull[s], nslice);
      mbar_init(&dempty[s], 1);
    }
    for (int s = 0; s < 2; s++) {
      mbar_init(&tfull[s], 2);
      mbar_init(&tempty[s], DW);
    }
    for (int s = 0; s < 4; s++) vflag[s] = 0;
    for (int s = 0; s < DW; s++) dprog[s] = 0;
    mbar_init(bar_fin, 1);
    *abort_f = 0;
    *nperiods = 0x7fffffff;
    fence_mbar_init();
  }
  // zero planes and unused columns stay zero: clear every digit slot once
  for (uint32_t o = tid * 16; o < DSLOTS * SLOT; o += THREADS * 16)
    *reinterpret_cast<uint4*>(dig + o) = make_uint4(0, 0, 0, 0);
  fence_proxy_async_smem();
  tc_before();
  __syncthreads();
  tc_after();
  const uint32_t tmem = *tslot;

  if (warp >= WPROD) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
    const int pw = warp == WPROD ? 0 : warp - WMMA;  // of 3 producer warps
    if (warp != WMMA && (pw == 0 || !allbulk)) {
      // ---- producer: FP64 rows of A and B into the stage ring -------------------------------------
      int issued = 0, rs = -1;
      uint32_t rph = 1;  // parity of the releases waited for: the round before
      for (int ls = 0; ls < nst; ls++) {
        if (++rs == R) {
          rs = 0;
          rph ^= 1u;
        }
        if (ls >= R) {
          int ok = 0;
          if (lane == 0) ok = wait_ab(&raw_empty[rs], rph, abort_f, p.err, 64);
          if (!__shfl_sync(0xffffffffu, ok, 0)) break;
        }
        const int64_t row0 = (s_begin + ls) * SR;
        const int rows = (int)min((int64_t)SR, p.K - row0);
        TI* dA = reinterpret_cast<TI*>(raw + (size_t)rs * p.raw_stage);
        TI* dB = dA + ROWS * W;
        if (allbulk) {
          if (lane == 0) {
            mbar_arrive_expect_tx(&raw_full[rs], (uint32_t)(rows * (Mb + (gram ? 0 : Nb)) * ES));
            bulk_g2s(dA, Ab + row0 * p.lda, (uint32_t)(rows * Mb * ES), &raw_full[rs]);
            if (!gram) bulk_g2s(dB, Bb + row0 * ldb, (uint32_t)(rows * Nb * ES), &raw_full[rs]);
          }
        } else {
          // a dense operand whose stage starts and ends on 16-byte boundaries (always but for an odd
          // last stage) is one bulk copy, announced on the barrier without an arrival; other rows are
          // copied by all lanes, 16 bytes each where the rows are aligned (a bulk copy per row costs
          // ~100 clocks: 3600 a stage of 32 rows), else element by element; one arrival per lane once
          // its copies have landed
          const bool sa = dense_a && (row0 * Mb * ES) % 16 == 0 && (rows * Mb * ES) % 16 == 0;
          const bool sb = !gram && dense_b && (row0 * Nb * ES) % 16 == 0 && (rows * Nb * ES) % 16 == 0;
          if (pw == 0 && lane == 0 && (sa || sb)) {
            mbar_expect_tx(&raw_full[rs], (uint32_t)(((sa ? rows * Mb : 0) + (sb ? rows * Nb : 0)) * ES));
            if (sa) bulk_g2s(dA, Ab + row0 * p.lda, (uint32_t)(rows * Mb * ES), &raw_full[rs]);
            if (sb) bulk_g2s(dB, Bb + row0 * ldb, (uint32_t)(rows * Nb * ES), &raw_full[rs]);
          }
          if (p.bulk) {
            const int ca = Mb * ES / 16, cb = Nb * ES / 16;  // <= 32
            if (!sa && lane < ca)
              for (int r = pw; r < rows; r += 3)
                cp_async16(dA + r * rsa + lane * (16 / ES), Ab + (row0 + r) * p.lda + lane * (16 / ES));
            if (!gram && !sb && lane < cb)
              for (int r = pw; r < rows; r += 3)
                cp_async16(dB + r * rsb + lane * (16 / ES), Bb + (row0 + r) * ldb + lane * (16 / ES));
          }
          if (!sa && !p.bulk)
            for (int e = 32 * pw + lane; e < rows * Mb; e += 96) {
              const int r = e / Mb, c = e - r * Mb;
              if constexpr (ES == 8)
                cp_async8(dA + r * rsa + c, Ab + (row0 + r) * p.lda + c);
              else
                cp_async4(dA + r * rsa + c, Ab + (row0 + r) * p.lda + c);
            }
          if (!gram && !sb && !p.bulk)
            for (int e = 32 * pw + lane; e < rows * Nb; e += 96) {
              const int r = e / Nb, c = e - r * Nb;
              if constexpr (ES == 8)
                cp_async8(dB + r * rsb + c, Bb + (row0 + r) * ldb + c);
              else
                cp_async4(dB + r * rsb + c, Bb + (row0 + r) * ldb + c);
            }
          cp_async_arrive(&raw_full[rs]);
        }
        issued = ls + 1;
      }
      // copies in flight must land before the CTA ends
      if (!allbulk) asm volatile("cp.async.wait_all;" ::: "memory");
      if (lane == 0)
        for (int ls = max(0, issued - R); ls < issued; ls++)
          mbar_wait_bounded(&raw_full[ls % R], (uint32_t)((ls / R) & 1), nullptr);
    } else if (warp == WMMA) {
      // ---- MMA issuer: one elected lane, descriptors from a base and constant offsets; opens and closes
      // the periods ---------------------------------------------------------------------------------------
      const uint32_t idesc = (1u << 4) | ((128u >> 3) << 17) | ((128u >> 4) << 24);  // F32 <- F16 x F16
      int ds = 0, periods = 0, ls = 0, pstart = 0, epoch = 0, epoch_periods = 0;
      uint32_t dph = 0;
      for (; ls < nst; ls++) {
        if (!__all_sync(0xffffffffu, wait_ab(&dfull[ds], dph, abort_f, p.err, 32))) break;
        const bool raised = vflag[ls & 3] == ls + 1;
        const bool start = ls == 0 || raised || ls - pstart >= PSTAGES || epoch_periods >= MAX_EPOCH_PERIODS;
        if (start) {
          if (raised || ls == 0 || epoch_periods >= MAX_EPOCH_PERIODS) {
            epoch++;
            epoch_periods = 0;
          }
          epoch_periods++;
          pstart = ls;
          const int buf = periods & 1;
          if (periods >= 2 &&
              !__all_sync(0xffffffffu, wait_ab(&tempty[buf], (uint32_t)(((periods >> 1) - 1) & 1), abort_f, p.err)))
            break;
          if (elect_one()) {
            if (periods) {  // the period before is complete
              mend[buf ^ 1] = ls;
              mma_commit(&tfull[buf ^ 1]);
              mbar_arrive(&tfull[buf ^ 1]);
            }
            mstart[buf] = ls;
            mepoch[buf] = epoch;
          }
          __syncwarp();
          periods++;
        }
        tc_after();
        const uint32_t a0 = smem_u32(dig) + ds * SLOT;
        if (elect_one()) {
          const uint32_t da = (uint32_t)desc(a0, LBO_A), db = (uint32_t)desc(a0 + SLOT_A, LBO_B);  // planes are 1024 bytes apart
          const uint32_t d0 = tmem + ((periods - 1) & 1) * 256;
  #pragma unroll
          for (int i = -3; i <= 4; i++) {
            const uint32_t ai = da + 64 * slot_a(i);
            if (i <= 2)  // both keys: planes 2 - i .. 5 - i
              mma_f16(d0, ai, db + 64 * (2 - i), idesc + (16u << 17), i == -3 ? !start : 1u);
            else
              mma_f16(d0 + 128, ai, db + 64 * (4 - i), idesc, 1u);
          }
          mma_commit(&dempty[ds]);
        }
        __syncwarp();
        if (++ds == DSLOTS) {
          ds = 0;
          dph ^= 1u;
        }
      }
      // (the set that the closing arrival is made on must have been drained: a drain warp that had not
      // yet seen its last period would otherwise wait for a phase that is past)
      if (periods >= 2) wait_ab(&tempty[periods & 1], (uint32_t)(((periods >> 1) - 1) & 1), abort_f, p.err);
      __syncwarp();
      if (elect_one()) {
        const int buf = periods & 1;
        if (periods) {
          mend[buf ^ 1] = ls;
          mma_commit(&tfull[buf ^ 1]);
          mbar_arrive(&tfull[buf ^ 1]);
          mma_commit(bar_fin);
        }
        *nperiods = periods;
        mbar_arrive(&tfull[buf]);
        mbar_arrive(&tfull[buf]);
      }
      __syncwarp();
      if (periods) mbar_wait_bounded(bar_fin, 0, nullptr);  // every MMA has finished before the TMEM is released
    }
  } else if (warp >= SW) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
    // ---- drain: TMEM -> one int64 word per cell and lane half; FP64 where an epoch ends ---------------
    // cells: TMEM lane 32 q + lane (q = warp % 4), C columns [32 nh, 32 nh + 32)
    const int q = warp & 3, nh = (warp >> 2) & 1;
    const int hm = q >> 1;                  // 0: levels 2..5, 1: levels 6..9
    const int m = (32 * q + lane) & 63;
    // cells this warp keeps: folded stages keep the two diagonal quadrants only
    const bool live = !FOLD || (q & 1) == nh;
    const int mv = FOLD ? (m & 31) : m, nlim = min(32, Nb - (FOLD ? 0 : 32 * nh));
    long long acc[32];
#pragma unroll
    for (int x = 0; x < 32; x++) acc[x] = 0;
    int acc_epoch = -1, ea = 0, eb = 0;  // exponents of row m; of column 32 nh + lane
    bool flushed = false;
    double* part = p.partials + ((size_t)(blk * nchunks + chunk) * 2 + hm) * 4096 + (32 * nh) * 64 + m;
    for (int idx = 0;; idx++) {
      const int buf = idx & 1;
      int ok = 1;
      if (lane == 0) ok = wait_ab(&tfull[buf], (uint32_t)((idx >> 1) & 1), abort_f, p.err, 300);
      ok = __shfl_sync(0xffffffffu, ok, 0);
      const bool last = !ok || *nperiods == idx;
      const int ep = last ? -2 : mepoch[buf];
      if (ep != acc_epoch) {  // warp-uniform: the words so far are complete
        // (by integer instructions unless the result could leave the normal range: a conversion and a
        // multiplication of every cell on the FP64 pipe took 7.2 us at 32 x 32, 12.5 at 64 x 64)
        if (live && (acc_epoch >= 0 || last)) {
#pragma unroll
          for (int x = 0; x < 32; x++) {
            const int ebx = __shfl_sync(0xffffffffu, eb, x) - 1040 - (hm ? 32 : 0), es = ea - 1040 + ebx;
            if (mv < Mb && x < nlim) {
              const double v = (unsigned)(es + 1022) <= 1980u ? window_int(acc[x], es + 1086)
                                                              : (double)acc[x] * pow2i(ea - 1040) * pow2i(ebx);
              part[x * 64] = flushed ? part[x * 64] + v : v;
            }
            acc[x] = 0;
          }
          flushed = true;
        }
        if (last) break;
        acc_epoch = ep;
        const uint32_t first = (uint32_t)mstart[buf];
        auto exponent = [&](int i) {
          const uint64_t r = rec[i];
          return (int)(first >= (uint32_t)(r >> 32) ? r & 0xFFFFu : (r >> 16) & 0xFFFFu);
        };
        ea = exponent(m);
        eb = exponent((gram ? 0 : 64) + 32 * nh + lane);
      }
      __syncwarp();
      if (lane == 0) dprog[warp - SW] = mend[buf];
      tc_after();
      const uint32_t tb = tmem + ((uint32_t)(32 * q) << 16) + buf * 256 + 32 * nh;
      if (live) {
#pragma unroll
        for (int hp = 0; hp < 8; hp++) {
          uint32_t s0[4], s1[4], s2[4], s3[4];
          tmem_ld4(tb + hp * 4, s0);          // key 2, columns j   : level 2 / 6
          tmem_ld4(tb + 64 + hp * 4, s1);     // key 2, columns j+1 : level 3 / 7
          tmem_ld4(tb + 128 + hp * 4, s2);    // key 4, columns j   : level 4 / 8
          tmem_ld4(tb + 192 + hp * 4, s3);    // key 4, columns j+1 : level 5 / 9
          tmem_wait_ld();
#pragma unroll
          for (int x = 0; x < 4; x++) {
            long long a = acc[hp * 4 + x] + __float2int_rn(__uint_as_float(s3[x]));
            a += (long long)__float2int_rn(__uint_as_float(s2[x])) * (1 << 8);
            a += (long long)__float2int_rn(__uint_as_float(s1[x])) * (1 << 16);
            a += (long long)__float2int_rn(__uint_as_float(s0[x])) * (1 << 24);
            acc[hp * 4 + x] = a;
          }
        }
      }
      tc_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty[buf]);
    }
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
    // ---- slicers --------------------------------------------------------------------------------------
    // slicing unit: column c of A or B and 4 rows (Gram: column c of A and 2 rows).  All 16 rows of a
    // column lie with one warp, so that its exponent is this warp's own affair: a warp that raises
    // one marks the stage, and the MMA warp begins a new period there.
    const bool isB = !gram && warp >= SW / 2;
    const int c = gram ? 4 * warp + (lane & 3) : 8 * (warp & 7) + (lane & 7);
    const int sub = gram ? lane >> 2 : lane >> 3;
    constexpr int NR = GR == 1 ? 2 : 4;  // rows read (Gram among other blocks: 2 of them count)
    const int nrow = gram ? 2 : 4;
    // folded stages: plane row c holds column c % 32 of the stage's row half c / 32
    const int cact = FOLD ? (c & 31) : c, r0 = (FOLD ? ROWS * (c >> 5) : 0) + sub * nrow;
    const bool cvalid = cact < (isB ? Nb : Mb);
    const int cofs = (c >> 3) * 128 + (c & 7) * 16;  // row c of a digit plane (8-row core groups)
    // the column's exponent; unused columns read column 0 and never raise theirs
    uint32_t Ecur = cvalid ? 0u : 4000u;
    // FP64 exponent fields = own fields + EOFS; columns up to EMIN (zeros, subnormal numbers in
    // range) are sliced by the general code
    constexpr bool F32 = ES == 4;
    constexpr uint32_t EOFS = F32 ? 896 : 0, EMIN = EOFS + 64;
    // (FP32 columns that reach 2^124 too: infinities keep the exponent field of their FP64 value)
    bool slow = true;  // warp-uniform: a column of this warp is such a one
    const int rstr = isB ? rsb : rsa;
    const int tofs = (isB ? ROWS * W : 0) + r0 * rstr + (cvalid ? cact : 0);

    struct Unit {
      uint32_t hi[NR], lo[NR];  // the elements' bits (FP32: hi)
    };
    auto value = [](const Unit& u, int k) {
      return F32 ? (double)__uint_as_float(u.hi[k]) : __hiloint2double((int)u.hi[k], (int)u.lo[k]);
    };
    auto field = [](const Unit& u, int k) { return F32 ? (u.hi[k] >> 23) & 0xFFu : (u.hi[k] >> 20) & 0x7FFu; };
    int rs = -1, ds = -1, ok = 1, raised = 0;  // ok: every wait has ended in time; raised: stage of the last raise
    uint32_t rph = 1, dph = 1;
    const bool wvalid = __any_sync(0xffffffffu, cvalid);  // (a warp without a column has nothing to do)
    for (int ls = 0; wvalid && ls < nst; ls++) {
      Unit cur;
      if (++rs == R) rs = 0;
      if (rs == 0) rph ^= 1u;
      if (++ds == DSLOTS) ds = 0;
      if (ds == 0) dph ^= 1u;
      ok &= mbar_wait_warp(&raw_full[rs], rph, abort_f);
      const int rows = (int)min((int64_t)SR, p.K - (s_begin + ls) * SR);
      const TI* T = reinterpret_cast<const TI*>(raw + (size_t)rs * p.raw_stage) + tofs;
      auto get = [&](int k) {
        if constexpr (F32) {
          cur.hi[k] = __float_as_uint(T[k * rstr]);
        } else {
          const double x = T[k * rstr];
          cur.hi[k] = (uint32_t)__double2hiint(x);
          cur.lo[k] = (uint32_t)__double2loint(x);
        }
      };
#pragma unroll
      for (int k = 0; k < NR; k++) cur.hi[k] = cur.lo[k] = 0;
      if (rows == SR) {
#pragma unroll
        for (int k = 0; k < NR; k++)
          if (GR < 2 || k < nrow) get(k);
      } else {
#pragma unroll
        for (int k = 0; k < NR; k++)
          if ((GR < 2 || k < nrow) && r0 + k < rows) get(k);
      }
      // does an element exceed its column's exponent?
      int over = 0;
      if (!slow) {
#pragma unroll
        for (int k = 0; k < NR; k++) over |= (int)(Ecur - EOFS - field(cur, k));
        over = over < 0;
      } else {
#pragma unroll
        for (int k = 0; k < NR; k++) over |= exp_field(value(cur, k)) > Ecur;
      }
      over = __any_sync(0xffffffffu, over && cvalid);
      if (lane == 0) mbar_arrive(&raw_empty[rs]);
      if (over) {  // rare: raise the exponents that are exceeded
        uint32_t e = 0;
#pragma unroll
        for (int k = 0; k < NR; k++) e = max(e, exp_field(value(cur, k)));
        if (gram) e = max(e, __shfl_xor_sync(0xffffffffu, e, 4));
        e = max(e, __shfl_xor_sync(0xffffffffu, e, 8));
        e = max(e, __shfl_xor_sync(0xffffffffu, e, 16));
        // a record keeps two exponents: the drain of the periods before this warp's last raise has
        // read what it needs (those periods ended there, whatever this stage holds)
        for (uint32_t i = 0;; i++) {
          int done = 1;
#pragma unroll
          for (int w = 0; w < DW; w++) done &= dprog[w] >= raised;
          if (done || *abort_f) break;
          if (i >= (1u << 22)) {
            ok = 0;
            break;
          }
          __nanosleep(64);
        }
        __syncwarp();
        if (cvalid && e > Ecur) {
          const uint32_t raise = e > EMAX ? (uint32_t)NONFINITE : min(e + HEAD, EMAX);
          if (sub == 0) rec[(isB ? 64 : 0) + c] = ((uint64_t)(uint32_t)ls << 32) | (uint64_t)((Ecur << 16) | raise);
          Ecur = raise;
        }
        raised = ls;
        vflag[ls & 3] = ls + 1;
        slow = __any_sync(0xffffffffu, Ecur <= EMIN || (F32 && Ecur > EOFS + 254 && cvalid));
      }
      if (ls >= DSLOTS) ok &= mbar_wait_warp(&dempty[ds], dph ^ 1u, abort_f);
      // slice: digits relative to Ecur into slot ds
      unsigned char* sa = dig + (size_t)ds * SLOT;
      unsigned char* sb = sa + SLOT_A;
      if (cvalid) {
        uint64_t g[NR];
        if (!slow) {
#pragma unroll
          for (int k = 0; k < NR; k++)
            g[k] = fixed_fast<TI>(cur.hi[k], cur.lo[k], Ecur - EOFS - field(cur, k));
        } else {
#pragma unroll
          for (int k = 0; k < NR; k++) {
            uint32_t gh, gl;
            g_words(value(cur, k), Ecur, gh, gl);
            g[k] = ((uint64_t)gh << 32) | gl;
          }
        }
        SignPair sg[NR / 2];
#pragma unroll
        for (int pp = 0; pp < NR / 2; pp++) sg[pp] = sign_pair(cur.hi[2 * pp], cur.hi[2 * pp + 1]);
        // digits d = 2 gi + 1 and d + 1 of each element pair
        auto digits = [&](int gi, uint32_t (&w1)[NR / 2], uint32_t (&w2)[NR / 2]) {
#pragma unroll
          for (int pp = 0; pp < NR / 2; pp++) {
            const uint32_t x = gi < 2 ? (uint32_t)(g[2 * pp] >> 32) : (uint32_t)g[2 * pp];
            const uint32_t y = gi < 2 ? (uint32_t)(g[2 * pp + 1] >> 32) : (uint32_t)g[2 * pp + 1];
            digit_pairs2(x, y, gi & 1, sg[pp], w1[pp], w2[pp]);
          }
        };
        if (GR == 1 || (GR == 2 && gram)) {
          unsigned char* da = sa + (sub >> 2) * LBO_A + cofs + (sub & 3) * 4;
          unsigned char* db = sb + (sub >> 2) * LBO_B + cofs + (sub & 3) * 4;
#pragma unroll
          for (int gi = 0; gi < 4; gi++) {
            uint32_t w1[NR / 2], w2[NR / 2];
            digits(gi, w1, w2);
            const int d = 2 * gi + 1;
            *reinterpret_cast<uint32_t*>(da + slot_a(d) * 1024) = w1[0];
            *reinterpret_cast<uint32_t*>(db + d * 1024) = w1[0];
            *reinterpret_cast<uint32_t*>(da + slot_a(d + 1) * 1024) = w2[0];
            *reinterpret_cast<uint32_t*>(db + (d + 1) * 1024) = w2[0];
          }
        } else if constexpr (NR == 4) {
          unsigned char* dst = (isB ? sb + (sub >> 1) * LBO_B : sa + (sub >> 1) * LBO_A) + cofs + (sub & 1) * 8;
#pragma unroll
          for (int gi = 0; gi < 4; gi++) {
            uint32_t w1[NR / 2], w2[NR / 2];
            digits(gi, w1, w2);
            const int d = 2 * gi + 1;
            *reinterpret_cast<uint2*>(dst + (isB ? d : slot_a(d)) * 1024) = make_uint2(w1[0], w1[1]);
            *reinterpret_cast<uint2*>(dst + (isB ? d + 1 : slot_a(d + 1)) * 1024) = make_uint2(w2[0], w2[1]);
          }
        }
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&dfull[ds]);
      if (!__all_sync(0xffffffffu, ok)) {  // a wait ran out, here or in another warp
        *abort_f = 1;
        if (lane == 0) atomicExch(p.err, SKINNY_DEVERR_TIMEOUT);
        break;
      }
    }
  }

  tc_before();
  __syncthreads();
  // back to the registers of the launch (a warpgroup's warps have met since the first change)
  if (warp >= SW && warp < WPROD)
    asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
  else
    asm volatile("setmaxnreg.inc.sync.aligned.u32 72;");
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
  if (*abort_f) return;

  // the CTA's sum of a cell: levels 2..5 (half 0) plus levels 6..9 (half 1), into half 0; with
  // folded stages plus the second row half's quadrant
  double* part = p.partials + (size_t)(blk * nchunks + chunk) * 8192;
  for (int e = tid; e < Mb * Nb; e += THREADS) {
    const int cell = (e / Mb) * 64 + e % Mb;
    double v = part[cell] + part[4096 + cell];
    if (FOLD) v += part[cell + 32 * 64 + 32] + part[4096 + cell + 32 * 64 + 32];
    part[cell] = v;
  }

  // ---- cross-CTA finish, two levels: the last CTA of each group of GROUP chunks sums the group's
  // partials in chunk order; the last group to finish sums the group sums in group order and
  // applies alpha and beta (deterministic; the work is spread over the group finishers) -----------
  __threadfence();
  __syncthreads();
  __shared__ int s_last;
  const int ngroups = (nchunks + GROUP - 1) / GROUP, grp = chunk / GROUP;
  const int gsize = min(GROUP, nchunks - grp * GROUP);
  unsigned* gcount = p.counter + blk * 16;  // [grp] per group, [15] for the block
  if (tid == 0) s_last = (atomicAdd(gcount + grp, 1u) == (unsigned)(gsize - 1));
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  const double* P = p.partials + (size_t)blk * nchunks * 8192;           // [chunk][2][4096], half 0 = CTA sum
  double* G = p.partials + (size_t)gridDim.x * 8192 + (size_t)blk * 15 * 4096;  // [group][4096]
  for (int e = tid; e < Mb * Nb; e += THREADS) {
    const int cell = (e / Mb) * 64 + e % Mb;
    double v[GROUP];
#pragma unroll
    for (int i = 0; i < GROUP; i++) v[i] = i < gsize ? __ldcg(P + (size_t)(grp * GROUP + i) * 8192 + cell) : 0.0;
    double sum = 0.0;
#pragma unroll
    for (int i = 0; i < GROUP; i++)
      if (i < gsize) sum += v[i];
    G[(size_t)grp * 4096 + cell] = sum;
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) {
    gcount[grp] = 0u;
    s_last = (atomicAdd(gcount + 15, 1u) == (unsigned)(ngroups - 1));
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  for (int e = tid; e < Mb * Nb; e += THREADS) {
    const int mm = e % Mb, nn = e / Mb, cell = nn * 64 + mm;
    double v[15];
#pragma unroll
    for (int i = 0; i < 15; i++) v[i] = i < ngroups ? __ldcg(G + (size_t)i * 4096 + cell) : 0.0;
    double sum = 0.0;
#pragma unroll
    for (int i = 0; i < 15; i++)
      if (i < ngroups) sum += v[i];
    const int64_t ci = (int64_t)(W * bj + nn) * p.ldc + W * bi + mm;
    const int64_t cmi = (int64_t)(W * bi + mm) * p.ldc + W * bj + nn;
    const bool mirror = p.sym && bi < bj;  // Gram: the mirrored block holds the same sums
    if (p.out_f32) {  // the one rounding of an FP32 result
      float* C = static_cast<float*>(p.C);
      C[ci] = (float)(p.beta_zero ? p.alpha * sum : (double)C[ci] * p.beta + sum * p.alpha);
      if (mirror) C[cmi] = (float)(p.beta_zero ? p.alpha * sum : (double)C[cmi] * p.beta + sum * p.alpha);
    } else {
      double* C = static_cast<double*>(p.C);
      C[ci] = p.beta_zero ? p.alpha * sum : C[ci] * p.beta + sum * p.alpha;
      if (mirror) C[cmi] = p.beta_zero ? p.alpha * sum : C[cmi] * p.beta + sum * p.alpha;
    }
  }
  if (tid == 0) gcount[15] = 0u;
}

}  // namespace splitw

skinny_status split_wide(skinny_handle h, int64_t M, int64_t N, int64_t K, const double* A, int64_t lda,
                         const void* alpha, const double* B, int64_t ldb, const void* beta, double* C,
                         int64_t ldc, cudaStream_t st) {
  return split_wide_t(h, false, false, M, N, K, A, lda, alpha, B, ldb, beta, C, ldc, st);
}

// Row chunks of each of nblk blocks at most, and the workspace they take: two halves of 4096 cells a CTA, then the
// group sums.  Asked for whatever the rows, so that a capture with more of them finds it.
static int64_t split_wide_chunks(skinny_handle h, int64_t nblk) {
  return std::max<int64_t>(1, std::min<int64_t>(h->dev.sms / nblk, (int64_t)15 * splitw::GROUP));
}
static size_t split_wide_bytes(skinny_handle h, int64_t nblk) {
  return (size_t)(split_wide_chunks(h, nblk) * nblk * 2 + nblk * 15) * 4096 * 8;
}

// A product that AUTO leaves to the CUDA-core kernels for its few rows (4096 at least) allocates what more rows will
// take here, so that these can be captured into a graph after it on the same stream, as before the rule counted rows.
// False, and nothing allocated, in a capture or below 4096 rows.
bool split_wide_reserve(skinny_handle h, int64_t M, int64_t N, int64_t K, bool sym, cudaStream_t st) {
  using namespace splitw;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (K < 4096 || cudaStreamIsCapturing(st, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) {
    cudaGetLastError();
    return false;
  }
  const int64_t bm = (M + W - 1) / W, bn = (N + W - 1) / W, nblk = sym ? bm * (bm + 1) / 2 : bm * bn;
  workspace_ensure(h->ws[st], split_wide_bytes(h, nblk), st);  // (without room: as the larger call finds it)
  return true;
}

skinny_status split_wide_t(skinny_handle h, bool in_f32, bool out_f32, int64_t M, int64_t N, int64_t K,
                           const void* A, int64_t lda, const void* alpha, const void* B, int64_t ldb,
                           const void* beta, void* C, int64_t ldc, cudaStream_t st) {
  using namespace splitw;
  const int64_t es = in_f32 ? 4 : 8;
  if (M > 128 || N > 128) {
    set_error("split precision TSMTTSM: M, N <= 128");
    return SKINNY_UNSUPPORTED;
  }
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
  a.sym = (A == B) && (lda == ldb) && (M == N);
  a.bm = (int)((M + W - 1) / W);
  const int bn = (int)((N + W - 1) / W);
  a.nblk = a.sym ? a.bm * (a.bm + 1) / 2 : a.bm * bn;
  // bulk copies: 16-byte aligned rows whose block widths are 16-byte multiples
  const int64_t per16 = 16 / es;
  const bool aligned =
      (uintptr_t)A % 16 == 0 && (uintptr_t)B % 16 == 0 && lda % per16 == 0 && ldb % per16 == 0;
  a.bulk = aligned && M % per16 == 0 && N % per16 == 0;
  a.abase16 = (uintptr_t)A % 16 == 0;
  a.bbase16 = (uintptr_t)B % 16 == 0;
  a.raw_stage = (a.sym && a.nblk == 1) ? RAW_OP : 2 * RAW_OP;
  const bool fold = M <= W / 2 && N <= W / 2;  // 32-row stages folded into the 64-row planes
  const int64_t fixed = HDR + (int64_t)DSLOTS * SLOT;
  a.rstages = (int)std::min<int64_t>(MAXR, (h->dev.smem_optin - fixed) / a.raw_stage);
  if (a.rstages < 2) {
    set_error("split precision: stages do not fit in shared memory");
    return SKINNY_UNSUPPORTED;
  }
  const int smem = (int)(fixed + (int64_t)a.rstages * a.raw_stage);
  const int64_t srows = fold ? 2 * ROWS : ROWS;
  a.nstages = (K + srows - 1) / srows;
  const int64_t nchunks = std::max<int64_t>(1, std::min(a.nstages, split_wide_chunks(h, a.nblk)));
  const int64_t grid = nchunks * a.nblk;
  Workspace& ws = h->ws[st];
  skinny_status s = workspace_ensure(ws, split_wide_bytes(h, a.nblk), st);
  if (s != SKINNY_OK) return s;
  a.partials = (double*)ws.partials;
  a.counter = ws.counter;
  a.err = h->err;
  static SmemAttr attr[12];
  auto launch = [&](auto kernel, SmemAttr& at) {
    ensure_smem_attr(kernel, smem, at);
    kernel<<<(int)grid, THREADS, smem, st>>>(a);
  };
  const int gk = !a.sym ? 0 : (a.nblk == 1 ? 1 : 2);  // folded products have one block
#define SK_WIDE(T, I)                                                                                 \
  {                                                                                                   \
    if (fold)                                                                                         \
      gk ? launch(split_wide_kernel<T, true, 1>, attr[I]) : launch(split_wide_kernel<T, true, 0>, attr[I + 1]); \
    else if (gk == 0)                                                                                 \
      launch(split_wide_kernel<T, false, 0>, attr[I + 2]);                                            \
    else                                                                                              \
      gk == 1 ? launch(split_wide_kernel<T, false, 1>, attr[I + 3])                                   \
              : launch(split_wide_kernel<T, false, 2>, attr[I + 4]);                                  \
  }
  if (!in_f32) SK_WIDE(double, 0) else SK_WIDE(float, 6)
#undef SK_WIDE
  count_launch();
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_error(std::string("split wide tsmttsm launch: ") + cudaGetErrorString(e));
    return SKINNY_DEVICE_ERROR;
  }
  return SKINNY_OK;
}

}  // namespace skinny
