// S/H contraction on the 5th-generation tensor cores (tcgen05, sm_100a).
//
// For every job (A panel of 128 V rows, B panel of NB = 32 or 64 V rows, walker
// split) the kernel accumulates
//   D[r][h*NB + c] = sum_w V[a0+r][w] * W_h(w) * V[b0+c][w],   h = 0,1,2
// with W_0 = w1, W_1 = w1 sum|z|^2, W_2 = w1 sum|z|^4: one set of M=128 x N=3 NB
// MMAs produces the S, H2 and H4 blocks at once.  Complex Gram entries are
// recovered from the real products of the [Re; Im] row planes afterwards.
//
// Precision: each FP32 operand x is split x = hi + lo into two 16-bit terms,
// FP16 for LEMC_GRAM_TF32X3 (11 + 11 significant bits, as two TF32 terms carry, at
// twice their MMA rate and half their operand bytes) or BF16, and the products
// hi*hi + hi*lo + lo*hi (+ lo*lo) are summed.  FP16's range is met by a power-of-two
// scale per V row and per weight plane, from the row's largest magnitude (a bound
// on it, see row_bound_kernel), which puts the row's top at 2^15; terms below
// 2^-25 of that scale are lost, i.e. 2^-40 of the row's largest value, where a
// row's root mean square is at least its largest value over sqrt(walkers).  The
// scales are undone in FP64.  Measured against FP64 sums of the same V (largest
// normalised entry; FP16 here, TF32 before): N=50, 65536 walkers 4.9e-7, 5.6e-7;
// N=200, 8192 walkers 5.7e-7, 7.5e-7; N=100, 16384 walkers 8.6e-7, 9.3e-7.
// The tensor core's accumulation truncates (about -4e-8 per MMA step), so every
// `flush_every` K-chunks (default one: 64 walkers, four steps) the epilogue warps
// move the accumulators out of tensor memory into FP32 register sums
// (round-to-nearest; two buffers let the MMAs continue meanwhile).  NB = 32 keeps
// the corrections in columns of their own; NB = 64 has no room for them and adds
// them first, while the accumulator is small.  At the end each job adds its sums,
// in FP64, to its private slot in global memory.
//
// MMA shape: with A in tensor memory an MMA costs about 97 cycles for any N up to
// 128 and 106 at N=192, so NB = 64 issues three N=192 MMAs a K step and NB = 32 one
// N=192 (A_hi times the stacked [B_hi; B_lo]) and one N=96.
//
// Operand placement.  The A operand (hi and lo, 128 rows x one K-chunk) lives
// in tensor memory: the A converters write it with tcgen05.st and the MMAs
// read it from there, so shared memory only carries the raw TMA stages and
// the (weighted, split) B operand.
//
// Pipeline (896 threads, one CTA per SM, register shares moved by setmaxnreg):
//   warp 25      loader: tiled TMA loads per half K-chunk of 32 walkers (A panel,
//                B panel in 128-byte-swizzled rows, weight planes; rows past the
//                end are zero-filled by the TMA unit) into a ring of raw stages;
//   warps 8-15   A converters: thread = A row (TMEM lane) of one half of every
//                chunk; raw FP32 -> scaled hi/lo, stored with tcgen05.st;
//   warps 16-23  B converters: raw FP32 -> weighted, split hi/lo B operands in
//                128-byte-swizzled K-major shared-memory layout;
//   warp 24      allocates 512 TMEM columns, one lane issues tcgen05.mma;
//   warp 26      scheduler: makes the issuer's barrier waits and hands each
//                K-chunk to it through a named barrier;
//   warps 0-7    epilogue: TMEM lane quarter = warp % 4, column half = warp / 4.
// Tensor memory columns: accumulator buffers at 0 and 192, A stages at 384 and
// 448 (hi at +0, lo at +32).
//
// What bounds it: shared-memory bandwidth.  A 64-walker chunk at NB = 64 moves
// about 217 KB through it (TMA writes 49, converter reads 48, B operands 48 written
// and 72 read by the MMAs), 1700 cycles at 128 B/cycle against 1285 of MMA issue
// and about 2700 measured; feeding the loads from L2 alone changes nothing.
// Measured (B200, 65536 walkers): 2713 states 6.75 -> 3.0 ms, 526 states 0.76 ->
// 0.39 ms, 272 states (NB = 32) 0.256 -> 0.152 ms.  One converter warp per scheduler
// and operand: 4.1 ms; shared memory through generic pointers: 3.4 ms; slot updates
// by each thread along its own row: 0.2 ms a job.
// No load uses cluster multicast; every source is this GPU's own memory.
// Every mbarrier wait is bounded in time; on expiry the kernel records
// LEMC_ERR_TIMEOUT in the error word, skips its output and unwinds: the loader
// first waits (bounded) for the TMA copies it has in flight and the issuer for
// the MMAs it has committed, then the CTA frees its tensor memory and exits.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "lemc_internal.h"

namespace lemc {
namespace {

constexpr int kM = 128;            // A panel rows (MMA M)
constexpr int kPanel = 32;         // B rows of one tile of the tile list
constexpr int kPanelCols = 3 * kPanel;  // its output columns: [weight][row]
constexpr int KC = 64;             // samples per K-chunk: one 128-byte operand row
constexpr int kHalf = 32;          // samples per raw stage (half a K-chunk)
constexpr int kOpRowBytes = 128;   // one swizzle-128B row of split operands
constexpr int kOpStages = 2;
constexpr int kEpiWarps = 8;
constexpr int kAConvWarp0 = 8;     // warps 8-15: A converters (lane quarter = warp % 4)
constexpr int kBConvWarp0 = 16;    // warps 16-23: B converters
constexpr int kRawReaders = 8;     // converter warps that read one raw stage (4 A, 4 B)
constexpr int kConvWarps = 16;     // converter warps that fill one operand stage
constexpr int kMmaWarp = 24;
constexpr int kLoadWarp = 25;
constexpr int kSchedWarp = 26;     // does the issuer's barrier waits (see the MMA issuer)
constexpr int kThreads = 28 * 32;  // seven warpgroups; warp 27 only fills the last one
// Register shares after the roles split (setmaxnreg): 896 threads start with 72
// each, and 256 x 120 + 512 x 56 + 128 x 40 = 896 x 72.
constexpr int kLaunchRegs = 72, kEpiRegs = 120, kConvRegs = 56, kMiscRegs = 40;
static_assert(256 * kEpiRegs + 512 * kConvRegs + 128 * kMiscRegs <= kThreads * kLaunchRegs,
              "register split exceeds the launch's registers");
constexpr int kTmemCols = 512;
constexpr uint32_t kBufCols = 192; // accumulator buffers at columns 0 and 192
constexpr uint32_t kColA = 384;    // A stages at 384 + 64 s (hi +0, lo +32)
static_assert(2 * kBufCols <= kColA, "accumulator buffers overlap the A stages");
constexpr long long kWaitCycles = 4000000000LL;  // default wait bound, ~2 s at 1.9 GHz

// NB = B rows of a job: 64 (two adjacent tiles) or 32 (one).
template <int NB>
struct Cfg {
  static constexpr int N = 3 * NB;                      // output columns
  static constexpr int B_TILE = N * kOpRowBytes;        // bytes of the hi (or lo) B operand
  static constexpr int A_BYTES = kM * kHalf * 4;
  static constexpr int B_BYTES = NB * kHalf * 4;
  static constexpr int W_BYTES = 3 * kHalf * 4;
  static constexpr int RAW_STAGE = A_BYTES + B_BYTES + 1024;  // weights padded to 1 KB
  static constexpr int RAW_STAGES = NB == 64 ? 5 : 8;
};

template <int NB>
struct Smem {
  uint8_t raw[Cfg<NB>::RAW_STAGES][Cfg<NB>::RAW_STAGE];  // 1024-aligned stages
  uint8_t bop[kOpStages][2 * Cfg<NB>::B_TILE];           // B hi | B lo
  uint64_t raw_full[Cfg<NB>::RAW_STAGES];
  uint64_t raw_empty[Cfg<NB>::RAW_STAGES];
  uint64_t op_full[kOpStages];
  uint64_t op_empty[kOpStages];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint64_t done;
  int row_exp[kM];                // scale exponents of the A rows and output columns
  int col_exp[Cfg<NB>::N];
  uint32_t tmem_base;
  int abort_flag;
};
static_assert(sizeof(float) * kM * (Cfg<64>::N + 1) <= sizeof(Smem<64>::raw) &&
                  sizeof(float) * kM * (Cfg<32>::N + 1) <= sizeof(Smem<32>::raw), "output staging");

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void mbar_arrive_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}

// CTA named barriers (0 is __syncthreads), 64 threads each: ids 1/2 hand
// K-chunk c (by parity) from the scheduler warp to the MMA warp ("ready"),
// ids 3/4 return it ("issued"), so neither warp can run two chunks ahead of
// the other and every barrier completes with exactly 32 + 32 threads.
__device__ __forceinline__ void named_arrive(int id) {
  asm volatile("bar.arrive %0, 64;" ::"r"(id) : "memory");
}
__device__ __forceinline__ void named_sync(int id) {
  asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory");
}

// One test of a barrier phase; the hardware may suspend the thread up to the hint,
// which keeps the waiting warps from filling the issue slots with polls.
constexpr uint32_t kWaitHintNs = 20000;
__device__ __forceinline__ bool mbar_try(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity), "r"(kWaitHintNs)
      : "memory");
  return ok != 0;
}

// Bounded wait; returns false (raising the CTA abort flag and the global error
// word) when the phase does not complete within `limit` cycles or another
// role gave up.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int* abort_flag, int* err,
                                          long long limit) {
  // a few tests for each look at the clock and the flag: up to two dozen warps
  // wait at a time, and their polls take issue slots from the converters
  auto test = [&]() {
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (mbar_try(bar, parity)) return true;
    return false;
  };
  if (test()) return true;
  const long long t0 = clock64();
  while (!test()) {
    if (*(volatile int*)abort_flag) return false;
    if (clock64() - t0 > limit) {
      *(volatile int*)abort_flag = 1;
      if (err) atomicExch(err, LEMC_ERR_TIMEOUT);
      return false;
    }
  }
  return true;
}

// Bounded wait for this CTA's own asynchronous work (its TMA copies, its
// committed MMAs) that does not give up when another role aborted: those
// operations complete by themselves, and the CTA must not release shared or
// tensor memory while they are in flight.
__device__ __forceinline__ void mbar_drain(uint64_t* bar, uint32_t parity, int* err, long long limit) {
  const long long t0 = clock64();
  while (!mbar_try(bar, parity)) {
    if (clock64() - t0 > limit) {
      if (err) atomicExch(err, LEMC_ERR_TIMEOUT);
      return;
    }
  }
}

// Tiled 2D TMA load (no multicast) completing on an mbarrier transaction count.
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y,
                                            uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar))
      : "memory");
}

// UMMA shared-memory descriptor: K-major, 128-byte swizzle, 8-row groups
// 1024 bytes apart (SBO), LBO 1 (unused for swizzled K-major), version 1.
__device__ __forceinline__ uint64_t sw128_desc(uint32_t saddr) {
  uint64_t d = 0;
  d |= uint64_t((saddr >> 4) & 0x3FFF);
  d |= uint64_t(1) << 16;
  d |= uint64_t((1024 >> 4) & 0x3FFF) << 32;
  d |= uint64_t(1) << 46;
  d |= uint64_t(2) << 61;
  return d;
}

// Instruction descriptor: dense, FP32 accumulate, A/B K-major, M=128, N=n.
__host__ __device__ constexpr uint32_t make_idesc(uint32_t ab_format, int n) {
  return (1u << 4) | (ab_format << 7) | (ab_format << 10) | (uint32_t(n >> 3) << 17) |
         (uint32_t(kM >> 4) << 24);
}

// D (TMEM) += A (TMEM, 128 lanes x K) * B (shared memory descriptor), 16-bit operands
__device__ __forceinline__ void mma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc,
                                       uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
      "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate));
}

// 16 consecutive 32-bit columns of this thread's TMEM lane
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
      "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]),
      "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_wait_st() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   smem_u32(bar))
               : "memory");
}

__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void fence_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait_ld() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// byte offset of 16-byte chunk `c` of row `r` in a 128B-swizzled K-major tile
__device__ __forceinline__ uint32_t sw128_off(int r, int c) {
  return uint32_t((r >> 3) * 1024 + (r & 7) * 128 + ((c ^ (r & 7)) << 4));
}

// Two samples x0, x1 as packed 16-bit pairs hi + lo: hi = x rounded to nearest,
// lo = x - hi (exact in FP32) rounded to nearest.  FP16 (22 significant bits) or
// BF16 (16).
template <bool HALF>
__device__ __forceinline__ void split2(float2 x, uint32_t& hi, uint32_t& lo) {
  const float2 m1 = make_float2(-1.f, -1.f);
  if (HALF) {
    const __half2 h = __float22half2_rn(x);
    const float2 r = __ffma2_rn(__half22float2(h), m1, x);  // x - hi, exact
    const __half2 l = __float22half2_rn(r);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = *reinterpret_cast<const uint32_t*>(&l);
  } else {
    const __nv_bfloat162 h = __float22bfloat162_rn(x);
    const float2 r = __ffma2_rn(__bfloat1622float2(h), m1, x);
    const __nv_bfloat162 l = __float22bfloat162_rn(r);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = *reinterpret_cast<const uint32_t*>(&l);
  }
}

// Power-of-two scales: a row (or weight plane) whose largest magnitude has the
// FP32 bits `max_bits` is multiplied by 2^row_exp, which brings the maximum into
// [2^14, 2^15) (weights: below 1), inside FP16's range; both steps and the
// division afterwards are exact.  A zero row keeps 1; an infinite or NaN one
// stays non-finite.
constexpr int kRowTop = 14;
__device__ __forceinline__ int scale_exp(uint32_t max_bits, int top) {
  if (max_bits == 0u) return 0;
  const int k = top - (int(max_bits >> 23) - 127);
  return max(-126, min(126, k));
}
__device__ __forceinline__ float pow2f(int k) { return __uint_as_float(uint32_t(k + 127) << 23); }
__device__ __forceinline__ double pow2d(int k) {
  return __longlong_as_double((long long)(k + 1023) << 52);
}

struct TcArgs {
  const float* V;
  int ldv;
  int total_rows;
  const float* rec_w;   // weight planes, stride ldw (256-byte aligned rows)
  int ldw;
  const TcTile* tiles;
  const uint32_t* range;  // bits of max |V row| [total_rows], then of max |W_h| [3]
  double* partials;
  int n_chunks_total;   // K-chunks over the padded walker range
  int n_splits;
  int flush_every;
  int passes;           // 3 or 4
  int* err;
  long long wait_cycles;  // bound of every mbarrier wait
  int hold_loads;         // test hook: the loader issues nothing (the waits then expire)
};

template <int R>
__device__ __forceinline__ void regs_inc() {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(R));
}
template <int R>
__device__ __forceinline__ void regs_dec() {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(R));
}

template <bool HALF, int NB>
__global__ void __launch_bounds__(kThreads, 1)
gram_tc_kernel(const TcArgs a, const __grid_constant__ CUtensorMap tmA,
               const __grid_constant__ CUtensorMap tmB, const __grid_constant__ CUtensorMap tmW) {
  using C = Cfg<NB>;
  constexpr int NKSTEP = kOpRowBytes / 32;   // one MMA consumes 32 bytes (16 samples) of K
  constexpr uint32_t IDESC = make_idesc(HALF ? 0u : 1u, C::N);
  constexpr uint32_t IDESC2 = make_idesc(HALF ? 0u : 1u, 192);
  constexpr int RS = C::RAW_STAGES;

  extern __shared__ __align__(1024) uint8_t smem_raw[];
  // aligned by an offset, not by rounding a pointer through an integer: that
  // loses the address space, and every access becomes a generic one
  Smem<NB>* sm = reinterpret_cast<Smem<NB>*>(smem_raw + (-smem_u32(smem_raw) & 1023u));

  const TcTile tile = a.tiles[blockIdx.x];
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int per = (a.n_chunks_total + a.n_splits - 1) / a.n_splits;
  const int c_beg = tile.ksplit * per;
  const int c_end = min(a.n_chunks_total, c_beg + per);
  const int nch = max(0, c_end - c_beg);
  const int F = a.flush_every;
  const int nint = (nch + F - 1) / F;

  if (threadIdx.x == 0) {
    for (int s = 0; s < RS; ++s) {
      mbar_init(&sm->raw_full[s], 1);
      mbar_init(&sm->raw_empty[s], kRawReaders);
    }
    for (int s = 0; s < kOpStages; ++s) {
      mbar_init(&sm->op_full[s], kConvWarps);
      mbar_init(&sm->op_empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&sm->acc_full[b], 1);
      mbar_init(&sm->acc_empty[b], kEpiWarps);
    }
    mbar_init(&sm->done, 1);
    sm->abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (threadIdx.x < C::N) {
    const int h = int(threadIdx.x) / NB, rb = tile.col0 + int(threadIdx.x) % NB;
    const int eb = rb < a.total_rows ? scale_exp(a.range[rb], kRowTop) : 0;
    sm->col_exp[threadIdx.x] = eb + scale_exp(a.range[a.total_rows + h], -1);
  }
  if (threadIdx.x < kM) {
    const int row = tile.row0 + int(threadIdx.x);
    sm->row_exp[threadIdx.x] = row < a.total_rows ? scale_exp(a.range[row], kRowTop) : 0;
  }
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&sm->tmem_base)),
                 "r"(kTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sm->tmem_base;
  int* abort_flag = &sm->abort_flag;
  // warp-uniform bounded wait
  auto wait_all = [&](uint64_t* bar, uint32_t parity) {
    return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag, a.err, a.wait_cycles)) != 0;
  };
  // one arrival per warp, after every lane's part is done
  auto arrive_warp = [&](uint64_t* bar) {
    __syncwarp();
    if (lane == 0) mbar_arrive(bar);
  };

  if (warp >= kMmaWarp) {
    regs_dec<kMiscRegs>();
    if (warp == kLoadWarp) {
      // ------------------------------- loader ------------------------------
      if (lane == 0) {
        constexpr uint32_t tx_bytes = uint32_t(C::A_BYTES + C::B_BYTES + C::W_BYTES);
        const int nh = 2 * nch;
        int issued = 0, s = 0;
        uint32_t ph = 1u;
        for (int hc = 0; hc < nh && !a.hold_loads; ++hc) {
          if (!mbar_wait(&sm->raw_empty[s], ph, abort_flag, a.err, a.wait_cycles)) break;
          const int k0 = c_beg * KC + hc * kHalf;
          uint8_t* dst = sm->raw[s];
          mbar_arrive_tx(&sm->raw_full[s], tx_bytes);
          tma_load_2d(dst, &tmA, k0, tile.row0, &sm->raw_full[s]);
          tma_load_2d(dst + C::A_BYTES, &tmB, k0, tile.col0, &sm->raw_full[s]);
          tma_load_2d(dst + C::A_BYTES + C::B_BYTES, &tmW, k0, 0, &sm->raw_full[s]);
          ++issued;
          if (++s == RS) {
            s = 0;
            ph ^= 1u;
          }
        }
        // the copies still in flight land before the CTA may exit, whatever the
        // other roles did: the last one issued into each stage
        for (int hc = max(0, issued - RS); hc < issued; ++hc)
          mbar_drain(&sm->raw_full[hc % RS], uint32_t(hc / RS) & 1u, a.err, a.wait_cycles);
      }
      __syncwarp();
    } else if (warp == kSchedWarp) {
      // ----------------------------- scheduler -----------------------------
      // An mbarrier test made by the thread that has just issued tcgen05.commit
      // stalls until the committed MMAs retire, which drains the tensor pipe every
      // K-chunk.  So this warp makes the issuer's waits (operand stage full;
      // accumulator buffer empty at the start of a flush group) and hands each chunk
      // over through a named barrier, which needs no shared-memory access.  It
      // arrives once per chunk whatever happens (after an abort without
      // waiting), so the issuer's barrier always completes.
      int s = 0, b = 0, f = 0;
      uint32_t ph_op = 0, ph_acc = 0;
      for (int c = 0; c < nch; ++c) {
        if (c >= 2) named_sync(3 + (c & 1));  // chunk c-2 issued: ids 1/2 are free again
        if (lane == 0 && !*(volatile int*)abort_flag) {
          bool ok = true;
          if (f == 0) {
            ok = mbar_wait(&sm->acc_empty[b], ((ph_acc >> b) & 1u) ^ 1u, abort_flag, a.err, a.wait_cycles);
            ph_acc ^= 1u << b;
          }
          if (ok) mbar_wait(&sm->op_full[s], ph_op, abort_flag, a.err, a.wait_cycles);
        }
        __syncwarp();
        named_arrive(1 + (c & 1));
        if (++f == F || c == nch - 1) {
          f = 0;
          b ^= 1;
        }
        if (++s == kOpStages) {
          s = 0;
          ph_op ^= 1u;
        }
      }
      for (int c = max(0, nch - 2); c < nch; ++c) named_sync(3 + (c & 1));
    } else if (warp == kMmaWarp) {
      // ---------------------------- MMA issuer -----------------------------
      // One thread issues every MMA, so its per-MMA instruction count bounds the
      // tensor-core issue rate: all descriptors and TMEM addresses are formed
      // once per stage, a K step only adds a constant, and the flush schedule is
      // kept in counters.  Its waits are made by the scheduler warp.
      const bool four = a.passes > 3;
      static_assert(kOpStages == 2, "the issuer keeps one descriptor per operand stage");
      const uint64_t bdesc0 = sw128_desc(smem_u32(sm->bop[0]));
      const uint64_t bdesc1 = sw128_desc(smem_u32(sm->bop[1]));
      constexpr uint64_t kLoDesc = uint64_t(C::B_TILE >> 4);  // B lo tile, in descriptor units
      int s = 0, b = 0, f = 0;          // operand stage, accumulator buffer, chunk within flush group
      int issued = 0;
      for (int c = 0; c < nch; ++c) {
        named_sync(1 + (c & 1));
        const bool go = !*(volatile int*)abort_flag;
        if (lane == 0 && go) {
          tc_fence_after();
          const uint64_t bh = s ? bdesc1 : bdesc0, bl = bh + kLoDesc;
          const uint32_t ahi = tmem + kColA + uint32_t(s * 64), alo = ahi + 32;
          const uint32_t d = tmem + uint32_t(b) * kBufCols;
          // the first MMA of a flush group overwrites the buffer.  K step ks: B
          // advances 32 bytes (2 descriptor units), A 8 TMEM columns
          const uint32_t acc_d = f == 0 ? 0u : 1u;
          if constexpr (NB == 64) {
            // the small products first, while the accumulator is small
#pragma unroll
            for (int ks = 0; ks < NKSTEP; ++ks) {
              mma_ts(d, ahi + 8 * ks, bl + 2 * ks, IDESC, ks == 0 ? acc_d : 1u);
              mma_ts(d, alo + 8 * ks, bh + 2 * ks, IDESC, 1u);
              if (four) mma_ts(d, alo + 8 * ks, bl + 2 * ks, IDESC, 1u);
            }
#pragma unroll
            for (int ks = 0; ks < NKSTEP; ++ks) mma_ts(d, ahi + 8 * ks, bh + 2 * ks, IDESC, 1u);
          } else {
            // hi*hi | corrections side by side; the B hi and lo tiles are
            // contiguous, so bh with N=192 spans both
            const uint32_t dc = d + C::N;
#pragma unroll
            for (int ks = 0; ks < NKSTEP; ++ks) {
              mma_ts(d, ahi + 8 * ks, bh + 2 * ks, IDESC2, ks == 0 ? acc_d : 1u);
              mma_ts(dc, alo + 8 * ks, bh + 2 * ks, IDESC, 1u);
              if (four) mma_ts(dc, alo + 8 * ks, bl + 2 * ks, IDESC, 1u);
            }
          }
          umma_commit(&sm->op_empty[s]);
          if (f + 1 == F || c == nch - 1) umma_commit(&sm->acc_full[b]);
          ++issued;
        }
        __syncwarp();
        named_arrive(3 + (c & 1));
        if (++f == F || c == nch - 1) {
          f = 0;
          b ^= 1;
        }
        if (++s == kOpStages) s = 0;
      }
      if (lane == 0 && issued > 0) {
        // every issued MMA must retire before TMEM is released
        umma_commit(&sm->done);
        mbar_drain(&sm->done, 0u, a.err, a.wait_cycles);
      }
      __syncwarp();
    }
  } else if (warp >= kAConvWarp0) {
    // Four warps of each kind take the first half of every K-chunk, four the
    // second: one warp per scheduler and operand is latency-bound (about five
    // cycles an instruction), 2330 cycles a chunk for B against 1370 of MMAs.
    regs_dec<kConvRegs>();
    const int half = (warp >> 2) & 1;
    int rs = half;  // raw stage of (chunk c, half): 2 c + half
    uint32_t ph_raw = 0u, ph_op = 1u;
    if (warp < kBConvWarp0) {
      // --------------------------- A converters ----------------------------
      // Thread = A row r = TMEM lane; its raw row segment is a 128-byte
      // swizzled row (16-byte chunk j of row r at r*128 + ((j ^ (r & 7)) << 4)).
      const int quarter = warp & 3;
      const int r = quarter * 32 + lane;
      const uint32_t a_col = tmem + (uint32_t(quarter * 32) << 16) + kColA + uint32_t(half * 16);
      const float sc1 = pow2f(sm->row_exp[r]);
      const float2 sc = make_float2(sc1, sc1);
      for (int c = 0; c < nch; ++c) {
        const int os = c & 1;
        if (!wait_all(&sm->raw_full[rs], ph_raw)) break;
        const uint8_t* raw = sm->raw[rs] + r * 128;
        // 16 TMEM columns of 2 samples each
        uint32_t hv[16], lv[16];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const float4 f = *reinterpret_cast<const float4*>(raw + ((q ^ (r & 7)) << 4));
          split2<HALF>(__fmul2_rn(make_float2(f.x, f.y), sc), hv[2 * q], lv[2 * q]);
          split2<HALF>(__fmul2_rn(make_float2(f.z, f.w), sc), hv[2 * q + 1], lv[2 * q + 1]);
        }
        arrive_warp(&sm->raw_empty[rs]);
        if ((rs += 2) >= RS) {
          rs -= RS;
          ph_raw ^= 1u;
        }
        if (!wait_all(&sm->op_empty[os], ph_op)) break;
        ph_op ^= uint32_t(os);
        tc_fence_after();
        tmem_st16(a_col + uint32_t(os * 64), hv);
        tmem_st16(a_col + uint32_t(os * 64) + 32, lv);
        tmem_wait_st();
        tc_fence_before();
        arrive_warp(&sm->op_full[os]);
      }
    } else {
      // --------------------------- B converters ----------------------------
      // NB rows x 4 operand chunks (8 samples) x 3 weight planes per raw stage.
      // A thread's items share one column range, so the weight products are
      // formed once; eight consecutive lanes hold eight rows of one chunk, which
      // the 128-byte swizzle spreads over all banks, reading and writing.
      const int t = threadIdx.x & 127;
      constexpr int kItems = NB / 32;
      const int ch = (t >> 3) & 3, rb0 = (t & 7) + 8 * (t >> 5);
      float sc[kItems], ws[3];
#pragma unroll
      for (int q = 0; q < kItems; ++q) {
        const int row = tile.col0 + rb0 + 32 * q;
        sc[q] = pow2f(row < a.total_rows ? scale_exp(a.range[row], kRowTop) : 0);
      }
#pragma unroll
      for (int h = 0; h < 3; ++h) ws[h] = pow2f(scale_exp(a.range[a.total_rows + h], -1));
      for (int c = 0; c < nch; ++c) {
        const int os = c & 1;
        if (!wait_all(&sm->op_empty[os], ph_op)) break;
        ph_op ^= uint32_t(os);
        uint8_t* b_hi = sm->bop[os];
        uint8_t* b_lo = b_hi + C::B_TILE;
        if (!wait_all(&sm->raw_full[rs], ph_raw)) break;
        const uint8_t* rawb = sm->raw[rs] + C::A_BYTES;
        const float4* rw = reinterpret_cast<const float4*>(rawb + C::B_BYTES) + 2 * ch;
        float2 x[kItems][4];
#pragma unroll
        for (int q = 0; q < kItems; ++q) {
          const int rb = rb0 + 32 * q;
          const float2 sq = make_float2(sc[q], sc[q]);
#pragma unroll
          for (int v = 0; v < 2; ++v) {
            const float4 g = *reinterpret_cast<const float4*>(
                rawb + rb * 128 + (((2 * ch + v) ^ (rb & 7)) << 4));
            x[q][2 * v] = __fmul2_rn(make_float2(g.x, g.y), sq);
            x[q][2 * v + 1] = __fmul2_rn(make_float2(g.z, g.w), sq);
          }
        }
#pragma unroll
        for (int h = 0; h < 3; ++h) {
          const float2 wsh = make_float2(ws[h], ws[h]);
          float2 ww[4];
#pragma unroll
          for (int v = 0; v < 2; ++v) {
            const float4 o = rw[v];
            ww[2 * v] = make_float2(o.x, o.y);
            ww[2 * v + 1] = make_float2(o.z, o.w);
            if (h > 0) {
              const float4 f = rw[h * (kHalf / 4) + v];
              ww[2 * v] = __fmul2_rn(ww[2 * v], make_float2(f.x, f.y));
              ww[2 * v + 1] = __fmul2_rn(ww[2 * v + 1], make_float2(f.z, f.w));
            }
            ww[2 * v] = __fmul2_rn(ww[2 * v], wsh);
            ww[2 * v + 1] = __fmul2_rn(ww[2 * v + 1], wsh);
          }
#pragma unroll
          for (int q = 0; q < kItems; ++q) {
            uint32_t hi[4], lo[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) split2<HALF>(__fmul2_rn(x[q][e], ww[e]), hi[e], lo[e]);
            const uint32_t off = sw128_off(h * NB + rb0 + 32 * q, half * 4 + ch);
            *reinterpret_cast<uint4*>(b_hi + off) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
            *reinterpret_cast<uint4*>(b_lo + off) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
          }
        }
        arrive_warp(&sm->raw_empty[rs]);
        if ((rs += 2) >= RS) {
          rs -= RS;
          ph_raw ^= 1u;
        }
        fence_async_smem();
        arrive_warp(&sm->op_full[os]);
      }
    }
  } else {
    // ------------------------------- epilogue ------------------------------
    regs_inc<kEpiRegs>();
    constexpr int EC = C::N / 2;                // output columns per thread
    const int quarter = warp & 3;
    const int part0 = (warp >> 2) * EC;         // first output column of this thread
    // Plain FP32 running sums (round-to-nearest, unbiased): over n flushes the
    // relative rounding error is ~2^-24 sqrt(n) / 3 per split, and the FP64
    // sum over splits averages it down further.
    float2 sum[EC / 2];
#pragma unroll
    for (int i = 0; i < EC / 2; ++i) sum[i] = make_float2(0.f, 0.f);
    const uint32_t lane_base = uint32_t(quarter * 32) << 16;
    bool ok = true;
    for (int q = 0; q < nint; ++q) {
      const int b = q & 1;
      if (!(ok = wait_all(&sm->acc_full[b], uint32_t(q >> 1) & 1u))) break;
      tc_fence_after();
      const uint32_t ta = tmem + lane_base + uint32_t(b) * kBufCols + uint32_t(part0);
#pragma unroll
      for (int part = 0; part < EC / 16; ++part) {
        uint32_t v0[16], v1[16];
        tmem_ld16(ta + part * 16, v0);
        // NB == 32: column j's corrections sit at j + 96
        if constexpr (NB == 32) tmem_ld16(ta + C::N + part * 16, v1);
        tmem_wait_ld();
        if (part == EC / 16 - 1) {
          // every column of this buffer is in registers: the MMAs may reuse it
          tc_fence_before();
          arrive_warp(&sm->acc_empty[b]);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          float2& t = sum[part * 8 + i];
          t = __fadd2_rn(t, make_float2(__uint_as_float(v0[2 * i]), __uint_as_float(v0[2 * i + 1])));
          if constexpr (NB == 32)
            t = __fadd2_rn(t, make_float2(__uint_as_float(v1[2 * i]), __uint_as_float(v1[2 * i + 1])));
        }
      }
    }
    // Stage the sums in the raw buffers (every copy into them has landed and been
    // read once the last accumulator is full), then undo the scales (exact powers
    // of two) in FP64 and add them to the slots along rows: a thread's own
    // row-wise update touches 32 rows, 768 bytes apart, per warp access, and
    // cost 60 us a job.
    if (nch > 0) {
      float* out = reinterpret_cast<float*>(sm->raw);
      if (ok) {
        float* mine = out + (quarter * 32 + lane) * (C::N + 1) + part0;
#pragma unroll
        for (int j = 0; j < EC / 2; ++j) {
          mine[2 * j] = sum[j].x;
          mine[2 * j + 1] = sum[j].y;
        }
      }
      asm volatile("bar.sync 5, %0;" ::"n"(kEpiWarps * 32) : "memory");
      if (ok && !*(volatile int*)abort_flag) {
        double* slot = a.partials + (size_t)tile.slot * (kM * kPanelCols);
#pragma unroll 4
        for (int e = threadIdx.x; e < tile.panels * kM * kPanelCols; e += kEpiWarps * 32) {
          const int i = (e / kPanelCols) % kM, j = e % kPanelCols;
          const int col = j / kPanel * NB + e / (kM * kPanelCols) * kPanel + j % kPanel;  // [h][rb]
          // one CTA per slot and launch: the reduction keeps the sum deterministic
          // and needs no round trip to L2
          atomicAdd(slot + e, double(out[i * (C::N + 1) + col]) *
                                  pow2d(-(sm->row_exp[i] + sm->col_exp[col])));
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols));
  }
}

// Fold the partial slots into the per-sector complex Gram planes:
//   G_h[a][b] += sum_splits [C(re a, re b) + C(im a, im b)]
//              + i [C(re a, im b) - C(im a, re b)]
// with C(r1, r2) read from the tile that covers A row r1 and B row r2, or
// from the tile of C(r2, r1) when that one was skipped by symmetry.  Each
// sector knows its tiles: first tile index, A/B row origins and the number
// of B panels (TcSector); A slice x of a sector holds B panels 4x .. nb-1.
__global__ void gram_tc_reduce_kernel(const double* __restrict__ partials,
                                      const TcTile* __restrict__ tiles,
                                      const TcSector* __restrict__ secs, int n_sec, int n_tiles,
                                      int n_splits, double* __restrict__ gram, size_t plane) {
  const int s = blockIdx.y;
  if (s >= n_sec) return;
  const TcSector sc = secs[s];
  const int D = sc.dim;
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= D * D) return;
  const int a = idx / D, b = idx % D;
  auto C = [&](int r1, int r2, int h) {
    // A slice x holds B panels y >= 4 x only (the others are transposes)
    if ((r2 - sc.b_base) / kPanel < 4 * ((r1 - sc.a_base) / kM)) {
      const int r = r1;
      r1 = r2;
      r2 = r;
    }
    const int x = (r1 - sc.a_base) / kM, y = (r2 - sc.b_base) / kPanel;
    const int t = sc.tile0 + x * sc.n_bpanels - 2 * x * (x - 1) + (y - 4 * x);
    double v = 0.0;
    if (t < 0 || t >= n_tiles) return v;
    const TcTile tl = tiles[t];
    const int i = r1 - tl.row0, j = r2 - tl.col0;
    if (i < 0 || i >= kM || j < 0 || j >= kPanel) return v;
    for (int sp = 0; sp < n_splits; ++sp) {
      const double* slot = partials + (size_t)(sp * n_tiles + t) * (kM * kPanelCols);
      v += slot[i * kPanelCols + h * kPanel + j];
    }
    return v;
  };
  const int ra = sc.row + a, ia = sc.row + D + a, rb = sc.row + b, ib = sc.row + D + b;
  for (int h = 0; h < 3; ++h) {
    const double re = C(ra, rb, h) + C(ia, ib, h);
    const double im = C(ra, ib, h) - C(ia, rb, h);
    const size_t o = 2 * ((size_t)sc.goff + (size_t)a * D + b) + 2 * plane * h;
    gram[o] += re;
    gram[o + 1] += im;
  }
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link
// dependency on libcuda).
using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                   const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                   const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

// 2D FP32 map over a row-major [rows][ld] array, box = box_x samples x box_y rows,
// rows past `rows` read as zero; swizzle128 stores each 128-byte box row with
// its 16-byte chunks XOR-permuted by (row % 8) (box_x must then be 32).
bool make_map(CUtensorMap* m, const float* base, int ld, int rows, int box_x, int box_y,
              bool swizzle128) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  const cuuint64_t dims[2] = {cuuint64_t(ld), cuuint64_t(rows)};
  const cuuint64_t strides[1] = {cuuint64_t(ld) * sizeof(float)};
  const cuuint32_t box[2] = {cuuint32_t(box_x), cuuint32_t(box_y)};
  const cuuint32_t estr[2] = {1, 1};
  return fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(base), dims, strides, box,
            estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            swizzle128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <bool HALF, int NB>
int launch_t(const TcArgs& a, int n_jobs, cudaStream_t st) {
  const size_t smem = sizeof(Smem<NB>) + 1024;
  if (smem > 227 * 1024) return LEMC_ERR_CAPACITY;
  CUtensorMap tmA, tmB, tmW;
  if (!make_map(&tmA, a.V, a.ldv, a.total_rows, kHalf, kM, true) ||
      !make_map(&tmB, a.V, a.ldv, a.total_rows, kHalf, NB, true) ||
      !make_map(&tmW, a.rec_w, a.ldw, 3, kHalf, 3, false))
    return LEMC_ERR_CUDA;
  cudaFuncAttributes fa;
  // the register split after launch assumes exactly kLaunchRegs per thread
  if (cudaFuncGetAttributes(&fa, gram_tc_kernel<HALF, NB>) != cudaSuccess || fa.numRegs != kLaunchRegs ||
      cudaFuncSetAttribute(gram_tc_kernel<HALF, NB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           int(smem)) != cudaSuccess)
    return LEMC_ERR_CUDA;
  gram_tc_kernel<HALF, NB><<<n_jobs, kThreads, smem, st>>>(a, tmA, tmB, tmW);
  return cudaPeekAtLastError() == cudaSuccess ? LEMC_OK : LEMC_ERR_CUDA;
}

// range[r] = bits of max |V[r][w]| over the padded walkers, range[rows + h] of
// max |W_h|, by unsigned maxima of the sign-cleared bits (NaN above infinity).
// One read of V; the arrays were cleared before the launch.
constexpr int kRangeThreads = 256, kRangeSpan = 8192;

__global__ void __launch_bounds__(kRangeThreads)
row_range_kernel(const float* __restrict__ V, int ldv, int rows, const float* __restrict__ rec_w,
                 int ldw, int Wpad, uint32_t* __restrict__ range) {
  const int r = blockIdx.y;
  const int w0 = blockIdx.x * kRangeSpan, w1 = min(Wpad, w0 + kRangeSpan);
  uint32_t m = 0u;
  auto take = [&](float x) { m = max(m, __float_as_uint(x) & 0x7FFFFFFFu); };
  if (r < rows) {
    const float4* p = reinterpret_cast<const float4*>(V + (size_t)r * ldv);
    for (int q = w0 / 4 + threadIdx.x; q < w1 / 4; q += kRangeThreads) {
      const float4 f = p[q];
      take(f.x); take(f.y); take(f.z); take(f.w);
    }
  } else {
    const int h = r - rows;
    for (int w = w0 + threadIdx.x; w < w1; w += kRangeThreads) {
      const float one = rec_w[w];
      take(h == 0 ? one : one * rec_w[(size_t)h * ldw + w]);
    }
  }
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0 && m) atomicMax(range + r, m);
}

// Host-side settings of the bounded waits (lemc_debug_gram_wait).
long long g_wait_cycles = kWaitCycles;
int g_hold_loads = 0;

}  // namespace

int set_gram_wait(long long cycles, int hold_loads) {
  if (cycles < 0) return LEMC_ERR_ARG;
  g_wait_cycles = cycles > 0 ? cycles : kWaitCycles;
  g_hold_loads = hold_loads != 0;
  return LEMC_OK;
}

int launch_gram_tc_rows(const float* V, int ldv, int total_rows, const float* rec_w, int ldw,
                        int Wpad, const TcTile* tiles, int n_jobs, int panels, int n_splits,
                        uint32_t* range, bool have_range, double* partials, int mode, int flush_every, int* err, cudaStream_t st) {
  if (mode != LEMC_GRAM_BF16X3 && mode != LEMC_GRAM_BF16X4 && mode != LEMC_GRAM_TF32X3)
    return LEMC_ERR_ARG;
  if (ldv % 64 != 0 || ldw % 64 != 0 || Wpad % 64 != 0 || n_jobs <= 0 || Wpad > ldv || Wpad > ldw)
    return LEMC_ERR_ARG;
  if (reinterpret_cast<uintptr_t>(V) % 256 != 0 || reinterpret_cast<uintptr_t>(rec_w) % 256 != 0)
    return LEMC_ERR_ARG;
  const bool half = (mode == LEMC_GRAM_TF32X3);
  TcArgs a;
  a.V = V;
  a.ldv = ldv;
  a.total_rows = total_rows;
  a.rec_w = rec_w;
  a.ldw = ldw;
  a.tiles = tiles;
  a.range = range;
  a.partials = partials;
  a.n_chunks_total = Wpad / KC;
  a.n_splits = n_splits;
  // flush_every counts 32-walker chunks for TF32X3 (eight steps of two terms, as
  // four 16-sample steps of two chunks) and K-chunks for BF16, whose 16-bit
  // representation limits it, so a longer interval costs nothing there
  a.flush_every = flush_every > 0 ? (half ? (flush_every > 1 ? flush_every / 2 : 1) : flush_every)
                                  : (half ? 1 : 4);
  a.passes = (mode == LEMC_GRAM_BF16X4) ? 4 : 3;
  a.err = err;
  a.wait_cycles = g_wait_cycles;
  a.hold_loads = g_hold_loads;
  if (!have_range) {
    if (cudaMemsetAsync(range, 0, sizeof(uint32_t) * (size_t(total_rows) + 3), st) != cudaSuccess)
      return LEMC_ERR_CUDA;
    row_range_kernel<<<dim3((Wpad + kRangeSpan - 1) / kRangeSpan, total_rows + 3), kRangeThreads, 0,
                       st>>>(V, ldv, total_rows, rec_w, ldw, Wpad, range);
  }
  if (panels == 2) return half ? launch_t<true, 64>(a, n_jobs, st) : launch_t<false, 64>(a, n_jobs, st);
  return half ? launch_t<true, 32>(a, n_jobs, st) : launch_t<false, 32>(a, n_jobs, st);
}

int launch_gram_tc_reduce(const double* partials, const TcTile* tiles, const TcSector* secs,
                          int n_sec, int n_tiles, int n_splits, int max_dim, double* gram,
                          size_t plane, cudaStream_t st) {
  dim3 grid((max_dim * max_dim + 255) / 256, n_sec);
  gram_tc_reduce_kernel<<<grid, 256, 0, st>>>(partials, tiles, secs, n_sec, n_tiles, n_splits,
                                              gram, plane);
  return cudaPeekAtLastError() == cudaSuccess ? LEMC_OK : LEMC_ERR_CUDA;
}

}  // namespace lemc
