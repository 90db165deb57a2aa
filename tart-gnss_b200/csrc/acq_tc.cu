// Tensor-core correlator (sm_100a, tcgen05): reduced-precision search.
//
// The inverse transform of every product Z * conj(C) (length Lc = R1 x 31 x
// GR, R1 = 33, 44, 55 and GR = 1, 3, 2 x 3 for Lc = 1023, 4092, 10230) is a
// Good-Thomas prime-factor transform.  The two large radices run on the
// 5th-generation tensor cores as GEMMs, the digits of 2 and 3 as butterflies
// in FP32 on the values the warps hold anyway:
//
//   P1  FP16 products, stored as the N x K operand B of stage 1: one K entry
//       per (R1-digit, re / im), columns (left-over digits or residues, 31-digit)
//   M1  D1 = A1 B, A1 the inverse DFT-R1 as a real matrix, rows (t1, re / im)
//   P2  D1 from TMEM, DFT-2 (Lc = 10230), FP16 rounding, back to TMEM as the
//       operand A2 of stage 2: rows (t1, h), K = (re / im, 31-digit)
//   M2  D2 = A2 B2, B2 the inverse DFT-31, over the columns of D1
//   P4  DFT-3 (Lc = 4092, 10230) and the row maximum of |y|^2
//
// The prime-factor map needs the digit contracted next to move from the rows
// (TMEM lanes) or columns of one GEMM to the K dimension of the next.  With
// the data as operand B in the first stage and as operand A in the second,
// D1's lanes hold t1 and its columns the 31-digit, which is A2's K as it
// stands: no transposition passes through shared memory.  A2's row needs the
// real and the imaginary part of one t1, which D1 has in two lanes; rows are
// ordered so that these are lanes r and r + 8 of a group of 16, and the
// 16x128b form of tcgen05.ld hands a thread exactly such pairs of lanes, the
// 16x128b form of tcgen05.st takes the FP16 words of lanes r (h = 0) and r + 8
// (h = 1).  h is the digit of 2 at Lc = 10230, one
// of two code-phase residues otherwise.
//
// Scaling: Z and conj(C) are stored as Z 2^-kz and conj(C) 2^-kd with
// kz + kd = k and 4 S Lc^2 2^-k <= 32768.  Then |Z 2^-kz| <= 4 S Lc 2^-kz and
// |C 2^-kd| <= Lc 2^-kd stay inside FP16, every product is below 32768 and so
// is every value of a partly inverted transform (a mean of correlation
// values); stage outputs are rounded with satfinite.
// Keys carry the row maximum of |y|^2 2^-2k (the lag bits are zero) and are
// only compared: every row of an (antenna, PRN) whose key lies within the
// FP16 error bound of its best is re-evaluated in FP32 afterwards
// (launch_tc_candidates, launch_correlate_listed), so the chosen row, and
// the reported peak, lag and second peak, are those of the FP32 search.
//
// One CTA per SM (the kernel takes the SM's TMEM).  A work item is one
// (antenna, bin, hypothesis) row and RES code-phase residues; a step is one
// PRN (non-coherent search: one block of one PRN) of an item.  Steps
// rotate over two or three chains (operand buffer and D region each), and the
// phases belong to different warps: 4 R1 product threads (P1; the item's FP16
// Z stays in their registers for all PRNs), 4 or 8 warps per chain for its P2
// and P4, so that one chain's P4 runs beside the other's P2, and one warp that
// issues M1 and fetches the code blocks.  M2 is issued by the first of its
// chain's warps: a thread's barrier test queues behind its own MMAs, so one
// issuer for both stages would see A2 late (measured: 1000 cycles).  Which
// barrier tells that an A2 region is free is tc_steps.h's.  Every wait is
// bounded (1 s): on expiry a role sets *err, drains (again bounded) and leaves
// its loop.
//
// What bounds it (Lc = 10230, per step, of about 2550 cycles measured over the
// whole 24-antenna search): the shared-memory data path, about 1600 cycles (P1
// reads 42 KB of code and writes 42 KB, the code copies write 42 KB, M1 and M2
// read 78 KB); the tensor cores 1120 (an M = 128, K = 16 MMA takes N / 2
// cycles; 686 for M1, 432 for M2); the FP32 pipe about 900 (DFT-2, DFT-3 and
// |y|^2: 8 operations per point).  Long runs sit at the 1000 W power limit.
// Measured against the three-stage design before it, which transposed through
// shared memory twice (24 antennas, 41 bins, --all): 62.2 -> 35.3 ms at Lc =
// 10230, 11.2 -> 6.1 at 4092, 3.65 -> 3.4 at 1023; non-coherent, one antenna,
// 100 ms: 81.1 -> 43.2, 16.6 -> 7.4 and 10.4 -> 4.5 ms; weak signals (24
// antennas, 201 bins, 10 blocks) 44.0 -> 28.8 ms.  RMS error of the FP16 row
// keys 8.8e-5 -> 6.9e-5 of the largest row (one rounding of the data less).
//
// The same kernel (NCB) runs the non-coherent search: each chain takes a PRN
// through all its coherent blocks (the Z of a block is loaded once for both
// PRNs), and the |y|^2 of the blocks are summed in the registers of the P4
// threads (each output of the transform has its thread) before the maximum.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <cstring>
#include <type_traits>
#include <vector>

#include "engine.h"
#include "pfa_common.cuh"
#include "tc_steps.h"

namespace tga {

namespace {

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(slot)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// mbarriers (and the operands of the product warps) go by their 32-bit shared
// addresses: a 64-bit generic pointer costs two registers and a conversion
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ uint32_t mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
  return done;
}
// The same test with a suspend-time hint: a thread whose phase has not
// completed sleeps until it completes or `ns` nanoseconds pass, instead of
// returning at once to poll again, so waiting warps leave their
// sub-partition's issue slots to the warps that work.
__device__ __forceinline__ uint32_t mbar_try_wait_sleep(uint32_t bar, uint32_t parity, uint32_t ns) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done)
      : "r"(bar), "r"(parity), "r"(ns)
      : "memory");
  return done;
}
__device__ __forceinline__ uint4 ld_shared(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void st_shared(uint32_t a, uint4 v) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
// D[tmem] (+)= A[smem desc] * B[smem desc], kind::f16, no lanes masked.
__device__ __forceinline__ void mma_f16(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc) {
  const uint32_t z = 0;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}" ::"r"(tmem_d),
      "l"(da), "l"(db), "r"(idesc), "r"(acc), "r"(z), "r"(z), "r"(z), "r"(z)
      : "memory");
}
__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// bulk copy global -> this CTA's shared memory, completing `bytes` of the
// barrier's transaction count (both addresses 16-byte aligned, bytes % 16 == 0)
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

// the same with operand A in TMEM (one lane per row, two K entries per column)
__device__ __forceinline__ void mma_f16_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t idesc, uint32_t acc) {
  const uint32_t z = 0;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %6, %7, %8}, p;\n\t}" ::"r"(tmem_d),
      "r"(tmem_a), "l"(db), "r"(idesc), "r"(acc), "r"(z), "r"(z), "r"(z), "r"(z)
      : "memory");
}
// True in one lane of a converged warp.  Measured at M = 128, N = 64, K = 16
// with A in TMEM: an MMA issues every 54 cycles behind a lane test, every 36
// behind elect.sync.
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "elect.sync _|q, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(p));
  return p != 0;
}
// 16 columns of 16 lanes: thread t gets, for i = 0 .. 3, column 4 i + t % 4 of
// lane t / 4 in r[2 i] and of lane t / 4 + 8 in r[2 i + 1]
__device__ __forceinline__ void tmem_ld_pairs(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.16x128b.x4.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
// 8 columns of 16 lanes: thread t writes, for i = 0, 1, column 4 i + t % 4 of
// lane t / 4 from r[2 i] and of lane t / 4 + 8 from r[2 i + 1]
__device__ __forceinline__ void tmem_st_pairs(uint32_t taddr, const uint32_t (&r)[4]) {
  asm volatile("tcgen05.st.sync.aligned.16x128b.x2.b32 [%0], {%1, %2, %3, %4};" ::"r"(taddr), "r"(r[0]), "r"(r[1]),
               "r"(r[2]), "r"(r[3])
               : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, uint32_t (&r)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, uint32_t (&r)[8]) { tmem_ld8(taddr, r); }
__device__ __forceinline__ void tmem_st_zero8(uint32_t taddr) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %1, %1, %1, %1, %1, %1, %1};" ::"r"(taddr), "r"(0u)
               : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// B2 in the K-major layout with the 128-byte swizzle: rows of 64 K entries,
// 8-row groups of 1024 bytes, the 16-byte chunk j of row r at chunk j ^ (r & 7)
__host__ __device__ __forceinline__ uint32_t sw128_off(int r, int j) {
  return (uint32_t)((r >> 3) * 1024 + (r & 7) * 128 + ((j ^ (r & 7)) << 4));
}
__device__ __forceinline__ uint64_t desc_sw128(uint32_t addr) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
// Un-swizzled operands are 8 x 16-byte cores of 128 contiguous bytes; lead and
// stride are the byte distances between cores along K and along the rows
// (K-major, A1), or along K and along the columns (MN-major, the products).
__device__ __forceinline__ uint64_t desc_cores(uint32_t addr, uint32_t lead, uint32_t stride) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lead >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((stride >> 4) & 0x3FFFu) << 32) | ((uint64_t)1 << 46);
}

// instruction descriptor: kind::f16, A = B = FP16, D = FP32, A K-major, M = 128;
// b_mn: B is MN-major
constexpr uint32_t idesc_f16(int n, bool b_mn) {
  return (1u << 4) | (b_mn ? 1u << 16 : 0u) | ((uint32_t)(n >> 3) << 17) | ((128u >> 4) << 24);
}
constexpr int pad16(int x) { return (x + 15) / 16 * 16; }

// Warp roles.  The first warps do P2 and P4, a group of them per chain: a warp
// reaches the TMEM lanes of quadrant warp % 4, so a group is a multiple of 4.  Then the product warps (Tc::PROD_WARPS) and the M1 warp.
constexpr int kTcTmemCols = 512;
constexpr long long kWaitPolls = 1LL << 22;
constexpr unsigned long long kWaitNs = 1000000000ull;  // 1 s per wait on the tensor cores
constexpr uint32_t kSuspendNs = 20000;                  // longest sleep of one test (20 us)

__device__ __forceinline__ unsigned long long globaltimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// polls the mbarrier phase until it completes, at most kWaitPolls times and
// kWaitNs nanoseconds; after the first test each one may sleep up to
// kSuspendNs (woken when the phase completes), so the bound is on the timer
__device__ __forceinline__ uint32_t bounded_wait(uint32_t bar, uint32_t phase) {
  uint32_t done = mbar_try_wait(bar, phase);
  if (done) return done;  // the common case reads no timer
  const unsigned long long t0 = globaltimer_ns();
  for (long long k = 0; k < kWaitPolls && !done; ++k) {
    done = mbar_try_wait_sleep(bar, phase, kSuspendNs);
    if (!done && (k & 7) == 7 && globaltimer_ns() - t0 > kWaitNs) break;
  }
  return done;
}
// the same for a whole warp: true when all its lanes saw the phase complete
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t phase) {
  if (__all_sync(0xffffffffu, mbar_try_wait(bar, phase))) return true;
  return __all_sync(0xffffffffu, bounded_wait(bar, phase)) != 0;
}
// Two phases at once: a test costs 150 to 300 cycles from issue to answer even
// when its phase has long completed, so both go out before either is looked at.
// A phase that its test saw complete is not tested again.
__device__ __forceinline__ bool warp_wait2(uint32_t bar0, uint32_t phase0, uint32_t bar1, uint32_t phase1) {
  const uint32_t a = mbar_try_wait(bar0, phase0), b = mbar_try_wait(bar1, phase1);
  if (__all_sync(0xffffffffu, a & b)) return true;
  return __all_sync(0xffffffffu, (a || bounded_wait(bar0, phase0)) && (b || bounded_wait(bar1, phase1))) != 0;
}

// Per code length: NB blocks of 2 x 32 columns (h, 31-digit) in D1; H2 / B3
// whether h / the block is a digit of 2 / 3 of the transform (a residue
// otherwise); NCH chains; A2S operand regions A2 (step s has region s % A2S: two
// where the 512 columns allow it); code slots.  An MMA of M = 128 rows costs the same for any R1 <=
// 64, hence the largest R1 that leaves 31 and digits of 2 and 3.
template <int M, bool NCB>
struct TcCfg;
template <bool NCB>
struct TcCfg<1, NCB> {
  // short steps, bound by the latency of their phases: a third chain where the
  // registers allow it (NCB holds a sum per output)
  static constexpr int NB = 2, NCH = NCB ? 2 : 3, A2S = 2, SLOTS = 4;
  static constexpr bool H2 = false, B3 = false;
};
template <bool NCB>
struct TcCfg<4, NCB> {
  static constexpr int NB = 3, NCH = 2, A2S = 1, SLOTS = 4;
  static constexpr bool H2 = false, B3 = true;
};
template <bool NCB>
struct TcCfg<10, NCB> {
  static constexpr int NB = 3, NCH = 2, A2S = 1, SLOTS = 2;
  static constexpr bool H2 = true, B3 = true;
};

template <int M, bool NCB>
struct Tc {
  using C = TcCfg<M, NCB>;
  using U = TcUnits<M>;
  // TMEM warps of a chain, PARTS per lane quadrant
  static constexpr int PARTS = NCB ? 2 : 1, CHAIN_WARPS = 4 * PARTS, NCH = C::NCH, TMEM_WARPS = NCH * CHAIN_WARPS;
  static_assert(!NCB || NCH == 2, "a round of the non-coherent search is a pair of PRNs");
  static constexpr int R1 = U::R1, NB = C::NB, A2S = C::A2S, SLOTS = C::SLOTS;
  static constexpr bool H2 = C::H2, B3 = C::B3;
  // code-phase residues of a step
  static constexpr int RES = (H2 ? 1 : 2) * (B3 ? 1 : NB);
  static_assert(RES * U::GR == 2 * NB, "column groups: residues x left-over digits");
  // stage 1: K1 = (re / im, R1-digit) padded, N1 columns, column 32 cg + d2
  // with column group cg = 2 b + h
  static constexpr int K1 = pad16(2 * R1), KH = K1 / 2, N1 = 64 * NB;
  static_assert(KH == U::R1P && 2 * R1 <= 128, "stage 1 rows, units");
  // rows: block i = t1 / 8 of eight t1 in the 16 lanes of group phys(i): the
  // blocks spread over the four quadrants first
  static constexpr int BLK = (R1 + 7) / 8;
  __host__ __device__ static constexpr int phys(int i) { return i < 4 ? 2 * i : 2 * (i - 4) + 1; }
  static_assert(BLK >= 4 && BLK <= 8, "eight groups of 16 lanes");
  // products: 16-byte rows (one K entry, eight columns), the K entries of eight
  // columns contiguous
  static constexpr int STRIDE_B = K1 * 16, B_BYTES = (8 * NB * STRIDE_B + 1023) / 1024 * 1024;
  static constexpr int A1_BYTES = 128 * K1 * 2, B2_BYTES = 64 * 128;
  static_assert(A1_BYTES % 1024 == 0, "1024-byte aligned regions");
  // one (PRN, hypothesis) block of code units
  static constexpr int CODE_BYTES = U::PER_SEQ * 16, CODE_REGION = (CODE_BYTES + 1023) / 1024 * 1024;
  // TMEM columns: a region of D per chain (stage 2 writes over stage 1), then A2
  static constexpr int A2_COL = NCH * N1, A2_COLS = 32 * NB;
  static_assert(A2_COL + A2S * A2_COLS <= kTcTmemCols, "TMEM");
  // product threads: one per (R1-digit with padding, j); slot gr of a thread is
  // its unit (gr 4 + j) R1P + d1, for every residue
  static constexpr int PROD_THREADS = 4 * U::R1P, PROD_WARPS = PROD_THREADS / 32;
  static_assert(PROD_THREADS % 32 == 0, "whole product warps");
  static constexpr int M1_WARP = TMEM_WARPS + PROD_WARPS, THREADS = 32 * (M1_WARP + 1);
  // NCB: all but the last slot's Z units stay in registers (GRK slots); the
  // last slot's go to shared memory, 16 bytes per thread and word, read back
  // only by the thread that wrote them: with all of them in registers the
  // 24-warp kernel spilled, and beside 210 KB of shared memory spills fall out
  // of L1
  static constexpr bool ZSM = NCB && U::GR > 1;
  static constexpr int GRK = ZSM ? U::GR - 1 : U::GR;
  static constexpr int ZS_BYTES = ZSM ? RES * 2 * PROD_THREADS * 16 : 0;
  // the K steps of A1 that the free TMEM columns hold (8 columns each); the
  // others are read from shared memory by every M1
  static constexpr int A1_COL = A2_COL + A2S * A2_COLS;
  static constexpr int A1_KS = (kTcTmemCols - A1_COL) / 8 < K1 / 16 ? (kTcTmemCols - A1_COL) / 8 : K1 / 16;
  static constexpr int SMEM_RAW = NCH * B_BYTES + A1_BYTES + B2_BYTES + SLOTS * CODE_REGION + ZS_BYTES + 1024;
  // more than half of the SM's shared memory: one CTA, and so one 512-column
  // TMEM allocation, per SM
  static constexpr int SMEM = SMEM_RAW > 120 * 1024 ? SMEM_RAW : 120 * 1024;
  static_assert(SMEM <= 227 * 1024, "shared memory");
};

__device__ __forceinline__ uint32_t h2_bits(__half2 h) { return *reinterpret_cast<uint32_t*>(&h); }
__device__ __forceinline__ __half2 bits_h2(uint32_t u) { return *reinterpret_cast<__half2*>(&u); }
__device__ __forceinline__ float2 f2_bits(uint32_t a, uint32_t b) {
  return make_float2(__uint_as_float(a), __uint_as_float(b));
}
// round two FP32 values to FP16, clamping to +-65504 instead of overflowing
__device__ __forceinline__ uint32_t pack_h2_sat(float2 v) {
  uint32_t d;
  asm("cvt.rn.satfinite.f16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(v.y), "f"(v.x));
  return d;
}
// (re, im) = (cr zr - ci zi, cr zi + ci zr) of two values, the products cr zr
// and cr zi rounded first
__device__ __forceinline__ void cmul_h2(uint32_t zr, uint32_t zi, uint32_t cr, uint32_t ci, uint32_t& re, uint32_t& im) {
  const __half2 a = bits_h2(zr), b = bits_h2(zi), c = bits_h2(cr), d = bits_h2(ci);
  re = h2_bits(__hfma2(d, __hneg2(b), __hmul2(c, a)));
  im = h2_bits(__hfma2(d, a, __hmul2(c, b)));
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }

// The constant operands, built on the host in double precision and rounded
// once to FP16: entries of exp(+2 pi i t d / R) as real 2 x 2 blocks.
// A1: row (t1, c) at lane 16 phys(t1 / 8) + t1 % 8 + 8 c, K = KH (re | im) + d1.
// B2: row 4 (t2 / 2) + 2 c + t2 % 2 (two adjacent outputs' real parts, then
// their imaginary parts), K = 32 (re | im) + 8 (d2 / 8) + 2 (d2 % 4) + (d2 /
// 4) % 2: a thread of P2 holds every fourth column and packs two of them.
template <int M>
std::vector<unsigned char> build_matrices() {
  using T = Tc<M, false>;
  const double kTwoPi = 6.283185307179586;
  std::vector<unsigned char> m((size_t)(T::A1_BYTES + T::B2_BYTES), 0);
  auto put = [&](size_t at, int c, int cc, int t, int d, int R) {
    const double ang = kTwoPi * (double)((t * d) % R) / (double)R;
    const double v = c == cc ? std::cos(ang) : (c == 0 ? -std::sin(ang) : std::sin(ang));
    const __half h = __float2half_rn((float)v);
    std::memcpy(m.data() + at, &h, 2);
  };
  for (int t = 0; t < T::R1; ++t)
    for (int c = 0; c < 2; ++c)
      for (int cc = 0; cc < 2; ++cc)
        for (int d = 0; d < T::R1; ++d) {
          const int row = 16 * T::phys(t / 8) + t % 8 + 8 * c, k = T::KH * cc + d;
          put((size_t)(k / 8) * 2048 + (size_t)row * 16 + (size_t)(k % 8) * 2, c, cc, t, d, T::R1);
        }
  for (int t = 0; t < 31; ++t)
    for (int c = 0; c < 2; ++c)
      for (int cc = 0; cc < 2; ++cc)
        for (int d = 0; d < 31; ++d) {
          const int row = 4 * (t / 2) + 2 * c + t % 2, k = 32 * cc + 8 * (d / 8) + 2 * (d % 4) + (d / 4) % 2;
          put((size_t)T::A1_BYTES + sw128_off(row, k / 8) + (size_t)(k % 8) * 2, c, cc, t, d, 31);
        }
  return m;
}

// FP16 operands (TcUnits) of spectra in the FP32 engine's digit layout; the
// forward transform writes those of Z itself, this packs the code spectra.
template <int M>
__global__ void __launch_bounds__(256) tc_pack_kernel(const float2* __restrict__ src, uint4* __restrict__ dst,
                                                      long long n_units, float scale) {
  using U = TcUnits<M>;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < n_units;
       e += (long long)gridDim.x * blockDim.x) {
    const long long seq = e / U::UNITS;
    const int u = (int)(e - seq * U::UNITS);
    const float2* s = src + seq * U::LC;
    float2 v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      v[i] = make_float2(0.f, 0.f);
      if (U::filled(u, i)) {
        v[i] = __ldg(s + U::src_offset(u, i));
        v[i].x *= scale;
        v[i].y *= scale;
      }
    }
    uint4* d = dst + seq * U::PER_SEQ + u;
    pack_unit(v, d[0], d[U::UNITS]);
  }
}

struct TcParams {
  const uint4* mats;  // A1 and B2 in their shared-memory layouts
  const uint4* z16;   // [n_ab*2][S] sequences (NCB: [n_ab][B][S])
  const uint4* d16;   // [n_prn][2] sequences
  unsigned long long* keys;
  int* err;
  int n_items;  // rows x groups: (row, residue group) work items
  int groups;   // ceil(S / RES)
  // work units: item u / split, rounds [r0, r1) of part u % split; a round is
  // one PRN (NCB: a pair of PRNs, one per chain)
  int split;
  int step_w, step_r;  // NCB: gridDim.x units on, in items and rounds
  int n_rounds, n_prn, S;
  int B;            // coherent blocks summed non-coherently (1: the drop-in search)
  int skip_commit;  // test hook: see TGA_TEST_TC_SKIP_COMMIT
};

// The CTA's units in order: item w, rounds [r0, r1).
template <bool NCB>
struct Units {
  const TcParams& p;
  int u, w, r0, r1;
  __device__ __forceinline__ explicit Units(const TcParams& q) : p(q), u(blockIdx.x) {
    w = u / p.split;
    set(u - w * p.split);
  }
  __device__ __forceinline__ bool more() const { return w < p.n_items; }
  __device__ __forceinline__ void next() {
    if (NCB) {  // one round per unit: no division per round
      r0 += p.step_r;
      w += p.step_w;
      if (r0 >= p.split) r0 -= p.split, ++w;
      r1 = r0 + 1;
    } else {
      u += gridDim.x;
      w = u / p.split;
      set(u - w * p.split);
    }
  }

 private:
  __device__ __forceinline__ void set(int part) {
    r0 = NCB ? part : part * p.n_rounds / p.split;  // (split <= 32)
    r1 = NCB ? part + 1 : (part + 1) * p.n_rounds / p.split;
  }
};

// mbarriers of the CTA and who completes them.  Step s is chain s % NCH's use
// s / NCH; a barrier of a chain is in phase (s / NCH) & 1.
template <class T>
struct Bars {
  using Turn = A2Turn<T::NCH, T::A2S>;
  // byte offsets from the CTA's first mbarrier
  static constexpr uint32_t PER = 8 * T::NCH;
  static constexpr uint32_t PROD = 0;         // P1 -> M1: the chain's products are stored (every product warp)
  static constexpr uint32_t M1 = PER;         // M1 done (commit): D1 is there, the products' buffer is free
  static constexpr uint32_t A2 = 2 * PER;     // P2 -> M2: A2 is there (the chain's TMEM warps)
  static constexpr uint32_t M2 = 3 * PER;     // M2 done (commit): D2 is there, A2 is free
  static constexpr uint32_t DFREE = 4 * PER;  // P4 -> M1: D is read (the chain's TMEM warps)
  static constexpr uint32_t A1 = 5 * PER;     // A1's first K steps are in TMEM (4 warps, once)
  static constexpr uint32_t CODE = A1 + 8;    // code block n (slot n % SLOTS) has landed
  static constexpr uint32_t AFREE = CODE + 8 * T::SLOTS;  // M2 of the region's step done (commit): the region is free
  static constexpr int COUNT = 5 * T::NCH + 1 + T::SLOTS + Turn::REGION_BARS;
};

// The M1 warp's thread.  M1 of step s needs its products and the D region that
// P4 of step s - NCH read.  When the products of a PRN's last step are there,
// its code slot is free: the thread fetches the block of the PRN SLOTS further
// on into it.
template <int M, bool NCB>
__device__ __forceinline__ bool m1_role(const TcParams& p, uint32_t bars, uint32_t A1, uint32_t PROD, uint32_t CODE,
                                        uint32_t tmem) {
  using T = Tc<M, NCB>;
  using Br = Bars<T>;
  const int B = NCB ? p.B : 1;
  constexpr int PER_ROUND = NCB ? 2 : 1;  // code blocks of a round
  // ---- code blocks in order: block `fetched` is chain fx of round fr of unit fu ----
  Units<NCB> fu(p);
  int fr = fu.r0, fx = 0, fetched = 0;
  auto fetch = [&]() {
    if (!fu.more()) return;
    const int hyp = NCB ? 0 : (fu.w / p.groups) & 1;
    int prn = NCB ? 2 * fr + fx : fr;
    if (prn >= p.n_prn) prn = p.n_prn - 1;  // an odd PRN number: the last one on both chains
    const int slot = fetched % T::SLOTS;
    mbar_arrive_expect_tx(bars + Br::CODE + 8u * (uint32_t)slot, (uint32_t)T::CODE_BYTES);
    bulk_g2s(CODE + (uint32_t)(slot * T::CODE_REGION), p.d16 + ((size_t)prn * 2 + hyp) * T::U::PER_SEQ,
             (uint32_t)T::CODE_BYTES, bars + Br::CODE + 8u * (uint32_t)slot);
    ++fetched;
    if (++fx == PER_ROUND) {
      fx = 0;
      if (++fr == fu.r1) {
        fu.next();
        fr = fu.r0;
      }
    }
  };
  for (int i = 0; i < T::SLOTS; ++i) fetch();
  const uint64_t da = desc_cores(A1, 2048, 128);
  const uint64_t db = desc_cores(PROD, 128, T::STRIDE_B);
  auto issue = [&](auto xc) {
    constexpr int x = decltype(xc)::value;
#pragma unroll
    for (int ks = 0; ks < T::K1 / 16; ++ks) {
      const uint64_t dbk = db + (uint64_t)(x * (T::B_BYTES >> 4) + ks * (256 >> 4));
      if (ks < T::A1_KS)
        mma_f16_ta(tmem + (uint32_t)(x * T::N1), tmem + (uint32_t)(T::A1_COL + 8 * ks), dbk, idesc_f16(T::N1, true),
                   ks > 0 ? 1u : 0u);
      else
        mma_f16(tmem + (uint32_t)(x * T::N1), da + (uint64_t)(ks * (4096 >> 4)), dbk, idesc_f16(T::N1, true),
                ks > 0 ? 1u : 0u);
    }
    mma_commit(bars + Br::M1 + 8u * (uint32_t)x);
  };
  int s = 0, commits = 0;
  bool ok = bounded_wait(bars + Br::A1, 0u) != 0;
  for (Units<NCB> u(p); u.more() && ok; u.next()) {
    const int n = (u.r1 - u.r0) * PER_ROUND * B;
    int left = NCB ? PER_ROUND * B : 1;  // steps of the round (of its code blocks) from here on
#pragma unroll 1
    for (int i = 0; i < n; ++i, ++s) {
      const int use = s / T::NCH, x = s - use * T::NCH;
      const uint32_t ph = (uint32_t)use & 1u;
      {
        const uint32_t prod = bars + Br::PROD + 8u * (uint32_t)x, dfree = bars + Br::DFREE + 8u * (uint32_t)x;
        const uint32_t a = mbar_try_wait(prod, ph), f = mbar_try_wait(dfree, ph ^ 1u);
        ok = (a & f) || (bounded_wait(prod, ph) && bounded_wait(dfree, ph ^ 1u));
      }
      if (!ok) break;
      tc_fence_after();
      // test hook (TGA_TEST_TC_SKIP_COMMIT): issue nothing, so the other
      // roles' waits run out with no tensor-core work in flight
      if (!p.skip_commit) {
        if (x == 0)
          issue(std::integral_constant<int, 0>());
        else if (x == 1)
          issue(std::integral_constant<int, 1>());
        else
          issue(std::integral_constant<int, T::NCH - 1>());
        ++commits;
      }
      if (left <= PER_ROUND) fetch();
      if (--left == 0) left = NCB ? PER_ROUND * B : 1;
    }
  }
  // drain: the last commit (after a timeout it may still be in flight; it
  // covers the MMAs before it), and the last copy into each slot
  if (commits > 0) {
    const int use = (commits - 1) / T::NCH, x = commits - 1 - use * T::NCH;
    bounded_wait(bars + Br::M1 + 8u * (uint32_t)x, (uint32_t)use & 1u);
  }
  for (int i = fetched > T::SLOTS ? fetched - T::SLOTS : 0; i < fetched; ++i)
    bounded_wait(bars + Br::CODE + 8u * (uint32_t)(i % T::SLOTS), (uint32_t)(i / T::SLOTS) & 1u);
  return ok;
}

template <int M, bool NCB>
__global__ void __launch_bounds__(Tc<M, NCB>::THREADS, 1) pfa_tc_kernel(const __grid_constant__ TcParams p) {
  using T = Tc<M, NCB>;
  using U = TcUnits<M>;
  using Br = Bars<T>;
  constexpr int NB = T::NB, RES = T::RES, GR = U::GR;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ uint64_t s_bar[Br::COUNT];
  __shared__ uint32_t s_tmem;
  // 32-bit shared addresses of the regions, from a 1024-byte boundary
  const uint32_t raw = smem_addr(smem_raw), A1 = (raw + 1023u) & ~1023u;
  const uint32_t B2 = A1 + T::A1_BYTES, PROD = B2 + T::B2_BYTES, CODE = PROD + T::NCH * T::B_BYTES;
  const uint32_t ZS = CODE + T::SLOTS * T::CODE_REGION;
  const uint32_t bars = smem_addr(s_bar);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int S = p.S, B = NCB ? p.B : 1;

  if (warp == 0) {
    tmem_alloc(&s_tmem, kTcTmemCols);
    tmem_relinquish();
  }
  if (tid == 0) {
    for (uint32_t x = 0; x < 8 * T::NCH; x += 8) {
      mbar_init(bars + Br::PROD + x, T::PROD_WARPS);
      mbar_init(bars + Br::M1 + x, 1);
      mbar_init(bars + Br::A2 + x, T::CHAIN_WARPS);
      mbar_init(bars + Br::M2 + x, 1);
      mbar_init(bars + Br::DFREE + x, T::CHAIN_WARPS);
    }
    mbar_init(bars + Br::A1, 4);
    for (uint32_t x = 0; x < 8 * T::SLOTS; x += 8) mbar_init(bars + Br::CODE + x, 1);
    for (int r = 0; r < Br::Turn::REGION_BARS; ++r) mbar_init(bars + Br::AFREE + 8u * (uint32_t)r, 1);
  }
  for (int i = tid; i < (T::A1_BYTES + T::B2_BYTES) / 16; i += T::THREADS)
    st_shared(A1 + 16u * (uint32_t)i, __ldg(p.mats + i));
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, s_tmem, 0);
  bool ok = true;

  if (warp < T::TMEM_WARPS) {
    // ---------------- P2 and P4 of chain x ----------------
    const int x = warp / T::CHAIN_WARPS, quad = warp & 3, part = (warp >> 2) % T::PARTS;
    const uint32_t bar = bars + 8u * (uint32_t)x;  // the chain's
    const uint32_t lanes = tmem + ((uint32_t)(quad * 32) << 16);
    // of the warp's first task: with two warps per quadrant the second takes
    // the upper halves of the 31-digits
    const uint32_t d_col = lanes + (uint32_t)(x * T::N1);
    const uint32_t a_col = lanes + (uint32_t)T::A2_COL;
    const uint32_t p2_d = d_col + (uint32_t)(16 * part), p2_a = a_col + (uint32_t)(8 * part);
    // A2's lanes that no row fills stay zero (so their outputs are zero and
    // the maximum may run over all lanes)
    if (part == 0 && x == 0) {
#pragma unroll
      for (int c = 0; c < T::A2S * T::A2_COLS; c += 8) tmem_st_zero8(a_col + (uint32_t)c);
      tmem_wait_st();
    }
    // A1's first K steps: this lane's row, two K entries per column
    if (x == 0 && part == 0) {
#pragma unroll
      for (int c = 0; c < 2 * T::A1_KS; ++c) {
        const uint4 w = ld_shared(A1 + (uint32_t)(c * 2048 + (quad * 32 + lane) * 16));
        asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(
                         lanes + (uint32_t)(T::A1_COL + 4 * c)),
                     "r"(w.x), "r"(w.y), "r"(w.z), "r"(w.w)
                     : "memory");
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bars + Br::A1);
    }
    asm volatile("bar.sync 1, %0;" ::"n"(32 * T::TMEM_WARPS) : "memory");
    // ---- P2: tasks (16-lane group lg, block, half of its 31-digits) of the
    // quadrant, every PARTS-th one, PB at a time: the loads of a batch go out
    // before the batch before is rounded and stored.  All TMEM addresses are the
    // warp's base plus a constant (tcgen05.ld takes a uniform register; a
    // rolled loop that computed them took 1.4 times the kernel's time) ----
    constexpr int TASKS = 4 * NB / T::PARTS, PB = NCB ? 1 : 2;
    const bool two = quad + 4 < T::BLK;  // the quadrant's second lane group has rows
    uint32_t pv[2][PB][2][8];
    // task i of the warp: c = 2 block + half
    auto task = [&](int i, int& lg, int& c) {
      const int t = T::PARTS * i;
      lg = t / (2 * NB);
      c = t - lg * 2 * NB;
    };
    auto p2_load = [&](int i0) {
#pragma unroll
      for (int i = 0; i < PB; ++i) {
        int lg, c;
        task(i0 + i, lg, c);
        if (i0 + i < TASKS && (lg == 0 || two)) {
          const uint32_t a = p2_d + ((uint32_t)(16 * lg) << 16) + (uint32_t)(64 * (c >> 1) + 16 * (c & 1));
          tmem_ld_pairs(a, pv[(i0 / PB) & 1][i][0]);
          tmem_ld_pairs(a + 32, pv[(i0 / PB) & 1][i][1]);
        }
      }
    };
    auto p2_store = [&](int i0, uint32_t region) {
#pragma unroll
      for (int i = 0; i < PB; ++i) {
        int lg, c;
        task(i0 + i, lg, c);
        if (i0 + i < TASKS && (lg == 0 || two)) {
          const uint32_t(&v0)[8] = pv[(i0 / PB) & 1][i][0], (&v1)[8] = pv[(i0 / PB) & 1][i][1];
          uint32_t re[4], im[4];
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            // (re, im) of columns x and x + 4, for h = 0 and 1
            float2 a0 = f2_bits(v0[4 * k], v0[4 * k + 1]), b0 = f2_bits(v0[4 * k + 2], v0[4 * k + 3]);
            float2 a1 = f2_bits(v1[4 * k], v1[4 * k + 1]), b1 = f2_bits(v1[4 * k + 2], v1[4 * k + 3]);
            if (T::H2) {
              const float2 as = add2(a0, a1), bs = add2(b0, b1);
              a1 = sub2(a0, a1);
              b1 = sub2(b0, b1);
              a0 = as;
              b0 = bs;
            }
            re[2 * k] = pack_h2_sat(make_float2(a0.x, b0.x));
            re[2 * k + 1] = pack_h2_sat(make_float2(a1.x, b1.x));
            im[2 * k] = pack_h2_sat(make_float2(a0.y, b0.y));
            im[2 * k + 1] = pack_h2_sat(make_float2(a1.y, b1.y));
          }
          const uint32_t a = p2_a + region + ((uint32_t)(16 * lg) << 16) + (uint32_t)(32 * (c >> 1) + 8 * (c & 1));
          tmem_st_pairs(a, re);
          tmem_st_pairs(a + 16, im);
        }
      }
    };
    auto p2 = [&](uint32_t region) {
      p2_load(0);
#pragma unroll
      for (int i0 = 0; i0 < TASKS; i0 += PB) {
        tmem_wait_ld();
        if (i0 + PB < TASKS) p2_load(i0 + PB);
        p2_store(i0, region);
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar + Br::A2);
    };
    // ---- M2, by the chain's first warp ----
    const uint64_t db2 = desc_sw128(B2);
    auto m2 = [&](auto xc, int reg) {
      constexpr int cx = decltype(xc)::value;
      const uint32_t region = (uint32_t)(reg * T::A2_COLS);
#pragma unroll
      for (int k = 0; k < NB; ++k)
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)
          mma_f16_ta(tmem + (uint32_t)(cx * T::N1 + 64 * k),
                     tmem + region + (uint32_t)(T::A2_COL + 32 * k + 8 * ks),
                     db2 + (uint64_t)(2 * ks), idesc_f16(64, false), ks > 0 ? 1u : 0u);
      mma_commit(bars + Br::M2 + 8u * cx);
      if (Br::Turn::REGION_BARS) mma_commit(bars + Br::AFREE + 8u * (uint32_t)reg);
    };
    // ---- P4: the warp's 1 / PARTS of the outputs t2 of every block, for the
    // thread's row; two adjacent outputs are one packed value ----
    constexpr int COLS = 64 / T::PARTS, PCOLS = NCB ? 4 : 8, PIECES = COLS / PCOLS, PK = PCOLS / 4;
    static_assert(PIECES % 2 == 0, "two buffers");
    float2 sums[NCB ? NB : 1][COLS / 4];
    auto p4_load = [&](int pc, uint32_t(&v)[NB][PCOLS]) {
      const uint32_t d = d_col + (uint32_t)(COLS * part + PCOLS * pc);
#pragma unroll
      for (int b = 0; b < NB; ++b) tmem_ld_cols(d + (uint32_t)(64 * b), v[b]);
    };
    auto p4_piece = [&](int pc, const uint32_t(&v)[NB][PCOLS], bool first, bool last, float& best) {
#pragma unroll
      for (int k = 0; k < PK; ++k) {
        float2 re[NB], im[NB];
#pragma unroll
        for (int b = 0; b < NB; ++b) {
          re[b] = f2_bits(v[b][4 * k], v[b][4 * k + 1]);
          im[b] = f2_bits(v[b][4 * k + 2], v[b][4 * k + 3]);
        }
        if constexpr (T::B3) {
          // inverse DFT-3 over the blocks
          const float2 mh = make_float2(-0.5f, -0.5f), sp = make_float2(0.8660254f, 0.8660254f),
                       sm = make_float2(-0.8660254f, -0.8660254f);
          const float2 tr = add2(re[1], re[2]), ti = add2(im[1], im[2]);
          const float2 ur = sub2(re[1], re[2]), ui = sub2(im[1], im[2]);
          const float2 mr = __ffma2_rn(tr, mh, re[0]), mi = __ffma2_rn(ti, mh, im[0]);
          re[0] = add2(re[0], tr);
          im[0] = add2(im[0], ti);
          re[1] = __ffma2_rn(ui, sm, mr);
          im[1] = __ffma2_rn(ur, sp, mi);
          re[2] = __ffma2_rn(ui, sp, mr);
          im[2] = __ffma2_rn(ur, sm, mi);
        }
#pragma unroll
        for (int b = 0; b < NB; ++b) {
          if constexpr (NCB) {
            // these sums only rank rows for the FP32 re-evaluation, which
            // recomputes the chosen values
            float2& sum = sums[b][PK * pc + k];
            const float2 z = make_float2(0.f, 0.f);
            sum = __ffma2_rn(re[b], re[b], __ffma2_rn(im[b], im[b], first ? z : sum));
            if (last) best = fmaxf(best, fmaxf(sum.x, sum.y));
          } else {
            const float2 pw = __ffma2_rn(re[b], re[b], __fmul2_rn(im[b], im[b]));
            best = fmaxf(best, fmaxf(pw.x, pw.y));
          }
        }
      }
    };
    auto p4 = [&](bool first, bool last) -> float {
      float best = 0.f, best2 = 0.f;
      uint32_t va[NB][PCOLS], vb[NB][PCOLS];
      p4_load(0, va);
#pragma unroll
      for (int pc = 0; pc < PIECES; pc += 2) {
        tmem_wait_ld();
        p4_load(pc + 1, vb);
        p4_piece(pc, va, first, last, best);
        tmem_wait_ld();
        if (pc + 2 < PIECES) {
          p4_load(pc + 2, va);
        } else {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar + Br::DFREE);
        }
        p4_piece(pc + 1, vb, first, last, best2);
      }
      return fmaxf(best, best2);
    };
    uint32_t use = 0;  // of the chain
    int s = 0;         // chain of the next step (drop-in search: steps run on across units)
    for (Units<NCB> u(p); u.more() && ok; u.next()) {
      const int ab_h = u.w / p.groups;
      for (int r = u.r0; r < u.r1 && ok; ++r) {
        if (!NCB) {
          const bool mine = s == x;
          s = s + 1 == T::NCH ? 0 : s + 1;
          if (!mine) continue;
        }
#pragma unroll 1
        for (int blk = 0; blk < B; ++blk, ++use) {
          // D1 is there, and the step's A2 is free (A2Turn)
          const int step = (int)use * T::NCH + x, reg = Br::Turn::region(step);
          if (Br::Turn::WAITS)
            ok = warp_wait2(bar + Br::M1, use & 1u,
                            bars + (Br::Turn::REGION_BARS ? Br::AFREE : Br::M2) + 8u * (uint32_t)Br::Turn::bar(step),
                            Br::Turn::parity(step));
          else
            ok = warp_wait(bar + Br::M1, use & 1u);
          if (!ok) break;
          tc_fence_after();
          p2((uint32_t)(reg * T::A2_COLS));
          if (warp == x * T::CHAIN_WARPS) {
            if (!(ok = warp_wait(bar + Br::A2, use & 1u))) break;
            tc_fence_after();
            if (elect_one()) {
              if (x == 0)
                m2(std::integral_constant<int, 0>(), reg);
              else if (x == 1)
                m2(std::integral_constant<int, 1>(), reg);
              else
                m2(std::integral_constant<int, T::NCH - 1>(), reg);
            }
            __syncwarp();
          }
          if (!(ok = warp_wait(bar + Br::M2, use & 1u))) break;
          tc_fence_after();
          const float best = p4(blk == 0, blk + 1 == B);
          if (blk + 1 == B) {
            // non-negative floats order like their bit patterns
            const unsigned bits = __reduce_max_sync(0xffffffffu, __float_as_uint(best));
            int prn = NCB ? 2 * r + x : r;
            if (prn >= p.n_prn) prn = p.n_prn - 1;
            if (lane == 0 && bits != 0u)
              atomicMax(p.keys + (size_t)ab_h * p.n_prn + prn, (unsigned long long)bits << 32);
          }
        }
      }
    }
    // drain: the commit on a region's barrier that no later step waits for (of
    // the CTA's n steps the last ones of every region)
    if (Br::Turn::REGION_BARS > 0 && ok && use > 0 && warp == x * T::CHAIN_WARPS) {
      const int n = ((int)use - (x < s ? 1 : 0)) * T::NCH + s, last = ((int)use - 1) * T::NCH + x;
      if (last >= n - T::A2S)
        ok = warp_wait(bars + Br::AFREE + 8u * (uint32_t)Br::Turn::region(last), (uint32_t)(last / T::A2S) & 1u);
    }
  } else if (warp < T::M1_WARP) {
    // ---------------- P1: FP16 products ----------------
    // thread (j, d1): its slots are T::PROD_THREADS units apart, and their
    // rows in the products a whole column group (4 strides)
    const int pt = tid - 32 * T::TMEM_WARPS, j = pt / U::R1P, d1 = pt - j * U::R1P;
    const uint32_t dst0 = PROD + (uint32_t)(j * T::STRIDE_B + d1 * 16), code0 = CODE + 16u * (uint32_t)pt;
    const uint32_t zs = ZS + 16u * (uint32_t)pt;
    uint4 z[T::GRK][RES][2];
    auto load_z = [&](int w, int blk) {
      const int ab_h = w / p.groups, rho0 = (w - ab_h * p.groups) * RES;
      const uint4* seq = p.z16 + (((size_t)ab_h * B + blk) * S + rho0) * U::PER_SEQ + pt;
#pragma unroll
      for (int r = 0; r < RES; ++r)
#pragma unroll
        for (int k = GR - 1; k >= 0; --k) {
          uint4 v[2] = {make_uint4(0u, 0u, 0u, 0u), make_uint4(0u, 0u, 0u, 0u)};
          if (rho0 + r < S) {
            const uint4* src = seq + r * U::PER_SEQ + k * T::PROD_THREADS;
            // the drop-in search reads its Z once (evict first); the
            // non-coherent search reads each block again for every PRN
            v[0] = NCB ? __ldcg(src) : __ldcs(src);
            v[1] = NCB ? __ldcg(src + U::UNITS) : __ldcs(src + U::UNITS);
          }
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            if (k < T::GRK)
              z[k][r][c] = v[c];
            else
              st_shared(zs + (uint32_t)((2 * r + c) * T::PROD_THREADS * 16), v[c]);
          }
        }
    };
    // the products of step s with code block n
    auto products = [&](int s, int n, bool new_code) -> bool {
      const uint32_t use = (uint32_t)s / T::NCH, x = (uint32_t)s - use * T::NCH, slot = (uint32_t)n % T::SLOTS;
      // the code block, and the buffer (M1 of step s - NCH; before that the phase
      // ahead of the barrier's first counts as complete)
      const uint32_t m1 = bars + Br::M1 + 8u * x, m1_ph = (use & 1u) ^ 1u;
      if (new_code ? !warp_wait2(bars + Br::CODE + 8u * slot, (uint32_t)(n / T::SLOTS) & 1u, m1, m1_ph)
                   : !warp_wait(m1, m1_ph))
        return false;
      {
        const uint32_t dst = dst0 + x * T::B_BYTES, code = code0 + slot * T::CODE_REGION;
        // the next unit's code is loaded ahead of this one's products (a load
        // does not pass the stores before it)
        uint4 cr = ld_shared(code), ci = ld_shared(code + 16 * U::UNITS);
#pragma unroll
        for (int k = 0; k < GR; ++k) {
          uint4 nr = cr, ni = ci;
          if (k + 1 < GR) {
            nr = ld_shared(code + 16 * (k + 1) * T::PROD_THREADS);
            ni = ld_shared(code + 16 * (k + 1) * T::PROD_THREADS + 16 * U::UNITS);
          }
#pragma unroll
          for (int r = 0; r < RES; ++r) {
            const uint4 zr = k < T::GRK ? z[k][r][0] : ld_shared(zs + (uint32_t)(2 * r * T::PROD_THREADS * 16));
            const uint4 zi = k < T::GRK ? z[k][r][1] : ld_shared(zs + (uint32_t)((2 * r + 1) * T::PROD_THREADS * 16));
            uint4 re, im;
            cmul_h2(zr.x, zi.x, cr.x, ci.x, re.x, im.x);
            cmul_h2(zr.y, zi.y, cr.y, ci.y, re.y, im.y);
            cmul_h2(zr.z, zi.z, cr.z, ci.z, re.z, im.z);
            cmul_h2(zr.w, zi.w, cr.w, ci.w, re.w, im.w);
            // column group of (left-over digits k, residue r)
            const int cg = M == 10 ? k : M == 4 ? 2 * k + r : r;
            st_shared(dst + (uint32_t)(cg * 4 * T::STRIDE_B), re);
            st_shared(dst + (uint32_t)(cg * 4 * T::STRIDE_B + T::KH * 16), im);
          }
          cr = nr;
          ci = ni;
        }
      }
      fence_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(bars + Br::PROD + 8u * x);
      return true;
    };
    int s = 0, n = 0;
    Units<NCB> u(p);
    if (u.more()) load_z(u.w, 0);
    while (u.more() && ok) {
      for (int r = u.r0; r < u.r1 && ok; ++r) {
        if constexpr (NCB) {
#pragma unroll 1
          for (int blk = 0; blk < B && ok; ++blk, s += 2) {
            ok = products(s, n, blk == 0) && products(s + 1, n + 1, blk == 0);
            // the next block's Z, while the products' buffers are in use
            if (blk + 1 < B) load_z(u.w, blk + 1);
          }
          n += 2;
        } else {
          ok = products(s, n, true);
          ++s;
          ++n;
        }
      }
      u.next();
      if (u.more()) load_z(u.w, 0);
    }
  } else {
    if (elect_one()) ok = m1_role<M, NCB>(p, bars, A1, PROD, CODE, tmem);
  }
  if (!ok) atomicExch(p.err, 1);
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0) tmem_dealloc(tmem, kTcTmemCols);
}

template <int M, bool NCB>
cudaError_t run_tc(const PolyClass& pc, const SearchDims& dims, int B, const void* d_mats, const void* d_z16,
                   const void* d_d16, unsigned long long* d_keys, int* d_err, int test_flags, int num_sms,
                   cudaStream_t st) {
  using T = Tc<M, NCB>;
  TcParams p = {};
  p.skip_commit = test_flags & 1;
  p.mats = static_cast<const uint4*>(d_mats);
  p.z16 = static_cast<const uint4*>(d_z16);
  p.d16 = static_cast<const uint4*>(d_d16);
  p.keys = d_keys;
  p.err = d_err;
  p.n_prn = dims.n_prn;
  p.S = pc.S;
  p.groups = (pc.S + T::RES - 1) / T::RES;
  p.B = NCB ? B : 1;
  p.n_items = dims.n_ant * dims.nb * (NCB ? 1 : 2) * p.groups;
  if (p.n_items < 1 || p.n_prn < 1) return cudaSuccess;
  p.n_rounds = NCB ? (p.n_prn + 1) / 2 : p.n_prn;
  // Non-coherent: a unit is one round, so the CTAs take neighbouring rounds at
  // any time and share an item's Z (read for every round) in L2, and no CTA has
  // more than one round more than another.  Whole items, split only when there
  // were fewer than SMs, left up to 43 % of the SMs idle in a last pass (one
  // antenna, 21 bins, 100 blocks: 8.2 -> 4.5 ms at Lc = 1023, 9.0 -> 7.4 at 4092,
  // 45.1 -> 43.2 at 10230, which the power limit holds by then).
  // Drop-in: Z is read once per unit, so as few parts as the SMs' shares allow:
  // a unit costs its rounds and about two more to change Z.
  // One antenna, 41 bins: 186 -> 154 us at Lc = 1023, 285 -> 264 at 4092.
  p.split = p.n_rounds;
  if (!NCB) {
    double best = 0.0;
    for (int split = 1; split <= 32 && split <= p.n_rounds; ++split) {
      const long long per_sm = ((long long)p.n_items * split + num_sms - 1) / num_sms;
      const double cost = (double)per_sm * ((p.n_rounds + split - 1) / split + 2.0);
      if (split == 1 || cost < best) {
        best = cost;
        p.split = split;
      }
    }
  }
  auto kern = pfa_tc_kernel<M, NCB>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, T::SMEM);
  if (e != cudaSuccess) return e;
  // one CTA per SM: T::SMEM is above half of the SM's shared memory, so the
  // 512-column TMEM allocation never meets another one
  int grid = num_sms;
  if (grid > p.n_items * p.split) grid = p.n_items * p.split;
  p.step_w = grid / p.split;
  p.step_r = grid % p.split;
  kern<<<grid, T::THREADS, T::SMEM, st>>>(p);
  kernel_launch_add(1);
  return cudaGetLastError();
}

// FP16 scale exponents (kz, kd) of Z and the code spectra, kz + kd = k with
// 4 S Lc^2 2^-k <= 32768
void tc_scales(const PolyClass& pc, int* kz, int* kd) {
  const double bound = 4.0 * pc.S * (double)pc.Lc * (double)pc.Lc;
  int k = 0;
  while (bound / (double)(1ull << k) > 32768.0 && k < 60) ++k;
  *kz = (k + 1) / 2;
  *kd = k - *kz;
}

template <int M>
cudaError_t run_pack(const float2* src, long long n_seq, void* dst, float scale, int num_sms, cudaStream_t st) {
  const long long n_units = n_seq * TcUnits<M>::UNITS;
  if (n_units == 0) return cudaSuccess;
  long long blocks = (n_units + 255) / 256;
  if (blocks > (long long)num_sms * 16) blocks = (long long)num_sms * 16;
  tc_pack_kernel<M><<<(int)blocks, 256, 0, st>>>(src, static_cast<uint4*>(dst), n_units, scale);
  kernel_launch_add(1);
  return cudaGetLastError();
}

}  // namespace

size_t tc_operand_bytes(const PolyClass& pc, long long n_seq) {
  const int units = pc.M == 1 ? TcUnits<1>::PER_SEQ : pc.M == 4 ? TcUnits<4>::PER_SEQ : TcUnits<10>::PER_SEQ;
  return (size_t)n_seq * units * sizeof(uint4);
}

std::vector<unsigned char> tc_dft_matrices(int M) {
  switch (M) {
    case 1: return build_matrices<1>();
    case 4: return build_matrices<4>();
    case 10: return build_matrices<10>();
  }
  return {};
}

double tc_key_amplitude(const PolyClass& pc) {
  int kz = 0, kd = 0;
  tc_scales(pc, &kz, &kd);
  return (double)(1ull << (kz + kd));
}

float tc_z_scale(const PolyClass& pc) {
  int kz = 0, kd = 0;
  tc_scales(pc, &kz, &kd);
  return (float)(1.0 / (double)(1ull << kz));
}

cudaError_t launch_tc_pack(const PolyClass& pc, const float2* d_src, long long n_seq, bool code, void* d_dst,
                           int num_sms, cudaStream_t st) {
  int kz = 0, kd = 0;
  tc_scales(pc, &kz, &kd);
  const float scale = (float)(1.0 / (double)(1ull << (code ? kd : kz)));
  switch (pc.M) {
    case 1: return run_pack<1>(d_src, n_seq, d_dst, scale, num_sms, st);
    case 4: return run_pack<4>(d_src, n_seq, d_dst, scale, num_sms, st);
    case 10: return run_pack<10>(d_src, n_seq, d_dst, scale, num_sms, st);
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_correlate_tc(const PolyClass& pc, const SearchDims& dims, const void* d_mats, const void* d_z16,
                                const void* d_d16, unsigned long long* d_keys, int* d_err, int test_flags,
                                int num_sms, cudaStream_t st) {
  switch (pc.M) {
    case 1: return run_tc<1, false>(pc, dims, 1, d_mats, d_z16, d_d16, d_keys, d_err, test_flags, num_sms, st);
    case 4: return run_tc<4, false>(pc, dims, 1, d_mats, d_z16, d_d16, d_keys, d_err, test_flags, num_sms, st);
    case 10: return run_tc<10, false>(pc, dims, 1, d_mats, d_z16, d_d16, d_keys, d_err, test_flags, num_sms, st);
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_correlate_tc_nc(const PolyClass& pc, const SearchDims& dims, int B, const void* d_mats,
                                   const void* d_z16, const void* d_d16, unsigned long long* d_keys, int* d_err,
                                   int test_flags, int num_sms, cudaStream_t st) {
  if (B < 1) return cudaErrorInvalidValue;
  switch (pc.M) {
    case 1: return run_tc<1, true>(pc, dims, B, d_mats, d_z16, d_d16, d_keys, d_err, test_flags, num_sms, st);
    case 4: return run_tc<4, true>(pc, dims, B, d_mats, d_z16, d_d16, d_keys, d_err, test_flags, num_sms, st);
    case 10: return run_tc<10, true>(pc, dims, B, d_mats, d_z16, d_d16, d_keys, d_err, test_flags, num_sms, st);
  }
  return cudaErrorInvalidValue;
}

}  // namespace tga
