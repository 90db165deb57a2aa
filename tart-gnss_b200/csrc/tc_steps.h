// Order of the tensor-core correlator's steps (acq_tc.cu): which barrier and
// phase a step waits for before it writes its operand region.  Plain C++, so
// that the protocol can be checked on the host.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define TGA_TC_HD __host__ __device__ __forceinline__
#else
#define TGA_TC_HD inline
#endif

namespace tga {

// Steps rotate over NCH chains and A2S operand regions: step s is chain s %
// NCH's and writes region s % A2S, which the second GEMM of step s - A2S reads.
// A waiting warp sees the parity of a barrier's phase alone, so the phase after
// the awaited one must not be able to complete before that warp has seen the
// awaited one.
//  * A2S == NCH: the region is the chain's own, whose last M2 its warps have
//    waited for already.
//  * A2S == 1: the M2 barrier of the chain of step s - 1.  Its next phase is
//    step s - 1 + NCH's, which cannot pass step s: they share the region.
//  * otherwise a barrier per region, which M2 of every step of the region
//    completes: its next phase is step s's own.  The M2 barrier of step s - A2S's
//    chain will not do: with NCH = 3 and A2S = 2 its next phase is step s + 1's,
//    which uses the other region and waits for no warp of step s.
template <int NCH, int A2S>
struct A2Turn {
  static_assert(A2S >= 1 && A2S <= NCH, "regions");
  static constexpr bool WAITS = A2S < NCH;
  static constexpr int REGION_BARS = WAITS && A2S > 1 ? A2S : 0;
  static TGA_TC_HD constexpr int region(int s) { return s % A2S; }
  // the barrier (of a region if REGION_BARS, else a chain's M2) and the parity
  // of the phase; before the first the phase ahead of the barrier's first,
  // which counts as complete
  static TGA_TC_HD constexpr int bar(int s) { return REGION_BARS ? s % A2S : (s + NCH - A2S) % NCH; }
  static TGA_TC_HD constexpr uint32_t parity(int s) {
    return (uint32_t)(REGION_BARS ? s / A2S + 1 : (s + NCH - A2S) / NCH + 1) & 1u;
  }
};

}  // namespace tga

#undef TGA_TC_HD
