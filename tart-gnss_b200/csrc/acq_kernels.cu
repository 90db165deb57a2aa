// CUDA kernels of the B200 acquisition engine (sm_100a).
//
// Fused path.  For a window of two code periods (N = 2P) the reference's
// dual-hypothesis correlation (correlate.rs:91-183) is rewritten exactly:
//
//  1. Fold:  f = x[0:P] + x[P:2P] gives the [c,c] correlation; the [c,-c]
//     correlation is the negacyclic correlation of g = x[0:P] - x[P:2P].
//  2. Polyphase: the resampled code is c(n) = chip((n / S) mod Lc) * pulse(n % S)
//     (S samples per chip, P = S * Lc).  Then for every lag tau = rho + S*t
//        r(tau) = sum_m chip(m) z_rho(m + t),   z_rho(j) = sum_s pulse(s) f(S j + rho + s)
//     i.e. S independent circular correlations of length Lc (the chip count,
//     1023 / 4092 / 10230) instead of one of length 2P.  The negacyclic
//     branch is made cyclic by the twist v(j) = exp(i pi j / Lc).
//  3. Every Lc is 31 * 33 * M (M = 1, 4, 10), pairwise coprime, so each
//     length-Lc DFT is a twiddle-free Good-Thomas transform: a DFT-31 stage
//     fed straight from global memory (Z * conj(D) formed in registers), a
//     DFT-33 stage and a DFT-M stage through shared memory.  The last stage
//     feeds |y|^2 straight into the argmax; no correlation vector ever
//     leaves the SM.
//
// Frequency-domain arrays use the digit layout [k31][kM][k33]; time-domain
// lag digits map to natural lags by the Chinese remainder theorem.
//
// Generic path (any N, generic_kernels.cu): the reference algorithm on the GPU,
// with mixed-radix FFTs of length N, or Bluestein's where N has a large prime.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include <atomic>
#include <cstdint>
#include <cstdio>
#include <mutex>

#include "dft.cuh"
#include "engine.h"
#include "gnss_tables.h"
#include "pfa_common.cuh"

namespace tga {

// Launches of the calling host thread: a search runs on the thread that
// called the entry point, so a per-thread count is that call's count even
// when several contexts run on several threads at once.
static thread_local int g_launches = 0;
int kernel_launch_count_reset() {
  int v = g_launches;
  g_launches = 0;
  return v;
}
int kernel_launch_count() { return g_launches; }
void kernel_launch_add(int n) { g_launches += n; }

#define TGA_LAUNCHED() (++g_launches, cudaGetLastError())

// ---------------------------------------------------------------------------
// antenna means: mean of the +-1 samples over the whole row (acquisition.rs:285)
// ---------------------------------------------------------------------------
// One CTA per row, bound by the latency of its loads: 16-byte words from the
// first aligned byte on, four of them in flight per thread, and the bytes
// before and after one by one (a row may start anywhere).  Byte loads for
// rows off an 8-byte boundary took 141 us in a search where this takes 10.
__global__ void __launch_bounds__(1024) antenna_means_kernel(const uint8_t* __restrict__ bits, size_t row_bytes,
                                                             double* __restrict__ mean) {
  const uint8_t* row = bits + (size_t)blockIdx.x * row_bytes;
  unsigned long long ones = 0;
  const size_t head = min(row_bytes, (size_t)(-(uintptr_t)row & 15));
  const size_t n_words = (row_bytes - head) / 16;
  const uint4* w = reinterpret_cast<const uint4*>(row + head);
#pragma unroll 4
  for (size_t i = threadIdx.x; i < n_words; i += blockDim.x) {
    const uint4 v = __ldg(w + i);
    ones += __popc(v.x) + __popc(v.y) + __popc(v.z) + __popc(v.w);
  }
  if (threadIdx.x < head) ones += __popc(row[threadIdx.x]);
  const size_t tail = head + n_words * 16 + threadIdx.x;
  if (tail < row_bytes) ones += __popc(row[tail]);
  for (int o = 16; o > 0; o >>= 1) ones += __shfl_xor_sync(0xffffffffu, ones, o);
  __shared__ unsigned long long part[32];
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = ones;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long t = 0;
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) t += part[i];
    const double n = (double)(row_bytes * 8);
    // sum of +-1 over the row is the exact integer 2*ones - n
    mean[blockIdx.x] = (double)(2.0 * (double)t - n) / n;
  }
}

cudaError_t launch_antenna_means(const uint8_t* d_bits, int n_rows, size_t row_bytes, double* d_mean,
                                 cudaStream_t st) {
  if (n_rows <= 0) return cudaSuccess;
  antenna_means_kernel<<<n_rows, 1024, 0, st>>>(d_bits, row_bytes, d_mean);
  return TGA_LAUNCHED();
}

// ---------------------------------------------------------------------------
// front end: carrier wipe-off (correlate.rs:110-115), fold, polyphase boxcar
// ---------------------------------------------------------------------------
struct FrontParams {
  SampleSource src;
  const double* fc;
  int nb, P, S, Lc;
  float pulse[kMaxPulse];
  // pulse shape: 0 any, 1 constant w0, 2 w0 for the first S / 2 samples and
  // -w0 for the rest (BOC(1, 1)); 1 and 2 let the polyphase sums run
  int pulse_kind;
  float pulse_w0;
  int n_grp;  // antennas per CTA
  float2* z;
};

constexpr int kFrontJ = 64;  // chips per CTA

// carrier phasor of sample n (as double, nd): exp(i (p * freq) as f32)
template <bool BITS>
__device__ __forceinline__ float2 carrier(const FrontParams& p, int n, double nd, double f) {
  const double ph = BITS ? (p.src.pc * nd) * f : __ldg(p.src.pp + n) * f;  // phasepoint * freq
  float sn, cs;
  sincos_phase(__double2float_rn(ph), &sn, &cs);
  return make_float2(cs, sn);
}

// One CTA: kFrontJ chips of one Doppler bin, folded samples in shared memory,
// polyphase sums from there.  Bound by issue slots, the phasors more than the
// sums with one antenna.  The phasor of a sample is the same for every antenna:
// with p.n_grp > 1 a CTA computes its phasors once, keeps them in shared memory,
// and takes n_grp antennas one after the other (24 antennas, all bins: 3.2 ms
// when every antenna computed them, 1.9 ms).
template <bool BITS, bool GROUP>
__global__ void __launch_bounds__(256) frontend_kernel(FrontParams p) {
  extern __shared__ __align__(16) float2 fsm[];
  const int S = p.S, P = p.P, Lc = p.Lc;
  const int grp = blockIdx.y / p.nb, bin = blockIdx.y - grp * p.nb;
  const int ant0 = GROUP ? grp * p.n_grp : grp, ant1 = GROUP ? min(ant0 + p.n_grp, p.src.n_ant) : ant0 + 1;
  const double f = p.fc[bin];
  const int j0 = blockIdx.x * kFrontJ;
  const int nj = min(kFrontJ, Lc - j0);
  const int cnt = nj * S + S - 1;
  const int span = kFrontJ * S + S;
  float2* fsh = fsm;                         // padded: index i + i/S
  float2* gsh = fsm + span + span / S + 1;
  float2* tw = gsh + span + span / S + 1;    // twist per chip
  float2* ph0 = tw + kFrontJ;                // GROUP: phasors of samples m and m + P
  float2* ph1 = ph0 + span;
  for (int jj = threadIdx.x; jj < nj; jj += blockDim.x) {
    double sn, cs;
    sincospi((double)(j0 + jj) / (double)Lc, &sn, &cs);
    tw[jj] = make_float2((float)cs, (float)sn);
  }
  if (GROUP) {
    double nd = (double)(S * j0 + (int)threadIdx.x);
    for (int i = threadIdx.x; i < cnt; i += 256, nd += 256.0) {
      int m = S * j0 + i;
      double md = nd;
      if (m >= P) m -= P, md -= (double)P;
      ph0[i] = carrier<BITS>(p, m, md, f);
      ph1[i] = carrier<BITS>(p, m + P, md + (double)P, f);
    }
  }
  for (int ant_slot = ant0; ant_slot < ant1; ++ant_slot) {
    if (GROUP && ant_slot != ant0) __syncthreads();  // the sums have read the last antenna's samples
    const int ab = ant_slot * p.nb + bin;
    const int row = p.src.ant[ant_slot];
    float s_one = 0.f, s_zero = 0.f;
    const uint8_t* bits = nullptr;
    const float* sig = nullptr;
    if (BITS) {  // (v - mean) as f32, v = +-1
      const double mean = __ldg(p.src.mean + row);
      s_one = (float)(1.0 - mean);
      s_zero = (float)(-1.0 - mean);
      bits = p.src.bits + (size_t)row * p.src.row_bytes;
    } else {
      sig = p.src.sig + (size_t)row * p.src.n_samples;
    }
    auto sample = [&](int n) {
      return BITS ? ((__ldg(bits + (n >> 3)) >> (7 - (n & 7))) & 1 ? s_one : s_zero) : __ldg(sig + n);
    };
    {
      // i / S and i mod S, carried along
      const int dq = 256 / S, dr = 256 - dq * S;
      int iq = threadIdx.x / S, ir = threadIdx.x - iq * S;
      double nd = (double)(S * j0 + (int)threadIdx.x);
      for (int i = threadIdx.x; i < cnt; i += 256) {
        int m = S * j0 + i;
        float sign = 1.f;
        if (m >= P) {  // wrap of the last chip: f is P-periodic, g antiperiodic
          m -= P;
          sign = -1.f;
        }
        float2 c0, c1;
        if (GROUP) {
          c0 = ph0[i];
          c1 = ph1[i];
        } else {
          const double md = sign < 0.f ? nd - (double)P : nd;
          c0 = carrier<BITS>(p, m, md, f);
          c1 = carrier<BITS>(p, m + P, md + (double)P, f);
          nd += 256.0;
        }
        const float s0 = sample(m), s1 = sample(m + P);
        const float2 x0 = make_float2(c0.x * s0, c0.y * s0);
        const float2 x1 = make_float2(c1.x * s1, c1.y * s1);
        const int pi = i + iq;
        fsh[pi] = cadd(x0, x1);
        const float2 g = csub(x0, x1);
        gsh[pi] = make_float2(g.x * sign, g.y * sign);
        iq += dq;
        ir += dr;
        if (ir >= S) ir -= S, ++iq;
      }
    }
    __syncthreads();
    const size_t seqA = ((size_t)ab * 2 + 0) * S, seqB = ((size_t)ab * 2 + 1) * S;
    if (p.pulse_kind != 0 && S >= 4) {
      // runs of L = S / 4 residues per thread: the first sum directly, each
      // next one from the previous (2 or 3 samples instead of S):
      //   constant w0:   z(rho + 1) = z(rho) + w0 (f[a + S] - f[a])
      //   w0 / -w0:      z(rho + 1) = z(rho) + w0 (2 f[a + S/2] - f[a] - f[a + S])
      // with a = jj S + rho; sample i sits at padded index i + i / S
      const int L = (S + 3) / 4;
      const float w0 = p.pulse_w0;
      const bool boc = p.pulse_kind == 2;
      const int H = S / 2;
      for (int o = threadIdx.x; o < 4 * nj; o += blockDim.x) {
        const int k = o / nj, jj = o - k * nj;
        const int rho0 = k * L, rho1 = min(rho0 + L, S);
        if (rho0 >= S) continue;
        float2 za = make_float2(0.f, 0.f), zb = make_float2(0.f, 0.f);
        const int base = jj * S + rho0 + jj;
        auto taps = [&](int s0, int s1, int at) {
#pragma unroll 4
          for (int s = s0; s < s1; ++s) {
            const float2 w = make_float2(p.pulse[s], p.pulse[s]);
            za = __ffma2_rn(w, fsh[at + s], za);
            zb = __ffma2_rn(w, gsh[at + s], zb);
          }
        };
        taps(0, S - rho0, base);  // up to the next chip's padding
        taps(S - rho0, S, base + 1);
        const int j = j0 + jj;
        p.z[(seqA + rho0) * Lc + j] = za;
        p.z[(seqB + rho0) * Lc + j] = cmul(zb, tw[jj]);
        for (int rho = rho0; rho + 1 < rho1; ++rho) {
          const int a = jj * S + rho;
          const int pa = a + jj, pe = a + S + jj + 1;
          if (boc) {
            const int pm = a + H + jj + (rho + H >= S ? 1 : 0);
            za.x += w0 * (2.f * fsh[pm].x - fsh[pa].x - fsh[pe].x);
            za.y += w0 * (2.f * fsh[pm].y - fsh[pa].y - fsh[pe].y);
            zb.x += w0 * (2.f * gsh[pm].x - gsh[pa].x - gsh[pe].x);
            zb.y += w0 * (2.f * gsh[pm].y - gsh[pa].y - gsh[pe].y);
          } else {
            za.x += w0 * (fsh[pe].x - fsh[pa].x);
            za.y += w0 * (fsh[pe].y - fsh[pa].y);
            zb.x += w0 * (gsh[pe].x - gsh[pa].x);
            zb.y += w0 * (gsh[pe].y - gsh[pa].y);
          }
          p.z[(seqA + rho + 1) * Lc + j] = za;
          p.z[(seqB + rho + 1) * Lc + j] = cmul(zb, tw[jj]);
        }
      }
      continue;
    }
    for (int o = threadIdx.x; o < S * nj; o += blockDim.x) {
      const int rho = o / nj, jj = o - rho * nj;
      float2 za = make_float2(0.f, 0.f), zb = make_float2(0.f, 0.f);
      // tap s reads sample i = jj S + rho + s at padded index i + i / S, and
      // i / S = jj + (rho + s >= S) since rho + s < 2 S: no division per tap
      const int base = jj * S + rho + jj;
      for (int s = 0; s < S; ++s) {
        const int pi = base + s + (rho + s >= S ? 1 : 0);
        const float w = p.pulse[s];
        za.x = fmaf(w, fsh[pi].x, za.x);
        za.y = fmaf(w, fsh[pi].y, za.y);
        zb.x = fmaf(w, gsh[pi].x, zb.x);
        zb.y = fmaf(w, gsh[pi].y, zb.y);
      }
      const int j = j0 + jj;
      p.z[(seqA + rho) * Lc + j] = za;
      p.z[(seqB + rho) * Lc + j] = cmul(zb, tw[jj]);
    }
  }
}

cudaError_t launch_frontend(const SampleSource& src, const SearchDims& dims, const PolyClass& pc,
                            float2* d_z, cudaStream_t st) {
  FrontParams p;
  p.src = src;
  p.fc = dims.fc;
  p.nb = dims.nb;
  p.P = pc.P;
  p.S = pc.S;
  p.Lc = pc.Lc;
  for (int i = 0; i < kMaxPulse; ++i) p.pulse[i] = pc.pulse[i];
  // the pulse's shape (see FrontParams)
  p.pulse_w0 = pc.pulse[0];
  bool constant = true, boc = pc.S % 2 == 0;
  for (int i = 0; i < pc.S; ++i) {
    constant = constant && pc.pulse[i] == pc.pulse[0];
    boc = boc && pc.pulse[i] == (i < pc.S / 2 ? pc.pulse[0] : -pc.pulse[0]);
  }
  p.pulse_kind = constant ? 1 : (boc ? 2 : 0);
  p.z = d_z;
  const int span = kFrontJ * pc.S + pc.S;
  const size_t smem = (size_t)(2 * (span + span / pc.S + 1) + kFrontJ) * sizeof(float2);
  const int tiles = (pc.Lc + kFrontJ - 1) / kFrontJ;
  // antennas per CTA: as many as leave kFrontCtas CTAs, about three waves
  constexpr int kFrontCtas = 2048;
  p.n_grp = 1;
  if (src.bits)
    p.n_grp = (int)std::min<long long>(
        dims.n_ant, std::max<long long>(1, (long long)tiles * dims.nb * dims.n_ant / kFrontCtas));
  const dim3 grid(tiles, (dims.n_ant + p.n_grp - 1) / p.n_grp * dims.nb);
  auto run = [&](auto kern, size_t bytes) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return e;
    kern<<<grid, 256, bytes, st>>>(p);
    return TGA_LAUNCHED();
  };
  const size_t group_smem = smem + (size_t)2 * span * sizeof(float2);
  if (!src.bits) return run(frontend_kernel<false, false>, smem);
  return p.n_grp > 1 ? run(frontend_kernel<true, true>, group_smem) : run(frontend_kernel<true, false>, smem);
}

// ---------------------------------------------------------------------------
// prime-factor transform engine
// ---------------------------------------------------------------------------
template <int M, int BC, int NT, int MINB, int MODE>
__global__ void __launch_bounds__(NT, MINB) pfa_kernel(PfaParams p) {
  using G = Geo<M>;
  constexpr int COLS = G::COLS, LC = G::LC, NC = G::NC;
  constexpr bool INV = (MODE == CORR || MODE == SECOND || MODE == CAND);
  constexpr bool ARGMAX = (MODE == CORR || MODE == CAND);
  extern __shared__ __align__(16) float2 buf[];
  __shared__ unsigned long long s_key;
  __shared__ unsigned int s_p2;
  __shared__ unsigned int s_floor;
  __shared__ bool s_last;
  // CAND with p2rows: for every residue of the row and every warp that
  // scanned it, its four largest |y|^2 as (value bits << 32) | lag, after
  // the transform buffer (TOP_WPS warps per residue)
  constexpr bool TOP = MODE == CAND;
  constexpr int TOP_WPS = NT / 32 / BC >= 1 ? NT / 32 / BC : 1;
  static_assert(TOP_WPS <= kTopWarps, "lists of a split row");
  unsigned long long* s_res = reinterpret_cast<unsigned long long*>(buf + BC * LC);
  const bool keep_top = TOP && p.p2rows != nullptr;
  const int tid = threadIdx.x;
  const int S = p.S;
  const int groups = INV ? (S + BC - 1) / BC : 1;
  // Work units: row w / split, residue groups [g0, g1) of part w % split.  With
  // fewer rows than CTAs in flight a row's groups are shared out (one row took
  // its 16 groups of Lc = 10230 one after the other on one SM: 115 us for the
  // second peak of one PRN, 15 us so, and 133 against 79 us for its 42 rows);
  // the parts meet in an atomic maximum, which keeps the tie rule (keys order
  // by value, then lag).  CORR's split comes from the host, which zeroes the
  // keys; CAND's from the number of rows listed.
  const int rows = MODE == CAND ? min(p.n_items, *p.cand_count) : p.n_items;
  const int split = MODE == CAND ? (rows > 0 ? max(1, min(groups, (int)gridDim.x / rows)) : 1) : max(1, p.split);
  const int n_work = INV ? rows * split : (p.n_seq + BC - 1) / BC;

  for (int unit = blockIdx.x; unit < n_work; unit += gridDim.x) {
    const int w = INV ? unit / split : unit, part = INV ? unit - w * split : 0;
    const int g0 = INV ? part * groups / split : 0, g1 = INV ? (part + 1) * groups / split : groups;
    int ab_h = 0, prn = 0, tau_star = 0;
    if (MODE == CORR) {
      ab_h = w / p.n_prn;
      prn = w - ab_h * p.n_prn;
    } else if (MODE == SECOND) {
      const BestRow b = p.best[w];
      ab_h = b.ab * 2 + b.hyp;
      prn = w % p.n_prn;
      tau_star = b.tau;
    } else if (MODE == CAND) {
      const int2 c = p.cand[w];
      ab_h = c.x;
      prn = c.y;
    }
    // where the item's key goes: CORR's item w is the row ab_h * n_prn + prn
    const int key_at = MODE == CAND ? ab_h * p.n_prn + prn : w;
    const int hyp = ab_h & 1;
    // CORR: running maximum of |y|^2 and a compact code of its position
    // ((rho*31 + a)*33 + b)*16 + c; the lag is decoded only on ties and once
    // per item, which keeps the per-output epilogue to a compare and selects.
    float pmax = -1.f;
    int cmax = 0;
    auto lag_of = [&](int code) -> int {
      const int c = code & 15, q = code >> 4;
      const int b = q % 33, q2 = q / 33;
      const int a = q2 % 31, rho = q2 / 31;
      return rho + S * G::natural(a, b, c);
    };
    float pws[NC];
    float floor_pw = -1.f;
    float pbest = 0.f;
    if (tid == 0) {
      s_key = 0ull;
      s_p2 = 0u;
      s_floor = 0u;
    }

    for (int g = g0; g < g1; ++g) {
      if (ARGMAX && NC > 1 && g > g0) floor_pw = fmaxf(floor_pw, __uint_as_float(s_floor));
      // sequence of slot s in this group, or -1 when idle
      auto seq_of = [&](int s) -> int {
        if (INV) {
          const int rho = g * BC + s;
          return rho < S ? rho : -1;
        }
        const int q = w * BC + s;
        return q < p.n_seq ? q : -1;
      };
      auto peak = [&](int code, float pw) {
        if (pw == pmax) {
          // exact tie: the reference keeps the later lag (Iterator::max_by)
          if (lag_of(code) > lag_of(cmax)) cmax = code;
        }
        cmax = pw > pmax ? code : cmax;
        pmax = fmaxf(pw, pmax);
      };
      // epilogue for output (s, a, b, c)
      auto epilogue = [&](int s, int a, int b, int c, float2 v) {
        if (!INV) {
          // the last stage reads and writes the same positions of its thread
          buf[s * LC + G::offset(a, b, c)] = MODE == FWD_Z ? v : make_float2(v.x, -v.y);
        } else {
          const float pw = fmaf(v.x, v.x, v.y * v.y);
          if (ARGMAX) {
            const int code = ((seq_of(s) * 31 + a) * 33 + b) * 16 + c;
            if (NC == 1)
              peak(code, pw);
            else
              pws[c] = pw;
            // kept in place for the second peak: the stage read its inputs
            // from these positions into registers before any output
            if (keep_top) reinterpret_cast<float*>(buf)[2 * (s * LC + G::offset(a, b, c))] = pw;
          } else {
            const int tau = seq_of(s) + S * G::natural(a, b, c);
            int d = tau - tau_star;
            d = d < 0 ? -d : d;
            const int dist = min(d, p.P - d);
            if (dist > p.chip_width) pbest = fmaxf(pbest, pw);
          }
        }
      };

      // CORR / CAND: the outputs of one DFT-M.  Only a value at or above the
      // largest of the CTA's earlier groups can be the row's, so one comparison
      // of their maximum does for nearly all of them (compares and selects per
      // output took a tenth of the instructions: Lc = 10230 and 4092 take 4 %
      // less time so; the 33 outputs of Lc = 1023 would cost registers, 8 % more)
      auto peaks = [&](int s, int a, int b) {
        float m = pws[0];
#pragma unroll
        for (int c = 1; c < NC; ++c) m = fmaxf(m, pws[c]);
        if (m < floor_pw) return;
#pragma unroll
        for (int c = 0; c < NC; ++c) peak(((seq_of(s) * 31 + a) * 33 + b) * 16 + c, pws[c]);
        floor_pw = fmaxf(floor_pw, pmax);
      };

      // ---- FWD_Z: the unit's sequences into buf as they are, 16 bytes at a
      // time (a unit starts on 16 bytes: BC or LC is even), and back in order at
      // the end.  Columns gathered from global memory and rows stored 8 bytes
      // apart kept the load / store queue full: 6.57 ms for 771840 sequences of
      // 1023 with their FP16 units, 4.41 so; 1.72 and 1.52 for 31488 of 10230.
      if (MODE == FWD_Z) {
        static_assert(BC * LC % 2 == 0, "units of whole 16-byte pieces");
        const int n = min(BC, p.n_seq - w * BC) * LC;
        const float2* src = p.z + (size_t)w * BC * LC;
        for (int i = 2 * tid; i < n; i += 2 * NT) {
          const unsigned dst = (unsigned)__cvta_generic_to_shared(buf + i);
          if (i + 1 < n)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src + i) : "memory");
          else
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src + i) : "memory");
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
      }
      // ---- FWD_D: chips, element n at its digits; the twist of hypothesis 1
      // in double (31 sincospi per column spilled: 23 against 13 us for one PRN
      // of 1023 chips, 59 against 38 for 126 of 10230) ----
      if (MODE == FWD_D) {
        for (int i = tid; i < BC * LC; i += NT) {
          const int s = BC == 1 ? 0 : i / LC, n = i - s * LC;
          const int q = seq_of(s);
          if (q < 0) continue;
          const float v = (float)__ldg(p.chips + (size_t)(q >> 1) * LC + n);
          double sn = 0.0, cs = 1.0;
          if (q & 1) sincospi((double)n / (double)LC, &sn, &cs);
          buf[s * LC + G::offset(n % 31, n % 33, NC == 1 ? 0 : n % NC)] = make_float2(v * (float)cs, v * (float)sn);
        }
        __syncthreads();
      }

      // ---- stage 1: DFT-31 over digit a; INV: input straight from global ----
      static_assert(BC * COLS <= NT, "one column per thread");
      if constexpr (MODE == FWD_Z) {
        // columns are read across the whole sequence: all of them before any
        // is written (threads without a column read the first).  Thread t has
        // the column through element 31 t: an odd stride, no bank conflicts
        // (in the order of b, 31 EB is a multiple of 16 elements for Lc = 4092)
        const bool on = tid < BC * COLS && seq_of(tid / COLS) >= 0;
        const int u = on ? tid : 0, s = u / COLS, t = u - s * COLS;
        float2 x[31];
#pragma unroll
        for (int a = 0; a < 31; ++a) x[a] = buf[s * LC + (31 * t + a * G::EA) % LC];
        __syncthreads();
        float2* dst = buf + s * LC + (31 * t) % NC * 33 + (31 * t) % 33;
        if (on) dft_odd<31, INV>(x, [&](int ta, float2 v) { dst[ta * COLS] = v; });
      } else if (tid < BC * COLS && seq_of(tid / COLS) >= 0) {
        const int s = tid / COLS, col = tid - s * COLS;
        const int q = seq_of(s);
        float2 x[31];
        if (INV) {
          const float2* zs = p.z + ((size_t)ab_h * S + q) * LC + col;
          const float2* ds = p.D + ((size_t)prn * 2 + hyp) * LC + col;
#pragma unroll
          // Z is read once per (row, rho): keep it out of L1 so the code
          // spectrum D, reused by every rho of the row, stays there.
          for (int a = 0; a < 31; ++a) x[a] = cmul(__ldcg(zs + a * COLS), __ldg(ds + a * COLS));
        } else {
#pragma unroll
          for (int a = 0; a < 31; ++a) x[a] = buf[s * LC + a * COLS + col];
        }
        float2* dst = buf + s * LC + col;
        dft_odd<31, INV>(x, [&](int ta, float2 v) { dst[ta * COLS] = v; });
      }
      __syncthreads();

      // ---- stage 2: DFT-33 over digit b ----
      for (int u = tid; u < BC * 31 * NC; u += NT) {
        const int s = u / (31 * NC), r = u - s * 31 * NC;
        const int a = r / NC, c = r - a * NC;
        if (seq_of(s) < 0) continue;
        float2* base = buf + s * LC + a * COLS + c * 33;
        float2 x[33];
#pragma unroll
        for (int b = 0; b < 33; ++b) x[b] = base[b];
        if constexpr (NC == 1) {
          dft33<INV>(x, [&](int tb, float2 v) { epilogue(s, a, tb, 0, v); });
        } else {
          dft33<INV>(x, [&](int tb, float2 v) { base[tb] = v; });
        }
      }

      // ---- stage 3: DFT-M over digit c ----
      if constexpr (NC > 1) {
        __syncthreads();
        for (int u = tid; u < BC * 1023; u += NT) {
          const int s = u / 1023, gi = u - s * 1023;
          const int a = gi / 33, b = gi - a * 33;
          if (seq_of(s) < 0) continue;
          const float2* base = buf + s * LC + a * COLS + b;
          float2 x[NC];
#pragma unroll
          for (int c = 0; c < NC; ++c) x[c] = base[c * 33];
          dft_small<NC, INV>(x, [&](int tc, float2 v) { epilogue(s, a, b, tc, v); });
          if (ARGMAX) peaks(s, a, b);
        }
      }
      if (ARGMAX && NC > 1 && g + 1 < g1) {
        const unsigned mine = __reduce_max_sync(0xffffffffu, pmax > 0.f ? __float_as_uint(pmax) : 0u);
        if ((tid & 31) == 0 && mine > s_floor) atomicMax(&s_floor, mine);
      }
      __syncthreads();
      // CAND with p2rows: the four largest |y|^2 of every residue of the
      // group (kept in place in buf) with their lags.  TOP_WPS warps scan a
      // residue; each takes the fourth largest of its lanes' maxima as a
      // lower bound on its four largest values, keeps per lane the four
      // largest values at or above it, and stores the warp's four largest.
      if (TOP && keep_top) {
        const int warp = tid >> 5, lane = tid & 31;
        const int sl = warp / TOP_WPS, sub = warp - sl * TOP_WPS;
        if (sl < BC && seq_of(sl) >= 0) {  // uniform over the warp
          const float* pws = reinterpret_cast<const float*>(buf + sl * LC);
          unsigned mb = 0u;
          for (int i = sub * 32 + lane; i < LC; i += TOP_WPS * 32) mb = max(mb, __float_as_uint(pws[2 * i]));
          unsigned thr = 0u;
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            thr = __reduce_max_sync(0xffffffffu, mb);
            const unsigned h = __ballot_sync(0xffffffffu, mb == thr);
            if (lane == __ffs(h) - 1) mb = 0u;
          }
          Top4 t;
          for (int i = sub * 32 + lane; i < LC; i += TOP_WPS * 32) {
            const float x = pws[2 * i];
            if (__float_as_uint(x) >= thr) t.add(x, i);
          }
          const int rho = seq_of(sl);
          unsigned long long* dst = s_res + ((size_t)rho * TOP_WPS + sub) * 4;
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            const unsigned vb = __float_as_uint(t.v[0]);
            const unsigned x = __reduce_max_sync(0xffffffffu, vb);
            const unsigned h = __ballot_sync(0xffffffffu, vb == x);
            const int src = __ffs(h) - 1;
            const int i = __shfl_sync(0xffffffffu, t.i[0], src);
            if (lane == src) t.pop();
            if (lane == r) {
              unsigned long long k = 0ull;
              if (x != 0u) {
                const int a = i / COLS, rem = i - a * COLS, c = rem / 33, b = rem - c * 33;
                k = ((unsigned long long)x << 32) | (unsigned)(rho + S * G::natural(a, b, c));
              }
              dst[r] = k;
            }
          }
        }
        // the next group's stage 1 overwrites the values scanned here
        __syncthreads();
      }
      // spectra to global memory in order
      if (!INV) {
        const int n = min(BC, p.n_seq - w * BC) * LC;
        float2* dst = (MODE == FWD_Z ? p.z : p.Dout) + (size_t)w * BC * LC;
        for (int i = 2 * tid; i < n; i += 2 * NT) {
          if (i + 1 < n)
            *reinterpret_cast<float4*>(dst + i) = *reinterpret_cast<const float4*>(buf + i);
          else
            dst[i] = buf[i];
        }
      }
      // tensor-core operands: FP16 units straight from the transformed
      // sequences in shared memory (the work of tc_pack_kernel, without
      // reading the FP32 spectra back from memory)
      if (MODE == FWD_Z && p.z16) {
        using U = TcUnits<M>;
        for (int e = tid; e < BC * U::UNITS; e += NT) {
          const int s = e / U::UNITS, r = e - s * U::UNITS;
          const int q = seq_of(s);
          if (q < 0) continue;
          const uint4 m = __ldg(p.z16_map + r);
          const unsigned off[8] = {m.x & 0xffffu, m.x >> 16, m.y & 0xffffu, m.y >> 16,
                                   m.z & 0xffffu, m.z >> 16, m.w & 0xffffu, m.w >> 16};
          float2 v[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            v[i] = make_float2(0.f, 0.f);
            if (off[i] != 0xffffu) {
              v[i] = buf[s * LC + (int)off[i]];
              v[i].x *= p.z16_scale;
              v[i].y *= p.z16_scale;
            }
          }
          uint4* dst = p.z16 + (size_t)q * U::PER_SEQ + r;
          pack_unit(v, dst[0], dst[U::UNITS]);
        }
        __syncthreads();
      }
    }

    if (ARGMAX) {
      unsigned long long kbest =
          pmax < 0.f ? 0ull : (((unsigned long long)__float_as_uint(pmax) << 32) | (unsigned)lag_of(cmax));
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long other = __shfl_xor_sync(0xffffffffu, kbest, o);
        kbest = other > kbest ? other : kbest;
      }
      if ((tid & 31) == 0) atomicMax(&s_key, kbest);
      __syncthreads();
      if (tid == 0) {
        if (split > 1)
          atomicMax(p.keys + key_at, s_key);
        else
          p.keys[key_at] = s_key;
      }
      // CAND with p2rows: the row's second peak against its own maximum, the
      // largest |y|^2 more than chip_width lags (circularly) from it.  At most
      // ceil((2 chip_width + 1) / S) <= 3 lags of a residue lie that close, so
      // the four largest of each residue (among the lists of the warps that
      // scanned it) hold it.  A split row's lists go through global memory, and
      // the part that finishes last looks at all of them.
      if (TOP && keep_top) {
        const int n_top = S * TOP_WPS * 4;
        unsigned long long* lists = p.top_lists + (size_t)w * n_top;
        bool mine = true;
        if (split > 1) {
          const int e0 = min(g0 * BC, S) * TOP_WPS * 4, e1 = min(g1 * BC, S) * TOP_WPS * 4;
          for (int e = e0 + tid; e < e1; e += NT) lists[e] = s_res[e];
          __threadfence();
          __syncthreads();
          if (tid == 0) {
            s_last = atomicAdd(p.top_done + w, 1) == split - 1;
            __threadfence();
          }
          __syncthreads();
          mine = s_last;
        }
        if (mine && tid < 32) {
          const unsigned long long kb = split > 1 ? __ldcg(p.keys + key_at) : s_key;
          const int tau_star = (int)(unsigned)kb;
          float p2 = 0.f;
          if (kb != 0ull)
            for (int e = tid; e < n_top; e += 32) {
              const unsigned long long k = split > 1 ? __ldcg(lists + e) : s_res[e];
              int d = (int)(unsigned)k - tau_star;
              d = d < 0 ? -d : d;
              if (k != 0ull && min(d, p.P - d) > p.chip_width) p2 = fmaxf(p2, __uint_as_float((unsigned)(k >> 32)));
            }
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) p2 = fmaxf(p2, __shfl_xor_sync(0xffffffffu, p2, o));
          if (tid == 0) p.p2rows[key_at] = p2;
        }
      }
    } else if (MODE == SECOND) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) pbest = fmaxf(pbest, __shfl_xor_sync(0xffffffffu, pbest, o));
      if ((tid & 31) == 0) atomicMax(&s_p2, __float_as_uint(pbest));
      __syncthreads();
      // (the bin reduction left 0 there)
      if (tid == 0) atomicMax(reinterpret_cast<int*>(&p.best[w].p2), (int)s_p2);
    }
    __syncthreads();
  }
}

// Launch configurations: (third digit M, slots per CTA, threads, min CTAs/SM).
// Variant 0 is the default; variant 1 doubles the polyphase branches (slots)
// and threads of a CTA at one CTA per SM, so more branches of one (row, PRN)
// item share the code spectrum in L1.  The correlation modes take the
// variant of the class (PolyClass::variant, set by tga_set_variant or
// tga_autotune); the forward transforms always run variant 0.
template <int M, int V>
struct PfaCfg;
template <>
struct PfaCfg<1, 0> {
  static constexpr int BC = 8, NT = 288, MINB = 2;  // 8 x 33 DFT-31 columns
};
template <>
struct PfaCfg<1, 1> {
  static constexpr int BC = 16, NT = 576, MINB = 1;
};
template <>
struct PfaCfg<4, 0> {
  static constexpr int BC = 2, NT = 288, MINB = 2;  // 2 x 132 columns
};
template <>
struct PfaCfg<4, 1> {
  static constexpr int BC = 4, NT = 576, MINB = 1;
};
template <>
struct PfaCfg<10, 0> {
  static constexpr int BC = 1, NT = 352, MINB = 2;  // 330 columns
};
template <>
struct PfaCfg<10, 1> {
  static constexpr int BC = 2, NT = 704, MINB = 1;  // two rho slots share D in L1
};

template <int M, int V, int MODE>
static cudaError_t run_pfa(const PfaParams& p, int n_work_slots, int num_sms, cudaStream_t st) {
  using C = PfaCfg<M, V>;
  constexpr int LC = Geo<M>::LC;
  size_t smem = (size_t)C::BC * LC * sizeof(float2);
  // CAND with p2rows: the four largest |y|^2 per residue and scanning warp
  if (MODE == CAND && p.p2rows) {
    constexpr int WPS = C::NT / 32 / C::BC >= 1 ? C::NT / 32 / C::BC : 1;
    smem += (size_t)p.S * WPS * 4 * sizeof(unsigned long long);
  }
  auto kern = pfa_kernel<M, C::BC, C::NT, C::MINB, MODE>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  int per_sm = 1;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, C::NT, smem);
  if (per_sm < 1) per_sm = 1;
  // FWD modes: n_work_slots counts sequences, grouped BC per work unit
  const int n_work = (MODE == FWD_Z || MODE == FWD_D) ? (n_work_slots + C::BC - 1) / C::BC : n_work_slots;
  int grid = num_sms * per_sm;
  PfaParams q = p;
  if (MODE == CORR || MODE == SECOND) {
    const int groups = (p.S + C::BC - 1) / C::BC;
    q.split = n_work > 0 ? std::max(1, std::min(groups, grid / n_work)) : 1;
    if (MODE == CORR && q.split > 1) {
      e = cudaMemsetAsync(p.keys, 0, (size_t)n_work * sizeof(unsigned long long), st);
      if (e != cudaSuccess) return e;
    }
    if (grid > n_work * q.split) grid = n_work * q.split;
  } else if (MODE == CAND) {
    if (grid > kMaxSplitRows) grid = kMaxSplitRows;
  } else if (grid > n_work) {
    grid = n_work;
  }
  if (grid < 1) return cudaSuccess;
  kern<<<grid, C::NT, smem, st>>>(q);
  return TGA_LAUNCHED();
}

template <int MODE>
static cudaError_t dispatch_pfa(const PolyClass& pc, const PfaParams& p, int n_work_slots, int num_sms,
                                cudaStream_t st) {
  if constexpr (MODE == CORR || MODE == SECOND || MODE == CAND) {
    if (pc.variant == 1) {
      switch (pc.M) {
        case 1: return run_pfa<1, 1, MODE>(p, n_work_slots, num_sms, st);
        case 4: return run_pfa<4, 1, MODE>(p, n_work_slots, num_sms, st);
        case 10: return run_pfa<10, 1, MODE>(p, n_work_slots, num_sms, st);
      }
      return cudaErrorInvalidValue;
    }
  }
  switch (pc.M) {
    case 1: return run_pfa<1, 0, MODE>(p, n_work_slots, num_sms, st);
    case 4: return run_pfa<4, 0, MODE>(p, n_work_slots, num_sms, st);
    case 10: return run_pfa<10, 0, MODE>(p, n_work_slots, num_sms, st);
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_forward_z(const PolyClass& pc, int n_ab, float2* d_z, int num_sms, cudaStream_t st) {
  PfaParams p = {};
  p.z = d_z;
  p.n_seq = n_ab * 2 * pc.S;
  p.S = pc.S;
  p.P = pc.P;
  return dispatch_pfa<FWD_Z>(pc, p, p.n_seq, num_sms, st);
}

std::vector<uint16_t> tc_unit_map(int M) {
  auto build = [](auto u) {
    using U = decltype(u);
    std::vector<uint16_t> t((size_t)U::UNITS * 8);
    for (int r = 0; r < U::UNITS; ++r) {
      for (int i = 0; i < 8; ++i)
        t[(size_t)r * 8 + i] = U::filled(r, i) ? (uint16_t)U::src_offset(r, i) : (uint16_t)0xffffu;
    }
    return t;
  };
  switch (M) {
    case 1: return build(TcUnits<1>());
    case 4: return build(TcUnits<4>());
    case 10: return build(TcUnits<10>());
  }
  return {};
}

cudaError_t launch_forward_z_tc(const PolyClass& pc, int n_ab, float2* d_z, void* d_z16, const void* d_map,
                                float z16_scale, int num_sms, cudaStream_t st) {
  PfaParams p = {};
  p.z = d_z;
  p.z16 = static_cast<uint4*>(d_z16);
  p.z16_map = static_cast<const uint4*>(d_map);
  p.z16_scale = z16_scale;
  p.n_seq = n_ab * 2 * pc.S;
  p.S = pc.S;
  p.P = pc.P;
  return dispatch_pfa<FWD_Z>(pc, p, p.n_seq, num_sms, st);
}

cudaError_t launch_forward_seqs_tc(const PolyClass& pc, long long n_seq, float2* d_z, void* d_z16, const void* d_map,
                                   float z16_scale, int num_sms, cudaStream_t st) {
  if (n_seq > 0x7fffffffLL) return cudaErrorInvalidValue;
  PfaParams p = {};
  p.z = d_z;
  p.z16 = static_cast<uint4*>(d_z16);
  p.z16_map = static_cast<const uint4*>(d_map);
  p.z16_scale = z16_scale;
  p.n_seq = (int)n_seq;
  p.S = pc.S;
  p.P = pc.P;
  return dispatch_pfa<FWD_Z>(pc, p, p.n_seq, num_sms, st);
}

cudaError_t launch_forward_seqs(const PolyClass& pc, long long n_seq, float2* d_z, int num_sms, cudaStream_t st) {
  if (n_seq > 0x7fffffffLL) return cudaErrorInvalidValue;
  PfaParams p = {};
  p.z = d_z;
  p.n_seq = (int)n_seq;
  p.S = pc.S;
  p.P = pc.P;
  return dispatch_pfa<FWD_Z>(pc, p, p.n_seq, num_sms, st);
}

cudaError_t launch_code_spectra(const PolyClass& pc, const int8_t* d_chips, int n_prn, float2* d_D,
                                int num_sms, cudaStream_t st) {
  PfaParams p = {};
  p.chips = d_chips;
  p.Dout = d_D;
  p.n_seq = n_prn * 2;
  p.S = pc.S;
  p.P = pc.P;
  return dispatch_pfa<FWD_D>(pc, p, p.n_seq, num_sms, st);
}

cudaError_t launch_correlate(const PolyClass& pc, const SearchDims& dims, const float2* d_Z,
                             const float2* d_D, unsigned long long* d_keys, int num_sms,
                             cudaStream_t st) {
  PfaParams p = {};
  p.z = const_cast<float2*>(d_Z);
  p.D = d_D;
  p.keys = d_keys;
  p.n_prn = dims.n_prn;
  p.S = pc.S;
  p.P = pc.P;
  p.n_items = dims.n_ant * dims.nb * 2 * dims.n_prn;
  return dispatch_pfa<CORR>(pc, p, p.n_items, num_sms, st);
}

cudaError_t launch_second_peak(const PolyClass& pc, const SearchDims& dims, const float2* d_Z,
                               const float2* d_D, BestRow* d_best, int chip_width, int num_sms,
                               cudaStream_t st) {
  PfaParams p = {};
  p.z = const_cast<float2*>(d_Z);
  p.D = d_D;
  p.best = d_best;
  p.n_prn = dims.n_prn;
  p.S = pc.S;
  p.P = pc.P;
  p.chip_width = chip_width;
  p.n_items = dims.n_ant * dims.n_prn;
  return dispatch_pfa<SECOND>(pc, p, p.n_items, num_sms, st);
}

size_t split_scratch_bytes(const PolyClass& pc) {
  // per row a counter and S x kTopWarps x 4 list entries
  return (size_t)kMaxSplitRows * (sizeof(int) + (size_t)pc.S * kTopWarps * 4 * sizeof(unsigned long long));
}

cudaError_t launch_correlate_listed(const PolyClass& pc, const SearchDims& dims, const float2* d_Z,
                                    const float2* d_D, const int2* d_cand, const int* d_count, int capacity,
                                    unsigned long long* d_keys, int num_sms, cudaStream_t st, void* d_scratch,
                                    float* d_p2rows, int chip_width) {
  PfaParams p = {};
  if (d_p2rows) {
    p.top_lists = static_cast<unsigned long long*>(d_scratch);
    p.top_done = reinterpret_cast<int*>(p.top_lists + (size_t)kMaxSplitRows * pc.S * kTopWarps * 4);
    const cudaError_t e = cudaMemsetAsync(p.top_done, 0, kMaxSplitRows * sizeof(int), st);
    if (e != cudaSuccess) return e;
  }
  p.p2rows = d_p2rows;
  p.chip_width = chip_width;
  p.z = const_cast<float2*>(d_Z);
  p.D = d_D;
  p.keys = d_keys;
  p.cand = d_cand;
  p.cand_count = d_count;
  p.n_prn = dims.n_prn;
  p.S = pc.S;
  p.P = pc.P;
  p.n_items = capacity;
  return dispatch_pfa<CAND>(pc, p, p.n_items, num_sms, st);
}

// The second peak of each cell from the re-evaluated rows: the cell's
// chosen row is always one of them (its FP32 key is the cell's maximum; when
// every key is 0, every row was listed).
__global__ void second_from_rows_kernel(int n_cells, int n_hyp, int n_prn, const float* __restrict__ p2rows,
                                        BestRow* __restrict__ best) {
  const int w = blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= n_cells) return;
  const BestRow b = best[w];
  best[w].p2 = p2rows[(size_t)(b.ab * n_hyp + b.hyp) * n_prn + (w % n_prn)];
}

cudaError_t launch_second_from_rows(const SearchDims& dims, int n_hyp, const float* d_p2rows, BestRow* d_best,
                                    cudaStream_t st) {
  const int n = dims.n_ant * dims.n_prn;
  if (n <= 0) return cudaSuccess;
  second_from_rows_kernel<<<(n + 255) / 256, 256, 0, st>>>(n, n_hyp, dims.n_prn, d_p2rows, d_best);
  return TGA_LAUNCHED();
}

// Rows of a reduced-precision search to re-evaluate in FP32.  Per (antenna,
// PRN), with K the largest reduced-precision key of its 2 nb rows, every row
// whose key is at least keep * K is listed (keep * K = 0 lists all rows).
// If every row's amplitude error is at most e and keep = (1 - 2 e / sqrt(K))^2
// or less, the row holding the FP32 maximum is always listed: its key is at
// least (sqrt(V) - e)^2 with V the FP32 maximum, and sqrt(K) <= sqrt(V) + e.
// Rows not listed hold FP32 values below V, so the FP32 keys of the listed
// rows alone give the FP32 search's choice under the same tie rules.
// Rows are [ant][bin][hyp] with n_hyp hypotheses (2 in the drop-in search,
// 1 in the non-coherent one); a listed row is (its row index, prn).
//
// Both kernels below read one 8-byte key per row and cell, a chain of nb
// loads in a chain when one thread walks a cell's rows (10 to 30 us; 7 to 10
// so).  A CTA takes 32 cells, whose keys are neighbours, and kRowLanes warps
// share their rows.
constexpr int kRowLanes = 16;

__global__ void __launch_bounds__(32 * kRowLanes)
    tc_candidates_kernel(int n_ant, int n_rows, int n_prn, const unsigned long long* __restrict__ keys, float keep,
                         int2* __restrict__ cand, int* __restrict__ count) {
  __shared__ float s_max[kRowLanes][32];
  const int i = blockIdx.x * 32 + threadIdx.x;
  const bool on = i < n_ant * n_prn;
  const int ant = on ? i / n_prn : 0, prn = on ? i - ant * n_prn : 0;
  const size_t row0 = (size_t)ant * n_rows;
  auto key = [&](int r) { return __uint_as_float((unsigned)(__ldg(keys + (row0 + r) * n_prn + prn) >> 32)); };
  float kmax = 0.f;
  if (on) {
#pragma unroll 4
    for (int r = threadIdx.y; r < n_rows; r += kRowLanes) kmax = fmaxf(kmax, key(r));
  }
  s_max[threadIdx.y][threadIdx.x] = kmax;
  __syncthreads();
#pragma unroll
  for (int y = 0; y < kRowLanes; ++y) kmax = fmaxf(kmax, s_max[y][threadIdx.x]);
  const float t = kmax * keep;
  if (on) {
#pragma unroll 4
    for (int r = threadIdx.y; r < n_rows; r += kRowLanes)
      if (key(r) >= t) cand[atomicAdd(count, 1)] = make_int2((int)(row0 + r), prn);
  }
}

cudaError_t launch_tc_candidates(const SearchDims& dims, int n_hyp, const unsigned long long* d_keys, float keep,
                                 int2* d_cand, int* d_count, cudaStream_t st) {
  const int n = dims.n_ant * dims.n_prn;
  if (n <= 0) return cudaSuccess;
  tc_candidates_kernel<<<(n + 31) / 32, dim3(32, kRowLanes), 0, st>>>(dims.n_ant, dims.nb * n_hyp, dims.n_prn,
                                                                      d_keys, keep, d_cand, d_count);
  return TGA_LAUNCHED();
}

// ---------------------------------------------------------------------------
// reduction over hypotheses and Doppler bins (correlate.rs:125-154)
// ---------------------------------------------------------------------------
template <int HYP>
__global__ void __launch_bounds__(32 * kRowLanes)
    reduce_bins_kernel(int n_ant, int nb, int n_prn, const unsigned long long* __restrict__ keys,
                       BestRow* __restrict__ best) {
  __shared__ unsigned long long s_best[kRowLanes][32];
  const int i = blockIdx.x * 32 + threadIdx.x;
  const bool on = i < n_ant * n_prn;
  const int ant = on ? i / n_prn : 0, prn = on ? i - ant * n_prn : 0;
  auto key = [&](int bin, int h) { return __ldg(keys + (((size_t)ant * nb + bin) * HYP + h) * n_prn + prn); };
  // (value, bin, hypothesis): the largest is the last bin of the largest
  // value (Iterator::max_by keeps the last maximum).  A NaN is never above
  // another value, and nothing is above a NaN in bin 0.
  unsigned long long top = 0ull;
  if (on) {
#pragma unroll 4
    for (int bin = threadIdx.y; bin < nb; bin += kRowLanes) {
      float pr = __uint_as_float((unsigned)(key(bin, 0) >> 32));
      int h = 0;
      if (HYP == 2) {
        const float pB = __uint_as_float((unsigned)(key(bin, HYP - 1) >> 32));
        // hypotheses: [c,-c] replaces [c,c] only when strictly stronger
        if (pB > pr) pr = pB, h = 1;
      }
      const unsigned v = pr >= 0.f ? __float_as_uint(pr) : bin == 0 ? 0xffffffffu : 0u;
      const unsigned long long k = ((unsigned long long)v << 32) | (unsigned)(bin * 2 + h);
      if (v != 0u || pr >= 0.f) top = k > top ? k : top;
    }
  }
  s_best[threadIdx.y][threadIdx.x] = top;
  __syncthreads();
  if (threadIdx.y != 0 || !on) return;
#pragma unroll
  for (int y = 0; y < kRowLanes; ++y) top = s_best[y][threadIdx.x] > top ? s_best[y][threadIdx.x] : top;
  const int bin = (int)(unsigned)top >> 1, h = (int)top & 1;
  const unsigned long long k = key(bin, h);
  BestRow r;
  r.ab = ant * nb + bin;
  r.hyp = h;
  r.tau = (int)(unsigned)(k & 0xffffffffull);
  r.p = __uint_as_float((unsigned)(k >> 32));
  r.p2 = 0.f;
  best[i] = r;
}

cudaError_t launch_reduce_bins(const SearchDims& dims, int n_hyp, const unsigned long long* d_keys, BestRow* d_best,
                               cudaStream_t st) {
  const int n = dims.n_ant * dims.n_prn;
  if (n <= 0) return cudaSuccess;
  const int grid = (n + 31) / 32;
  const dim3 block(32, kRowLanes);
  if (n_hyp == 2)
    reduce_bins_kernel<2><<<grid, block, 0, st>>>(dims.n_ant, dims.nb, dims.n_prn, d_keys, d_best);
  else
    reduce_bins_kernel<1><<<grid, block, 0, st>>>(dims.n_ant, dims.nb, dims.n_prn, d_keys, d_best);
  return TGA_LAUNCHED();
}

// ---------------------------------------------------------------------------
// ACR C/N0 (acr.rs:49-84) and result finalisation (acquisition.rs:237-247)
// ---------------------------------------------------------------------------
__constant__ double kAcrGps[59][2];
__constant__ double kAcrGal[71][2];
__constant__ double kAcrBds[79][2];
__constant__ double kAcrL1c[79][2];
// The tables are uploaded once per device, on the first call that needs them
// (with that device current).  Host threads making their first calls at
// once are serialised by the mutex; later calls only read the flag.
constexpr int kAcrMaxDevices = 64;
static std::atomic<bool> g_acr_uploaded[kAcrMaxDevices];
static std::mutex g_acr_mutex;

static cudaError_t upload_acr_tables() {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const bool cached = dev >= 0 && dev < kAcrMaxDevices;
  if (cached && g_acr_uploaded[dev].load(std::memory_order_acquire)) return cudaSuccess;
  std::lock_guard<std::mutex> lock(g_acr_mutex);
  if (cached && g_acr_uploaded[dev].load(std::memory_order_relaxed)) return cudaSuccess;
  e = cudaMemcpyToSymbol(kAcrGps, TGA_GPS_L1_CA_ACR_TABLE, sizeof(kAcrGps));
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(kAcrGal, TGA_GALILEO_E1C_ACR_TABLE, sizeof(kAcrGal));
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(kAcrBds, TGA_BEIDOU_B1C_ACR_TABLE, sizeof(kAcrBds));
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(kAcrL1c, TGA_GPS_L1C_ACR_TABLE, sizeof(kAcrL1c));
  if (e == cudaSuccess && cached) g_acr_uploaded[dev].store(true, std::memory_order_release);
  return e;
}

__device__ bool estimate_cn0_dev(double r_a, int table, double* out) {
  const double(*t)[2];
  int n;
  switch (table) {
    case 0: t = kAcrGps; n = 59; break;
    case 1: t = kAcrGal; n = 71; break;
    case 2: t = kAcrBds; n = 79; break;
    default: t = kAcrL1c; n = 79; break;
  }
  if (!(r_a > 1.0) || !isfinite(r_a)) return false;
  if (r_a <= t[0][0]) { *out = t[0][1]; return true; }
  if (r_a >= t[n - 1][0]) { *out = t[n - 1][1]; return true; }
  int lo = 0, hi = n;  // first index with r >= r_a
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (t[mid][0] < r_a) lo = mid + 1; else hi = mid;
  }
  if (lo == 0) { *out = t[0][1]; return true; }
  if (lo >= n) { *out = t[n - 1][1]; return true; }
  const double la = log(t[lo - 1][0]), lb = log(t[lo][0]);
  const double tt = (log(r_a) - la) / (lb - la);
  double v = t[lo - 1][1] + tt * (t[lo][1] - t[lo - 1][1]);
  v = v < 20.0 ? 20.0 : (v > 70.0 ? 70.0 : v);
  *out = v;
  return true;
}

__global__ void finalize_kernel(int n_cells, int nb, int n_prn, int P, int Lc, const double* __restrict__ fc,
                                double center, const BestRow* __restrict__ best, const int8_t* __restrict__ tables,
                                int want_cn0, CellOut* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_cells) return;
  const BestRow b = best[i];
  const double scale = sqrt(2.0 * (double)P) / (double)Lc;
  const float vm = (float)(sqrt((double)b.p) * scale);
  float vs = (float)(sqrt((double)fmaxf(b.p2, 0.f)) * scale);
  if (vs <= 0.f) vs = 1e-6f;  // correlate.rs:173-175
  const int bin = b.ab % nb;
  CellOut o;
  o.strength = (double)vm;
  o.second = (double)vs;
  o.codephase_frac = (double)b.tau / (double)P;
  o.frequency = fc[bin] - center;
  o.bin = bin;
  o.tau = b.tau;
  o.hyp = b.hyp;
  o.cn0 = 0.0;
  o.cn0_valid = 0;
  if (want_cn0) {
    const double m = o.strength, s = o.second;
    if (s > 0.0 && m > s) {
      const double q = m / s;
      double c;
      if (estimate_cn0_dev(q * q, tables[i % n_prn], &c)) {
        o.cn0 = c;
        o.cn0_valid = 1;
      }
    }
  }
  out[i] = o;
}

cudaError_t launch_finalize(const PolyClass& pc, const SearchDims& dims, const BestRow* d_best,
                            double center_freq, const int8_t* d_tables, int want_cn0, CellOut* d_out,
                            cudaStream_t st) {
  cudaError_t e = upload_acr_tables();
  if (e != cudaSuccess) return e;
  const int n = dims.n_ant * dims.n_prn;
  if (n <= 0) return cudaSuccess;
  finalize_kernel<<<(n + 127) / 128, 128, 0, st>>>(n, dims.nb, dims.n_prn, pc.P, pc.Lc, dims.fc,
                                                   center_freq, d_best, d_tables, want_cn0, d_out);
  return TGA_LAUNCHED();
}

__global__ void acr_batch_kernel(const double* __restrict__ ra, int n, int table, double* __restrict__ cn0,
                                 uint8_t* __restrict__ valid) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double c = 0.0;
  const bool ok = estimate_cn0_dev(ra[i], table, &c);
  cn0[i] = ok ? c : 0.0;
  valid[i] = ok ? 1 : 0;
}

cudaError_t launch_acr_batch(const double* d_ra, int n, int table, double* d_cn0, uint8_t* d_valid,
                             cudaStream_t st) {
  cudaError_t e = upload_acr_tables();
  if (e != cudaSuccess) return e;
  if (n <= 0) return cudaSuccess;
  acr_batch_kernel<<<(n + 255) / 256, 256, 0, st>>>(d_ra, n, table, d_cn0, d_valid);
  return TGA_LAUNCHED();
}

// ---------------------------------------------------------------------------
// antenna cross-correlation counts (observation.rs:175-195):
// counts[i*n+j] = number of samples where antennas i and j agree
// ---------------------------------------------------------------------------
__global__ void xcorr_kernel(const uint8_t* __restrict__ bits, int n_ant, size_t row_bytes,
                             unsigned long long* __restrict__ counts) {
  const int i = blockIdx.y, j = blockIdx.x;
  if (j < i) return;
  const uint8_t* a = bits + (size_t)i * row_bytes;
  const uint8_t* b = bits + (size_t)j * row_bytes;
  unsigned long long diff = 0;
  const bool aligned = ((((uintptr_t)a) | ((uintptr_t)b)) & 15) == 0;
  size_t done = 0;
  if (aligned) {
    const size_t nv = row_bytes / 16;
    const uint4* av = reinterpret_cast<const uint4*>(a);
    const uint4* bv = reinterpret_cast<const uint4*>(b);
    for (size_t k = threadIdx.x; k < nv; k += blockDim.x) {
      const uint4 x = __ldg(av + k), y = __ldg(bv + k);
      diff += __popc(x.x ^ y.x) + __popc(x.y ^ y.y) + __popc(x.z ^ y.z) + __popc(x.w ^ y.w);
    }
    done = nv * 16;
  }
  for (size_t k = done + threadIdx.x; k < row_bytes; k += blockDim.x) diff += __popc((unsigned)(a[k] ^ b[k]));
  for (int o = 16; o > 0; o >>= 1) diff += __shfl_xor_sync(0xffffffffu, diff, o);
  __shared__ unsigned long long part[32];
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = diff;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long t = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += part[w];
    const unsigned long long agree = (unsigned long long)row_bytes * 8ull - t;
    counts[(size_t)i * n_ant + j] = agree;
    counts[(size_t)j * n_ant + i] = agree;
  }
}

cudaError_t launch_xcorr_matrix(const uint8_t* d_bits, int n_ant, size_t row_bytes, unsigned long long* d_counts,
                                cudaStream_t st) {
  if (n_ant <= 0) return cudaSuccess;
  xcorr_kernel<<<dim3(n_ant, n_ant), 256, 0, st>>>(d_bits, n_ant, row_bytes, d_counts);
  return TGA_LAUNCHED();
}

}  // namespace tga
