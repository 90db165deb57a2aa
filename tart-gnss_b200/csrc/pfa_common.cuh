// Shared definitions of the prime-factor transform kernels (FP32 SIMT and
// tensor-core variants).
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "engine.h"

namespace tga {

constexpr int modinv_c(int a, int m) {
  a %= m;
  for (int x = 1; x < m; ++x)
    if ((a * x) % m == 1) return x;
  return 0;
}

// Geometry of the Lc = 31 * 33 * M prime-factor transform.
template <int M>
struct Geo {
  static constexpr int NC = M;
  static constexpr int COLS = 33 * M;  // columns of the DFT-31 stage
  static constexpr int LC = 31 * COLS;
  // natural index n = (a*EA + b*EB + c*EC) mod LC for digits (a, b, c)
  static constexpr int EA = (LC / 31) * modinv_c((LC / 31) % 31, 31);
  static constexpr int EB = (LC / 33) * modinv_c((LC / 33) % 33, 33);
  static constexpr int EC = (M == 1) ? 0 : (LC / M) * modinv_c((LC / M) % M, M);
  __device__ static __forceinline__ int natural(int a, int b, int c) {
    return (int)((unsigned)(a * EA + b * EB + c * EC) % (unsigned)LC);
  }
  // digit-layout offset of (a, b, c): [a][c][b]
  __device__ static __forceinline__ int offset(int a, int b, int c) { return a * COLS + c * 33 + b; }
};

// FP16 operands of the tensor-core search.  Lc = R1 x 31 x GR with R1 = 33,
// 44, 55 for M = 1, 4, 10; GR counts the digits left over (1; 3; 2 x 3).
// Unit u = (gr 4 + j) R1P + d1 of a sequence holds the spectrum at 31-digits
// 8 j .. 8 j + 7 (zero for digit 31), R1-digit d1 (zero from R1 on: R1P is R1
// padded so that eight units from d1 = 0 on are 128 aligned bytes, one
// shared-memory wavefront) and left-over digits gr
// (M = 10: gr = 2 b + h, b of 3 and h of 2) as eight FP16 real parts (16
// bytes, in the first plane of PER_SEQ / 2 units) and eight imaginary parts
// (the same place in the second plane).  A unit is then one 16-byte row of
// the first stage's operand (8 columns of one K entry), and the products of
// two units are packed FP16 operations on whole registers.  A frequency
// digit d of radix R stands for the natural frequencies k = d (Lc / R) (mod
// R); src_offset is where the FP32 engine's digit layout [a][c][b] of the
// (31, 33, M) map holds the same frequency.
__device__ __forceinline__ void pack_unit(const float2 (&v)[8], uint4& re, uint4& im) {
  uint32_t r[4], i[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const __half2 a = __floats2half2_rn(v[2 * k].x, v[2 * k + 1].x);
    const __half2 b = __floats2half2_rn(v[2 * k].y, v[2 * k + 1].y);
    r[k] = *reinterpret_cast<const uint32_t*>(&a);
    i[k] = *reinterpret_cast<const uint32_t*>(&b);
  }
  re = make_uint4(r[0], r[1], r[2], r[3]);
  im = make_uint4(i[0], i[1], i[2], i[3]);
}

template <int M>
struct TcUnits {
  static constexpr int R1 = M == 1 ? 33 : M == 4 ? 44 : 55, GR = M == 1 ? 1 : M == 4 ? 3 : 6;
  static constexpr int R1P = (2 * R1 + 15) / 16 * 8;  // 40, 48, 56
  static constexpr int LC = 1023 * M, UNITS = GR * 4 * R1P, PER_SEQ = 2 * UNITS;
  static_assert(R1 * 31 * GR == LC, "factorisation");
  static constexpr int digit(int R) { return (LC / R) * modinv_c((LC / R) % R, R); }
  static constexpr int UB = modinv_c((LC / 33) % 33, 33);
  static constexpr int UC = M == 1 ? 0 : modinv_c((LC / M) % M, M);
  __host__ __device__ static constexpr int freq_part(int d, int R, int E) { return ((d * (LC / R)) % R) * E; }
  // 31-digit i of unit u holds a value (not padding)
  __host__ __device__ static __forceinline__ bool filled(int u, int i) {
    return u % R1P < R1 && 8 * ((u / R1P) & 3) + i < 31;
  }
  // digit-layout offset of the frequency at 31-digit i of unit u
  __host__ __device__ static __forceinline__ int src_offset(int u, int i) {
    constexpr int E1 = digit(R1), E31 = digit(31), E3 = M == 1 ? 0 : digit(3), E2 = M == 10 ? digit(2) : 0;
    const int q = u / R1P, d1 = u - q * R1P, gr = q >> 2, d2 = 8 * (q & 3) + i;
    const int b = M == 10 ? gr >> 1 : gr, h = M == 10 ? gr & 1 : 0;
    int k = freq_part(d1, R1, E1) + freq_part(d2, 31, E31);
    if (M != 1) k += freq_part(b, 3, E3);
    if (M == 10) k += freq_part(h, 2, E2);
    k %= LC;
    const int kb = (UB * k) % 33, kc = M == 1 ? 0 : (UC * k) % M;
    return d2 * 33 * M + kc * 33 + kb;  // the 31-digit is the same in both layouts
  }
};

// The four largest (value, index) pairs seen by a thread, largest first;
// values are non-negative |y|^2 (as bits they order like unsigned
// integers), an empty place holds 0.
struct Top4 {
  float v[4] = {0.f, 0.f, 0.f, 0.f};
  int i[4] = {0, 0, 0, 0};
  __device__ __forceinline__ void add(float x, int k) {
    if (!(x > v[3])) return;
    const bool g0 = x > v[0], g1 = x > v[1], g2 = x > v[2];
    v[3] = g2 ? v[2] : x;
    i[3] = g2 ? i[2] : k;
    v[2] = g1 ? v[1] : (g2 ? x : v[2]);
    i[2] = g1 ? i[1] : (g2 ? k : i[2]);
    v[1] = g0 ? v[0] : (g1 ? x : v[1]);
    i[1] = g0 ? i[0] : (g1 ? k : i[1]);
    v[0] = g0 ? x : v[0];
    i[0] = g0 ? k : i[0];
  }
  __device__ __forceinline__ void pop() {
    v[0] = v[1], i[0] = i[1];
    v[1] = v[2], i[1] = i[2];
    v[2] = v[3], i[2] = i[3];
    v[3] = 0.f;
  }
};

// CAND is CORR over a device-built list of rows (the candidates of a
// reduced-precision search, re-evaluated in FP32): row i of the list is
// (ab * 2 + hyp, prn), the list holds *cand_count rows, and each row's key
// goes where CORR would write it.
enum PfaMode { FWD_Z = 0, FWD_D = 1, CORR = 2, SECOND = 3, CAND = 4 };

struct PfaParams {
  float2* z;                  // FWD_Z: sequences, transformed in place; CORR/SECOND: Z
  const float2* D;            // CORR/SECOND: conjugated code spectra
  float2* Dout;               // FWD_D output
  const int8_t* chips;        // FWD_D input [n_prn][Lc]
  int n_seq;                  // FWD modes
  int n_items;                // CORR: n_ab*2*n_prn rows; SECOND: n_ant*n_prn; CAND: list capacity
  int n_prn, S, P, chip_width;
  unsigned long long* keys;   // CORR / CAND output, one per row ([ab * 2 + hyp][prn])
  BestRow* best;              // SECOND in/out
  const int2* cand;           // CAND: the rows to evaluate
  const int* cand_count;      // CAND: their number (device)
  int split;                  // CORR / SECOND: CTAs that share a row's residue groups
  unsigned long long* top_lists;  // CAND with p2rows, split rows: their residues' lists
  int* top_done;              // and the parts finished (zeroed), both for kMaxSplitRows rows
  float* p2rows;              // CAND (optional): each listed row's second peak
                              // against its own maximum, where its key goes
  uint4* z16;                 // FWD_Z (optional): the transformed sequences also as TcUnits, x z16_scale
  const uint4* z16_map;       // per unit: the 8 src_offset values as 16-bit fields (0xffff: zero)
  float z16_scale;
};

}  // namespace tga
