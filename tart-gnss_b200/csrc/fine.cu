// Fine acquisition: correlation of a band-limited code replica at a
// continuous code delay and carrier frequency, with its first and second
// derivatives, over many antennas in one pass.
//
// The reference's only precedent is optimize_fit (junk/acquisition.py:403-445),
// which refines the frequency by a scalar search and the code phase by a
// Gaussian fit to three correlation samples.  Here the refinement is a Newton
// iteration on the coherent multi-antenna power
//
//   P(tau, f, phi) = | sum_a exp(-i phi_a) R_a(tau, f) |^2,
//   R_a(tau, f)    = (1/N) sum_n s_a[n] exp(+i 2 pi f (n - n0) / fs) c(n - tau),
//
// s_a the de-meaned +-1 samples of antenna a (the reference's wipe-off sign
// convention, correlate.rs:110-115), c the code as a sequence of
// rectangular (sub)chips of T samples whose edges are smoothed by a Gaussian
// of standard deviation sigma samples (a front-end filter model; without it a
// fractional delay is not observable at an integer number of samples per
// chip).  The kernel returns, per (task, antenna), the six complex sums
//
//   R, dR/dtau, dR/df, d2R/dtau2, d2R/df2, d2R/dtau df
//
// from which the host forms P, its gradient with respect to (tau, f, phi_a)
// and its Hessian: the gradient of |S|^2 is the adjoint contraction
// 2 Re(conj(S) dS), which needs exactly these tangents of S.
#include <cuda_runtime.h>

#include <cstdint>

#include "chip_index.h"
#include "engine.h"

namespace tga {

namespace {

constexpr int kFineThreads = 256;
constexpr int kFineChunk = 1024;  // samples per block of the sums
constexpr int kScanSub = 256;     // samples of the scan's shared-memory tile
constexpr int kScanTiles = 4;     // tiles per block of the scan
// frequencies and antennas of the scan's tile, one (frequency, antenna pair) per
// thread: the default scan of a 10 ms window on the receiver's 24 antennas fills
// 252 of 256.  A narrower scan or fewer antennas leave threads of the products
// idle, more of either repeats a tile's replicas; against the six sums at every
// frequency it is still ahead everywhere (4 satellites, 100 ms, 129 frequencies:
// 1 antenna 20.4 -> 4.1 ms, 9 antennas 33.4 -> 7.0, 25 antennas 54.4 -> 14.5, 48
// antennas 89 -> 23; one satellite, 10 ms, 2 antennas 478 -> 406 us a call).
constexpr int kScanK = 21, kScanAnt = 24;

// replica value and its first two derivatives at continuous time t (samples)
// from the four edges around t: c(t) = seq[k] + sum_m d_m (Phi(u_m) - [u_m >= 0])
__device__ __forceinline__ void replica(const int8_t* __restrict__ seq, int L, double T, double inv_sigma, double t,
                                        float& c, float& c1, float& c2) {
  const double k = floor(t / T);
  const int kk = chip_index(k, L);
  auto wrap = [&](int m) -> int { return m < 0 ? m + L : m >= L ? m - L : m; };  // L >= 1023
  c = (float)__ldg(seq + kk);
  c1 = 0.f;
  c2 = 0.f;
  const float is = (float)inv_sigma;
#pragma unroll
  for (int dm = -1; dm <= 2; ++dm) {
    const float d = (float)(__ldg(seq + wrap(kk + dm)) - __ldg(seq + wrap(kk + dm - 1)));  // jump at edge kk + dm
    if (d == 0.f) continue;
    const float u = (float)((t - (k + (double)dm) * T) * inv_sigma);
    const float pdf = 0.3989422804014327f * __expf(-0.5f * u * u);
    c += d * (normcdff(u) - (u >= 0.f ? 1.f : 0.f));
    c1 += d * pdf * is;
    c2 -= d * u * pdf * is * is;
  }
}

// Sums of every antenna over one chunk.  The seven per-sample weights go to
// shared memory; a warp then takes NQ antennas through the chunk, so that each
// weight read serves all of them (one antenna at a time the loop was bound by
// those reads: 127 -> 90 us for 12 satellites x 24 antennas x 163680 samples,
// index arithmetic in 32 bits included).  NQ is chosen so that the block's eight
// warps cover the antennas in one go where they can: 1 up to 8 antennas, 2 up to
// 16, 3 beyond.  The order of each antenna's additions does not depend on NQ.
template <int NQ>
__global__ void __launch_bounds__(kFineThreads) fine_sums_kernel(const uint8_t* __restrict__ bits, int n_ant,
                                                                 size_t row_bytes, const double* __restrict__ mean,
                                                                 const FineTask* __restrict__ tasks,
                                                                 double* __restrict__ out) {
  __shared__ float s_w[7][kFineChunk];  // per sample: a0 (2), a1 (2), a2 (2), x
  const FineTask tk = tasks[blockIdx.y];
  const long long c0 = (long long)blockIdx.x * kFineChunk;
  if (c0 >= tk.length) return;
  const int cn = (int)min((long long)kFineChunk, tk.length - c0);
  const double inv_sigma = 1.0 / tk.sigma;
  for (int i = threadIdx.x; i < cn; i += kFineThreads) {
    const long long n = tk.start + c0 + i;
    const double dn = (double)n - tk.n0;
    // carrier phase reduced in f64 before the single-precision sincos
    double cyc = tk.f_over_fs * dn;
    cyc -= floor(cyc);
    float sn, cs;
    sincospif((float)(2.0 * cyc), &sn, &cs);
    float c, c1, c2;
    replica(tk.seq, tk.seq_len, tk.T, inv_sigma, (double)n - tk.tau, c, c1, c2);
    s_w[0][i] = cs * c;
    s_w[1][i] = sn * c;
    s_w[2][i] = -cs * c1;  // d/dtau of c(n - tau) = -c'
    s_w[3][i] = -sn * c1;
    s_w[4][i] = cs * c2;
    s_w[5][i] = sn * c2;
    s_w[6][i] = (float)(dn * tk.two_pi_over_fs);
  }
  __syncthreads();

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int g = warp; g * NQ < n_ant; g += kFineThreads / 32) {
    const int ant0 = g * NQ;
    const uint8_t* row[NQ];
    float hi[NQ], lo[NQ], acc[NQ][12];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const int ant = min(ant0 + q, n_ant - 1);
      row[q] = bits + (size_t)ant * row_bytes;
      const float m = (float)mean[ant];
      hi[q] = 1.f - m;
      lo[q] = -1.f - m;
#pragma unroll
      for (int j = 0; j < 12; ++j) acc[q][j] = 0.f;
    }
    for (int i = lane; i < cn; i += 32) {
      const long long n = tk.start + c0 + i;
      const float a0r = s_w[0][i], a0i = s_w[1][i], a1r = s_w[2][i], a1i = s_w[3][i];
      const float a2r = s_w[4][i], a2i = s_w[5][i], x = s_w[6][i];
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        const int bit = (__ldg(row[q] + (n >> 3)) >> (7 - (int)(n & 7))) & 1;
        const float s = bit ? hi[q] : lo[q];
        const float sx = s * x, sxx = sx * x;
        acc[q][0] = fmaf(s, a0r, acc[q][0]);  // R
        acc[q][1] = fmaf(s, a0i, acc[q][1]);
        acc[q][2] = fmaf(s, a1r, acc[q][2]);  // dR/dtau
        acc[q][3] = fmaf(s, a1i, acc[q][3]);
        acc[q][4] = fmaf(-sx, a0i, acc[q][4]);  // dR/df / (2 pi / fs) folded in x: i x a0
        acc[q][5] = fmaf(sx, a0r, acc[q][5]);
        acc[q][6] = fmaf(s, a2r, acc[q][6]);  // d2R/dtau2
        acc[q][7] = fmaf(s, a2i, acc[q][7]);
        acc[q][8] = fmaf(-sxx, a0r, acc[q][8]);  // d2R/df2: -x^2 a0
        acc[q][9] = fmaf(-sxx, a0i, acc[q][9]);
        acc[q][10] = fmaf(-sx, a1i, acc[q][10]);  // d2R/dtau df: i x a1
        acc[q][11] = fmaf(sx, a1r, acc[q][11]);
      }
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      if (ant0 + q >= n_ant) break;  // uniform over the warp
      float mine = 0.f;
#pragma unroll
      for (int j = 0; j < 12; ++j) {
        float v = acc[q][j];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == j) mine = v;
      }
      if (lane < 12) atomicAdd(out + ((size_t)tk.slot * n_ant + ant0 + q) * 12 + lane, (double)mine);
    }
  }
}

// R alone (the first of the six sums) at n_k frequencies f_over_fs + (k - k0)
// df_over_fs: what the frequency scan needs, out[slot + k][antenna][2].  The
// replica does not depend on the frequency, so it is evaluated once per sample;
// then R[a][k] = sum_n s_a[n] w[n][k] is a small matrix product from shared
// memory, two antennas and one frequency per thread: 12 satellites x 21
// frequencies x 24 antennas x 163680 samples took 2.38 ms as 252 evaluations
// of the six sums, and take 0.39 ms so (half of it the 21 phasors per sample).
// Bound by the shared-memory path (its wavefronts 71 % of peak, issue 52 %).  FP32
// over 32 samples, then f64.
__global__ void __launch_bounds__(kFineThreads) fine_scan_kernel(const uint8_t* __restrict__ bits, int n_ant,
                                                                 size_t row_bytes, const double* __restrict__ mean,
                                                                 const FineScan* __restrict__ tasks,
                                                                 double* __restrict__ out) {
  extern __shared__ __align__(16) float2 s_mem[];
  float2* s_w = s_mem;                               // [kScanSub][kScanK]
  float2* s_s = s_mem + (size_t)kScanSub * kScanK;   // [kScanSub][kScanAnt / 2]: two antennas' samples
  const FineScan sc = tasks[blockIdx.y];
  const FineTask tk = sc.task;
  const int k_lo = (int)blockIdx.z * kScanK;
  const long long c0 = (long long)blockIdx.x * kScanSub * kScanTiles;
  if (c0 >= tk.length || k_lo >= sc.n_k) return;
  const int nk = min(kScanK, sc.n_k - k_lo);
  const double inv_sigma = 1.0 / tk.sigma;
  for (int ant0 = 0; ant0 < n_ant; ant0 += kScanAnt) {
    const int na = min(kScanAnt, n_ant - ant0), pairs = (na + 1) / 2;
    const int item = threadIdx.x, k = item % kScanK, pr = item / kScanK;
    const bool mine = k < nk && pr < pairs;
    double sum[4] = {0.0, 0.0, 0.0, 0.0};
    for (int tile = 0; tile < kScanTiles; ++tile) {
      const long long t0 = c0 + (long long)tile * kScanSub;
      if (t0 >= tk.length) break;
      const int cn = (int)min((long long)kScanSub, tk.length - t0);
      __syncthreads();
      for (int i = threadIdx.x; i < kScanSub; i += kFineThreads) {
        float c = 0.f, c1, c2;
        const long long n = tk.start + t0 + i;
        const double dn = (double)n - tk.n0;
        if (i < cn) replica(tk.seq, tk.seq_len, tk.T, inv_sigma, (double)n - tk.tau, c, c1, c2);
        for (int kq = 0; kq < nk; ++kq) {
          double cyc = (tk.f_over_fs + (double)(k_lo + kq - sc.k0) * sc.df_over_fs) * dn;
          cyc -= floor(cyc);
          float sn, cs;
          sincospif((float)(2.0 * cyc), &sn, &cs);
          s_w[i * kScanK + kq] = make_float2(cs * c, sn * c);
        }
      }
      for (int e = threadIdx.x; e < kScanSub * pairs; e += kFineThreads) {
        const int pq = e / kScanSub, i = e - pq * kScanSub;
        float v[2] = {0.f, 0.f};
        if (i < cn) {
          const long long n = tk.start + t0 + i;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int ant = ant0 + 2 * pq + h;
            if (ant < n_ant) {
              const int bit = (__ldg(bits + (size_t)ant * row_bytes + (n >> 3)) >> (7 - (int)(n & 7))) & 1;
              const float m = (float)mean[ant];
              v[h] = bit ? 1.f - m : -1.f - m;
            }
          }
        }
        s_s[i * (kScanAnt / 2) + pq] = make_float2(v[0], v[1]);
      }
      __syncthreads();
      if (mine) {
        for (int i0 = 0; i0 < kScanSub; i0 += 32) {
          float r0 = 0.f, q0 = 0.f, r1 = 0.f, q1 = 0.f;
#pragma unroll 8
          for (int i = i0; i < i0 + 32; ++i) {
            const float2 w = s_w[i * kScanK + k], sv = s_s[i * (kScanAnt / 2) + pr];
            r0 = fmaf(sv.x, w.x, r0);
            q0 = fmaf(sv.x, w.y, q0);
            r1 = fmaf(sv.y, w.x, r1);
            q1 = fmaf(sv.y, w.y, q1);
          }
          sum[0] += (double)r0;
          sum[1] += (double)q0;
          sum[2] += (double)r1;
          sum[3] += (double)q1;
        }
      }
    }
    if (mine) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int ant = ant0 + 2 * pr + h;
        if (ant >= n_ant) break;
        double* dst = out + ((size_t)(tk.slot + k_lo + k) * n_ant + ant) * 2;
        atomicAdd(dst, sum[2 * h]);
        atomicAdd(dst + 1, sum[2 * h + 1]);
      }
    }
  }
}

}  // namespace

cudaError_t launch_fine_sums(const uint8_t* d_bits, int n_ant, size_t row_bytes, const double* d_mean,
                             const FineTask* d_tasks, int n_tasks, long long max_length, double* d_out,
                             cudaStream_t st) {
  if (n_tasks <= 0 || max_length <= 0) return cudaSuccess;
  cudaError_t e = cudaMemsetAsync(d_out, 0, (size_t)n_tasks * n_ant * 12 * sizeof(double), st);
  if (e != cudaSuccess) return e;
  const long long chunks = (max_length + kFineChunk - 1) / kFineChunk;
  if (chunks > 0x7fffffffLL || n_tasks > 65535) return cudaErrorInvalidValue;
  dim3 grid((unsigned)chunks, (unsigned)n_tasks);
  auto kern = n_ant <= 8 ? fine_sums_kernel<1> : n_ant <= 16 ? fine_sums_kernel<2> : fine_sums_kernel<3>;
  kern<<<grid, kFineThreads, 0, st>>>(d_bits, n_ant, row_bytes, d_mean, d_tasks, d_out);
  kernel_launch_add(1);
  return cudaGetLastError();
}

cudaError_t launch_fine_scan(const uint8_t* d_bits, int n_ant, size_t row_bytes, const double* d_mean,
                             const FineScan* d_tasks, int n_tasks, int n_points, int max_k, long long max_length,
                             double* d_out, cudaStream_t st) {
  if (n_tasks <= 0 || max_length <= 0) return cudaSuccess;
  cudaError_t e = cudaMemsetAsync(d_out, 0, (size_t)n_points * n_ant * 2 * sizeof(double), st);
  if (e != cudaSuccess) return e;
  constexpr long long kChunk = (long long)kScanSub * kScanTiles;
  const long long chunks = (max_length + kChunk - 1) / kChunk, kt = (max_k + kScanK - 1) / kScanK;
  if (chunks > 0x7fffffffLL || n_tasks > 65535 || kt > 65535) return cudaErrorInvalidValue;
  constexpr size_t smem = (size_t)kScanSub * (kScanK + kScanAnt / 2) * sizeof(float2);
  static_assert(kScanK * (kScanAnt / 2) <= kFineThreads, "one item per thread");
  e = cudaFuncSetAttribute(fine_scan_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  fine_scan_kernel<<<dim3((unsigned)chunks, (unsigned)n_tasks, (unsigned)kt), kFineThreads, smem, st>>>(
      d_bits, n_ant, row_bytes, d_mean, d_tasks, d_out);
  kernel_launch_add(1);
  return cudaGetLastError();
}

}  // namespace tga
