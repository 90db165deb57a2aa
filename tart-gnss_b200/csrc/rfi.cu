// Narrowband RFI scan per antenna (tart-gnss-acquire --rfi, rfi.rs:91-168).
//
// For every antenna row of packed bits:
//   * z = (+-1 samples) - mean over the whole row (rfi.rs:145-147);
//   * its spectrum in f64 (rfi.rs:100-106: FFT of the whole record, powers of
//     the first n/2 bins), with this library's own f64 FFT (fft64.cu) over
//     all antennas at once;
//   * the median bin power, exactly: a radix select over the bit patterns of
//     the non-negative powers (RfiBufs), no sorting.  24 rows of 818400 bins: the
//     eight histogram passes and their serial digit searches took 0.41 ms;
//     the first digit is counted where the powers are made, the second and the
//     gathering of the few bins left are a pass each, 0.08 ms in all (rows of
//     equal powers, which leave too many bins: rfi_median_kernel);
//   * local maxima p[k] > p[k-1], p[k] >= p[k+1] with 10 log10(p / floor) >
//     15 dB (rfi.rs:113-123), appended to a per-antenna list that the host
//     clusters (10 kHz, strongest first, at most 3 lines; rfi.rs:125-139);
//   * the autocorrelation at lags 1, 3 and 16 (rfi.rs:84-87) exactly from
//     popcounts: sum z_i z_{i+L} = sum s s' - m (sum s_head + sum s_tail)
//     + (n - L) m^2 with sum s s' = (n - L) - 2 popcount(b_i xor b_{i+L}).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <string>

#include "engine.h"

namespace tga {

namespace {

// the digit holding rank[a] among kRfiDigits counts, one block per antenna:
// narrows the prefix and the rank, and says how many bins share the prefix
__global__ void __launch_bounds__(256) rfi_select_kernel(const unsigned* __restrict__ hist, int digit, int shift,
                                                         unsigned rank0, unsigned long long* __restrict__ prefix,
                                                         unsigned* __restrict__ rank, unsigned* __restrict__ n_same) {
  __shared__ unsigned part[256];
  constexpr int PER = kRfiDigits / 256;
  const int a = blockIdx.x, t = threadIdx.x;
  const unsigned* h = hist + ((size_t)a * 2 + digit) * kRfiDigits + t * PER;
  unsigned sum = 0;
  for (int i = 0; i < PER; ++i) sum += h[i];
  part[t] = sum;
  __syncthreads();
  for (int o = 1; o < 256; o <<= 1) {  // inclusive scan
    const unsigned v = t >= o ? part[t - o] : 0u;
    __syncthreads();
    part[t] += v;
    __syncthreads();
  }
  const unsigned r = digit == 0 ? rank0 : rank[a];
  unsigned cum = part[t] - sum;
  __syncthreads();
  if (r >= cum && r < cum + sum) {
    int d = 0;
    while (cum + h[d] <= r) cum += h[d++];
    prefix[a] = (digit == 0 ? 0ull : prefix[a]) | ((unsigned long long)(t * PER + d) << shift);
    rank[a] = r - cum;
    n_same[a] = h[d];
  }
}

// f(bits) for every power of antenna a's row (an even number of them, rows
// 16-byte aligned): four 16-byte loads in flight per thread
template <class F>
__device__ __forceinline__ void for_powers(const double* __restrict__ p, unsigned half, int a, F&& f) {
  const double2* row = reinterpret_cast<const double2*>(p + (size_t)a * half);
  const unsigned n = half / 2, stride = gridDim.x * 256;
  for (unsigned k = blockIdx.x * 256 + threadIdx.x; k < n; k += 4 * stride) {
    double2 v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (k + i * stride < n) v[i] = __ldg(row + k + i * stride);
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (k + i * stride < n) {
        f((unsigned long long)__double_as_longlong(v[i].x));
        f((unsigned long long)__double_as_longlong(v[i].y));
      }
  }
}

// histogram of the second digit over the bins whose first digit is the prefix's
__global__ void __launch_bounds__(256) rfi_hist_kernel(const double* __restrict__ p, unsigned half,
                                                       const unsigned long long* __restrict__ prefix,
                                                       unsigned* __restrict__ hist) {
  __shared__ unsigned sh[kRfiDigits];
  const int a = blockIdx.y;
  for (int i = threadIdx.x; i < kRfiDigits; i += 256) sh[i] = 0;
  __syncthreads();
  const unsigned long long pre = prefix[a] >> kRfiShift0;
  for_powers(p, half, a, [&](unsigned long long u) {
    if (u >> kRfiShift0 == pre) atomicAdd(&sh[(u >> kRfiShift1) & (kRfiDigits - 1)], 1u);
  });
  __syncthreads();
  for (int i = threadIdx.x; i < kRfiDigits; i += 256)
    if (sh[i]) atomicAdd(hist + ((size_t)a * 2 + 1) * kRfiDigits + i, sh[i]);
}

// the bins that share both digits, where the list holds them
__global__ void __launch_bounds__(256) rfi_gather_kernel(const double* __restrict__ p, unsigned half,
                                                         const unsigned long long* __restrict__ prefix,
                                                         const unsigned* __restrict__ n_same,
                                                         unsigned* __restrict__ n_list,
                                                         unsigned long long* __restrict__ list) {
  const int a = blockIdx.y;
  if (n_same[a] > (unsigned)kRfiList) return;
  const unsigned long long pre = prefix[a] >> kRfiShift1;
  for_powers(p, half, a, [&](unsigned long long u) {
    if (u >> kRfiShift1 == pre) list[(size_t)a * kRfiList + atomicAdd(n_list + a, 1u)] = u;
  });
}

// The element of rank[a] among the gathered bins, one cluster per antenna: its
// first CTA ranks the list.  More bins than the list holds (a constant row, whose
// powers are all 0, or one with few samples off): three more digits over the
// whole row by the cluster, each CTA counting its share and summing an eighth
// of the digits over all.  One row of 818400 equal powers: the scan of one
// antenna takes 246 us; with one CTA for the digits, and the bins gathered
// before they were counted, 1074.
constexpr int kMedianCtas = 8, kMedianThreads = kRfiDigits / kMedianCtas;

__global__ void __cluster_dims__(kMedianCtas, 1, 1) __launch_bounds__(kMedianThreads)
    rfi_median_kernel(const double* __restrict__ p, unsigned half, const unsigned* __restrict__ n_same,
                      const unsigned long long* __restrict__ list, const unsigned* __restrict__ rank,
                      unsigned long long* __restrict__ prefix) {
  namespace cg = cooperative_groups;
  __shared__ unsigned sh[kRfiDigits];
  __shared__ unsigned s_warp[kMedianThreads / 32], s_total;
  __shared__ unsigned long long s_pre;
  __shared__ unsigned s_rank;
  cg::cluster_group cluster = cg::this_cluster();
  const int a = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned me = cluster.block_rank(), n = n_same[a];
  if (n <= (unsigned)kRfiList) {
    if (me != 0) return;
    const unsigned r = rank[a];
    const unsigned long long* l = list + (size_t)a * kRfiList;
    for (unsigned i = tid; i < n; i += kMedianThreads) {
      unsigned less = 0, same = 0;
      for (unsigned k = 0; k < n; ++k) {
        less += l[k] < l[i] ? 1u : 0u;
        same += l[k] == l[i] ? 1u : 0u;
      }
      if (r >= less && r < less + same) prefix[a] = l[i];  // equal elements write the same value
    }
    return;
  }
  if (tid == 0) {
    s_pre = prefix[a];
    s_rank = rank[a];
  }
  const double2* row = reinterpret_cast<const double2*>(p + (size_t)a * half);
  constexpr unsigned stride = kMedianCtas * kMedianThreads;
  for (int shift = kRfiShift1 - 13; shift > -13; shift -= 13) {
    const int lo = shift < 0 ? 0 : shift, width = shift < 0 ? 13 + shift : 13;
    for (int i = tid; i < kRfiDigits; i += kMedianThreads) sh[i] = 0;
    __syncthreads();
    const unsigned long long pre = s_pre;
    const unsigned left = s_rank;
    // equal digits of a warp are counted at once
    auto add = [&](double v, bool on) {
      const unsigned long long u = (unsigned long long)__double_as_longlong(v);
      const unsigned d = on && u >> (lo + width) == pre >> (lo + width) ? (unsigned)(u >> lo) & ((1u << width) - 1) : ~0u;
      const unsigned d0 = __shfl_sync(0xffffffffu, d, 0);
      if (__all_sync(0xffffffffu, d == d0)) {
        if (lane == 0 && d != ~0u) atomicAdd(&sh[d], 32u);
      } else if (d != ~0u) {
        atomicAdd(&sh[d], 1u);
      }
    };
    for (unsigned w = me * kMedianThreads + 32 * warp; w < half / 2; w += 4 * stride) {
      double2 v[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        v[i] = make_double2(0.0, 0.0);
        if (w + lane + i * stride < half / 2) v[i] = __ldg(row + w + lane + i * stride);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const bool on = w + lane + i * stride < half / 2;
        add(v[i].x, on);
        add(v[i].y, on);
      }
    }
    cluster.sync();
    // digit me kMedianThreads + tid of the whole row, and the counts up to it
    unsigned c = 0;
#pragma unroll
    for (int q = 0; q < kMedianCtas; ++q) c += *cluster.map_shared_rank(&sh[me * kMedianThreads + tid], q);
    unsigned upto = c;
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned v = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += v;
    }
    if (lane == 31) s_warp[warp] = upto;
    __syncthreads();
    for (int q = 0; q < warp; ++q) upto += s_warp[q];
    if (tid == kMedianThreads - 1) s_total = upto;
    cluster.sync();
    for (unsigned q = 0; q < me; ++q) upto += *cluster.map_shared_rank(&s_total, q);
    if (left < upto && left >= upto - c) {  // one thread of the cluster
      for (int q = 0; q < kMedianCtas; ++q) {
        *cluster.map_shared_rank(&s_pre, q) = pre | (unsigned long long)(me * kMedianThreads + tid) << lo;
        *cluster.map_shared_rank(&s_rank, q) = left - (upto - c);
      }
    }
    cluster.sync();
  }
  if (me == 0 && tid == 0) prefix[a] = s_pre;
}

__global__ void rfi_peaks_kernel(const double* __restrict__ p, long long half, const unsigned long long* __restrict__ floor_bits,
                                 double min_excess_db, int cap, unsigned* __restrict__ count,
                                 long long* __restrict__ bins, double* __restrict__ excess) {
  const int a = blockIdx.y;
  const double* row = p + (size_t)a * half;
  const double fl = __longlong_as_double((long long)floor_bits[a]);
  for (long long k = 1 + (long long)blockIdx.x * blockDim.x + threadIdx.x; k < half - 1;
       k += (long long)gridDim.x * blockDim.x) {
    const double v = row[k];
    // (15 dB is a factor of 31.62: the logarithm is taken only where it can matter)
    if (v > row[k - 1] && v >= row[k + 1] && v >= 31.6 * fl) {
      const double ex = 10.0 * log10(v / fl);
      if (ex > min_excess_db) {
        const unsigned idx = atomicAdd(&count[a], 1u);
        if (idx < (unsigned)cap) {
          bins[(size_t)a * cap + idx] = k;
          excess[(size_t)a * cap + idx] = ex;
        }
      }
    }
  }
}

__device__ __forceinline__ unsigned long long be_word(const uint8_t* row, size_t row_bytes, long long w) {
  unsigned long long v = 0;
  const long long b0 = w * 8;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const long long b = b0 + i;
    v = (v << 8) | (b < (long long)row_bytes ? (unsigned long long)__ldg(row + b) : 0ull);
  }
  return v;
}

// per antenna and lag L in {1, 3, 16}: popcounts of b_i xor b_{i+L}, of b_i
// and of b_{i+L} over i < n - L (big-endian words: sample 64 w + j is bit 63 - j)
__global__ void rfi_acf_kernel(const uint8_t* __restrict__ bits, size_t row_bytes, long long n,
                               unsigned long long* __restrict__ out /* [a][3][3] */) {
  const int a = blockIdx.y;
  const uint8_t* row = bits + (size_t)a * row_bytes;
  const long long words = (n + 63) / 64;
  const int lags[3] = {1, 3, 16};
  unsigned long long acc[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  for (long long w = (long long)blockIdx.x * blockDim.x + threadIdx.x; w < words; w += (long long)gridDim.x * blockDim.x) {
    const unsigned long long cur = be_word(row, row_bytes, w), nxt = be_word(row, row_bytes, w + 1);
#pragma unroll
    for (int l = 0; l < 3; ++l) {
      const int L = lags[l];
      const unsigned long long sh = (cur << L) | (nxt >> (64 - L));
      const long long vb = n - L - 64 * w;  // valid positions in this word
      const unsigned long long mask = vb >= 64 ? ~0ull : (vb <= 0 ? 0ull : (~0ull << (64 - vb)));
      acc[3 * l] += __popcll((cur ^ sh) & mask);
      acc[3 * l + 1] += __popcll(cur & mask);
      acc[3 * l + 2] += __popcll(sh & mask);
    }
  }
#pragma unroll
  for (int j = 0; j < 9; ++j) {
    unsigned long long v = acc[j];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(out + (size_t)a * 9 + j, v);
  }
}

}  // namespace

cudaError_t rfi_scan_device(const uint8_t* d_bits, int n_ant, size_t row_bytes, const double* d_mean, const RfiBufs& b,
                            int cap, int num_sms, cudaStream_t st, std::string* why) {
  const long long n = (long long)row_bytes * 8, half = n / 2;
  if (n_ant <= 0 || n < 8) return cudaSuccess;
  cudaError_t e;
  const size_t A = (size_t)n_ant;
  if ((e = cudaMemsetAsync(b.hist, 0, A * 2 * kRfiDigits * sizeof(unsigned), st)) != cudaSuccess) return e;
  if ((e = cudaMemsetAsync(b.n_list, 0, A * sizeof(unsigned), st)) != cudaSuccess) return e;
  if ((e = cudaMemsetAsync(b.count, 0, A * sizeof(unsigned), st)) != cudaSuccess) return e;
  if ((e = cudaMemsetAsync(b.acf, 0, A * 9 * sizeof(unsigned long long), st)) != cudaSuccess) return e;
  // powers of the first n/2 bins of every antenna's f64 spectrum
  e = real_power_spectrum(d_bits, row_bytes, d_mean, b.z, b.X, b.work, n_ant, b.p, b.hist, num_sms, st, why);
  if (e != cudaSuccess) return e;
  // median bin power: rank half / 2 (rfi.rs:110-111)
  const unsigned h = (unsigned)half;
  const dim3 g((unsigned)std::min<long long>(std::max(32, 8 * num_sms / n_ant), (half + 2047) / 2048), (unsigned)n_ant);
  rfi_select_kernel<<<n_ant, 256, 0, st>>>(b.hist, 0, kRfiShift0, h / 2, b.prefix, b.rank, b.n_same);
  rfi_hist_kernel<<<g, 256, 0, st>>>(b.p, h, b.prefix, b.hist);
  rfi_select_kernel<<<n_ant, 256, 0, st>>>(b.hist, 1, kRfiShift1, 0u, b.prefix, b.rank, b.n_same);
  rfi_gather_kernel<<<g, 256, 0, st>>>(b.p, h, b.prefix, b.n_same, b.n_list, b.list);
  rfi_median_kernel<<<dim3(kMedianCtas, (unsigned)n_ant), kMedianThreads, 0, st>>>(b.p, h, b.n_same, b.list, b.rank,
                                                                                  b.prefix);
  rfi_peaks_kernel<<<dim3(256, (unsigned)n_ant), 256, 0, st>>>(b.p, half, b.prefix, 15.0, cap, b.count, b.bins,
                                                               b.excess);
  rfi_acf_kernel<<<dim3(64, (unsigned)n_ant), 256, 0, st>>>(d_bits, row_bytes, n, b.acf);
  kernel_launch_add(7);
  return cudaGetLastError();
}

}  // namespace tga
