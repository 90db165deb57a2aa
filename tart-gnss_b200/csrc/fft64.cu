// Double-precision FFT of any length for the RFI scan (rfi.rs:91-106 takes
// the f64 spectrum of a whole record per antenna).
//
// Mixed-radix Stockham autosort passes (the formulation of Govindaraju et
// al., SC'08, generalised from radix 2 to any radix R): with the
// sub-transforms of length Ns done, one pass writes
//
//   out[q Ns R + r Ns + k] = sum_{s < R} in[q Ns + k + s L / R] W_L^{s (k + r Ns) L / (Ns R)}
//
// (k < Ns, r < R, W_L = exp(-2 pi i / L)), so after the passes of all
// factors of L the result is in natural order.  Each pass reads and writes
// the whole batch, so what counts is their number (a pass runs at 4 to 6 TB/s,
// HBM half busy: 7 to 10 warps per SM, which the butterfly's registers allow,
// wait for their loads): the factors are gathered into radices of up to 33 (32; 33 = 3 x 11
// and 15 = 3 x 5 without twiddles; 25; 31, ...), one whole butterfly per thread in
// registers, and the first pass reads the packed bits themselves.  24 rows of
// 1636800 samples (L = 32 x 25 x 33 x 31): the seven passes of radices 16, 2,
// 3, 5, 5, 11, 31 with R-term sums took 4.2 ms, the four passes 0.41 ms.
// Other prime factors up to kMaxRadix run as one output per thread, an R-term
// sum.  Twiddles come from one table W_L^m, m < L, built in double precision
// with sincospi; a butterfly loads about 2 sqrt(R) of them and forms the
// others as products of two.  A length with a prime factor above kMaxRadix is
// transformed by Bluestein's chirp-z identity over a power-of-two convolution.
//
// The real record of n samples is transformed as n/2 complex points z[m] =
// x[2m] + i x[2m+1] (the layout the record already has as doubles), then
//   X[k] = (Z[k] + conj(Z[L-k])) / 2 - i W_n^k (Z[k] - conj(Z[L-k])) / 2,
// L = n/2, of which the scan keeps |X[k]|^2 for k < n/2.
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <string>
#include <vector>

#include "engine.h"
#include "mixed_radix.cuh"

namespace tga {

namespace {

constexpr int kMaxRadix = 1024;

// tw[m] = exp(-2 pi i m / L), m < L
__global__ void twiddle64_kernel(double2* __restrict__ tw, long long L) {
  for (long long m = (long long)blockIdx.x * blockDim.x + threadIdx.x; m < L; m += (long long)gridDim.x * blockDim.x) {
    double s, c;
    sincospi(2.0 * (double)m / (double)L, &s, &c);
    tw[m] = make_double2(c, -s);
  }
}

// One pass of radix R, one butterfly per thread; blockIdx.y is the sequence.
// FIRST (Ns = 1): the input is the row's samples, complex point m = (sample
// 2 m) + i (sample 2 m + 1), each +-1 - mean; a thread's R outputs are
// contiguous, so the block's go out through shared memory in order.
struct FirstSource {
  const uint8_t* bits;
  size_t row_bytes;
  const double* mean;
};
constexpr int kPassThreads = 128;

template <int R, bool FIRST>
__global__ void __launch_bounds__(kPassThreads) pass64_kernel(const double2* __restrict__ in, FirstSource src,
                                                              double2* __restrict__ out,
                                                              const double2* __restrict__ tw, unsigned L,
                                                              unsigned Ns) {
  extern __shared__ __align__(16) double2 s_out[];
  const unsigned LR = L / R, j = blockIdx.x * kPassThreads + threadIdx.x;
  const size_t seq = (size_t)blockIdx.y * L;
  double2 v[R];
  if (j < LR) {
    if constexpr (FIRST) {
      const uint8_t* row = src.bits + (size_t)blockIdx.y * src.row_bytes;
      const double m = src.mean[blockIdx.y], hi = 1.0 - m, lo = -1.0 - m;
#pragma unroll
      for (int s = 0; s < R; ++s) {
        const unsigned i = j + s * LR;  // samples 2 i and 2 i + 1
        const unsigned two = (unsigned)__ldg(row + (i >> 2)) >> (6 - 2 * (i & 3u));
        v[s] = make_double2(two & 2u ? hi : lo, two & 1u ? hi : lo);
      }
      double2* o = s_out + threadIdx.x * (R + 1);
      mr_dft<R>(v, [&](int r, double2 y) { o[r] = y; });
    } else {
      const unsigned q = j / Ns, k = j - q * Ns, b = k * (L / (Ns * R));  // twiddle of s: W_L^{s b}
      const double2* x = in + seq + j;
#pragma unroll
      for (int s = 0; s < R; ++s) v[s] = x[(size_t)s * LR];
      // W^{s b} = W^{(s % G) b} W^{(s - s % G) b}
      constexpr int G = R <= 4 ? R : R <= 9 ? 3 : R <= 16 ? 4 : 6;
      double2 lowp[G];
#pragma unroll
      for (int s = 1; s < G; ++s) lowp[s] = __ldg(tw + (size_t)s * b);
#pragma unroll
      for (int g = 0; g < R; g += G) {
        double2 h = make_double2(1.0, 0.0);
        if (g > 0) h = __ldg(tw + (size_t)g * b);
#pragma unroll
        for (int s = 0; s < G; ++s) {
          if (g + s >= R || g + s == 0) continue;
          const double2 w = s == 0 ? h : g == 0 ? lowp[s] : mr_cmul(h, lowp[s]);
          v[g + s] = mr_cmul(v[g + s], w);
        }
      }
      double2* y = out + seq + (size_t)q * Ns * R + k;
      mr_dft<R>(v, [&](int r, double2 t) { y[(size_t)r * Ns] = t; });
    }
  }
  if constexpr (FIRST) {
    __syncthreads();
    const unsigned j0 = blockIdx.x * kPassThreads, n = min((unsigned)kPassThreads, LR - j0) * R;
    double2* y = out + seq + (size_t)j0 * R;
    for (unsigned i = threadIdx.x; i < n; i += kPassThreads) y[i] = s_out[i + i / R];
  }
}

// One pass of any radix R, one output per thread (an R-term sum).
__global__ void __launch_bounds__(256) pass_any_kernel(const double2* __restrict__ in, double2* __restrict__ out,
                                                       const double2* __restrict__ tw, long long L, int R,
                                                       long long Ns, long long total) {
  const long long LR = L / R, NsR = Ns * R, step = L / NsR;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const long long a = i / L, o = i - a * L;
    const long long q = o / NsR, rem = o - q * NsR, r = rem / Ns, k = rem - r * Ns;
    const double2* x = in + a * L + q * Ns + k;
    const long long base = (k + r * Ns) * step;  // < L
    double2 acc = make_double2(0.0, 0.0);
    long long m = 0;
    for (int s = 0; s < R; ++s) {
      const double2 u = x[s * LR], w = __ldg(tw + m);
      acc.x += u.x * w.x - u.y * w.y;
      acc.y += u.x * w.y + u.y * w.x;
      m += base;
      if (m >= L) m -= L;
    }
    out[i] = acc;
  }
}

int grid_for(long long work, int num_sms) {
  long long g = (work + 255) / 256;
  const long long cap = (long long)num_sms * 32;
  return (int)(g < 1 ? 1 : (g > cap ? cap : g));
}

template <int R, bool FIRST>
cudaError_t run_pass64(const double2* x, const FirstSource& src, double2* y, const double2* tw, long long L, int batch,
                       long long Ns, cudaStream_t st) {
  const size_t smem = FIRST ? (size_t)kPassThreads * (R + 1) * sizeof(double2) : 0;
  auto kern = pass64_kernel<R, FIRST>;
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  const dim3 grid((unsigned)((L / R + kPassThreads - 1) / kPassThreads), (unsigned)batch);
  kern<<<grid, kPassThreads, smem, st>>>(x, src, y, tw, (unsigned)L, (unsigned)Ns);
  return cudaGetLastError();
}

// Stockham passes over `batch` sequences of length L (below 2^30) in a
// (ping-pong with b); *result is the buffer holding the result.  With src the
// first pass reads the rows' bits and a is only written.
cudaError_t stockham(double2* a, double2* b, const FirstSource* src, const double2* tw, long long L, int batch,
                     const std::vector<int>& radices, int num_sms, cudaStream_t st, double2** result) {
  long long Ns = 1;
  double2* x = a;
  double2* y = b;
  const FirstSource none = {};
  for (int R : radices) {
    cudaError_t e;
    const bool first = Ns == 1 && src;
    switch (R) {
#define TGA_PASS(RR)                                                                          \
  case RR:                                                                                    \
    e = run_pass64<RR, false>(x, none, y, tw, L, batch, Ns, st);                              \
    break;
#define TGA_PASS2(RR)                                                                         \
  case RR:                                                                                    \
    e = first ? run_pass64<RR, true>(x, *src, y, tw, L, batch, Ns, st)                        \
              : run_pass64<RR, false>(x, none, y, tw, L, batch, Ns, st);                      \
    break;
      TGA_PASS2(32) TGA_PASS2(16) TGA_PASS2(8) TGA_PASS2(4) TGA_PASS(2)
      TGA_PASS(33) TGA_PASS(25) TGA_PASS(15) TGA_PASS(31) TGA_PASS(13) TGA_PASS(11) TGA_PASS(7) TGA_PASS(5) TGA_PASS(3)
#undef TGA_PASS
#undef TGA_PASS2
      default: {
        const long long total = L * batch;
        pass_any_kernel<<<grid_for(total, num_sms), 256, 0, st>>>(x, y, tw, L, R, Ns, total);
        e = cudaGetLastError();
      }
    }
    kernel_launch_add(1);
    if (e != cudaSuccess) return e;
    Ns *= R;
    double2* t = x;
    x = y;
    y = t;
  }
  *result = x;
  return cudaSuccess;
}

// ---- Bluestein: X[k] = c[k] sum_m (x[m] c[m]) conj(c[k - m]), c[m] = W_{2L}^{m^2}
__global__ void chirp64_kernel(double2* __restrict__ c, long long L) {
  for (long long m = (long long)blockIdx.x * blockDim.x + threadIdx.x; m < L; m += (long long)gridDim.x * blockDim.x) {
    const unsigned long long r = ((unsigned long long)m * (unsigned long long)m) % (2ull * (unsigned long long)L);
    double s, co;
    sincospi((double)r / (double)L, &s, &co);
    c[m] = make_double2(co, -s);
  }
}
// h = conj(c) wrapped circularly into length M (index M - m for m > 0), zero elsewhere
__global__ void chirp_filter64_kernel(const double2* __restrict__ c, long long L, long long M, double2* __restrict__ h) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < M; i += (long long)gridDim.x * blockDim.x) {
    long long m = -1;
    if (i < L) m = i;
    else if (i > M - L) m = M - i;
    h[i] = m >= 0 ? make_double2(c[m].x, -c[m].y) : make_double2(0.0, 0.0);
  }
}
__global__ void premul64_kernel(const double2* __restrict__ x, const double2* __restrict__ c, long long L, long long M,
                                double2* __restrict__ y) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < M; i += (long long)gridDim.x * blockDim.x)
    y[i] = i < L ? mr_cmul(x[i], c[i]) : make_double2(0.0, 0.0);
}
// conj(a * b): the inverse transform of the product runs as a forward one
__global__ void conjmul64_kernel(double2* __restrict__ a, const double2* __restrict__ b, long long M) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < M; i += (long long)gridDim.x * blockDim.x) {
    const double2 v = mr_cmul(a[i], b[i]);
    a[i] = make_double2(v.x, -v.y);
  }
}
__global__ void postmul64_kernel(const double2* __restrict__ y, const double2* __restrict__ c, long long L, long long M,
                                 double2* __restrict__ out) {
  const double inv = 1.0 / (double)M;
  for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < L; k += (long long)gridDim.x * blockDim.x) {
    const double2 v = make_double2(y[k].x * inv, -y[k].y * inv);  // conj of the forward transform, / M
    out[k] = mr_cmul(v, c[k]);
  }
}

// The rows' samples as doubles (Bluestein's input): +-1 - mean
__global__ void samples64_kernel(FirstSource src, long long n, double* __restrict__ z) {
  const uint8_t* row = src.bits + (size_t)blockIdx.y * src.row_bytes;
  const double m = src.mean[blockIdx.y];
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const int bit = (__ldg(row + (i >> 3)) >> (7 - (int)(i & 7))) & 1;
    z[(size_t)blockIdx.y * n + i] = (bit ? 1.0 : -1.0) - m;
  }
}

// |X[k]|^2 for k < L of the real record whose n = 2 L point spectrum is
// recovered from Z = FFT_L(z), z[m] = x[2m] + i x[2m+1] (L even), and the
// histogram of their top digits (first pass of the median's radix select).
// A thread takes bins k and L - k, which need the same two values of Z and one
// twiddle W_n^k = exp(-i pi k / L): the table's W_L^{k / 2}, times w1 = W_n for
// an odd k, or sincospi where there is no table.  The histogram costs no pass
// of its own over the powers.
constexpr int kPowerIters = 16;
__global__ void __launch_bounds__(256) real_power_kernel(const double2* __restrict__ Z, const double2* __restrict__ tw,
                                                         double2 w1, unsigned L, double* __restrict__ p,
                                                         unsigned* __restrict__ hist) {
  __shared__ unsigned sh[kRfiDigits];
  for (int i = threadIdx.x; i < kRfiDigits; i += 256) sh[i] = 0;
  __syncthreads();
  const double2* z = Z + (size_t)blockIdx.y * L;
  double* row = p + (size_t)blockIdx.y * L;
  auto put = [&](unsigned k, double v) {
    row[k] = v;
    atomicAdd(&sh[(unsigned)((unsigned long long)__double_as_longlong(v) >> kRfiShift0)], 1u);
  };
  for (int it = 0; it < kPowerIters; ++it) {
    const unsigned k = (blockIdx.x * kPowerIters + it) * 256 + threadIdx.x;
    if (k > L / 2) break;
    const double2 zk = z[k], zc = z[k == 0 ? 0 : L - k];
    const double2 e = make_double2(0.5 * (zk.x + zc.x), 0.5 * (zk.y - zc.y));  // (Z[k] + conj Z[L-k]) / 2
    const double2 o = make_double2(0.5 * (zk.x - zc.x), 0.5 * (zk.y + zc.y));  // (Z[k] - conj Z[L-k]) / 2
    double2 w;  // exp(-i pi k / L)
    if (tw) {
      w = __ldg(tw + k / 2);
      if (k & 1u) w = mr_cmul(w, w1);
    } else {
      double s, c;
      sincospi((double)k / (double)L, &s, &c);
      w = make_double2(c, -s);
    }
    const double2 wo = mr_cmul(w, o);
    // X[k] = e - i w o; X[L - k] = conj(e) - i conj(w o)
    const double ar = e.x + wo.y, ai = e.y - wo.x;
    put(k, ar * ar + ai * ai);
    if (k != 0 && 2 * k != L) {
      const double br = e.x - wo.y, bi = -e.y - wo.x;
      put(L - k, br * br + bi * bi);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < kRfiDigits; i += 256)
    if (sh[i]) atomicAdd(hist + (size_t)blockIdx.y * 2 * kRfiDigits + i, sh[i]);
}

long long next_pow2(long long v) {
  long long m = 1;
  while (m < v) m <<= 1;
  return m;
}

}  // namespace

size_t fft64_workspace_bytes(long long n, int batch) {
  const long long L = n / 2;
  std::vector<int> r;
  if (mr_radices(L, kMaxRadix, &r)) return (size_t)L * 16;  // the twiddle table
  const long long M = next_pow2(2 * L - 1);
  return (size_t)(M + L + 3 * M) * 16;  // table of M, chirp, filter spectrum, two work buffers
}

cudaError_t real_power_spectrum(const uint8_t* d_bits, size_t row_bytes, const double* d_mean, double* d_x, void* d_buf,
                                void* d_work, int batch, double* d_p, unsigned* d_hist, int num_sms, cudaStream_t st,
                                std::string* why) {
  const long long n = (long long)row_bytes * 8, L = n / 2;
  if (n < 8 || L >= (1LL << 30) || batch > 65535) {
    *why = "the RFI spectrum needs records of 8 samples up to 2^31 and at most 65535 antennas";
    return cudaErrorInvalidValue;
  }
  double2* z = reinterpret_cast<double2*>(d_x);
  double2* buf = static_cast<double2*>(d_buf);
  double2* work = static_cast<double2*>(d_work);
  const FirstSource src = {d_bits, row_bytes, d_mean};
  cudaError_t e = cudaSuccess;
  std::vector<int> radices;
  double2* Z = nullptr;
  const double2* tw = nullptr;
  if (mr_radices(L, kMaxRadix, &radices)) {
    // L is a multiple of 4, so the first radix is a power of two, at least 4
    twiddle64_kernel<<<grid_for(L, num_sms), 256, 0, st>>>(work, L);
    kernel_launch_add(1);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    tw = work;
    if ((e = stockham(z, buf, &src, work, L, batch, radices, num_sms, st, &Z)) != cudaSuccess) return e;
  } else {
    // Bluestein per sequence: convolution length M = 2^m >= 2L - 1
    const long long M = next_pow2(2 * L - 1);
    mr_radices(M, kMaxRadix, &radices);
    double2* twM = work;
    double2* chirp = twM + M;
    double2* H = chirp + L;
    double2* u = H + M;
    double2* v = u + M;
    samples64_kernel<<<dim3(256, (unsigned)batch), 256, 0, st>>>(src, n, d_x);
    twiddle64_kernel<<<grid_for(M, num_sms), 256, 0, st>>>(twM, M);
    chirp64_kernel<<<grid_for(L, num_sms), 256, 0, st>>>(chirp, L);
    chirp_filter64_kernel<<<grid_for(M, num_sms), 256, 0, st>>>(chirp, L, M, u);
    kernel_launch_add(4);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    double2* h = nullptr;
    if ((e = stockham(u, v, nullptr, twM, M, 1, radices, num_sms, st, &h)) != cudaSuccess) return e;
    if (h != H) e = cudaMemcpyAsync(H, h, (size_t)M * 16, cudaMemcpyDeviceToDevice, st);
    if (e != cudaSuccess) return e;
    for (int a = 0; a < batch; ++a) {
      premul64_kernel<<<grid_for(M, num_sms), 256, 0, st>>>(z + a * L, chirp, L, M, u);
      kernel_launch_add(1);
      double2 *y = nullptr, *w = nullptr;
      if ((e = stockham(u, v, nullptr, twM, M, 1, radices, num_sms, st, &y)) != cudaSuccess) return e;
      conjmul64_kernel<<<grid_for(M, num_sms), 256, 0, st>>>(y, H, M);
      kernel_launch_add(1);
      if ((e = stockham(y, y == u ? v : u, nullptr, twM, M, 1, radices, num_sms, st, &w)) != cudaSuccess) return e;
      postmul64_kernel<<<grid_for(L, num_sms), 256, 0, st>>>(w, chirp, L, M, buf + a * L);
      kernel_launch_add(1);
      if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    Z = buf;
  }
  const double half_step = 3.14159265358979323846 / (double)L;
  const unsigned blocks = (unsigned)((L / 2 + 1 + 256 * kPowerIters - 1) / (256 * kPowerIters));
  real_power_kernel<<<dim3(blocks, (unsigned)batch), 256, 0, st>>>(
      Z, tw, make_double2(std::cos(half_step), -std::sin(half_step)), (unsigned)L, d_p, d_hist);
  kernel_launch_add(1);
  return cudaGetLastError();
}

}  // namespace tga
