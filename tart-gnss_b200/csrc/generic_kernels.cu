// Generic acquisition path: the reference algorithm (correlate.rs:91-183) for
// any signal length N, on the GPU.
//
// Used when the fused polyphase kernels do not apply: windows that are not
// exactly two code periods, or codes that are not a whole number of samples
// per chip (e.g. 16 MHz sampling).  Per Doppler bin: carrier wipe-off,
// forward FFT of length N, for both hypotheses ([c,c] and [c,-c]) the product
// with the conjugated code spectrum, inverse FFT, |.|/sqrt(N), last-max
// argmax; then the hypothesis / bin reduction and the second peak.
//
// A length whose prime factors are at most kGenPrime (the usual ones: 32000 =
// 2^8 5^3 at 16 MHz) is transformed as it is, by mixed-radix Stockham passes
// with one butterfly per thread (mixed_radix.cuh).  Any other length uses
// Bluestein's chirp-z identity
//   X[k] = w[k] * sum_n (x[n] w[n]) conj(w[k-n]),  w[n] = exp(-i pi n^2 / N)
// evaluated as a circular convolution of length M = 2^m >= 2N-1 with the same
// passes.  Inverse transforms run as forward ones of conjugated data (only
// the magnitude of their results is used).  What bounds a call is the number
// of launches and, at tens of MB, L2: one GPS search at 16 MHz took 1.29 ms of
// device time in 150 kernels (every transform by Bluestein over radix-2 passes),
// and takes 0.105 ms in 13 (the whole call 167 us, with the copy of the signal
// and two read-backs).  RMS error of the peaks against 64 bits 1.8e-7 -> 7e-8.
#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "dft.cuh"
#include "engine.h"
#include "mixed_radix.cuh"

namespace tga {

#define TGA_GLAUNCHED() (kernel_launch_add(1), cudaGetLastError())

namespace {

constexpr int kGenPrime = 64;  // largest prime factor of a direct transform

// Workspace: two buffers of the transforms' batch (length F = N, or the
// Bluestein length M), twiddles W_F^m, and for Bluestein the chirp and its
// filter's spectrum.
struct Ws {
  float2 *tw, *a, *b, *w, *H;
};

bool direct_length(int N) {
  std::vector<int> r;
  return mr_radices(N, kGenPrime, &r);
}

Ws carve(float2* base, const GenericPlan& gp, int nb) {
  const size_t N = gp.N, F = direct_length(gp.N) ? N : (size_t)gp.Mpow2, batch = 2 * (size_t)nb + 2;
  Ws v;
  float2* p = base;
  v.tw = p; p += F;
  v.a = p; p += batch * F;
  v.b = p; p += batch * F;
  v.w = p; p += N;
  v.H = p;
  return v;
}

// tw[m] = exp(-2 pi i m / F)
__global__ void twiddle_kernel(int F, float2* __restrict__ tw) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= F) return;
  double s, c;
  sincospi(2.0 * (double)i / (double)F, &s, &c);
  tw[i] = make_float2((float)c, (float)-s);
}

__global__ void chirp_kernel(int N, float2* __restrict__ w) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  // exp(-i pi n^2 / N) with n^2 reduced mod 2N exactly in integers
  const long long r = ((long long)i * i) % (2LL * N);
  double s, c;
  sincospi((double)r / (double)N, &s, &c);
  w[i] = make_float2((float)c, (float)-s);
}

// h[m] = conj(w[m]) wrapped onto the length-M circle
__global__ void chirp_filter_kernel(int N, int M, const float2* __restrict__ w, float2* __restrict__ h) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= M) return;
  int n = -1;
  if (m < N) n = m;
  else if (m > M - N) n = M - m;
  h[m] = n >= 0 ? make_float2(w[n].x, -w[n].y) : make_float2(0.f, 0.f);
}

// One Stockham pass of radix R (see fft64.cu), one butterfly per thread;
// blockIdx.y is the sequence.  A pass with Ns = 1 of a power-of-two radix puts
// its block's R contiguous outputs per thread in order through shared memory.
constexpr int kGenThreads = 128;

template <int R, bool STAGE>
__global__ void __launch_bounds__(kGenThreads) pass32_kernel(const float2* __restrict__ in, float2* __restrict__ out,
                                                             const float2* __restrict__ tw, unsigned L, unsigned Ns) {
  extern __shared__ __align__(16) float2 s_out[];
  const unsigned LR = L / R, j = blockIdx.x * kGenThreads + threadIdx.x;
  const size_t seq = (size_t)blockIdx.y * L;
  if (j < LR) {
    float2 v[R];
    const float2* x = in + seq + j;
#pragma unroll
    for (int s = 0; s < R; ++s) v[s] = x[(size_t)s * LR];
    if constexpr (STAGE) {
      float2* o = s_out + threadIdx.x * (R + 1);
      mr_dft<R>(v, [&](int r, float2 y) { o[r] = y; });
    } else {
      const unsigned q = j / Ns, k = j - q * Ns, b = k * (L / (Ns * R));  // twiddle of s: W_L^{s b}
#pragma unroll
      for (int s = 1; s < R; ++s) v[s] = mr_cmul(v[s], __ldg(tw + (size_t)s * b));
      float2* y = out + seq + (size_t)q * Ns * R + k;
      mr_dft<R>(v, [&](int r, float2 t) { y[(size_t)r * Ns] = t; });
    }
  }
  if constexpr (STAGE) {
    __syncthreads();
    const unsigned j0 = blockIdx.x * kGenThreads;
    if (j0 < LR) {
      const unsigned n = min((unsigned)kGenThreads, LR - j0) * R;
      float2* y = out + seq + (size_t)j0 * R;
      for (unsigned i = threadIdx.x; i < n; i += kGenThreads) y[i] = s_out[i + i / R];
    }
  }
}

// One pass of any radix R, one output per thread (an R-term sum).
__global__ void __launch_bounds__(256) pass32_any_kernel(const float2* __restrict__ in, float2* __restrict__ out,
                                                         const float2* __restrict__ tw, unsigned L, int R,
                                                         unsigned Ns) {
  const unsigned o = blockIdx.x * 256 + threadIdx.x;
  if (o >= L) return;
  const unsigned LR = L / R, NsR = Ns * R, q = o / NsR, rem = o - q * NsR, r = rem / Ns, k = rem - r * Ns;
  const float2* x = in + (size_t)blockIdx.y * L + q * Ns + k;
  const unsigned base = (k + r * Ns) * (L / NsR);  // < L
  float2 acc = make_float2(0.f, 0.f);
  unsigned m = 0;
  for (int s = 0; s < R; ++s) {
    const float2 u = x[(size_t)s * LR], w = __ldg(tw + m);
    acc.x += u.x * w.x - u.y * w.y;
    acc.y += u.x * w.y + u.y * w.x;
    m += base;
    if (m >= L) m -= L;
  }
  out[(size_t)blockIdx.y * L + o] = acc;
}

template <int R, bool STAGE>
cudaError_t run_pass32(const float2* x, float2* y, const float2* tw, int L, int batch, int Ns, cudaStream_t st) {
  const dim3 grid((unsigned)((L / R + kGenThreads - 1) / kGenThreads), (unsigned)batch);
  const size_t smem = STAGE ? (size_t)kGenThreads * (R + 1) * sizeof(float2) : 0;
  pass32_kernel<R, STAGE><<<grid, kGenThreads, smem, st>>>(x, y, tw, (unsigned)L, (unsigned)Ns);
  return cudaGetLastError();
}

// forward transforms of `batch` sequences of length L in x (ping-pong with y);
// *result is the buffer holding them
cudaError_t fft32(float2* x, float2* y, const float2* tw, int L, int batch, const std::vector<int>& radices,
                  cudaStream_t st, float2** result) {
  int Ns = 1;
  for (int R : radices) {
    cudaError_t e;
    switch (R) {
#define TGA_PASS(RR)                                               \
  case RR:                                                         \
    e = run_pass32<RR, false>(x, y, tw, L, batch, Ns, st);         \
    break;
#define TGA_PASS2(RR)                                              \
  case RR:                                                         \
    e = Ns == 1 ? run_pass32<RR, true>(x, y, tw, L, batch, Ns, st) \
                : run_pass32<RR, false>(x, y, tw, L, batch, Ns, st); \
    break;
      TGA_PASS2(32) TGA_PASS2(16) TGA_PASS2(8) TGA_PASS2(4) TGA_PASS2(2)
      TGA_PASS(33) TGA_PASS(25) TGA_PASS(15) TGA_PASS(31) TGA_PASS(13) TGA_PASS(11) TGA_PASS(7) TGA_PASS(5) TGA_PASS(3)
#undef TGA_PASS
#undef TGA_PASS2
      default:
        pass32_any_kernel<<<dim3((unsigned)((L + 255) / 256), (unsigned)batch), 256, 0, st>>>(x, y, tw, (unsigned)L, R,
                                                                                             (unsigned)Ns);
        e = cudaGetLastError();
    }
    kernel_launch_add(1);
    if (e != cudaSuccess) return e;
    Ns *= R;
    float2* t = x;
    x = y;
    y = t;
  }
  *result = x;
  return cudaSuccess;
}

// (x w, padded to M) for Bluestein
__global__ void premul_kernel(const float2* __restrict__ in, int N, int M, const float2* __restrict__ w,
                              float2* __restrict__ out) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= M) return;
  const size_t s = blockIdx.y;
  out[s * M + m] = m < N ? cmul(in[s * N + m], w[m]) : make_float2(0.f, 0.f);
}

// conj(a h): the inverse transform of the product runs as a forward one
__global__ void pointwise_kernel(float2* __restrict__ a, const float2* __restrict__ h, int M) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= M) return;
  float2* p = a + (size_t)blockIdx.y * M + m;
  const float2 v = cmul(*p, h[m]);
  *p = make_float2(v.x, -v.y);
}

__global__ void postmul_kernel(const float2* __restrict__ c, int N, int M, const float2* __restrict__ w,
                               float2* __restrict__ out) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= N) return;
  const size_t s = blockIdx.y;
  const float2 u = c[s * M + k];
  const float2 v = cmul(make_float2(u.x, -u.y), w[k]);
  const float inv = 1.0f / (float)M;  // M is a power of two: exact
  out[s * N + k] = make_float2(v.x * inv, v.y * inv);
}

unsigned nblk(long long n, int t) { return (unsigned)((n + t - 1) / t); }

// Forward DFTs of nseq sequences of length N held in v.a (direct: of length N
// each, transformed in place of it; Bluestein: read from `in`); *result is
// where they are, N apart.
struct Transform {
  bool direct;
  std::vector<int> radices;  // of N, or of M
};
cudaError_t transform(const GenericPlan& gp, const Transform& t, const Ws& v, float2* in, float2* spare, int nseq,
                      cudaStream_t st, float2** result) {
  const int N = gp.N, M = gp.Mpow2;
  if (t.direct) return fft32(in, spare, v.tw, N, nseq, t.radices, st, result);
  // `in` and `spare` have room for nseq sequences of M
  cudaError_t e;
  const dim3 gm(nblk(M, 256), (unsigned)nseq), gn(nblk(N, 256), (unsigned)nseq);
  premul_kernel<<<gm, 256, 0, st>>>(in, N, M, v.w, spare);
  float2* r = nullptr;
  if ((e = fft32(spare, in, v.tw, M, nseq, t.radices, st, &r)) != cudaSuccess) return e;
  pointwise_kernel<<<gm, 256, 0, st>>>(r, v.H, M);
  float2* q = nullptr;
  if ((e = fft32(r, r == in ? spare : in, v.tw, M, nseq, t.radices, st, &q)) != cudaSuccess) return e;
  *result = q == in ? spare : in;
  postmul_kernel<<<gn, 256, 0, st>>>(q, N, M, v.w, *result);
  kernel_launch_add(3);
  return cudaGetLastError();
}

// Inputs of the forward transforms: sequences 0 and 1 the codes [c,c] and
// [c,-c] (sample n the (sub)chip floor(n / spc), the sign changing at `split`;
// correlate.rs:47-58, acquisition.rs:146-159 in f64 as there), 2 + b the signal
// wiped off for bin b (correlate.rs:110-115, f32 phase)
__global__ void inputs_kernel(GenericCode code, const float* __restrict__ sig, const double* __restrict__ pp,
                              const double* __restrict__ fc, int N, float2* __restrict__ X) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x, q = blockIdx.y;
  if (n >= N) return;
  float2 v;
  if (q < 2) {
    const long long i = (long long)floor((double)n / code.spc) % code.len;
    int c = __ldg(code.chips + (code.boc ? i >> 1 : i));
    if (code.boc && (i & 1)) c = -c;
    v = make_float2(q == 1 && n >= code.split ? (float)-c : (float)c, 0.f);
  } else {
    const float ph = __double2float_rn(pp[n] * fc[q - 2]);
    float sn, cs;
    sincos_phase(ph, &sn, &cs);
    const float s = sig[n];
    v = make_float2(cs * s, sn * s);
  }
  X[(size_t)q * N + n] = v;
}

// conj(X_b conj(C_h)) for every bin b and hypothesis h (q = 2 b + h): the
// magnitudes of its forward transform are those of the inverse transform of
// the product
__global__ void hyp_product_kernel(const float2* __restrict__ X, int N, float2* __restrict__ Y) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x, q = blockIdx.y;
  if (n >= N) return;
  const float2 c = X[(size_t)(q & 1) * N + n], x = X[(size_t)(2 + (q >> 1)) * N + n];
  const float2 v = cmul(x, make_float2(c.x, -c.y));
  Y[(size_t)q * N + n] = make_float2(v.x, -v.y);
}

// |.| * 1/sqrt(N) and last-max argmax per (bin, hypothesis) row (keys zeroed).
__global__ void __launch_bounds__(256) norm_argmax_kernel(const float2* __restrict__ Y, int N,
                                                          float* __restrict__ corr,
                                                          unsigned long long* __restrict__ keys) {
  const size_t q = blockIdx.y;
  const float scale = 1.0f / sqrtf((float)N);
  unsigned long long best = 0ull;
#pragma unroll 4
  for (int n = blockIdx.x * 256 + threadIdx.x; n < N; n += gridDim.x * 256) {
    const float2 v = Y[q * N + n];
    const float c = hypotf(v.x, v.y) * scale;  // Complex::norm() * scale
    corr[q * N + n] = c;
    const unsigned long long k = ((unsigned long long)__float_as_uint(c) << 32) | (unsigned)n;
    best = k > best ? k : best;
  }
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long t = __shfl_xor_sync(0xffffffffu, best, o);
    best = t > best ? t : best;
  }
  __shared__ unsigned long long part[8];
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = best;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) best = part[w] > best ? part[w] : best;
    if (best) atomicMax(keys + q, best);
  }
}

// second peak over the winning row (correlate.rs:156-175), found by every block
// for itself; res_f[1] (0 before, and after where there is none) collects the blocks' maxima.  The distances
// of 32000 samples kept one block's SM busy for 21.8 us; 32 blocks 6.1.
__global__ void select_second_kernel(const float* __restrict__ corr, const unsigned long long* __restrict__ keys, int N,
                                     int nb, int period, int chip_width, int* __restrict__ res_i,
                                     float* __restrict__ res_f) {
  __shared__ int s_q, s_idx;
  __shared__ float s_peak;
  if (threadIdx.x < 32) {
    // a bin's row is [c,-c]'s only when strictly stronger; the last bin of the
    // largest value wins.  A NaN is never above another value, and nothing is
    // above a NaN in bin 0.
    unsigned long long best = 0ull;  // (value bits, bin)
    for (int b = threadIdx.x; b < nb; b += 32) {
      const float pa = __uint_as_float((unsigned)(keys[2 * b] >> 32));
      const float pB = __uint_as_float((unsigned)(keys[2 * b + 1] >> 32));
      const float pr = pB > pa ? pB : pa;
      const unsigned v = pr >= 0.f ? __float_as_uint(pr) : b == 0 ? 0xffffffffu : 0u;
      const unsigned long long k = ((unsigned long long)v << 32) | (unsigned)b;
      if (pr >= 0.f || v != 0u) best = k > best ? k : best;
    }
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long t = __shfl_xor_sync(0xffffffffu, best, o);
      best = t > best ? t : best;
    }
    if (threadIdx.x == 0) {
      const int b = (int)(unsigned)best;
      const unsigned long long ka = keys[2 * b], kb = keys[2 * b + 1];
      const bool useB = __uint_as_float((unsigned)(kb >> 32)) > __uint_as_float((unsigned)(ka >> 32));
      s_q = 2 * b + (useB ? 1 : 0);
      s_idx = (int)(unsigned)((useB ? kb : ka) & 0xffffffffu);
      s_peak = __uint_as_float((unsigned)((useB ? kb : ka) >> 32));
    }
  }
  __syncthreads();
  const int main_cp = s_idx % period;
  float m = -1.f;  // below every |.|
  const float* row = corr + (long long)s_q * N;
#pragma unroll 4
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) {
    const float v = __ldg(row + i);  // read whether it counts or not: the loads do not wait for the distances
    const int cp = i % period;
    const int dist = cp >= main_cp ? min(cp - main_cp, period - cp + main_cp) : min(main_cp - cp, period - main_cp + cp);
    m = dist > chip_width ? fmaxf(m, v) : m;
  }
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  __shared__ float part[32];
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) m = fmaxf(m, part[w]);
    atomicMax(reinterpret_cast<int*>(res_f + 1), __float_as_int(m));  // (-1 stays below 0)
    if (blockIdx.x != 0) return;
    res_i[0] = s_q >> 1;
    res_i[1] = s_idx;
    res_i[2] = s_q & 1;
    res_f[0] = s_peak;
  }
}

// acquisition.rs:281-294 on the GPU: +-1 samples minus the row mean, first n
// as f32, and phase points TAU/fs * i in f64.
__global__ void bits_to_signal_kernel(const uint8_t* __restrict__ bits, size_t row_bytes, int row,
                                      const double* __restrict__ mean, int n, double pc, float* __restrict__ sig,
                                      double* __restrict__ pp) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint8_t byte = bits[(size_t)row * row_bytes + (i >> 3)];
  const double v = ((byte >> (7 - (i & 7))) & 1) ? 1.0 : -1.0;
  sig[i] = (float)(v - mean[row]);
  pp[i] = pc * (double)i;
}

}  // namespace

cudaError_t launch_bits_to_signal(const uint8_t* d_bits, size_t row_bytes, int row, const double* d_mean, int n,
                                  double pc, float* d_sig, double* d_pp, cudaStream_t st) {
  bits_to_signal_kernel<<<nblk(n, 256), 256, 0, st>>>(d_bits, row_bytes, row, d_mean, n, pc, d_sig, d_pp);
  return TGA_GLAUNCHED();
}

size_t generic_work_elems(const GenericPlan& gp, int nb) {
  const size_t N = gp.N, F = direct_length(gp.N) ? N : (size_t)gp.Mpow2, batch = 2 * (size_t)nb + 2;
  // twiddles, two buffers, chirp, filter, and the rows' keys at the end
  return F + 2 * batch * F + N + F + 2 * (size_t)nb;
}

cudaError_t launch_generic(const GenericPlan& gp, const float* d_sig, const double* d_pp, const double* d_fc, int nb,
                           const GenericCode& code, int period, double fs, float2* d_work, size_t work_elems,
                           float* d_corr, int* d_res_i, float* d_res_f, cudaStream_t st) {
  if (work_elems < generic_work_elems(gp, nb)) return cudaErrorInvalidValue;
  const int N = gp.N, M = gp.Mpow2;
  const Ws v = carve(d_work, gp, nb);
  unsigned long long* keys = reinterpret_cast<unsigned long long*>(d_work + generic_work_elems(gp, nb) - 2 * (size_t)nb);
  cudaError_t e;
  Transform t;
  t.direct = mr_radices(N, kGenPrime, &t.radices);
  const int F = t.direct ? N : M;
  twiddle_kernel<<<nblk(F, 256), 256, 0, st>>>(F, v.tw);
  kernel_launch_add(1);
  if (!t.direct) {
    mr_radices(M, kGenPrime, &t.radices);
    chirp_kernel<<<nblk(N, 256), 256, 0, st>>>(N, v.w);
    chirp_filter_kernel<<<nblk(M, 256), 256, 0, st>>>(N, M, v.w, v.a);
    kernel_launch_add(2);
    float2* h = nullptr;
    if ((e = fft32(v.a, v.b, v.tw, M, 1, t.radices, st, &h)) != cudaSuccess) return e;
    if ((e = cudaMemcpyAsync(v.H, h, (size_t)M * sizeof(float2), cudaMemcpyDeviceToDevice, st)) != cudaSuccess) return e;
  }
  if ((e = cudaMemsetAsync(keys, 0, 2 * (size_t)nb * sizeof(unsigned long long), st)) != cudaSuccess) return e;
  if ((e = cudaMemsetAsync(d_res_f, 0, 2 * sizeof(float), st)) != cudaSuccess) return e;
  // code spectra (correlate.rs:47-68), and the wipe-off and forward transform of every bin
  const dim3 g1(nblk(N, 256), (unsigned)(nb + 2)), g2(nblk(N, 256), (unsigned)(2 * nb));
  inputs_kernel<<<g1, 256, 0, st>>>(code, d_sig, d_pp, d_fc, N, v.a);
  float2 *X = nullptr, *Y = nullptr;
  if ((e = transform(gp, t, v, v.a, v.b, nb + 2, st, &X)) != cudaSuccess) return e;
  if (X != v.a) {  // the products go where the spectra are not
    hyp_product_kernel<<<g2, 256, 0, st>>>(X, N, v.a);
    e = transform(gp, t, v, v.a, v.b, 2 * nb, st, &Y);
  } else {
    hyp_product_kernel<<<g2, 256, 0, st>>>(X, N, v.b);
    e = transform(gp, t, v, v.b, v.a, 2 * nb, st, &Y);
  }
  if (e != cudaSuccess) return e;
  norm_argmax_kernel<<<dim3(nblk(N, 256 * 4), (unsigned)(2 * nb)), 256, 0, st>>>(Y, N, d_corr, keys);
  select_second_kernel<<<32, 256, 0, st>>>(d_corr, keys, N, nb, period, (int)ceil(fs / 1.023e6), d_res_i, d_res_f);
  kernel_launch_add(4);
  return cudaGetLastError();
}

}  // namespace tga
