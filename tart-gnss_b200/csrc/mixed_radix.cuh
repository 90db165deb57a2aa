// Register-resident forward DFTs of the mixed-radix FFTs (fft64.cu in double,
// generic_kernels.cu in single precision) and the choice of their radices.
#pragma once
#include <cuda_runtime.h>

#include <vector>

#include "mixed_radix_consts.cuh"

namespace tga {

template <class T> struct MrVec;
template <> struct MrVec<float> { using type = float2; };
template <> struct MrVec<double> { using type = double2; };

template <class V>
__device__ __forceinline__ V mr_cmul(V a, V b) {
  V r;
  r.x = a.x * b.x - a.y * b.y;
  r.y = a.x * b.y + a.y * b.x;
  return r;
}
template <class V, class T>
__device__ __forceinline__ V mr_make(T x, T y) {
  V r;
  r.x = x;
  r.y = y;
  return r;
}

template <class T, int R> struct MrConst;
#define TGA_MR_CONST(R)                                                             \
  template <> struct MrConst<double, R> {                                           \
    __device__ static __forceinline__ double c(int m) { return kCosD##R[m]; }       \
    __device__ static __forceinline__ double s(int m) { return kSinD##R[m]; }       \
  };                                                                                \
  template <> struct MrConst<float, R> {                                            \
    __device__ static __forceinline__ float c(int m) { return kCosF##R[m]; }        \
    __device__ static __forceinline__ float s(int m) { return kSinF##R[m]; }        \
  };
TGA_MR_CONST(3)
TGA_MR_CONST(5)
TGA_MR_CONST(7)
TGA_MR_CONST(11)
TGA_MR_CONST(13)
TGA_MR_CONST(25)
TGA_MR_CONST(31)
TGA_MR_CONST(32)
#undef TGA_MR_CONST

// Forward DFTs of register arrays, outputs streamed to st(k, value).
// Odd prime R: pairs s_n = x_n + x_{R-n}, d_n = x_n - x_{R-n} halve the terms.
template <int R, class V, class St>
__device__ __forceinline__ void mr_dft_prime(const V (&x)[R], St&& st) {
  using T = decltype(V::x);
  constexpr int H = (R - 1) / 2;
  V s[H], d[H];
#pragma unroll
  for (int n = 1; n <= H; ++n) {
    s[n - 1] = mr_make<V>(x[n].x + x[R - n].x, x[n].y + x[R - n].y);
    d[n - 1] = mr_make<V>(x[n].x - x[R - n].x, x[n].y - x[R - n].y);
  }
  V X0 = x[0];
#pragma unroll
  for (int n = 0; n < H; ++n) X0 = mr_make<V>(X0.x + s[n].x, X0.y + s[n].y);
  const V x0 = x[0];
  st(0, X0);
#pragma unroll
  for (int k = 1; k <= H; ++k) {
    V A = x0, B = mr_make<V>(T(0), T(0));
#pragma unroll
    for (int n = 1; n <= H; ++n) {
      const T c = MrConst<T, R>::c((n * k) % R), sn = MrConst<T, R>::s((n * k) % R);
      A.x = fma(s[n - 1].x, c, A.x);
      A.y = fma(s[n - 1].y, c, A.y);
      B.x = fma(d[n - 1].x, sn, B.x);
      B.y = fma(d[n - 1].y, sn, B.y);
    }
    st(k, mr_make<V>(A.x + B.y, A.y - B.x));      // A - i B
    st(R - k, mr_make<V>(A.x - B.y, A.y + B.x));  // A + i B
  }
}

// N a power of two up to 32: decimation in time over x[off + i stride]
template <int N, int STRIDE, int M, class V>
__device__ __forceinline__ void mr_dft_pow2(const V (&x)[M], int off, V (&y)[N]) {
  using T = decltype(V::x);
  if constexpr (N == 1) {
    y[0] = x[off];
  } else {
    V e[N / 2], o[N / 2];
    mr_dft_pow2<N / 2, 2 * STRIDE>(x, off, e);
    mr_dft_pow2<N / 2, 2 * STRIDE>(x, off + STRIDE, o);
#pragma unroll
    for (int k = 0; k < N / 2; ++k) {
      V t = o[k];
      if (4 * k == N)
        t = mr_make<V>(o[k].y, -o[k].x);  // times -i
      else if (k > 0)
        t = mr_cmul(o[k], mr_make<V>(MrConst<T, 32>::c(k * (32 / N)), -MrConst<T, 32>::s(k * (32 / N))));
      y[k] = mr_make<V>(e[k].x + t.x, e[k].y + t.y);
      y[k + N / 2] = mr_make<V>(e[k].x - t.x, e[k].y - t.y);
    }
  }
}

template <int R, class V, class St>
__device__ __forceinline__ void mr_dft(const V (&x)[R], St&& st) {
  using T = decltype(V::x);
  if constexpr ((R & (R - 1)) == 0) {
    V y[R];
    mr_dft_pow2<R, 1>(x, 0, y);
#pragma unroll
    for (int k = 0; k < R; ++k) st(k, y[k]);
  } else if constexpr (R == 33 || R == 15) {
    // 3 x P, coprime: n = (P n1 + 3 n2) mod R, k = (P (P^-1 mod 3) k1 + 3 (3^-1 mod P) k2) mod R
    constexpr int P = R / 3, E1 = P * (P % 3 == 1 ? 1 : 2), E2 = 3 * (P == 11 ? 4 : 2);
    V u[3][P];
#pragma unroll
    for (int n2 = 0; n2 < P; ++n2) {
      const V t[3] = {x[(3 * n2) % R], x[(P + 3 * n2) % R], x[(2 * P + 3 * n2) % R]};
      mr_dft_prime<3>(t, [&](int k1, V v) { u[k1][n2] = v; });
    }
#pragma unroll
    for (int k1 = 0; k1 < 3; ++k1) mr_dft_prime<P>(u[k1], [&](int k2, V v) { st((E1 * k1 + E2 * k2) % R, v); });
  } else if constexpr (R == 25) {
    // n = 5 n1 + n2, k = k1 + 5 k2, twiddles W_25^{n2 k1}
    V u[5][5];  // [k1][n2]
#pragma unroll
    for (int n2 = 0; n2 < 5; ++n2) {
      const V t[5] = {x[n2], x[5 + n2], x[10 + n2], x[15 + n2], x[20 + n2]};
      mr_dft_prime<5>(t, [&](int k1, V v) {
        u[k1][n2] = k1 * n2 == 0
                        ? v
                        : mr_cmul(v, mr_make<V>(MrConst<T, 25>::c(k1 * n2), -MrConst<T, 25>::s(k1 * n2)));
      });
    }
#pragma unroll
    for (int k1 = 0; k1 < 5; ++k1) mr_dft_prime<5>(u[k1], [&](int k2, V v) { st(k1 + 5 * k2, v); });
  } else {
    mr_dft_prime<R>(x, st);
  }
}

// Radices of L in pass order: the power of two in as few parts of at most 32 as
// there can be, then the odd primes, 5 with 5 and 3 with 11 or 5 together; false
// when a prime factor exceeds max_prime.
inline bool mr_radices(long long L, int max_prime, std::vector<int>* radices) {
  radices->clear();
  long long m = L;
  int twos = 0;
  while (m % 2 == 0) {
    m /= 2;
    ++twos;
  }
  for (int parts = (twos + 4) / 5; parts > 0; --parts) {
    const int t = (twos + parts - 1) / parts;
    radices->push_back(1 << t);
    twos -= t;
  }
  std::vector<int> odd;
  for (long long p = 3; p * p <= m || m > 1; p += 2) {
    if (p * p > m) p = m;  // m is prime
    while (m % p == 0) {
      if (p > max_prime) return false;
      odd.push_back((int)p);
      m /= p;
    }
    if (m == 1) break;
  }
  auto pair = [&](int p, int q) {
    for (;;) {
      size_t i = odd.size(), k = odd.size();
      for (size_t t = 0; t < odd.size(); ++t) {
        if (odd[t] == p && i == odd.size())
          i = t;
        else if (odd[t] == q)
          k = t;
      }
      if (i == odd.size() || k == odd.size()) return;
      odd.erase(odd.begin() + (long)(i > k ? i : k));
      odd.erase(odd.begin() + (long)(i > k ? k : i));
      radices->push_back(p * q);
    }
  };
  pair(5, 5);
  pair(3, 11);
  pair(3, 5);
  for (int p : odd) radices->push_back(p);
  return true;
}

}  // namespace tga
