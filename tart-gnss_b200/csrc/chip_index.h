// Place of a chip number in a periodic sequence.  Plain C++, so that it can be
// checked on the host over every double.
#pragma once
#include <cmath>
#include <cstdint>

#ifdef __CUDACC__
#define TGA_CI_HD __host__ __device__ __forceinline__
#else
#define TGA_CI_HD inline
#endif

namespace tga {

// k mod L of a whole number k held as a double, in [0, L) for every double: a
// code phase may be any finite number, and k indexes memory.  Below 2^52 the
// quotient's rounding moves the remainder by at most one L, and the product is
// exact; from there on (and for infinities and NaN) the 64-bit remainder of k,
// saturated.
TGA_CI_HD int chip_index(double k, int L) {
  if (fabs(k) < 4503599627370496.0) {
    const int r = (int)(k - floor(k / (double)L) * (double)L);
    return r < 0 ? r + L : r >= L ? r - L : r;
  }
  const long long n = k >= 9.2233720368547758e18    ? INT64_MAX
                      : k > -9.2233720368547758e18 ? (long long)k
                                                   : INT64_MIN;
  const int r = (int)(n % L);
  return r < 0 ? r + L : r;
}

}  // namespace tga

#undef TGA_CI_HD
