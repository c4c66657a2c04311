// pme_direct_math.h -- arithmetic of the pair kernel: exact sums of its force terms, each rounded once to
// 2^-40 (plain C++ beside CUDA, so that they can be checked without a GPU), and its reciprocal.
#pragma once

#include <cstring>

#ifdef __CUDACC__
#define PME_SUM_FN __host__ __device__ __forceinline__
#else
#define PME_SUM_FN inline
#endif

namespace pme {
namespace direct {

constexpr double kRoundMagic = 6755399441055744.0;   // 1.5 * 2^52: the low bits of v + kRoundMagic hold rint(v)

PME_SUM_FN unsigned long long bits_of(double v) {
#ifdef __CUDA_ARCH__
  return (unsigned long long)__double_as_longlong(v);
#else
  unsigned long long u;
  std::memcpy(&u, &v, sizeof(u));
  return u;
#endif
}

// Sum of integers rint(v), |v| < 2^51, given as v + kRoundMagic: every term adds the bits of kRoundMagic
// too, which are taken off once at the end.  All of it modulo 2^64, where the wrap is defined; the result
// is the sum's two's complement.
struct RoundedSum {
  unsigned long long bits = 0ull;
  PME_SUM_FN void add_rounded(double v_plus_magic) { bits += bits_of(v_plus_magic); }
  PME_SUM_FN void add(long long v) { bits += (unsigned long long)v; }
  PME_SUM_FN unsigned long long total(int rounded_terms) const {
    return bits - (unsigned long long)rounded_terms * bits_of(kRoundMagic);
  }
};

#ifdef __CUDACC__
// The hardware's approximation of 1 / x, |1 - x y| < 2^-19 (its 20 leading mantissa bits; measured in
// tests/test_gpu_direct_math.py).
__device__ __forceinline__ double reciprocal_guess(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}

// 1 / x by one third-order Newton (Halley-type) step y (1 + e + e^2), e = 1 - x y, from the guess: e^3 <
// 2^-57 is left, so the result is within an ulp of 1 / x.
__device__ __forceinline__ double reciprocal(double x) {
  const double y = reciprocal_guess(x), e = __fma_rn(-x, y, 1.0);
  return __fma_rn(y, __fma_rn(e, e, e), y);
}
#endif

}  // namespace direct
}  // namespace pme
