// line_quotient.cuh -- a / b from the reciprocal of b, for the line solver
// (lsgs.cu), and the tests that tell where it is a / b bit for bit.  Plain C++
// outside nvcc, so that its arithmetic can be checked on the host as it is.
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define FPSI_HD __host__ __device__ __forceinline__
#else
#define FPSI_HD inline
#endif

namespace fpsi {
namespace dev {

FPSI_HD uint32_t float_bits(float a) {
#ifdef __CUDA_ARCH__
  return __float_as_uint(a);
#else
  uint32_t u;
  std::memcpy(&u, &a, sizeof(u));
  return u;
#endif
}
FPSI_HD uint64_t double_bits(double a) {
#ifdef __CUDA_ARCH__
  return uint64_t(__double_as_longlong(a));
#else
  uint64_t u;
  std::memcpy(&u, &a, sizeof(u));
  return u;
#endif
}
FPSI_HD float fma_rn(float a, float b, float c) { return fmaf(a, b, c); }
FPSI_HD double fma_rn(double a, double b, double c) { return fma(a, b, c); }

// a / b from y = RN(1 / b): the reciprocal's own error is added back
// (y + yl = 1 / b to twice the precision), so q is within one ulp of a / b,
// and one correction by its exact remainder rounds it correctly (Markstein's
// theorem: Computation of elementary functions on the IBM RISC System/6000
// processor, IBM J. Res. Dev. 34, 1990).  Four dependent FMAs instead of a
// division's sequence; the result is that of a / b bit for bit while b and a
// are in the ranges of pivot_ok and tiny() (a zero keeps its value, not its
// sign).
template <class T>
FPSI_HD T quotient(T a, T b, T y) {
  const T yl = fma_rn(-b, y, T(1)) * y;
  const T q = fma_rn(a, y, a * yl);
  return fma_rn(fma_rn(-b, q, a), y, q);
}
// |b| in 2^-100 .. 2^28 (FP32), 2^-300 .. 2^300 (FP64)
FPSI_HD bool pivot_ok(float b) { return fabsf(b) >= 0x1p-100f && fabsf(b) <= 0x1p28f; }
FPSI_HD bool pivot_ok(double b) { return fabs(b) >= 0x1p-300 && fabs(b) <= 0x1p300; }
// the smallest nonzero |a| so far, as a key (twice its bits, less one; zero
// gives the largest key), and whether one below 2^-90 (2^-600) was among
// them: there the remainder or the reciprocal's second part may underflow.
// Above, an overflow ends in a NaN.
FPSI_HD uint32_t key_min(uint32_t k, float a) {
  const uint32_t n = 2u * float_bits(a) - 1u;
  return k < n ? k : n;
}
// the high word of twice its high word and its low word, less one: the low
// word's borrow tells zero from the values below 2^-1042 (two integer adds)
FPSI_HD uint32_t key_min(uint32_t k, double a) {
  const uint64_t u = double_bits(a), hi = u >> 32;
  const uint32_t n = uint32_t((((hi + hi) << 32 | (u & 0xffffffffu)) - 1u) >> 32);
  return k < n ? k : n;
}
template <class T>
FPSI_HD bool tiny(uint32_t k) {
  return k < (sizeof(T) == 4 ? 2u * ((127u - 90u) << 23) : 2u * ((1023u - 600u) << 20)) - 1u;
}

}  // namespace dev
}  // namespace fpsi
