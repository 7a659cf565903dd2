// 1 / (1 + e^-x) for the prompt GEMM's epilogue: one ex2 and one reciprocal.  Plain arithmetic beside these two, which the caller passes in: a test
// builds it with the host compiler and exact ones.
//
// e^-x = 2^(hi + lo), hi the product -x log2(e) rounded to fp32 and lo what that leaves: its rounding, and the part of log2(e) below its own fp32 value
// (without which the error grows by 1.3e-8 |x|, ten ulps at -88).  With exact ex2 and rcp the result is within 2^-22.5 of the sigmoid; ex2.approx and
// rcp.approx add their own few ulps.  From e^-x = 2^128 on the result is 0, as with expf; a NaN argument gives a number: callers multiply by x.
#pragma once
#ifdef __CUDACC__
#define MB_HD __host__ __device__ __forceinline__
#else
#include <cmath>
#define MB_HD inline
#endif

namespace mb200 {

template <class Ex2, class Rcp>
MB_HD float sigmoid_by(float x, Ex2 ex2, Rcp rcp) {
  constexpr float kLog2e = 1.44269502162933349609375f, kLog2eTail = 1.9259629911e-8f, kLn2 = 0.6931471805599453f;
  const float z = fminf(fmaxf(x, -120.f), 120.f);
  const float hi = z * -kLog2e, lo = fmaf(z, -kLog2eTail, fmaf(z, -kLog2e, -hi));
  float e = ex2(hi);
  e = hi >= 128.f ? e : fmaf(e, lo * kLn2, e);  // (infinity times a zero or negative lo must not turn into something else)
  return rcp(1.f + e);
}

}  // namespace mb200
