// FP32 values as integers over a common exponent, for exact sums without the FP64 pipe.
#pragma once
#include <cmath>

#if defined(__CUDACC__)
#define CFLBM_HD __host__ __device__ __forceinline__
#else
#define CFLBM_HD inline
#endif

namespace cflbm {

struct FloatLimbs {
  int a, b, c;
};

CFLBM_HD int limb_round(float x) {
#if defined(__CUDA_ARCH__)
  return __float2int_rn(x);
#else
  return (int)lrintf(x);
#endif
}

// v = (a + b 2^-24 + c 2^-48) 2^(e - 149) but for less than 2^-72 of 2^(e - 126), where
// |v| < 2^(e - 126); scale = 2^(149 - e).  |a|, |b|, |c| <= 2^23: 128 of each add up in
// 32 bits.
CFLBM_HD FloatLimbs float_limbs(float v, float scale) {
  FloatLimbs l;
  const float u = v * scale;
  l.a = limb_round(u);
  const float r = (u - (float)l.a) * 16777216.0f;
  l.b = limb_round(r);
  l.c = limb_round((r - (float)l.b) * 16777216.0f);
  return l;
}

}  // namespace cflbm
