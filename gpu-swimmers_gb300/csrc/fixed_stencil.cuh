// fixed_stencil.cuh -- Peskin weights in 64-bit integers (the default FP64 particle
// kernels; see fixed_site.cuh for why).
#pragma once
#include "fixed_site.cuh"

namespace lbswim {

// The four weights (peskin_weights4) of a stencil with dr = x - ceil(x - 2),
// 1 <= dr <= 2, in units of 2^-63, within 2^-60: with a = dr - 1 one square root
// s of v = 1 + 4 a (1 - a) in [1, 2], from a 22-bit reciprocal root and two
// Newton steps s + (v - s^2) / (2 s).
__host__ __device__ __forceinline__ void fixed_weights4(double dr, long long w[4]) {
  const double ad = dr - 1.0;  // exact
  const unsigned long long b = double_bits(ad);
  const int sh = 1023 + 1 - (int)(hi_word(b) >> 20);  // 1 for a = 1
  // a in units of 2^-62
  const unsigned long long a =
      sh > 60 ? 0ull : (((b << 11) | 0x8000000000000000ull) >> sh);
  // 4 a (1 - a) in units of 2^-62: the factors in units of 2^-64, where 1 wraps
  // to 0 (and the product is 0)
  const unsigned long long A = a << 2, B = 0ull - A;
#ifdef __CUDA_ARCH__
  const unsigned long long ab = __umul64hi(A, B);
#else
  const unsigned long long ab = (unsigned long long)(((unsigned __int128)A * B) >> 64);
#endif
  const unsigned long long v = (1ull << 62) + ab;
  const float vf = (float)(hi_word(v) >> 7) * 0x1p-23f;
#ifdef __CUDA_ARCH__
  float yf;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(yf) : "f"(vf));
#else
  float yf = 1.0f;
  for (int i = 0; i < 6; ++i) yf = yf * (1.5f - 0.5f * vf * yf * yf);
#endif
  unsigned y = (unsigned)(yf * 0x1p31f);  // 1 / s in units of 2^-31
  y = y < 0x7fffffffu ? y : 0x7fffffffu;
  long long s = (long long)(((unsigned long long)hi_word(v) * y) << 1);  // units of 2^-62
  const long long vq = (long long)(v >> 2);  // the residuals in units of 2^-60
  Digits d = digits(s);
  long long r = vq - mul_hi(d, d);
  s += ((long long)(int)(r >> 10) * (int)y) >> 20;
  d = digits(s);
  r = vq - mul_hi(d, d);
  s += ((long long)(int)r * (int)y) >> 30;
  // (3 - 2 a -+ s) / 8 and (1 + 2 a +- s) / 8, the sums in units of 2^-61
  const long long p = (3ll << 61) - (long long)a, q = (1ll << 61) + (long long)a;
  const long long h = (s + 1) >> 1;
  w[0] = (p - h) >> 1;
  w[1] = (long long)(((unsigned long long)p + (unsigned long long)h) >> 1);
  w[2] = (long long)(((unsigned long long)q + (unsigned long long)h) >> 1);
  w[3] = (q - h) >> 1;
}

}  // namespace lbswim
