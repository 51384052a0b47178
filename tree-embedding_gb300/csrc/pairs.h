// Pairs of floats for the Cholesky factorizations: sums of products to about
// 2^-41 on the fp32 pipes (fp64 runs at 2 FMAs a clock on an SM here).
#pragma once
#include <stdint.h>

namespace tsvd {

__device__ __forceinline__ float rsqrt_approx(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rcp_approx(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// ------------------------------------------------------------------ pairs of floats
// Sums of products to about 2^-41 of 1 in two floats, for sums that stay
// within [-1, 1]: s carries kAnchor + sum on the grid of its exponent, so what
// one fused multiply-add rounds away is exactly the product minus the change
// of s, which a second one recovers for c (six operations a term where the
// error-free product and TwoSum take twelve). (s, c) -= (ah, al) * (bh, bl):
constexpr float kAnchor = 3.f;
__device__ __forceinline__ void pair_fms(float &s, float &c, float ah, float al, float bh,
                                         float bl) {
  const float t = __fmaf_rn(-ah, bh, s);
  const float z = __fsub_rn(t, s);
  c = __fadd_rn(c, __fmaf_rn(-ah, bh, -z));
  c = __fmaf_rn(-ah, bl, c);
  c = __fmaf_rn(-al, bh, c);
  s = t;
}
// h + l, |h + l| <= 1, into that form.
__device__ __forceinline__ void pair_anchor(float &h, float &l) {
  const float s = __fadd_rn(kAnchor, h);
  l = __fadd_rn(l, __fsub_rn(h, __fsub_rn(s, kAnchor)));
  h = s;
}
__device__ __forceinline__ void pair_norm(float &s, float &c) {
  const float t = __fadd_rn(s, c);
  c = __fsub_rn(c, __fsub_rn(t, s));
  s = t;
}
// an anchored sum as a plain pair
__device__ __forceinline__ void pair_value(float &s, float &c) {
  s = __fsub_rn(s, kAnchor);
  const float t = __fadd_rn(s, c), z = __fsub_rn(t, s);
  c = __fadd_rn(__fsub_rn(s, __fsub_rn(t, z)), __fsub_rn(c, z));
  s = t;
}
// (s, c) *= (yh, yl)
__device__ __forceinline__ void pair_scale(float &s, float &c, float yh, float yl) {
  const float p = __fmul_rn(s, yh);
  float e = __fmaf_rn(s, yh, -p);
  e = __fmaf_rn(s, yl, e);
  e = __fmaf_rn(c, yh, e);
  s = p;
  c = e;
}

// The double with these bits, times 2^sc, as a pair of floats: the leading 23
// mantissa bits and the other 29. Integer work (the conversions and the
// arithmetic of doubles run at 2 a clock on an SM). Below 2^-100: zero.
__device__ __forceinline__ void pair_of(long long bits, int sc, float &hi, float &lo) {
  const uint32_t top = (uint32_t)(bits >> 32), bot = (uint32_t)bits;
  const int raw = (int)((top >> 20) & 0x7ffu), e = raw - 1023 + sc;
  const uint32_t sign = top & 0x80000000u;
  if (raw == 0 || e < -100) {
    hi = lo = 0.f;
    return;
  }
  if (raw == 0x7ff || e > 100) {  // not finite: no pivot is accepted from it
    hi = lo = __uint_as_float(0x7fffffffu);
    return;
  }
  const uint32_t lead = ((top & 0xfffffu) << 3) | (bot >> 29);
  hi = __uint_as_float(sign | ((uint32_t)(e + 127) << 23) | lead);
  const float rest = __uint2float_rn(bot & 0x1fffffffu) * 1.862645149230957e-9f;  // 2^-29
  lo = rest * __uint_as_float(sign | ((uint32_t)(e - 23 + 127) << 23));
}

}  // namespace tsvd
