// Phase factors in FP32 from phases in half turns.
#pragma once
#include <cstdint>

#include "fft_pack.cuh"

namespace sfxc {

// exp(i pi x) of each lane: x reduced to the nearest half integer (exact in
// FP32 for |x| < 2^21), the Taylor polynomials of sin(pi r) and cos(pi r) on
// |r| <= 1/4 (remainders below 2e-9), and the quadrant.  Each part is within
// 1.3e-7: the sine's product, its last sum and pi itself round by 1.5e-7 of at
// most 0.71, the cosine's last sum by 3e-8 and the terms before it, 0.31 in all,
// by 2e-7 of that.
__device__ __forceinline__ cpair phasor(float x0, float x1) {
  const float2 x = make_float2(x0, x1), magic = dup2(12582912.0f);  // 1.5 x 2^23: rounds to integers
  const float2 y = fma2(x, dup2(2.0f), magic);
  const float2 r = fma2(sub2(y, magic), dup2(-0.5f), x), u = mul2(r, r);
  float2 s = fma2(u, dup2(0.0821458866f), dup2(-0.599264529f));
  s = fma2(s, u, dup2(2.55016404f));
  s = fma2(s, u, dup2(-5.16771278f));
  s = mul2(fma2(s, u, dup2(3.14159265f)), r);
  float2 c = fma2(u, dup2(-0.0258068913f), dup2(0.235330630f));
  c = fma2(c, u, dup2(-1.33526277f));
  c = fma2(c, u, dup2(4.05871213f));
  c = fma2(c, u, dup2(-4.93480220f));
  c = fma2(c, u, dup2(1.0f));
  auto turn = [](float yy, float ss, float cc, float &re, float &im) {
    const uint32_t n = __float_as_uint(yy);  // quadrant in the low two bits
    const bool odd = n & 1;
    const uint32_t sn = (n << 30) & 0x80000000u, cn = ((n + 1) << 30) & 0x80000000u;
    im = __uint_as_float(__float_as_uint(odd ? cc : ss) ^ sn);
    re = __uint_as_float(__float_as_uint(odd ? ss : cc) ^ cn);
  };
  cpair e;
  turn(y.x, s.x, c.x, e.re.x, e.im.x);
  turn(y.y, s.y, c.y, e.re.y, e.im.y);
  return e;
}

}  // namespace sfxc
