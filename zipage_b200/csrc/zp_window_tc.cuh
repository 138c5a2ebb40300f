// The weights of capped scores, shared by the tcgen05 kernels over windows.
#pragma once
#include "zp_tc.cuh"
#include "zp_window_attn.cuh"

namespace zp {

using namespace tc;

// four raw products -> exp2(-2c / (1 + exp2(y s)) + off).  The exponent is held at 30: beyond, 1 / (1 + E) is below
// 2^-30 and the weight is 1 to fp32 accuracy, and the product of four stays finite.
__device__ __forceinline__ void weights4(const uint32_t* s, float y, float m2c, float off, float (&p)[4]) {
  const float2 yy = make_float2(y, y), one = make_float2(1.f, 1.f);
  const float2 u = fmul2(make_float2(__uint_as_float(s[0]), __uint_as_float(s[1])), yy), v = fmul2(make_float2(__uint_as_float(s[2]), __uint_as_float(s[3])), yy);
  const float2 ab = fadd2(make_float2(ex2_approx(fminf(u.x, 30.f)), ex2_approx(fminf(u.y, 30.f))), one), cd = fadd2(make_float2(ex2_approx(fminf(v.x, 30.f)), ex2_approx(fminf(v.y, 30.f))), one);
  const float2 prod = fmul2(make_float2(ab.x, cd.x), make_float2(ab.y, cd.y));
  const float r = rcp_approx(prod.x * prod.y) * m2c;
  const float2 rr = fmul2(make_float2(prod.y, prod.x), make_float2(r, r));      // m2c / ab, m2c / cd
  float2 lo = make_float2(off, off), hi = lo;
  ffma2(lo, make_float2(rr.x, rr.x), make_float2(ab.y, ab.x));
  ffma2(hi, make_float2(rr.y, rr.y), make_float2(cd.y, cd.x));
  p[0] = ex2_approx(lo.x); p[1] = ex2_approx(lo.y); p[2] = ex2_approx(hi.x); p[3] = ex2_approx(hi.y);
}

}  // namespace zp
