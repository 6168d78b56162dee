// 2^x of the attention kernels' softmax, split over two units of the SM.
//
// A 128 x 128 score tile needs 16384 exponentials, 1024 cycles of the special-function unit (16 per cycle and SM, measured;
// 2^x on a bf16 pair counts as two), which is as long as the tile's tensor-core products at head size 128 and twice as long at
// 64.  Some of the pairs therefore go through a polynomial on the FMA pipe: with all of a pair's work counted, a pair costs 16
// cycles of the special-function unit or 16 of the FMA pipe per warp and scheduler, and 4 of the FMA pipe in either case, so
// that some 7 of 16 pairs by polynomial would be the balance where nothing else shared the pipes.  Measured, 16384 tokens, 16
// heads of 64, not causal, forward: 1614 us with none, 1503 with 4, 1533 with 6, 1527 with 8 of 16.
#pragma once
#include "sm100.cuh"

namespace yv {

// max that keeps NaN
__device__ __forceinline__ float max_nan(float a, float b) {
  float d;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
  return d;
}

// 2^x for x <= 0 (anything below -127 gives 0) in packed fp32: x = n + f with n = round(x), f in [-1/2, 1/2];
// 2^f = 1 + f (c1 + f (c2 + f c3)), the cubic with p(0) = 1 that minimises the largest relative error (1.0e-4, a twentieth of
// the rounding to bf16 that follows).  With KEEP_NAN the exponent is a factor, and NaN or +infinity give NaN; without, it is
// an integer shift and add, one operation less, and the caller sees to NaN and infinities.
template <bool KEEP_NAN>
__device__ __forceinline__ float2 ex2_poly2(float2 x) {
  const float2 magic = make_float2(12582912.f, 12582912.f), unmagic = make_float2(-12582912.f, -12582912.f);  // 1.5 * 2^23
  x.x = KEEP_NAN ? max_nan(x.x, -127.f) : fmaxf(x.x, -127.f);
  x.y = KEEP_NAN ? max_nan(x.y, -127.f) : fmaxf(x.y, -127.f);
  const float2 r = __fadd2_rn(x, magic);                   // the low mantissa bits hold n
  const float2 n = __fadd2_rn(r, unmagic);
  const float2 f = __ffma2_rn(n, make_float2(-1.f, -1.f), x);
  float2 q = __ffma2_rn(make_float2(0.05500893294811249f, 0.05500893294811249f), f,
                        make_float2(0.2422109693288803f, 0.2422109693288803f));
  q = __ffma2_rn(q, f, make_float2(0.6932829022407532f, 0.6932829022407532f));
  q = __ffma2_rn(q, f, make_float2(1.f, 1.f));
  const int one = 0x3F800000;
  if (KEEP_NAN)
    return __fmul2_rn(q, make_float2(__int_as_float(one + (__float_as_int(r.x) << 23)),
                                     __int_as_float(one + (__float_as_int(r.y) << 23))));
  return make_float2(__int_as_float(__float_as_int(q.x) + (__float_as_int(r.x) << 23)),
                     __int_as_float(__float_as_int(q.y) + (__float_as_int(r.y) << 23)));
}

// Pair `i` of a row: POLY of every 16 consecutive pairs go through the polynomial, evenly spread.
template <int POLY, bool KEEP_NAN>
__device__ __forceinline__ float2 ex2_pair(int i, float2 x) {
  if (((i & 15) * POLY) % 16 < POLY) return ex2_poly2<KEEP_NAN>(x);
  return make_float2(ex2(x.x), ex2(x.y));
}

}  // namespace yv
