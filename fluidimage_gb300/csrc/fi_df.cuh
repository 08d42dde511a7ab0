// Double-float arithmetic: values as unevaluated pairs hi + lo of floats (about 48
// significant bits), computed on the FP32 pipe.  The error-free transformations use
// the _rn intrinsics so that no FMA contraction can merge a product into the
// following sum.
#pragma once

#include <cuda_runtime.h>

namespace fi {

__device__ __forceinline__ float2 df_split(double v) {
  const float hi = __double2float_rn(v);
  return make_float2(hi, __double2float_rn(v - (double)hi));
}

__device__ __forceinline__ double df_to_double(float2 a) { return (double)a.x + (double)a.y; }

// (a.x + a.y) + (b.x + b.y), renormalised
__device__ __forceinline__ float2 df_add(float2 a, float2 b) {
  const float s = __fadd_rn(a.x, b.x);
  const float bb = __fsub_rn(s, a.x);
  const float err = __fadd_rn(__fsub_rn(a.x, __fsub_rn(s, bb)), __fsub_rn(b.x, bb));
  const float lo = __fadd_rn(__fadd_rn(a.y, b.y), err);
  const float hi = __fadd_rn(s, lo);
  return make_float2(hi, __fsub_rn(lo, __fsub_rn(hi, s)));
}

// a - b of two pairs (an exact product by -1 in a fused multiply-add: one packed
// instruction, where the negation of a pair would take its own)
__device__ __forceinline__ float2 df_sub2(float2 a, float2 b) {
  return __ffma2_rn(b, make_float2(-1.f, -1.f), a);
}

// (sh.x, sl.x) += b * (zh.x + zl.x) and (sh.y, sl.y) += b * (zh.y + zl.y), b = b.x + b.y, by
// error-free products and sums in packed FP32x2 instructions (the lo * lo terms, 2^-48
// relative, are dropped).
__device__ __forceinline__ void df_mac_x2(float2 b, float2 zh, float2 zl, float2& sh,
                                          float2& sl) {
  const float2 bh = make_float2(b.x, b.x), nbh = make_float2(-b.x, -b.x);
  const float2 nbl = make_float2(-b.y, -b.y);
  const float2 p = __fmul2_rn(bh, zh);
  float2 ne = __ffma2_rn(nbh, zh, p);  // minus the error of the product
  ne = __ffma2_rn(nbh, zl, ne);
  ne = __ffma2_rn(nbl, zh, ne);
  const float2 t = __fadd2_rn(sh, p);
  const float2 bb = df_sub2(t, sh);
  const float2 err = __fadd2_rn(df_sub2(sh, df_sub2(t, bb)), df_sub2(p, bb));
  sl = __fadd2_rn(sl, df_sub2(err, ne));
  sh = t;
}

// (sh, sl) += (ah, al) in both lanes
__device__ __forceinline__ void df_acc_x2(float2 ah, float2 al, float2& sh, float2& sl) {
  const float2 t = __fadd2_rn(sh, ah);
  const float2 bb = df_sub2(t, sh);
  const float2 err = __fadd2_rn(df_sub2(sh, df_sub2(t, bb)), df_sub2(ah, bb));
  sl = __fadd2_rn(sl, __fadd2_rn(err, al));
  sh = t;
}

// renormalised: (sh, sl) with sl below half an ulp of sh
__device__ __forceinline__ void df_norm_x2(float2& sh, float2& sl) {
  const float2 hi = __fadd2_rn(sh, sl);
  sl = df_sub2(sl, df_sub2(hi, sh));
  sh = hi;
}

}  // namespace fi
