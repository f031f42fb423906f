// Double-single accumulation (value = hi + lo, two floats) by error-free
// transformations (Dekker / Knuth): the sum s + p = t + err exactly with TwoSum,
// the product a*b = p + e exactly.
#pragma once

namespace mnpbem {

struct DS { float hi, lo; };

// s.hi + a b -> s.hi, returning what that leaves out.  With u = t - s and Knuth's
// TwoSum of s and p = fl(a b), the rest is (s - (t - u)) + (p - u) + (a b - p); one
// fma(a, b, -u) gives its last two terms.  The intrinsics keep the compiler from
// contracting p into the sum, which would break the identity where |s| < |a b|.
__device__ __forceinline__ float ds_acc_prod(float& s, float a, float b) {
  const float t = __fadd_rn(s, __fmul_rn(a, b));
  const float u = __fsub_rn(t, s);
  const float rest = __fadd_rn(__fsub_rn(s, __fsub_rn(t, u)), __fmaf_rn(a, b, -u));
  s = t;
  return rest;
}
__device__ __forceinline__ DS ds_add(DS a, DS b) {
  const float t = a.hi + b.hi;
  const float bp = t - a.hi;
  const float err = (a.hi - (t - bp)) + (b.hi - bp);
  const float lo = a.lo + b.lo + err;
  DS r;
  r.hi = t + lo;                 // renormalise (FastTwoSum)
  r.lo = lo - (r.hi - t);
  return r;
}

// complex (ah + al) * (xh + xl) added to (re, im): exact products of the high
// parts, first-order corrections from the low parts (relative size 2^-24).  The
// double-single products are bound by these FP32 operations, 42 of them; with the
// product's error and the sum's formed apart they were 52, and the rms error of a
// sum of 4000 products 1.6 times as large.
__device__ __forceinline__ void ds_cfma(DS& re, DS& im, float2 ah, float2 al, float2 xh, float2 xl) {
  const float r = __fadd_rn(ds_acc_prod(re.hi, ah.x, xh.x), ds_acc_prod(re.hi, -ah.y, xh.y));
  const float i = __fadd_rn(ds_acc_prod(im.hi, ah.x, xh.y), ds_acc_prod(im.hi, ah.y, xh.x));
  const float lr = fmaf(-al.y, xh.y, fmaf(al.x, xh.x, fmaf(-ah.y, xl.y, ah.x * xl.x)));
  const float li = fmaf(al.y, xh.x, fmaf(al.x, xh.y, fmaf(ah.y, xl.x, ah.x * xl.y)));
  re.lo += r + lr;
  im.lo += i + li;
}

// double <-> (hi, lo) split; a complex128 value as float4 (hi.x, hi.y, lo.x, lo.y)
__device__ __forceinline__ float4 split4(double2 v) {
  const float hx = (float)v.x, hy = (float)v.y;
  return make_float4(hx, hy, (float)(v.x - (double)hx), (float)(v.y - (double)hy));
}
__device__ __forceinline__ double2 join4(float4 v) {
  return make_double2((double)v.x + (double)v.z, (double)v.y + (double)v.w);
}

}  // namespace mnpbem
