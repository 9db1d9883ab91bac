// Packed double-single arithmetic, as the FP64-accurate hopping operator computes with it (dhop_ds.cu): a
// complex number as two FP32 pairs, (re, im) of the leading parts in h and of the trailing parts in l, so
// that one FADD2 / FMUL2 / FFMA2 serves both components: half the instructions of the scalar form of
// dsfloat.cuh, the same error-free transformations step by step.  Compiles for the host too, where its tests run.
//
// Errors, relative to the sum S of the magnitudes added:
//   split2       2^-47 (the bits of ds_split where the trailing part is a normal number)
//   +            2^-46 (SloppyDWPlusDW)
//   dot2         n steps, then join2: each step rounds four times in e, which stays below (3 + n) 2^-24 S, and
//                drops the product of two trailing parts (2^-48 of its term): 4 n (3 + n) 2^-48 S, for the
//                six steps of a row of SU(3) below 2^-40 S
#pragma once
#include "dsfloat.cuh"

namespace gbdw {

#ifndef __CUDACC__
struct float2 {
  float x, y;
};
struct double2 {
  double x, y;
};
inline float2 make_float2(float x, float y) { return {x, y}; }
#endif

struct ds2 {
  float2 h, l;
};
GBDW_HD float2 add2(float2 a, float2 b) {
#ifdef __CUDA_ARCH__
  return __fadd2_rn(a, b);
#else
  return make_float2(a.x + b.x, a.y + b.y);
#endif
}
GBDW_HD float2 mul2(float2 a, float2 b) {
#ifdef __CUDA_ARCH__
  return __fmul2_rn(a, b);
#else
  return make_float2(a.x * b.x, a.y * b.y);
#endif
}
GBDW_HD float2 fma2(float2 a, float2 b, float2 c) {
#ifdef __CUDA_ARCH__
  return __ffma2_rn(a, b, c);
#else
  return make_float2(ds_detail::fma_(a.x, b.x, c.x), ds_detail::fma_(a.y, b.y, c.y));
#endif
}
GBDW_HD float2 sub2(float2 a, float2 b) { return fma2(b, make_float2(-1.f, -1.f), a); }  // exact product
GBDW_HD float2 swap2(float2 a) { return make_float2(a.y, a.x); }
// s + e = a + b exactly (Knuth)
GBDW_HD float2 two_sum2(float2 a, float2 b, float2& e) {
  const float2 s = add2(a, b), bb = sub2(s, a);
  e = add2(sub2(a, sub2(s, bb)), sub2(b, bb));
  return s;
}
// the pair (s, t) renormalised (Dekker)
GBDW_HD ds2 join2(float2 s, float2 t) {
  const float2 h = add2(s, t);
  return {h, sub2(t, sub2(h, s))};
}
// SloppyDWPlusDW
GBDW_HD ds2 operator+(ds2 a, ds2 b) {
  float2 e;
  const float2 s = two_sum2(a.h, b.h, e);
  return join2(s, add2(e, add2(a.l, b.l)));
}
// One step of a compensated dot product: s + e += a b with s the running sum of the leading products
// (every rounding error of which goes into e) and e plain FP32; a is the same real for both components
// up to sign.
GBDW_HD void dot2(float2 ah, float2 al, ds2 b, float2& s, float2& e) {
  const float2 p = mul2(ah, b.h);
  const float2 pe = fma2(ah, b.h, make_float2(-p.x, -p.y));  // exact
  e = fma2(ah, b.l, e);
  e = fma2(al, b.h, e);
  float2 f;
  s = two_sum2(s, p, f);
  e = add2(e, add2(pe, f));
}
// An FP64 complex number as pairs: h the leading 24 mantissa bits moved over by integer operations, l the
// other 29 rounded to 24 and scaled by 2^-52 of h's exponent.
GBDW_HD void split1(double d, float& h, float& l) {
  using namespace ds_detail;
  const uint64_t b = bits(d);
  const uint32_t hi = uint32_t(b >> 32), lo = uint32_t(b);
  const uint32_t t = (hi << 3) | (lo >> 29);
  const uint32_t hb = ((t & 0x7fffffffu) ^ 0x40000000u) | (hi & 0x80000000u);
  const uint32_t ah = hi & 0x7fffffffu;
  const float scale = mul_(from_bits(hb & 0xff800000u), 2.220446049250313e-16f);
  h = from_bits(hb);
  l = mul_(float(lo & 0x1fffffffu), scale);
  if (ah - 0x38100000u >= 0x0fe00000u) {  // below 2^-126 (zero) or beyond FP32 (infinity)
    h = from_bits((hi & 0x80000000u) | (ah < 0x38100000u ? 0u : 0x7f800000u));
    l = 0.f;
  }
}
GBDW_HD ds2 split2(double2 a) {
  float2 h, l;
  split1(a.x, h.x, l.x);
  split1(a.y, h.y, l.y);
  return join2(h, l);
}

}  // namespace gbdw
