// Arithmetic in unevaluated sums of two floats, and quotients with a shared reciprocal, for
// the places where the FP64 steps of the reference bound a kernel (this part issues FP64 at
// 1/64 of the FP32 rate).  Error-free sums and products: Dekker 1971, Knuth TAOCP 2 (4.2.2);
// division from a reciprocal: Markstein 1990.
#pragma once
#include <cuda_runtime.h>

namespace stspix {

struct FF {
  float h, l;
};
#define FF_CONST(x) FF{(float)(x), (float)((x) - (double)(float)(x))}

// RN(h + e) into *out; false when a value within `margin` of it may round elsewhere.
__device__ __forceinline__ bool ff_round(float h, float e, float margin, float* out) {
  const float up = h + (e + margin), dn = h + (e - margin);
  *out = up;
  return up == dn;
}
// The rounding error of s = a + b.
__device__ __forceinline__ float sum_err(float a, float b, float s) {
  const float bb = s - a;
  return (a - (s - bb)) + (b - bb);
}
// a k - p for p = RN(a.h k.h), k a constant pair.
__device__ __forceinline__ float mul_err(FF a, FF k, float p) {
  return fmaf(a.l, k.h, fmaf(a.h, k.l, fmaf(a.h, k.h, -p)));
}

// An unsigned integer below 2^60 as a pair: its leading 24 bits and the next 24 (at most
// 2^-47 of it is dropped).  32-bit conversions only: the 64-bit ones cost as FP64 does.
__device__ __forceinline__ FF ff_from_u60(unsigned long long u) {
  const int sh = max(40 - __clzll((long long)u), 0), sl = max(sh - 24, 0);
  const unsigned long long rest = u & ((1ULL << sh) - 1);
  return FF{(float)(unsigned)(u >> sh) * __int_as_float((127 + sh) << 23),
            (float)(unsigned)(rest >> sl) * __int_as_float((127 + sl) << 23)};
}

// (float)(a / 2^28 / n) as FP64 gives it (a fixed-point colour sum over 0 < n < 2^24 pixels,
// y = RN(1 / n)), without FP64: the quotient's pair errs by less than 2^-45, so unless it
// lies within 2^-42 of a rounding boundary both round to the same float.  false there, and
// for larger n or |a| >= 2^60.
__device__ __forceinline__ bool mean_ff(long long a, int n, float y, float* out) {
  const unsigned long long u = a < 0 ? 0ULL - (unsigned long long)a : (unsigned long long)a;
  if (n >= 1 << 24 || (u >> 60)) return false;
  const FF s = ff_from_u60(u);
  const float q = s.h * y;
  float m;
  const bool ok = ff_round(q, (fmaf(-q, (float)n, s.h) + s.l) * y, q * 0x1p-42f, &m);
  m *= 0x1p-28f;
  *out = a < 0 ? -m : m;
  return ok;
}

// (float)log(x) as FP64 gives it, without FP64: x = 2^e m with m in [0.707, 1.414],
// log m = 2 atanh(s), s = (m - 1) / (m + 1), by its series in s^2 (nine terms: the rest is
// below 2^-49), the first four terms and the sum with e log 2 in pairs.  The relative error
// is below 2^-41 outside |x - 1| < 2^-6 (below 2^-44 but near there, where the low part of
// m, rounded to 24 bits, counts); false there, outside the normal numbers, and within 2^-40 of a rounding boundary.
__device__ __forceinline__ bool log_ff(double x, float* out) {
  const int hi = __double2hiint(x);
  const unsigned lo = (unsigned)__double2loint(x);
  if (hi < 0x00100000 || hi >= 0x7ff00000) return false;
  int e = (hi >> 20) - 1023;
  float mh = __int_as_float(0x3f800000 | ((hi & 0xFFFFF) << 3) | (int)(lo >> 29));
  float ml = (float)(lo & 0x1FFFFFFFu) * 0x1p-52f;
  if (mh > 1.4140625f) { mh *= 0.5f; ml *= 0.5f; e++; }
  if (e == 0 && fabsf(mh - 1.f) < 0x1p-6f) return false;
  // s = (m - 1) / (m + 1)
  const float f = mh - 1.f;                    // exact
  const float nh = f + ml, nl = ml - (nh - f);
  const float dh = mh + 1.f, dl = (mh - (dh - 1.f)) + ml;
  const float y = __frcp_rn(dh), q = nh * y;
  const float ql = (fmaf(-q, dh, nh) + fmaf(-q, dl, nl)) * y;
  // z = s^2
  const float zh = q * q, zl = fmaf(q, q, -zh) + 2.f * (q * ql);
  float t = (float)(1.0 / 17);
  t = fmaf(t, zh, (float)(1.0 / 15));
  t = fmaf(t, zh, (float)(1.0 / 13));
  t = fmaf(t, zh, (float)(1.0 / 11));
  t = fmaf(t, zh, (float)(1.0 / 9));
  FF u{t, 0.f};
  auto step = [&](FF c) {                      // u = c + z u
    const float p = zh * u.h, pe = fmaf(zh, u.h, -p) + (zh * u.l + zl * u.h);
    const float s = c.h + p;
    u = FF{s, (p - (s - c.h)) + (c.l + pe)};
  };
  constexpr FF c7 = FF_CONST(1.0 / 7), c5 = FF_CONST(1.0 / 5), c3 = FF_CONST(1.0 / 3);
  step(c7);
  step(c5);
  step(c3);
  // log m = 2 (s + s z u)
  const float wh = zh * u.h, wl = fmaf(zh, u.h, -wh) + (zh * u.l + zl * u.h);
  const float p = q * wh, pe = fmaf(q, wh, -p) + (q * wl + ql * wh);
  const float lh = 2.f * (q + p), ll = 2.f * ((p - ((q + p) - q)) + (pe + ql));
  // + e log 2, log 2 = 355 / 512 (times e exact; the split of Cody and Waite 1980) + a pair
  constexpr FF k2 = FF_CONST(-2.121944400546905827679e-4);
  const float ef = (float)e;
  const float a = ef * 0.693359375f, b = ef * k2.h;
  const float s1 = a + b, s2 = s1 + lh;
  const float r = (sum_err(a, b, s1) + sum_err(s1, lh, s2)) +
                  (fmaf(ef, k2.h, -b) + (ef * k2.l + ll));
  return ff_round(s2, r, fabsf(s2) * 0x1p-40f, out);
}

// A non-negative integer as a double: below 2^52 by one addition (a conversion costs more).
__device__ __forceinline__ double to_double(long long a) {
  if ((unsigned long long)a >> 52) return (double)a;
  return __hiloint2double(0x43300000 | (int)(a >> 32), (int)a) - 0x1p52;
}
// RN(1 / d) for d > 0 of at most 34 significant bits (an integer below 2^34, say), d within
// the normal floats, f = d rounded to FP32: two Newton steps from the FP32 reciprocal.  The
// second errs by less than 2^-88 before its rounding, and 1 / d is at least 2^-87 (relative)
// from a rounding boundary, or on a power of two.  Other d: the division.
__device__ __forceinline__ double recip34(double d, float f) {
  if (((unsigned)__double2loint(d) & 0x7FFFFu) || !(f > 0x1p-100f && f < 0x1p100f)) return 1.0 / d;
  const int i = __float_as_int(__frcp_rn(f));
  // the float as a double: exponent bias 127 -> 1023
  const double r0 = __hiloint2double((i >> 3) + (896 << 20), i << 29);
  const double r1 = fma(r0, fma(-d, r0, 1.0), r0);
  return fma(r1, fma(-d, r1, 1.0), r1);
}
// RN(a / n) for integers a >= 0 and 0 < n < 2^31, ad = a, nd = n, y = RN(1 / n): a / n is at
// least 2^-32 units of its last place from a rounding boundary, the corrected quotient
// within 2^-51 of it before its rounding.
__device__ __forceinline__ double div_int(long long a, double ad, double nd, double y) {
  if ((unsigned long long)a >> 52) return ad / nd;
  const double q = ad * y;
  return fma(fma(-nd, q, ad), y, q);
}
// RN(x / d) with y = RN(1 / d): the first correction leaves a faithful quotient, so the
// second rounds correctly (Markstein's theorem) where nothing over- or underflows; there,
// and for zeros, infinities and NaN, the division.
__device__ __forceinline__ double div_recip(double x, double d, double y) {
  const double q0 = x * y;
  const int ex = (__double2hiint(x) >> 20) & 0x7ff, eq = (__double2hiint(q0) >> 20) & 0x7ff;
  if ((unsigned)(ex - 523) > 1000u || (unsigned)(eq - 523) > 1000u) return x / d;
  const double q = fma(fma(-d, q0, x), y, q0);
  return fma(fma(-d, q, x), y, q);
}
// floor of 0 <= m < 2^31 and whether m has a fraction.
__device__ __forceinline__ int floor_bits(double m, bool* frac) {
  const int hi = __double2hiint(m);
  const unsigned lo = (unsigned)__double2loint(m);
  const int e = (hi >> 20) - 1023;
  if (e < 0) {
    *frac = (hi | (int)lo) != 0;
    return 0;
  }
  const unsigned long long v = ((unsigned long long)((hi & 0xFFFFF) | 0x100000) << 32) | lo;
  *frac = (v << (12 + e)) != 0;
  return (int)(v >> (52 - e));
}

}  // namespace stspix
