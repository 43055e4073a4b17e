// Colour front end of the reference's frame pipeline (gauenk/st_spix
// st_spix/csrc/bist/rgb2lab.cu): sRGB -> CIELAB and back, and 8-bit frame ingest.
// Not called by bist_forward in the reference (pyapi.cu:95-102), so the drop-in path
// leaves frames as given; these serve callers that feed LAB, as the reference's
// command-line pipeline does, and the opt-in ingest conversion of the batched path
// (stspix_config.lab_ingest).
//
// The steps follow the reference exactly (they define the values callers compare
// against): the first channel is read as blue (rgb2lab.cu:64-66), the arithmetic is
// FP64 except that every power goes through the FP32 powf, L is stored divided by
// -100 and a, b by 100 in FP32, and pixels with a NaN channel are left unwritten.
// The colour constants are the CIE standard ones (D65 white, epsilon 0.008856,
// kappa 903.3, the sRGB transfer curve).
#include <cstdint>
#include <cuda_runtime.h>

#include "engine.h"
#include "ff.h"
#include "pdl.h"

namespace stspix {

// x / b for a constant b, correctly rounded, with y = RN(1 / b): one multiplication and two
// fused multiply-adds (Markstein 1990; Brisebarre, Muller and Raina 2004, algorithm 1) in
// place of a division's dozen FP64 instructions.  The last sum differs from x / b by less than
// 1.8 2^-53 of half an ulp, so only quotients nearest to a midpoint could round wrongly; for
// each constant below they are few, and right (tests/test_div_const.py tries them all).
// Values near overflow and NaN divide.
__device__ __forceinline__ double div_const(double x, double b, double y) {
  const double q = x * y;
  if (!(fabs(q) < 1e300)) return x / b;
  return fma(fma(-b, q, x), y, q);
}
#define DIV_CONST(x, b) div_const(x, b, 1.0 / (b))

// sRGB -> CIELAB of one pixel in FP64, as the reference's steps.
__device__ __noinline__ void rgb2lab_fp64(float cR, float cG, float cB, float* lab) {
  auto lin = [](double c) {
    return c <= 0.04045 ? DIV_CONST(c, 12.92)
                        : (double)powf((float)DIV_CONST(c + 0.055, 1.055), (float)2.4);
  };
  const double r = lin((double)cR), g = lin((double)cG), b = lin((double)cB);
  const double X = r * 0.4124564 + g * 0.3575761 + b * 0.1804375;
  const double Y = r * 0.2126729 + g * 0.7151522 + b * 0.0721750;
  const double Z = r * 0.0193339 + g * 0.1191920 + b * 0.9503041;
  const double eps = 0.008856, kappa = 903.3;
  auto f = [&](double v) {
    return v > eps ? (double)powf((float)v, (float)(1.0 / 3.0)) : DIV_CONST(kappa * v + 16.0, 116.0);
  };
  const double fx = f(DIV_CONST(X, 0.950456)), fy = f(Y), fz = f(DIV_CONST(Z, 1.088754));
  lab[0] = (float)(116.0 * fy - 16.0);
  lab[1] = (float)(500.0 * (fx - fy));
  lab[2] = (float)(200.0 * (fy - fz));
}

// The same values without FP64 for nearly every pixel (this part issues FP64 at 1/64 of
// the FP32 rate: the FP64 steps with divisions took 457 us for 1080x1920; now 46).  Every
// FP64 result of the steps above is rounded to FP32 before it is used (an argument of powf,
// or an output).  Each is computed here as an unevaluated sum h + e of two floats
// (error-free sums and products, Dekker 1971 and Knuth TAOCP 2; constants split the same
// way).  The arguments of powf so have a relative error below 2^-45, where the FP64 chain
// errs by less than 2^-50: unless h + e lies within 2^-43 of a rounding boundary both round
// to the same float (ff_round adds and subtracts the margin and compares).  The outputs are
// exact in both forms when f is a power (0.2 < f < 16: at most 37 bits); in the linear
// branch of f (dark colours) the pair of f errs by less than 2^-46, and the outputs' margins
// are absolute.  A pixel where a margin fails or a tristimulus value is at the edge of f's
// branches, with larger values or an infinity, takes the FP64 steps: about 1 pixel in 10^5
// of a bright frame; of the dark ones those of exactly equal channels (the differences
// cancel), but for black.
constexpr float kFFMargin = 0x1p-43f;

__device__ __forceinline__ bool lin_ff(float c, FF* r) {
  // (the largest float not above 0.04045 is its rounding)
  if (c <= 0.04045f) {
    constexpr FF k = FF_CONST(1.0 / 12.92);
    const float p = c * k.h;
    *r = FF{p, mul_err(FF{c, 0.f}, k, p)};
    return true;
  }
  constexpr FF a = FF_CONST(0.055), k = FF_CONST(1.0 / 1.055);
  const float s = c + a.h;
  const FF t{s, sum_err(c, a.h, s) + a.l};
  const float p = t.h * k.h;
  float x;
  const bool ok = ff_round(p, mul_err(t, k, p), p * kFFMargin, &x);
  *r = FF{powf(x, (float)2.4), 0.f};
  return ok;
}
// f(r kr + g kg + b kb); *dark: the linear branch.
__device__ __forceinline__ bool f_ff(FF r, FF g, FF b, FF kr, FF kg, FF kb, FF* f, bool* dark) {
  const float p0 = r.h * kr.h, p1 = g.h * kg.h, p2 = b.h * kb.h;
  const float s = p0 + p1, v = s + p2;
  const float e = ((mul_err(r, kr, p0) + mul_err(g, kg, p1)) + mul_err(b, kb, p2)) +
                  (sum_err(p0, p1, s) + sum_err(s, p2, v));
  const float mag = fabsf(p0) + fabsf(p1) + fabsf(p2);
  // (between 0.008855 and 0.008857 lie the branches' edge and its neighbours: FP64)
  *dark = v < 0.008855f;
  if (*dark) {
    constexpr FF kappa = FF_CONST(903.3), k = FF_CONST(1.0 / 116.0);
    const float p = v * kappa.h, t = p + 16.f;
    const FF w{t, mul_err(FF{v, e}, kappa, p) + sum_err(p, 16.f, t)};
    const float q = w.h * k.h;
    *f = FF{q, mul_err(w, k, q)};
    return mag < 0.02f;          // (no cancellation of larger terms)
  }
  float x;
  const bool ok = ff_round(v, e, mag * kFFMargin, &x);
  *f = FF{powf(x, (float)(1.0 / 3.0)), 0.f};
  return ok && x > 0.008857f && f->h < 16.f;
}
__device__ __forceinline__ bool rgb2lab_ff(float cR, float cG, float cB, float* lab) {
  if (cR == 0.f && cG == 0.f && cB == 0.f) {
    lab[0] = (float)(116.0 * ((903.3 * 0.0 + 16.0) / 116.0) - 16.0);
    lab[1] = lab[2] = 0.f;
    return true;
  }
  FF r, g, b;
  bool ok = lin_ff(cR, &r);
  ok &= lin_ff(cG, &g);
  ok &= lin_ff(cB, &b);
  constexpr FF xr = FF_CONST(0.4124564 / 0.950456), xg = FF_CONST(0.3575761 / 0.950456),
               xb = FF_CONST(0.1804375 / 0.950456);
  constexpr FF yr = FF_CONST(0.2126729), yg = FF_CONST(0.7151522), yb = FF_CONST(0.0721750);
  constexpr FF zr = FF_CONST(0.0193339 / 1.088754), zg = FF_CONST(0.1191920 / 1.088754),
               zb = FF_CONST(0.9503041 / 1.088754);
  FF fx, fy, fz;
  bool dx, dy, dz;
  ok &= f_ff(r, g, b, xr, xg, xb, &fx, &dx);
  ok &= f_ff(r, g, b, yr, yg, yb, &fy, &dy);
  ok &= f_ff(r, g, b, zr, zg, zb, &fz, &dz);
  const float p = 116.f * fy.h, s = p - 16.f;
  ok &= ff_round(s, fmaf(116.f, fy.l, fmaf(116.f, fy.h, -p)) + sum_err(p, -16.f, s),
                 dy ? 0x1p-38f : 0.f, &lab[0]);
  auto diff = [&](float k, FF a, FF c, float margin, float* out) {
    const float d = a.h - c.h, l = sum_err(a.h, -c.h, d) + (a.l - c.l), q = k * d;
    return ff_round(q, fmaf(k, l, fmaf(k, d, -q)), margin, out);
  };
  ok &= diff(500.f, fx, fy, dx || dy ? 0x1p-35f : 0.f, &lab[1]);
  ok &= diff(200.f, fy, fz, dy || dz ? 0x1p-35f : 0.f, &lab[2]);
  return ok;
}

// One pixel: first_blue: the first channel is blue (bist/rgb2lab.cu:64-66); 0: red
// (the legacy prop/rgb2lab.cu:42-44 reads the channels in RGB order, otherwise
// identical).  Returns false (nothing written) for a pixel with a NaN channel.
__device__ __forceinline__ bool rgb2lab_px(float c0, float c1, float c2, float* out,
                                           int first_blue) {
  const float sB = first_blue ? c0 : c2, sR = first_blue ? c2 : c0;
  if (c0 != c0 || c1 != c1 || c2 != c2) return false;
  float lab[3];
  if (!rgb2lab_ff(sR, c1, sB, lab)) rgb2lab_fp64(sR, c1, sB, lab);
  out[0] = lab[0] / (-100);
  out[1] = lab[1] / 100;
  out[2] = lab[2] / 100;
  return true;
}

// nan_copy 1: a pixel with a NaN channel gets its input values; 0: it is left unwritten, as
// the reference leaves it.
__global__ void __launch_bounds__(256) k_rgb2lab(const float* rgb, float* lab, long long npix,
                                                 int first_blue, int nan_copy) {
  pdl_enter();
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= npix) return;
  const float c0 = rgb[3 * t], c1 = rgb[3 * t + 1], c2 = rgb[3 * t + 2];
  if (!rgb2lab_px(c0, c1, c2, lab + 3 * t, first_blue) && nan_copy) {
    lab[3 * t] = c0; lab[3 * t + 1] = c1; lab[3 * t + 2] = c2;
  }
}

// Ingest of a batch with stspix_config.lab_ingest: every frame's colours converted
// once into the slot's engine buffer (img), which every later kernel reads.  A pixel
// with a NaN channel keeps its input values (the reference leaves it unwritten).
__global__ void kb_lab_ingest(const Slot* __restrict__ slots) {
  pdl_enter();
  const Slot& S = slots[blockIdx.y];
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (!S.img_src || t >= S.npix) return;
  float* out = const_cast<float*>(S.img) + 3 * t;
  const float* in = S.img_src + 3 * t;
  const float c0 = in[0], c1 = in[1], c2 = in[2];
  if (!rgb2lab_px(c0, c1, c2, out, 1)) {
    out[0] = c0;
    out[1] = c1;
    out[2] = c2;
  }
}

__global__ void k_lab2rgb(const float* __restrict__ lab, float* __restrict__ rgb, long long npix) {
  pdl_enter();
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= npix) return;
  const double L = lab[3 * t] * (-100);
  const double La = lab[3 * t + 1] * 100;
  const double Lb = lab[3 * t + 2] * 100;
  if (L != L || La != La || Lb != Lb) return;
  const double fy = (L + 16) / 116;
  const double fx = La / 500 + fy;
  const double fz = fy - Lb / 200;
  auto inv = [](double v) {
    const double c = (double)powf((float)v, (float)3);
    return c > 0.008856 ? c : (v - 16.0 / 116.0) / 7.787;
  };
  const double x = inv(fx), y = inv(fy), z = inv(fz);
  const double X = 0.950456 * x, Y = 1.000 * y, Z = 1.088754 * z;
  const double R = X * 3.2406 + Y * (-1.5372) + Z * (-0.4986);
  const double G = X * -0.9689 + Y * 1.8758 + Z * 0.0415;
  const double B = X * 0.0557 + Y * (-0.2040) + Z * 1.0570;
  auto gam = [](double c) {
    return c > 0.0031308 ? 1.055 * ((double)powf((float)c, (float)(1.0 / 2.4))) - 0.055 : 12.92 * c;
  };
  const double r = gam(R), g = gam(G), b = gam(B);
  // clamp to [0, 1] through float, written in RGB order
  float px = (float)fmin(1.0, b * 1.0), py = (float)fmin(1.0, g * 1.0), pz = (float)fmin(1.0, r * 1.0);
  px = (float)fmax(0.0, (double)px);
  py = (float)fmax(0.0, (double)py);
  pz = (float)fmax(0.0, (double)pz);
  rgb[3 * t] = pz;
  rgb[3 * t + 1] = py;
  rgb[3 * t + 2] = px;
}

// rescale_image_kernel (rgb2lab.cu:184-198): 8-bit frames to float, divided by mval.  Four
// values per thread where both pointers allow it (one byte per thread: 27 us for 1080x1920,
// now 9); the values left over by the last thread's.
__global__ void k_rescale_u8(const uint8_t* __restrict__ in, float* __restrict__ out,
                             long long nvals, float mval) {
  pdl_enter();
  const long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * 4;
  if (i >= nvals) return;
  if (i + 4 <= nvals && ((uintptr_t)in & 3) == 0 && ((uintptr_t)out & 15) == 0) {
    const uchar4 v = *(const uchar4*)(in + i);
    *(float4*)(out + i) = make_float4(v.x / mval, v.y / mval, v.z / mval, v.w / mval);
  } else {
    for (long long t = i; t < i + 4 && t < nvals; t++) out[t] = float(in[t] / mval);
  }
}

}  // namespace stspix
