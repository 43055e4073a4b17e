// Superpixel quality metrics on the device (gauenk/st_spix
// st_spix/spix_utils/evaluate.py:94-512): per-frame id sizes, temporal extent and
// size variation, explained variance (per frame and over the video), PSNR of the
// pooled video, and under-segmentation error / segmentation accuracy against a
// ground-truth segmentation.
//
// Two passes over the pixels, then small per-id kernels:
//   k_q_accum  per-frame id counts (int32), colour sums (FP64) and id x ground-truth
//              overlap counts (int32), by warp-block label rounds;
//   k_q_resid  per pixel: squared distance to the pixel's pooled colour, per frame;
//   k_q_id_time / k_q_mean / k_q_frame_ids / k_q_uesa  per id: size statistics over time,
//              pooled colours, pooled-vs-mean sums, overlap-based UE / SA sums
//              (integers, exact).
// Pooled colours follow sp_pooling.py:36 (sum / (count + 1e-8)) and
// sp_video_pooling.cu (sum / (count + 1e-10)).
#include <cstdint>
#include <climits>
#include <cuda_runtime.h>

#include "kernels.h"

namespace stspix {

__global__ void k_q_range_init(int* mm) {
  pdl_enter();
  if (threadIdx.x < 4) mm[threadIdx.x] = (threadIdx.x & 1) ? INT_MIN : INT_MAX;
}

// min / max of n labels into mm[0], mm[1] (grid-stride, block reduction); with a grid of
// two rows those of b into mm[2], mm[3].
__global__ void k_q_range(const int32_t* __restrict__ a, const int32_t* __restrict__ b,
                          long long n, int* mm) {
  pdl_enter();
  if (blockIdx.y) { a = b; mm += 2; }
  int lo = INT_MAX, hi = INT_MIN;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const int v = a[i];
    lo = min(lo, v);
    hi = max(hi, v);
  }
  for (int o = 16; o > 0; o >>= 1) {
    lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  __shared__ int slo[32], shi[32];
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) { slo[w] = lo; shi[w] = hi; }
  __syncthreads();
  if (w == 0) {
    const int nw = blockDim.x >> 5;
    lo = l < nw ? slo[l] : INT_MAX;
    hi = l < nw ? shi[l] : INT_MIN;
    for (int o = 16; o > 0; o >>= 1) {
      lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
      hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    if (l == 0) { atomicMin(&mm[0], lo); atomicMax(&mm[1], hi); }
  }
}

// A float's bits as a signed integer multiple of 2^(base - 150), base = the smallest
// exponent kept, in two parts: n = hi 2^20 + lo.  Exact for zero and exponents base ..
// base + 16 (m << 16 < 2^40).
__device__ __forceinline__ void q_parts(float v, int base, int& lo, int& hi) {
  const unsigned b = __float_as_uint(v);
  const int sh = (int)((b >> 23) & 255u) - base;
  const unsigned m = (b << 1) ? ((b & 0x7fffffu) | 0x800000u) : 0u;
  const int l = (int)((m << (sh & 31)) & 0xfffffu), h = (int)(m >> ((20 - sh) & 31));
  lo = (int)b < 0 ? -l : l;
  hi = (int)b < 0 ? -h : h;
}
// n 2^(base - 150) as a double, exact for |n| < 2^51: n is placed in the mantissa of
// 1.5 2^52 and the scale is a power of two.
__device__ __forceinline__ double q_scaled(long long n, int base) {
  const double d = __longlong_as_double(0x4338000000000000LL + n) - 6755399441055744.0;
  return d * __longlong_as_double((long long)(1023 + base - 150) << 52);
}
__device__ __forceinline__ double q_warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// label_rounds for colours: a warp whose first 16 rounds took fewer than three pixels each
// leaves the rest, which it returns, to be added pixel by pixel.  A round costs what three to
// four pixels' atomics do, and only noise leaves so few pixels to a label: 8 frames of 480x854
// with 2,000 random ids took 1761 us in rounds alone, now 320 (681 with scans of rows and
// atomics per run); superpixels of two pixels' width stay in rounds.
template <typename Body>
__device__ __forceinline__ unsigned q_label_rounds(const int (&key)[8], unsigned pend, Body body) {
  int k, src, left = 16;
  unsigned m;
  while (label_round(key, pend, k, m, src)) {
    body(k, m, src);
    if (--left == 0 && __reduce_add_sync(0xffffffffu, __popc(pend)) > 256 - 3 * 16) break;
  }
  return pend;
}

// Pass 1.  Ids are spix - off in [0, S) (others are skipped: the caller refuses them);
// ground-truth ids in [0, G1) (gt may be null, then G1 = 1 and J null).  COLOUR: vid is read.
// A frame is npix pixels in rows of W (H rows, the last one partial); a warp owns a 32 x 8
// block and takes its (id, ground-truth id) pairs one at a time (label_rounds), adding a
// pair's totals with one set of atomics.
// The colours of a block are summed as integers scaled to the block's largest exponent:
// exact when every value is zero or within 2^-16 of the largest (GB300 issues FP64 at
// 1/64 of the FP32 rate, and scans of doubles made this pass FP64-bound); a block with a
// wider range, a denormal, an infinity or a NaN sums in FP64.  Both are at least as
// accurate as FP64 sums in sequence.
// Bound: memory and issue.  8 frames of 480x854 with ground truth: 44 us (293 us with
// FP64 scans of 32-pixel row segments and atomics per run, frame and video sums included).
template <bool COLOUR>
__device__ __forceinline__ void q_accum(const float* __restrict__ vid,
                                        const int32_t* __restrict__ spix,
                                        const int32_t* __restrict__ gt, long long npix, int H,
                                        int W, int off, int S, int G1, int* __restrict__ cnt,
                                        double* __restrict__ fsum, int* __restrict__ J) {
  int gx, by;
  if (!warp_block(W, H, gx, by)) return;
  const int lane = threadIdx.x & 31;
  const int t = blockIdx.y;
  const size_t f0 = (size_t)t * npix;
  int key[8];
  float c[8][3];
  unsigned pend = 0, top = 0;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const long long p = (long long)(by + i) * W + gx;
    const bool in = gx < W && by + i < H && p < npix;
    const int k = in ? spix[f0 + p] - off : -1;
    const int g = in && gt ? gt[f0 + p] : 0;
    const bool ok = k >= 0 && k < S && g >= 0 && g < G1;
    key[i] = ok ? k * G1 + g : -1;                  // S G1 < 2^31
    if (ok) pend |= 1u << i;
    if (COLOUR) {
#pragma unroll
      for (int q = 0; q < 3; q++) {
        c[i][q] = ok ? vid[3 * (f0 + p) + q] : 0.f;
        top = max(top, __float_as_uint(c[i][q]) << 1);
      }
    }
  }
  auto count = [&](int pair, unsigned m, int src) {
    const int N = __reduce_add_sync(0xffffffffu, __popc(m));
    if (lane == src) {
      const int k = J ? pair / G1 : pair;
      atomicAdd(&cnt[(size_t)t * S + k], N);
      if (J) atomicAdd(&J[(size_t)t * S * G1 + pair], N);
    }
  };
  if (!COLOUR) {
    label_rounds(key, pend, count);
    return;
  }
  // the block's exponents: base .. base + 16
  const int base = max((int)(__reduce_max_sync(0xffffffffu, top) >> 24), 17) - 16;
  bool wide = base + 16 >= 255;
#pragma unroll
  for (int i = 0; i < 8; i++)
#pragma unroll
    for (int q = 0; q < 3; q++) {
      const unsigned b = __float_as_uint(c[i][q]) << 1;
      wide |= b != 0 && (int)(b >> 24) < base;
    }
  if (!__any_sync(0xffffffffu, wide)) {
    int lo[8][3], hi[8][3];
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
      for (int q = 0; q < 3; q++) q_parts(c[i][q], base, lo[i][q], hi[i][q]);
    pend = q_label_rounds(key, pend, [&](int pair, unsigned m, int src) {
      int l[3] = {0, 0, 0}, h[3] = {0, 0, 0};
#pragma unroll
      for (int i = 0; i < 8; i++)
        if ((m >> i) & 1u) {
#pragma unroll
          for (int q = 0; q < 3; q++) { l[q] += lo[i][q]; h[q] += hi[i][q]; }
        }
      // (a lane's parts stay below 2^24 in size, a warp's below 2^29)
      long long n[3];
#pragma unroll
      for (int q = 0; q < 3; q++)
        n[q] = (long long)__reduce_add_sync(0xffffffffu, h[q]) * 1048576LL +
               __reduce_add_sync(0xffffffffu, l[q]);
      count(pair, m, src);
      if (lane == src) {
        double* f = fsum + 3 * ((size_t)t * S + (J ? pair / G1 : pair));
#pragma unroll
        for (int q = 0; q < 3; q++) atomicAdd(f + q, q_scaled(n[q], base));
      }
    });
  } else {
    pend = q_label_rounds(key, pend, [&](int pair, unsigned m, int src) {
      double d[3] = {0, 0, 0};
#pragma unroll
      for (int i = 0; i < 8; i++)
        if ((m >> i) & 1u) { d[0] += c[i][0]; d[1] += c[i][1]; d[2] += c[i][2]; }
#pragma unroll
      for (int q = 0; q < 3; q++) d[q] = q_warp_sum(d[q]);
      count(pair, m, src);
      if (lane == src) {
        double* f = fsum + 3 * ((size_t)t * S + (J ? pair / G1 : pair));
#pragma unroll
        for (int q = 0; q < 3; q++) atomicAdd(f + q, d[q]);
      }
    });
  }
  // the pixels left over, read again (registers are short above)
#pragma unroll 1
  for (; pend; pend &= pend - 1) {
    const size_t p = f0 + (size_t)(by + __ffs(pend) - 1) * W + gx;
    const int k = spix[p] - off;
    atomicAdd(&cnt[(size_t)t * S + k], 1);
    if (J) atomicAdd(&J[((size_t)t * S + k) * G1 + (gt ? gt[p] : 0)], 1);
    double* f = fsum + 3 * ((size_t)t * S + k);
#pragma unroll
    for (int q = 0; q < 3; q++) atomicAdd(f + q, (double)vid[3 * p + q]);
  }
}

// Grid (64 x 32 tiles of a frame, T).
__global__ void __launch_bounds__(256, 4) k_q_accum(
    const float* __restrict__ vid, const int32_t* __restrict__ spix,
    const int32_t* __restrict__ gt, long long npix, int H, int W, int off, int S, int G1,
    int* __restrict__ cnt, double* __restrict__ fsum, int* __restrict__ J) {
  pdl_enter();
  q_accum<true>(vid, spix, gt, npix, H, W, off, S, G1, cnt, fsum, J);
}
__global__ void __launch_bounds__(256) k_q_count(const int32_t* __restrict__ spix, long long npix,
                                                 int H, int W, int off, int S,
                                                 int* __restrict__ cnt) {
  pdl_enter();
  q_accum<false>(nullptr, spix, nullptr, npix, H, W, off, S, 1, cnt, nullptr, nullptr);
}

__device__ __forceinline__ double q_block_sum(double v, double* sh) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) sh[w] = v;
  __syncthreads();
  double s = 0;
  if (w == 0) {
    s = l < (int)(blockDim.x >> 5) ? sh[l] : 0.0;
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  }
  return s;   // valid in thread 0
}

// Per id over time: frames alive, total size, the unbiased standard deviation of its size
// over the frames it is alive in (-1 if alive in fewer than two), and, when fsum is not
// null, its colour sums over the video.
__global__ void k_q_id_time(const int* __restrict__ cnt, const double* __restrict__ fsum, int T,
                            int S, long long* ntot, double* std_out, double* vsum) {
  pdl_enter();
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= S) return;
  long long n = 0, s1 = 0;
  __int128 s2 = 0;
  double v[3] = {0, 0, 0};
  for (int t = 0; t < T; t++) {
    const size_t ts = (size_t)t * S + s;
    const long long c = cnt[ts];
    if (c > 0) { n++; s1 += c; s2 += (__int128)(c * c); }
    if (fsum)
      for (int q = 0; q < 3; q++) v[q] += fsum[3 * ts + q];
  }
  ntot[s] = s1;
  if (fsum)
    for (int q = 0; q < 3; q++) vsum[3 * (size_t)s + q] = v[q];
  if (n > 1) {
    const __int128 num = (__int128)n * s2 - (__int128)s1 * s1;
    std_out[s] = sqrt((double)num / ((double)n * (double)(n - 1)));
  } else {
    std_out[s] = -1.0;
  }
}

// Grid (x blocks over ids, T): msum[t] += the frame's colour sums (over its ids), and the
// pooled colour of every id of the frame, mean = sum / (count + 1e-8).
__global__ void __launch_bounds__(256) k_q_mean(const int* __restrict__ cnt,
                                                const double* __restrict__ fsum, int S,
                                                double* __restrict__ mean, double* msum) {
  pdl_enter();
  __shared__ double sh[32];
  const size_t t = blockIdx.y;
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  double v[3] = {0, 0, 0};
  if (s < S) {
    const size_t ts = t * S + s;
    const double n = (double)cnt[ts] + 1e-8;
#pragma unroll
    for (int q = 0; q < 3; q++) {
      v[q] = fsum[3 * ts + q];
      mean[3 * ts + q] = v[q] / n;
    }
  }
#pragma unroll
  for (int q = 0; q < 3; q++) {
    const double a = q_block_sum(v[q], sh);
    if (threadIdx.x == 0) atomicAdd(&msum[3 * t + q], a);
  }
}

// A float as a double by integer moves (the conversion instruction runs at the FP64 rate);
// denormals, infinities and NaN convert.
__device__ __forceinline__ double q_widen(float v) {
  const unsigned b = __float_as_uint(v), e = (b >> 23) & 255u;
  if (e == 255u || (e == 0u && (b << 1))) return (double)v;
  const unsigned hi = (b & 0x80000000u) | ((b & 0x7fffffffu) >> 3);
  return __hiloint2double((int)(e ? hi + (896u << 20) : hi), (int)(b << 29));
}

// Pass 2, grid (x blocks, T): sse[t] += sum_c (v - pooled)^2, the pooled colours from `mean`.
// The squared distances to the frame's mean follow from it per id (k_q_frame_ids).  Bound by
// FP64: a subtraction and a multiply-add per value.  8 frames of 480x854: 65 us (441 us
// with three divisions a pixel, and two more sums).
__global__ void __launch_bounds__(256) k_q_resid(
    const float* __restrict__ vid, const int32_t* __restrict__ spix, int npix, int off, int S,
    const double* __restrict__ mean, double* sse) {
  pdl_enter();
  __shared__ double sh[32];
  const int t = blockIdx.y;
  const double* __restrict__ mt = mean + 3 * (size_t)t * S;
  double a0 = 0, a1 = 0, a2 = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < npix; i += gridDim.x * blockDim.x) {
    const size_t idx = (size_t)t * npix + i;
    const float* p = vid + 3 * idx;
    const double* u = mt + 3 * (size_t)(spix[idx] - off);
    const double d0 = q_widen(p[0]) - u[0], d1 = q_widen(p[1]) - u[1], d2 = q_widen(p[2]) - u[2];
    a0 = fma(d0, d0, a0);
    a1 = fma(d1, d1, a1);
    a2 = fma(d2, d2, a2);
  }
  const double a = q_block_sum(a0 + a1 + a2, sh);
  if (threadIdx.x == 0) atomicAdd(&sse[t], a);
}

// Grid (x blocks over ids, T): live ids per frame, and, when fsum is not null, with u = an
// id's pooled colour and m = the frame's mean: pool2 = sum n (u - m)^2, the cross term
// cross = sum (F - n u)(u - m) (zero up to the 1e-8 of the pooled means), so that the
// frame's sum of squared distances to its mean is sse + 2 cross + pool2, every term of it
// positive but the tiny cross; pool3 = the video pooling's sum (x255).
__global__ void __launch_bounds__(256) k_q_frame_ids(
    const int* __restrict__ cnt, const double* __restrict__ fsum,
    const double* __restrict__ mean, const double* __restrict__ vsum,
    const long long* __restrict__ ntot, const double* __restrict__ msum, int S, int npix,
    unsigned long long* live, double* pool2, double* cross, double* pool3) {
  pdl_enter();
  __shared__ double sh[32];
  const int t = blockIdx.y;
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  double a = 0, x = 0, b = 0;
  int alive = 0;
  if (s < S) {
    const size_t ts = (size_t)t * S + s;
    const int c = cnt[ts];
    if (c > 0) {
      alive = 1;
      if (fsum) {
        const double N = (double)ntot[s] + 1e-10;
#pragma unroll
        for (int q = 0; q < 3; q++) {
          const double m = msum[3 * t + q] / npix;
          const double u = mean[3 * ts + q], d = u - m;
          a += c * (d * d);
          x += fma(-(double)c, u, fsum[3 * ts + q]) * d;
          const double e = 255.0 * vsum[3 * (size_t)s + q] / N - 255.0 * m;
          b += c * (e * e);
        }
      }
    }
  }
  const unsigned nl = __popc(__ballot_sync(0xffffffffu, alive));
  if ((threadIdx.x & 31) == 0 && nl) atomicAdd(&live[t], (unsigned long long)nl);
  if (!fsum) return;
  a = q_block_sum(a, sh);
  if (threadIdx.x == 0) atomicAdd(&pool2[t], a);
  x = q_block_sum(x, sh);
  if (threadIdx.x == 0) atomicAdd(&cross[t], x);
  b = q_block_sum(b, sh);
  if (threadIdx.x == 0) atomicAdd(&pool3[t], b);
}

// Overlap scores (evaluate.py:436-468), one block per kQUesaIds ids and 256 ground-truth ids,
// in one grid dimension (either count may exceed the 65,535 of the others): a thread takes
// one ground-truth id g and kQUesaIds ids, and reads their overlaps of every frame
// (neighbouring threads neighbouring words).  Per frame: the corrected
// under-segmentation sum (min(out, in) over ids overlapping g), the accuracy sum (in over
// ids at least half inside g) and g's size; over the video: the same with in and out summed
// over the frames (out only where the id overlaps g in that frame).  Few pairs overlap, so
// the sums are added as they come.  8 frames, 900 ids, 400 ground-truth ids: 10 us (415 us
// in two kernels with a thread per id walking its rows).
__global__ void __launch_bounds__(256) k_q_uesa(
    const int* __restrict__ cnt, const int* __restrict__ J, const long long* __restrict__ ntot,
    int T, int S, int G1, unsigned long long* ue, unsigned long long* sa, unsigned long long* size,
    unsigned long long* ue3, unsigned long long* sa3) {
  pdl_enter();
  const unsigned ns = ((unsigned)S + kQUesaIds - 1) / kQUesaIds;   // blocks over the ids
  const int g = (int)(blockIdx.x / ns * blockDim.x + threadIdx.x);
  if (g >= G1) return;
  const int s0 = (int)(blockIdx.x % ns) * kQUesaIds;
  long long in[kQUesaIds], out[kQUesaIds];
#pragma unroll
  for (int i = 0; i < kQUesaIds; i++) in[i] = out[i] = 0;
  for (int t = 0; t < T; t++) {
    int j[kQUesaIds];
#pragma unroll
    for (int i = 0; i < kQUesaIds; i++)
      j[i] = s0 + i < S ? J[((size_t)t * S + s0 + i) * G1 + g] : 0;
    unsigned long long u = 0, a = 0, z = 0;
#pragma unroll
    for (int i = 0; i < kQUesaIds; i++) {
      if (j[i] <= 0) continue;
      const long long n = cnt[(size_t)t * S + s0 + i], o = n - j[i];
      in[i] += j[i];
      out[i] += o;
      u += (unsigned long long)min(o, (long long)j[i]);
      if (2LL * j[i] >= n) a += (unsigned long long)j[i];
      z += (unsigned long long)j[i];
    }
    const size_t tg = (size_t)t * G1 + g;
    if (u) atomicAdd(&ue[tg], u);
    if (a) atomicAdd(&sa[tg], a);
    if (z) atomicAdd(&size[tg], z);
  }
  unsigned long long u = 0, a = 0;
#pragma unroll
  for (int i = 0; i < kQUesaIds; i++) {
    if (in[i] <= 0) continue;
    u += (unsigned long long)min(out[i], in[i]);
    if (2 * in[i] >= ntot[s0 + i]) a += (unsigned long long)in[i];
  }
  if (u) atomicAdd(&ue3[g], u);
  if (a) atomicAdd(&sa3[g], a);
}

// sp_pooling (st_spix/sp_pooling.py:10-47) outputs: down[t][s] = colour sum / (count
// + 1e-8) for every id 0..S-1 of every frame, pooled[p] = down of the pixel's id.
// mm: the smallest and largest id; with ids outside [0, S) nothing is written (the caller
// refuses them, after these kernels are launched).
__device__ __forceinline__ bool q_in_range(const int* __restrict__ mm, int S) {
  return mm[0] >= 0 && mm[1] < S;
}
__global__ void k_q_down(const int* __restrict__ mm, int S, const int* __restrict__ cnt,
                         const double* __restrict__ fsum, long long TS, float* __restrict__ down) {
  pdl_enter();
  if (!q_in_range(mm, S)) return;
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= TS) return;
  const double n = (double)cnt[i] + 1e-8;
  for (int c = 0; c < 3; c++) down[3 * i + c] = (float)(fsum[3 * i + c] / n);
}

// A block writes the colours of kMarkPix consecutive pixels: gathered per pixel into shared
// memory, stored as consecutive 16-byte words (single values where `pooled` is not 16-byte
// aligned, and in the last block).
__global__ void __launch_bounds__(256) k_q_pool_write(const int* __restrict__ mm,
                                                      const int32_t* __restrict__ spix, int npix,
                                                      int S, long long n,
                                                      const float* __restrict__ down,
                                                      float* __restrict__ pooled) {
  pdl_enter();
  if (!q_in_range(mm, S)) return;
  __shared__ __align__(16) float v[3 * kMarkPix];
  const long long p0 = (long long)blockIdx.x * kMarkPix;
  const long long t0 = p0 / npix;
  const unsigned r0 = (unsigned)(p0 - t0 * npix);
#pragma unroll
  for (int j = 0; j < kMarkPix / 256; j++) {
    const unsigned k = threadIdx.x + 256 * j;
    float c[3] = {0.f, 0.f, 0.f};
    if (p0 + k < n) {
      const size_t ts = (size_t)(t0 + (r0 + k) / (unsigned)npix) * S + spix[p0 + k];
#pragma unroll
      for (int q = 0; q < 3; q++) c[q] = down[3 * ts + q];
    }
#pragma unroll
    for (int q = 0; q < 3; q++) v[3 * k + q] = c[q];
  }
  __syncthreads();
  float* dst = pooled + 3 * p0;
  if (p0 + kMarkPix <= n && ((uintptr_t)dst & 15) == 0) {
#pragma unroll
    for (int j = 0; j < 3 * kMarkPix / 4 / 256; j++) {
      const int i = threadIdx.x + 256 * j;
      ((float4*)dst)[i] = ((const float4*)v)[i];
    }
  } else {
    const long long left = n - p0;
    const int m = 3 * (int)(left < kMarkPix ? left : kMarkPix);
    for (int e = threadIdx.x; e < m; e += 256) dst[e] = v[e];
  }
}

}  // namespace stspix
