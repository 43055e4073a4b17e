// GB300 kernels of the per-frame BASS path: hex initialisation, compaction,
// sufficient statistics + posterior, boundary sweep, parameter read-out.
// Reference files cited per kernel (gauenk/st_spix, st_spix/csrc/bist/).
#include <cstdint>
#include <cuda_runtime.h>

#include "engine.h"
#include "ff.h"
#include "kernels.h"

namespace stspix {

// ---------------------------------------------------------------------------
// Hex initialisation (init_seg.cu:48-75).  The reference tests every centre per
// pixel and keeps the LAST centre at the minimum distance.
// Nearest hexagon centre of pixel (x, y) (InitHexSeg, init_seg.cu:63-75): the
// reference scans every centre in FP64 and keeps the last one at the smallest
// squared distance.  A point of the lattice's plane lies within one hexagon radius Hh of
// its nearest centre, rows of centres are 1.5 Hh apart and columns w = sqrt(3) Hh, so the
// nearest centre, and every centre at the same distance, lies in the rows floor(y / 1.5 Hh)
// and the next, in columns floor(x / w) and its two neighbours; the row before is scanned
// too, so that a rounded quotient next to an integer does not matter.
//
// An FP32 pass over the nine candidates finds the smallest squared distance and the next.
// With |dx|, |dy| < 3 hexagon sizes s and centre coordinates below x + y + 3s, the FP32
// squared distance errs by less than ~5e-6 s (x + y + 6s) + 1e-7 d2 px^2; the margin
// below exceeds twice that, so with the next distance outside the margin the nearest
// centre is settled (nearly every pixel), and otherwise the candidates inside it, every
// FP64 minimiser among them, are evaluated in FP64 with the reference's rule, in its scan
// order.  The label is the reference's.  Bound by FP64 before (this part issues it slowly):
// with 25 candidates, and all within 8 px^2 of the smallest in FP64, a 2160x3840 frame took
// 685 us; now 114.
// r0, c0: the search window's centre row floor(y / (1.5 Hh)) and column floor(x / w).
__device__ __forceinline__ int hex_label_rc(int x, int y, double Hh, double w, int nx, int ny,
                                           int r0, int c0) {
  const float wf = (float)w, hf = (float)(1.5 * Hh), half = (float)(0.5 * w);
  const float xf = (float)x, yf = (float)y;
  float mn = 3.0e38f, next = 3.0e38f;
  int best = 0;
#pragma unroll
  for (int i = -1; i <= 1; i++) {
    const int r = r0 + i;
    const float dy = yf - (float)r * hf;
    const float x0 = (r & 1) ? 0.f : half;
#pragma unroll
    for (int j = -1; j <= 1; j++) {
      const int c = c0 + j;
      const float dx = xf - ((float)c * wf + x0);
      float d2 = dx * dx + dy * dy;
      if (r < 0 || r >= ny || c < 0 || c >= nx) d2 = 3.0e38f;
      if (d2 < mn) { next = mn; mn = d2; best = r * nx + c; }
      else next = fminf(next, d2);
    }
  }
  const float sz = wf + hf;
  const float lim = mn + 1e-5f * mn + 1e-5f * sz * (xf + yf + 8.0f * sz);
  if (next > lim) return best;
  double D2 = 1.7976931348623157e308;
  for (int r = r0 - 1; r <= r0 + 1; r++) {
    if (r < 0 || r >= ny) continue;
    for (int c = c0 - 1; c <= c0 + 1; c++) {
      if (c < 0 || c >= nx) continue;
      const float dxf = xf - ((float)c * wf + ((r % 2 == 0) ? half : 0.f));
      const float dyf = yf - (float)r * hf;
      if (dxf * dxf + dyf * dyf > lim) continue;
      double xx = double(c) * w;
      double yy = double(r) * 1.5 * Hh;
      if (r % 2 == 0) xx = xx + 0.5 * w;
      double dx = (x - xx);
      double dy = (y - yy);
      double d2 = dx * dx + dy * dy;
      if (d2 <= D2) { D2 = d2; best = r * nx + c; }
    }
  }
  return best;
}
__device__ __forceinline__ int hex_label(int x, int y, double Hh, double w, int nx, int ny) {
  return hex_label_rc(x, y, Hh, w, nx, ny, (int)floor(y / (1.5 * Hh)), (int)floor(x / w));
}

__global__ void k_init_hex(int* __restrict__ seg, int H, int W, double Hh, double w, int nx,
                           int ny) {
  pdl_enter();
  int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= H * W) return;
  seg[idx] = hex_label(idx % W, idx / W, Hh, w, nx, ny);
}

// Grid: the 64 x 32 tiles of a slot.  The window row depends on y only and the window
// column on x only, so a block computes those of its 32 rows and 64 columns once (two
// FP64 divisions per row or column instead of per pixel; this part issues FP64 slowly).
__global__ void __launch_bounds__(256) kb_init_hex(const Slot* __restrict__ slots) {
  pdl_enter();
  SLOT_Y;
  __shared__ int r0s[32], c0s[64];
  const int W = S.W, H = S.H;
  const int tiles_x = (W + 63) / 64;
  if ((int)blockIdx.x >= tiles_x * ((H + 31) / 32)) return;
  const int tx0 = (blockIdx.x % tiles_x) * 64, ty0 = (blockIdx.x / tiles_x) * 32;
  const double Hh = S.hex_h, w = S.hex_w;
  if (threadIdx.x < 32) r0s[threadIdx.x] = (int)floor((ty0 + (int)threadIdx.x) / (1.5 * Hh));
  else if (threadIdx.x < 96) c0s[threadIdx.x - 32] = (int)floor((tx0 + (int)threadIdx.x - 32) / w);
  __syncthreads();
  for (int i = threadIdx.x; i < 64 * 32; i += blockDim.x) {
    const int lx = i & 63, ly = i >> 6;
    const int x = tx0 + lx, y = ty0 + ly;
    if (x < W && y < H)
      S.seg[(size_t)y * W + x] =
          hex_label_rc(x, y, Hh, w, S.hex_nx, S.hex_ny, r0s[ly], c0s[lx]);
  }
}

// ---------------------------------------------------------------------------
// Compaction (compact_spix.cu:41-122, 196-290): flags of live ids in [lo, hi],
// exclusive scan, remap.
// mode 0: hex ids [0, nraw); mode 1: ids [lo, max_spix] of the finished frame.
__global__ void kb_mark_present(const Slot* __restrict__ slots, int mode) {
  pdl_enter();
  SLOT_Y;
  const int lo = mode == 0 ? 0 : S.lo;
  const int hi = mode == 0 ? S.nraw - 1 : min(S.sc->max_spix, S.cap - 1);
  FOR_PIX(i, S.npix) {
    // one store per run of equal labels (the run's first pixel)
    const int v = S.seg[i];
    if (v >= lo && v <= hi && (i == 0 || S.seg[i - 1] != v)) S.flags[v - lo] = 1;
  }
}

// One block of 1024 threads per slot: exclusive scan of n byte flags (n up to a few 10^5),
// each counted as 0 or 1 (the split acceptance flags of propagated frames carry extra bits).
//   mode 0: hex-id presence (n = nraw)           -> total = live hex ids
//   mode 1: split acceptance (n = ids in use)    -> total = accepted splits
//   mode 2: relabel mint flags (n = ids in use)  -> total = minted ids
//   mode 3: final presence (n = max_spix+1-lo)   -> total = live new ids
// A thread takes 16 flags (one 16-byte load; the arrays start on 256-byte boundaries and end
// at least 2 entries past cap, so the tail is read byte by byte), a warp and then the block
// are scanned by shuffles.  Bound: two block-wide steps per 16384 flags.  Over all cap ids
// with serial chunks a scan took 82 us on a 2160x3840 frame (cap 400,000, 13,000 in use).
__global__ void __launch_bounds__(1024) kb_scan(const Slot* __restrict__ slots, int mode) {
  pdl_enter();
  const Slot& S = slots[blockIdx.x];
  if (mode == 2 && !S.mode) return;  // mint flags exist on propagated slots only
  __shared__ int part[32];
  const uint8_t* flags = (mode == 1) ? S.accept : (mode == 2) ? S.mint : S.flags;
  const int n = (mode == 0) ? S.nraw : (mode == 3) ? min(S.sc->max_spix + 1, S.cap) - S.lo
                                              : live_ids(S);
  int* excl = S.excl;
  int* total = (mode == 0) ? &S.sc->nspix : (mode == 3) ? &S.sc->tmp1 : &S.sc->tmp2;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int run = 0;
  for (int base = 0; base < n; base += 16 * 1024) {
    const int i = base + 16 * (int)threadIdx.x;
    unsigned bits = 0;                           // bit q: flag i + q
    if (i + 16 <= n) {
      const uint4 v = *(const uint4*)(flags + i);
      const unsigned w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int q = 0; q < 16; q++) bits |= (unsigned)(((w[q >> 2] >> (8 * (q & 3))) & 0xffu) != 0) << q;
    } else {
      for (int q = 0; q < 16 && i + q < n; q++) bits |= (unsigned)(flags[i + q] != 0) << q;
    }
    const int c = __popc(bits);
    int inc = c;
#pragma unroll
    for (int k = 1; k < 32; k <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, inc, k);
      if (lane >= k) inc += t;
    }
    if (lane == 31) part[warp] = inc;
    __syncthreads();
    int p = part[lane], pi = p;                  // every warp scans the 32 warp totals
#pragma unroll
    for (int k = 1; k < 32; k <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, pi, k);
      if (lane >= k) pi += t;
    }
    const int before = run + __shfl_sync(0xffffffffu, pi - p, warp) + inc - c;
#pragma unroll
    for (int q = 0; q < 16; q++)
      if (i + q < n) excl[i + q] = before + __popc(bits & ((1u << q) - 1u));
    run += __shfl_sync(0xffffffffu, pi, 31);
    __syncthreads();                             // part is free for the next tile
  }
  if (threadIdx.x == 0) {
    *total = run;
    if (mode == 0 && !S.mode) S.sc->max_spix = run - 1;     // the hex ids in use
    if (mode == 3) S.sc->nspix = S.lo + run;                // the compacted ids
  }
}

__global__ void kb_remap(const Slot* __restrict__ slots, int mode) {
  pdl_enter();
  SLOT_Y;
  const int lo = mode == 0 ? 0 : S.lo;
  FOR_PIX(i, S.npix) {
    const int v = S.seg[i];
    if (v >= lo) S.seg[i] = lo + S.excl[v - lo];
  }
}

// fill_new_params_from_old (compact_spix.cu:220-265): gather moved fields.
__global__ void kb_compact_gather(const Slot* __restrict__ slots) {
  pdl_enter();
  SLOT_Y;
  const SpDev& sp = S.sp;
  const SpDev& tmp = S.tmp;
  const uint8_t* flags = S.flags;
  const int* excl = S.excl;
  const int lo = S.lo;
  FOR_ID_FROM(v, lo, min(S.sc->max_spix + 1, sp.cap)) {
    if (!flags[v - lo]) continue;
    int j = excl[v - lo];
    for (int c = 0; c < 3; c++) {
      tmp.mu_app[3 * j + c] = sp.mu_app[3 * v + c];
      tmp.prior_mu_app[3 * j + c] = sp.prior_mu_app[3 * v + c];
      tmp.sigma_shape[3 * j + c] = sp.sigma_shape[3 * v + c];
      tmp.prior_sigma_shape[3 * j + c] = sp.prior_sigma_shape[3 * v + c];
      tmp.sample_sigma_shape[3 * j + c] = sp.sample_sigma_shape[3 * v + c];
    }
    for (int c = 0; c < 2; c++) {
      tmp.mu_shape[2 * j + c] = sp.mu_shape[2 * v + c];
      tmp.prior_mu_shape[2 * j + c] = sp.prior_mu_shape[2 * v + c];
    }
    tmp.logdet[j] = sp.logdet[v];
    tmp.count[j] = sp.count[v];
    tmp.prior_count[j] = sp.prior_count[v];
    tmp.valid[j] = sp.valid[v];
  }
}

// fill_old_params_from_new (compact_spix.cu:268-290).
__global__ void kb_compact_scatter(const Slot* __restrict__ slots) {
  pdl_enter();
  SLOT_Y;
  const SpDev& sp = S.sp;
  const SpDev& tmp = S.tmp;
  const int lo = S.lo;
  FOR_ID(j, min(S.sc->tmp1, sp.cap - lo)) {
    int d = lo + j;
    for (int c = 0; c < 3; c++) {
      sp.mu_app[3 * d + c] = tmp.mu_app[3 * j + c];
      sp.prior_mu_app[3 * d + c] = tmp.prior_mu_app[3 * j + c];
      sp.sigma_shape[3 * d + c] = tmp.sigma_shape[3 * j + c];
      sp.prior_sigma_shape[3 * d + c] = tmp.prior_sigma_shape[3 * j + c];
      sp.sample_sigma_shape[3 * d + c] = tmp.sample_sigma_shape[3 * j + c];
    }
    for (int c = 0; c < 2; c++) {
      sp.mu_shape[2 * d + c] = tmp.mu_shape[2 * j + c];
      sp.prior_mu_shape[2 * d + c] = tmp.prior_mu_shape[2 * j + c];
    }
    sp.logdet[d] = tmp.logdet[j];
    sp.count[d] = tmp.count[j];
    sp.prior_count[d] = tmp.prior_count[j];
    sp.valid[d] = tmp.valid[j];
  }
}

// ---------------------------------------------------------------------------
// init_sp_params_kernel + mark_active_contiguous (init_sparams.cu:45-166,
// 195-286) for a BASS frame; *nspix live ids, count = npix / nspix.
__global__ void kb_init_bass_params(const Slot* __restrict__ slots) {
  pdl_enter();
  SLOT_Y;
  if (S.mode) return;
  const int sp_size = S.sp_size;
  const SpDev& sp = S.sp;
  const int npix = S.npix;
  FOR_ID(k, sp.cap) {
    int nspix = S.sc->nspix;
    int count = (int)(npix / (1. * nspix));
    sp.prior_sigma_shape[3 * k] = 1.0 / sp_size;
    sp.prior_sigma_shape[3 * k + 1] = 0.;
    sp.prior_sigma_shape[3 * k + 2] = 1.0 / sp_size;
    sp.prior_icov[3 * k] = 1; sp.prior_icov[3 * k + 1] = 0; sp.prior_icov[3 * k + 2] = 1;
    sp.prop[k] = 0;
    sp.icount[k] = 0.f;
    sp.sm_count[k] = 0;
    for (int c = 0; c < 3; c++) {
      sp.mu_app[3 * k + c] = 0.f; sp.prior_mu_app[3 * k + c] = 0.f;
      sp.sigma_shape[3 * k + c] = 0.0; sp.sample_sigma_shape[3 * k + c] = 0.0;
    }
    for (int c = 0; c < 2; c++) { sp.mu_shape[2 * k + c] = 0.0; sp.prior_mu_shape[2 * k + c] = 0.0; }
    sp.logdet[k] = 0.0;
    sp.count[k] = 0;
    if (k < nspix) { sp.valid[k] = 1; sp.prior_count[k] = (float)count; }
    else { sp.valid[k] = 0; sp.prior_count[k] = 0.f; }
  }
}

// prior_mu_app := initial mean (calc_summ_stats, update_params.cu:142-203).
__global__ void kb_init_prior_mu(const Slot* __restrict__ slots) {
  pdl_enter();
  SLOT_Y;
  if (S.mode) return;
  const SpDev& sp = S.sp;
  FOR_ID(k, min(S.sc->nspix, sp.cap)) {
    int n = sp.count[k];
    double c = n;
    for (int ch = 0; ch < 3; ch++)
      sp.prior_mu_app[3 * k + ch] =
          n > 0 ? (float)(fx_unq(sp.acc[8 * k + ch], kFxAppShift) / c) : 0.f;
  }
}

// ---------------------------------------------------------------------------
// Sufficient statistics (sum_by_label, update_params.cu:89-130), R1.  A warp owns a
// 32 x 8 block of a frame: lane = column, and it holds the block's 8 labels and colours
// of its column in registers (every load issued before any is used).  The warp then
// takes the block's labels one at a time (label_rounds): each lane sums its pixels of
// that label, the warp adds the lanes' sums with full-warp reductions (colour sums in
// 24-bit parts, positions relative to the block so they fit 32 bits) and one lane adds
// the label's totals to its global sums with one set of 64-bit atomics.  A block holds
// a few labels, so a few reductions and atomic sets serve 256 pixels.  Colours in
// [0, 1] are summed in 32 bits (one conversion each); others wait in the warp's shared
// staging rows `cw` and are converted and summed in 64 bits in their label's round.
// Integer sums: the totals do not depend on the grouping or the order of the adds.
// ytab: row_sums of the 256 masks of rows.
__device__ __forceinline__ void block_stats(const Slot& S, int bx, int by, float (*cw)[3][32],
                                            const unsigned* ytab) {
  const int lane = threadIdx.x & 31;
  const int H = S.H, W = S.W;
  const SpDev& sp = S.sp;
  const int cap = sp.cap;
  const int gx = bx + lane;
  int lab[8];
  float c[8][3];
  unsigned pend = 0, top = 0;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const int gy = by + i;
    const bool in = gx < W && gy < H;
    const size_t g = (size_t)gy * W + gx;
    lab[i] = in ? S.seg[g] : -1;
#pragma unroll
    for (int ch = 0; ch < 3; ch++) {
      c[i][ch] = in ? S.img[3 * g + ch] : 0.f;
      top = max(top, __float_as_uint(c[i][ch]));
    }
    if (lab[i] >= 0 && lab[i] < cap) pend |= 1u << i;
  }
  // the warp's totals of label k given its colour sums: count and position moments
  // (relative to the block, two to a word), one set of atomics
  auto add = [&](int k, unsigned m, int src, const long long (&St)[3]) {
    const Moments b = block_moments(m, ytab[m], lane);
    if (lane == src) {
      unsigned long long* acc = (unsigned long long*)(sp.acc + 8 * (size_t)k);
      atomicAdd(&sp.count[k], b.n);
      atomicAdd(acc + 0, (unsigned long long)St[0]);
      atomicAdd(acc + 1, (unsigned long long)St[1]);
      atomicAdd(acc + 2, (unsigned long long)St[2]);
      add_moments(acc + 3, b, bx, by);
    }
  };
  if (__all_sync(0xffffffffu, unit_bits(top))) {
    unsigned q[8][3];
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
      for (int ch = 0; ch < 3; ch++) q[i][ch] = fx_unit(c[i][ch], kFxAppShift);
    label_rounds(lab, pend, [&](int k, unsigned m, int src) {
      unsigned s[3] = {0, 0, 0};
#pragma unroll
      for (int i = 0; i < 8; i++)
        if ((m >> i) & 1u) { s[0] += q[i][0]; s[1] += q[i][1]; s[2] += q[i][2]; }
      long long St[3];
      warp_sum3_u31(s, St);
      add(k, m, src, St);
    });
    return;
  }
  // other colours: 64-bit sums, the colours wait in shared memory and a lane converts
  // each of its pixels in the round of its label
#pragma unroll
  for (int i = 0; i < 8; i++)
#pragma unroll
    for (int ch = 0; ch < 3; ch++) cw[i][ch][lane] = c[i][ch];
  __syncwarp();
  label_rounds(lab, pend, [&](int k, unsigned m, int src) {
    long long s[3] = {0, 0, 0};
    for (unsigned mm = m; mm; mm &= mm - 1) {
      const int i = __ffs(mm) - 1;
#pragma unroll
      for (int ch = 0; ch < 3; ch++) s[ch] += fx_q(cw[i][ch][lane], kFxAppShift);
    }
#pragma unroll
    for (int ch = 0; ch < 3; ch++) s[ch] = warp_sum64(s[ch]);
    add(k, m, src, s);
  });
}

// Grid: the 64 x 32 tiles of the first B slots (a block finds its slot by binary
// search over the slots' first tiles); warp w takes the tile's 32 x 8 block
// (w & 1, w >> 1).
__global__ void __launch_bounds__(256, 4) kb_accumulate(const Slot* __restrict__ slots, int B) {
  pdl_enter();
  if (B <= 0) return;
  const int t = blockIdx.x;
  int lo = 0, hi = B - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (slots[mid].tile_base[1] <= t) lo = mid; else hi = mid - 1;
  }
  const Slot& S = slots[lo];
  const int tl = t - S.tile_base[1];
  const int tiles_x = (S.W + 63) / 64;
  const int warp = threadIdx.x >> 5;
  __shared__ float cs[8][8][3][32];   // [warp][row][channel][lane]
  __shared__ unsigned ytab[256];
  ytab[threadIdx.x] = row_sums(threadIdx.x);
  __syncthreads();
  block_stats(S, (tl % tiles_x) * 64 + (warp & 1) * 32, (tl / tiles_x) * 32 + (warp >> 1) * 8,
              cs[warp], ytab);
}

// Accumulator precision study: colour sums by per-pixel FP32 (mode 1, as the
// reference's sum_by_label, update_params.cu:115-117) or FP64 (mode 2) atomics into
// a scratch array (the compaction buffer's sums), then written over the int64 colour
// sums in 2^-28 units (exact for the magnitudes of colour sums), so the posterior sees
// the precision of that accumulator.  Counts and positions stay exact.
__global__ void kb_accumulate_fp(const Slot* __restrict__ slots, int mode) {
  pdl_enter();
  SLOT_Y;
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= S.npix) return;
  const int k = S.seg[t];
  if (k < 0 || k >= S.sp.cap) return;
  const float* p = S.img + 3 * (size_t)t;
  if (mode == 1) {
    float* f = (float*)S.tmp.acc;
    for (int c = 0; c < 3; c++) atomicAdd(&f[3 * (size_t)k + c], p[c]);
  } else {
    double* d = (double*)S.tmp.acc;
    for (int c = 0; c < 3; c++) atomicAdd(&d[3 * (size_t)k + c], (double)p[c]);
  }
}

__global__ void kb_accumulate_fp_store(const Slot* __restrict__ slots, int mode) {
  pdl_enter();
  SLOT_Y;
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= S.sp.cap) return;
  for (int c = 0; c < 3; c++) {
    const double v = mode == 1 ? (double)((const float*)S.tmp.acc)[3 * (size_t)k + c]
                               : ((const double*)S.tmp.acc)[3 * (size_t)k + c];
    S.sp.acc[8 * (size_t)k + c] = __double2ll_rn(ldexp(v, kFxAppShift));
  }
}

__global__ void kb_accumulate_fp_clear(const Slot* __restrict__ slots) {
  pdl_enter();
  SLOT_Y;
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= S.sp.cap) return;
  double* d = (double*)S.tmp.acc;
  for (int c = 0; c < 3; c++) d[3 * (size_t)k + c] = 0.0;
}

// Statistics of a labelling with a chosen accumulator (study entry point).
__global__ void k_label_stats(const float* __restrict__ img, const int* __restrict__ lab,
                              long long npix, int n, int mode, long long* iacc, float* facc,
                              double* dacc) {
  pdl_enter();
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= npix) return;
  const int k = lab[t];
  if (k < 0 || k >= n) return;
  const float* p = img + 3 * t;
  atomicAdd((unsigned long long*)&iacc[7 * (size_t)k], 1ull);
  for (int c = 0; c < 3; c++) {
    const float v = p[c];
    if (mode == 0) {
      atomicAdd((unsigned long long*)&iacc[7 * (size_t)k + 1 + c], (unsigned long long)fx_q(v, kFxAppShift));
      atomicAdd((unsigned long long*)&iacc[7 * (size_t)k + 4 + c], (unsigned long long)fx_q(v * v, kFxSqShift));
    } else if (mode == 1) {
      atomicAdd(&facc[7 * (size_t)k + 1 + c], v);
      atomicAdd(&facc[7 * (size_t)k + 4 + c], v * v);
    } else {
      atomicAdd(&dacc[7 * (size_t)k + 1 + c], (double)v);
      atomicAdd(&dacc[7 * (size_t)k + 4 + c], (double)v * (double)v);
    }
  }
}

__global__ void k_label_stats_out(int n, int mode, const long long* iacc, const float* facc,
                                  const double* dacc, double* out) {
  pdl_enter();
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  out[7 * (size_t)k] = (double)iacc[7 * (size_t)k];
  for (int c = 1; c < 7; c++) {
    double v;
    if (mode == 0) v = ldexp((double)iacc[7 * (size_t)k + c], c < 4 ? -kFxAppShift : -kFxSqShift);
    else if (mode == 1) v = facc[7 * (size_t)k + c];
    else v = dacc[7 * (size_t)k + c];
    out[7 * (size_t)k + c] = v;
  }
}

// ---------------------------------------------------------------------------
// Posterior (calc_simple_update, update_params.cu:220-381, with
// _add_sigma_smoothing :206-217) + clear_fields semantics for dead ids.
__device__ __forceinline__ void smooth_prior(double in_x, double in_y, double in_z, int count,
                                             float pc, int sp_size, double* ox, double* oy,
                                             double* oz) {
  int nf = 50;
  double total_count = 1. * (count + pc * nf);
  *ox = (pc * sp_size + count * in_x) / (total_count + 3.0);
  *oy = (count * in_y) / (total_count + 3.0);
  *oz = (pc * sp_size + count * in_z) / (total_count + 3.0);
}

// One block = 32 consecutive ids, four warps.  Every value is that of the reference's FP64
// expression, bit for bit, but an FP64 instruction here occupies its scheduler for 64 cycles
// (measured: a dependent or an independent one, one lane or 32; a division 564, log 2100),
// so their number on the longest warp is what a launch lasts.  The four warps sit on four
// schedulers and share the work out: warps 1 and 2 take the x and y means and scatters,
// warp 0 the mixed one, each then one entry of the smoothed covariance and of its inverse;
// warp 3 the prior, the reciprocal of the smoothing's denominator and the log determinant.
// Quotients of one divisor share its reciprocal (correctly rounded all the same, see ff.h),
// and where only a float is kept (colour means, the record's log determinant) it is computed
// in pairs of floats, FP64 only next to a rounding boundary.
//
// incremental: only the ids whose count or sums differ from those their posterior last saw
// (S.snap) are computed.  Between two posteriors of the outer loop only the sweeps run,
// which change no other input of the posterior (priors, flags and the sample covariance
// change in the split, merge and relabel steps and at the frame's set-up, whose posteriors
// are full), so an id with equal sums would get the values it already holds (the same
// expressions of the same inputs).  The prior shape term is read from S.pscache then, which
// the last full posterior wrote.
//
// merged: the sums come from a merge (S.tmp, see kb_merge_apply) and become the slot's.
//
// log64: sp.logdet in FP64 (the state read-out); otherwise its float, which is all that the
// records and the parameter read-out take of it.
//
// Every load of a group, the old record and the snapshot among them, is issued before any
// is used, and the ids are compared where they are computed: on most frames, with one group
// per block, a launch is the chain launch - slot - loads - FP64 - store.  With a work list of
// the changed ids built by a kernel of its own a posterior took 10.5 us on a 240x320 frame,
// 13.4 on 720x1280 and 17.1 on 8 frames of 480x854; without it, but with a division per
// quotient and the log in FP64, 5.7, 7.6 and 11.6 (and 32.4 on 16 frames of mixed sizes);
// now 5.0, 6.5, 7.9 (and 17.9; the last step the spread of the groups, see SLOT_X).
__global__ void __launch_bounds__(128) kb_posterior(const Slot* __restrict__ slots,
                                                    int incremental, int log64, int merged) {
  pdl_enter();
  SLOT_X;
  __shared__ double v_ps[3][32], v_den[3][32], v_m[2][32], v_s[3][32], v_ld[32];
  __shared__ float v_i[3][32];
  __shared__ int v_pos[2][32];
  __shared__ unsigned s_diff[3];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const SpDev& sp = S.sp;
  const int cap = sp.cap;
  const int last = min(cap - 1, S.sc->max_spix);
  // the sums and the covariance entry (xx, xy, yy) of a warp
  const int f0 = w == 0 ? 0 : w == 1 ? 3 : 4;
  const int f1 = w == 0 ? 6 : w == 1 ? 5 : 7, ent = w == 0 ? 1 : w == 1 ? 0 : 2;
  for (int g = blockIdx.y;; g += gridDim.y) {
    const int k = 32 * g + lane;
    int count_int = 0;
    uint8_t valid = 0, prop = 0;
    float pc = 0.f;
    long long a[4] = {0, 0, 0, 0}, o[4] = {0, 0, 0, 0}, ocount = 0;
    double q0 = 0, q1 = 0, q2 = 0, i0 = 0, i1 = 0, i2 = 0;
    uint4 orec[3];
    if (k < cap) {
      const long long* acc = (merged ? S.tmp.acc : sp.acc) + 8 * (size_t)k;
      const long long* snap = S.snap + 9 * (size_t)k;
      count_int = (merged ? S.tmp.count : sp.count)[k];
      valid = sp.valid[k];
      pc = sp.prior_count[k];
      if (w < 3) {
        a[0] = acc[f0]; o[0] = snap[f0];
        a[3] = acc[f1]; o[3] = snap[f1];
        if (incremental) q0 = S.pscache[3 * (size_t)k + ent];
        if (w == 0) {
          a[1] = acc[1]; o[1] = snap[1];
          a[2] = acc[2]; o[2] = snap[2];
          ocount = snap[8];
#pragma unroll
          for (int q = 0; q < 3; q++) orec[q] = ((const uint4*)&sp.rec[k])[q];
        }
      } else if (!incremental) {
        prop = sp.prop[k];
        q0 = sp.sample_sigma_shape[3 * k]; q1 = sp.sample_sigma_shape[3 * k + 1];
        q2 = sp.sample_sigma_shape[3 * k + 2];
        i0 = sp.prior_icov[3 * k]; i1 = sp.prior_icov[3 * k + 1]; i2 = sp.prior_icov[3 * k + 2];
      }
    }
    if (32 * g > last) return;                     // block-uniform
    const bool inr = k <= last;
    if (w < 3) {
      bool diff = !incremental;
#pragma unroll
      for (int f = 0; f < 4; f++) diff |= a[f] != o[f];
      if (w == 0) diff |= ocount != count_int;
      const unsigned m = __ballot_sync(0xffffffffu, inr && diff);
      if (lane == 0) s_diff[w] = m;
    }
    __syncthreads();
    const bool want = ((s_diff[0] | s_diff[1] | s_diff[2]) >> lane) & 1u;
    const bool live = want && valid && count_int > 0;
    const bool any = __any_sync(0xffffffffu, live);          // the same in every warp
    // (the sweeps of the next update score again only the pixels next to a changed record)
    if (w == 0 && inr && !live) S.recchg[k] = 0;
    double r0 = 0, nd = 0;
    float app[3] = {0.f, 0.f, 0.f};                // warp 0: the mean colour
    if (live) {
      nd = to_double(count_int);
      if (w == 0) {
        // colour means (fixed-point sums, R1)
        const float y = __frcp_rn((float)count_int);
#pragma unroll
        for (int c = 0; c < 3; c++)
          if (!mean_ff(a[c], count_int, y, &app[c]))
            app[c] = (float)(fx_unq(a[c], kFxAppShift) / nd);
        r0 = to_double(a[3]);
      } else if (w < 3) {
        // shape mean and scatter, of x or of y
        const double y = recip34(nd, (float)count_int), s = to_double(a[0]);
        const double m = div_int(a[0], s, nd, y);
        v_m[w - 1][lane] = m;
        r0 = to_double(a[3]) - nd * m * m;
        sp.mu_shape[2 * k + w - 1] = m;
        // floor and has-fraction, in the bits below and above
        bool frac;
        const int fl = floor_bits(m, &frac);
        v_pos[w - 1][lane] = (int)((unsigned)fl << 1) | (frac ? 1 : 0);
      } else {
        const double total_count = nd + pc * 50;
        const double den = total_count + 3.0;
        v_den[0][lane] = den;
        v_den[1][lane] = recip34(den, pc >= 0.f ? (float)count_int + pc * 50 + 3.f : 0.f);
        v_den[2][lane] = pc;
        // prior shape term (calc_simple_update with _add_sigma_smoothing)
        if (!incremental) {
          double px, py, pz;
          if (prop) {
            smooth_prior(q0, q1, q2, (int)pc, pc, S.sp_size, &px, &py, &pz);
          } else {
            px = i0; py = i1; pz = i2;
          }
          double pr_det = px * pz - py * py;
          if (!(pr_det > 0)) atomicExch(&S.sc->status, STSPIX_ERR_DEGENERATE);
          pr_det = sqrt(pr_det);
          const double t0 = pc / pr_det * px, t1 = pc / pr_det * py, t2 = pc / pr_det * pz;
          v_ps[0][lane] = t0; v_ps[1][lane] = t1; v_ps[2][lane] = t2;
          S.pscache[3 * (size_t)k] = t0; S.pscache[3 * (size_t)k + 1] = t1;
          S.pscache[3 * (size_t)k + 2] = t2;
        }
      }
    }
    __syncthreads();
    if (want) {
      // (behind the first barrier's reads, beside the FP64 work)
      long long* snap = S.snap + 9 * (size_t)k;
      if (w < 3) {
        snap[f0] = a[0];
        snap[f1] = a[3];
      }
      if (merged && w < 3) {
        long long* acc = sp.acc + 8 * (size_t)k;
        acc[f0] = a[0];
        acc[f1] = a[3];
        if (w == 0) { acc[1] = a[1]; acc[2] = a[2]; sp.count[k] = count_int; }
      }
      if (w == 0) {
        snap[1] = a[1];
        snap[2] = a[2];
        snap[8] = count_int;
        if (valid && count_int <= 0) sp.valid[k] = 0;
#pragma unroll
        for (int c = 0; c < 3; c++) sp.mu_app[3 * k + c] = app[c];
        if (!live) {
          for (int c = 0; c < 3; c++) sp.sigma_shape[3 * k + c] = 0.0;
          sp.mu_shape[2 * k] = 0.0; sp.mu_shape[2 * k + 1] = 0.0;
        }
      }
    }
    if (!any) continue;
    // the smoothed covariance, an entry per warp
    if (live && w < 3) {
      if (w == 0) r0 = r0 - nd * v_m[0][lane] * v_m[1][lane];
      const double ps = incremental ? q0 : v_ps[ent][lane];
      v_s[ent][lane] = div_recip(v_den[2][lane] * ps + r0, v_den[0][lane], v_den[1][lane]);
    }
    __syncthreads();
    // its inverse and log determinant
    if (live) {
      double sx = v_s[0][lane], sy = v_s[1][lane], sz = v_s[2][lane];
      double det = sx * sz - sy * sy;
      if (det <= 0) {
        sx = sx + 0.00001;
        sz = sz + 0.00001;
        det = sx * sz - sy * sy;
        if (det <= 0) det = 0.00001;
      }
      if (w < 3) {
        const double v = (w == 0 ? -sy : w == 1 ? sz : sx) / det;
        sp.sigma_shape[3 * k + ent] = v;
        v_i[ent][lane] = (float)v;
      } else {
        float l;
        v_ld[lane] = !log64 && log_ff(det, &l) ? (double)l : log(det);
      }
    }
    __syncthreads();
    if (live && w == 0) {
      const double ld = v_ld[lane];
      sp.logdet[k] = ld;
      SweepRec r;
      r.mu_r = app[0]; r.mu_g = app[1]; r.mu_b = app[2];
      r.logdet = (float)ld;
      const int px = v_pos[0][lane], py = v_pos[1][lane];
      r.mxi = (int)((unsigned)px >> 1); r.myi = (int)((unsigned)py >> 1);
      r.frac = (px & 1) | ((py & 1) << 1);
      r.isx = v_i[0][lane]; r.isy = v_i[1][lane]; r.isz = v_i[2][lane]; r.pad = 0.f;
      r.count = count_int;
      const uint4* nw = (const uint4*)&r;
      bool same = true;
#pragma unroll
      for (int q = 0; q < 3; q++)
        same &= orec[q].x == nw[q].x && orec[q].y == nw[q].y && orec[q].z == nw[q].z &&
                orec[q].w == nw[q].w;
      S.recchg[k] = same ? 0 : 1;
      sp.rec[k] = r;
    }
  }
}

// clear_fields + the helper memset (update_params.cu:54-88, :26): zero the counts and
// the sums of every slot, of all ids (once per frame) or of the ids in use.  An id that a
// step adds gets its sums from that step (kb_split_commit; for minted ids the merge's sums,
// which the posterior takes over), or from such a clear and a pass over the pixels (the
// FP32 and FP64 accumulators).
__global__ void kb_clear_stats(const Slot* __restrict__ slots, int all) {
  pdl_enter();
  SLOT_Y;
  const int n = all ? S.sp.cap : live_ids(S);
  ulonglong2* acc = (ulonglong2*)S.sp.acc;           // 8 sums, 64 bytes, per id
  FOR_ID(k, n) S.sp.count[k] = 0;
  FOR_ID(q, 4 * n) acc[q] = make_ulonglong2(0, 0);
}

// store_sample_sigma_shape_k (update_params.cu:397-438).
__global__ void kb_store_sample(const Slot* __restrict__ slots) {
  pdl_enter();
  SLOT_Y;
  const SpDev& sp = S.sp;
  const int n = min(sp.cap, S.sc->max_spix + 1);     // ids above are never valid
  FOR_SP(k, n) {
  if (!sp.valid[k]) continue;
  const long long* a = sp.acc + 8 * (size_t)k;
  double count = sp.count[k] * 1.0;
  double mx = a[3] / count, my = a[4] / count;
  sp.mu_shape[2 * k] = mx; sp.mu_shape[2 * k + 1] = my;
  double sx, sy, sz;
  if (count > 0) {
    sx = a[5] / count - mx * mx;
    sy = a[6] / count - mx * my;
    sz = a[7] / count - my * my;
  } else {
    sx = sp.prior_sigma_shape[3 * k]; sy = sp.prior_sigma_shape[3 * k + 1];
    sz = sp.prior_sigma_shape[3 * k + 2];
  }
  sp.sample_sigma_shape[3 * k] = sx;
  sp.sample_sigma_shape[3 * k + 1] = sy;
  sp.sample_sigma_shape[3 * k + 2] = sz;
  }
}

// ---------------------------------------------------------------------------
// Border masks (seg_utils.cu:164-195 and 218-257).
__global__ void k_find_border(const int* __restrict__ seg, uint8_t* __restrict__ border, int H,
                              int W) {
  pdl_enter();
  int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= H * W) return;
  int x = idx % W, y = idx / W;
  if (y < 1 || x < 1 || y >= H - 1 || x >= W - 1) { border[idx] = 1; return; }
  int C = seg[idx];
  border[idx] = (C != seg[idx - W] || C != seg[idx + W] || C != seg[idx + 1] ||
                 C != seg[idx - 1]) ? 1 : 0;
}

__global__ void kb_find_border(const Slot* __restrict__ slots) {
  pdl_enter();
  SLOT_Y;
  const int W = S.W, H = S.H;
  const int* seg = S.seg;
  FOR_PIX(idx, S.npix) {
    const int x = idx % W, y = idx / W;
    if (y < 1 || x < 1 || y >= H - 1 || x >= W - 1) { S.border[idx] = 1; continue; }
    const int C = seg[idx];
    S.border[idx] = (C != seg[idx - W] || C != seg[idx + W] || C != seg[idx + 1] ||
                     C != seg[idx - 1]) ? 1 : 0;
  }
}

__global__ void k_find_border_end(const int* __restrict__ seg, uint8_t* __restrict__ border,
                                  int H, int W, int nframes) {
  pdl_enter();
  long long gi = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  long long npix = (long long)H * W;
  if (gi >= npix * nframes) return;
  int idx = (int)(gi % npix);
  const int* s = seg + (gi - idx);
  int x = idx % W, y = idx / W;
  int C = s[idx];
  int N = -1, S = -1, E = -1, Wl = -1;
  if (y > 0) N = s[idx - W];
  if (x > 0) Wl = s[idx - 1];
  if (y < H - 1) S = s[idx + W];
  if (x < W - 1) E = s[idx + 1];
  uint8_t b = 0;
  if ((N >= 0 && C != N) || (S >= 0 && C != S) || (E >= 0 && C != E) || (Wl >= 0 && C != Wl)) {
    if (N >= 0 && C > N) b = 1;
    if (S >= 0 && C > S) b = 1;
    if (E >= 0 && C > E) b = 1;
    if (Wl >= 0 && C > Wl) b = 1;
  }
  border[gi] = b;
}

// get_marked_video in one pass (GetImageOverlaid, pyapi.cu:221-246, on the border rule of
// CudaFindBorderPixels_end): a pixel with a 4-neighbour of a smaller (non-negative) label
// takes the colour, the others their clamped values.
// A block takes kMarkPix consecutive pixels of the video: first their border bits, a thread
// four pixels a block width apart, as ballots in shared memory, while their 3 kMarkPix values
// are loaded as consecutive 16-byte words (single values where a pointer is not 16-byte
// aligned, and in the last block), so every load and store is coalesced although a pixel is
// 12 bytes.
// Bound by memory: 28 B a pixel (labels, colours, result) and the neighbour rows from L1 and
// L2.  8 frames of 480x854: 22 us; a pass took 100 us with a border mask and an
// overlay kernel in FP64, the mask's allocation and a cleared result (24 now).
// out may be vid (every value is read before it is written, by the same thread).
__global__ void __launch_bounds__(256) k_marked(float* out, const float* vid,
                                                const int* __restrict__ spix,
                                                const float* __restrict__ color, int H, int W,
                                                long long n) {
  pdl_enter();
  __shared__ unsigned bits[kMarkPix / 32];
  const long long p0 = (long long)blockIdx.x * kMarkPix;
  // row and column of the block's first pixel; H and W fit 32 bits
  const long long row0 = p0 / W;
  const unsigned x0 = (unsigned)(p0 - row0 * W), y0 = (unsigned)(row0 % H);
  const float* src = vid + 3 * p0;
  float* dst = out + 3 * p0;
  constexpr int kVec = 3 * kMarkPix / 4 / 256;
  const bool vec = p0 + kMarkPix <= n && (((uintptr_t)src | (uintptr_t)dst) & 15) == 0;
  float4 v[kVec];
  if (vec) {
#pragma unroll
    for (int j = 0; j < kVec; j++) v[j] = ((const float4*)src)[threadIdx.x + 256 * j];
  }
#pragma unroll
  for (int j = 0; j < kMarkPix / 256; j++) {
    const unsigned k = threadIdx.x + 256 * j;
    const long long p = p0 + k;
    bool b = false;
    if (p < n) {
      const unsigned r = (x0 + k) / (unsigned)W, x = (x0 + k) - r * (unsigned)W;
      const unsigned y = (y0 + r) % (unsigned)H;
      const int C = spix[p];
      auto below = [&](int v) { return v >= 0 && C > v; };
      if (y > 0) b |= below(spix[p - W]);
      if (x > 0) b |= below(spix[p - 1]);
      if (y + 1 < (unsigned)H) b |= below(spix[p + W]);
      if (x + 1 < (unsigned)W) b |= below(spix[p + 1]);
    }
    const unsigned m = __ballot_sync(0xffffffffu, b);
    if ((threadIdx.x & 31) == 0) bits[k >> 5] = m;
  }
  const float col[3] = {color[0], color[1], color[2]};
  __syncthreads();
  auto value = [&](unsigned e, float v) {
    const unsigned q = e / 3u, c = e - 3u * q;
    const float k = c == 0 ? col[0] : c == 1 ? col[1] : col[2];
    return ((bits[q >> 5] >> (q & 31)) & 1u) ? k : __saturatef(v);   // (a NaN becomes 0)
  };
  if (vec) {
#pragma unroll
    for (int j = 0; j < kVec; j++) {
      const unsigned i = threadIdx.x + 256 * j;
      ((float4*)dst)[i] = make_float4(value(4 * i, v[j].x), value(4 * i + 1, v[j].y),
                                      value(4 * i + 2, v[j].z), value(4 * i + 3, v[j].w));
    }
  } else {
    const long long left = n - p0;
    const unsigned m = 3u * (unsigned)(left < kMarkPix ? left : kMarkPix);
    for (unsigned e = threadIdx.x; e < m; e += 256) dst[e] = value(e, src[e]);
  }
}

// ---------------------------------------------------------------------------
// Boundary sweep (update_seg_subset, update_seg.cu:30-190; calc_joint :194-259;
// simple-point table seg_utils.h:15-79).
// Simple-point table (data, identical to the reference's bass_lut): bit i of the
// index is set when 3x3 neighbour i (NW,N,NE,W,E,SW,S,SE) carries the candidate
// label or lies outside the image.
constexpr unsigned char kSimpleLut[256] = {
    0, 0, 1, 1, 0, 0, 1, 1, 1, 1, 0, 1, 0, 0, 0, 1, 1, 0, 0, 0, 1, 0, 1, 1, 0, 0,
    0, 0, 0, 0, 0, 1, 0, 0, 0, 0, 0, 0, 0, 0, 1, 1, 0, 1, 0, 0, 0, 1, 0, 0, 0, 0,
    0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 1, 1, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0,
    0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 1, 0, 0, 0, 0, 0, 0, 0,
    1, 1, 0, 1, 0, 0, 0, 1, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0,
    0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 1, 0, 0, 0, 1, 0, 1, 1, 0, 0, 0, 0,
    0, 0, 0, 1, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0,
    0, 0, 0, 0, 0, 0, 0, 0, 0, 1, 1, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0,
    1, 0, 0, 0, 1, 0, 1, 1, 0, 0, 0, 0, 0, 0, 0, 0, 1, 0, 0, 0, 0, 0, 0, 0, 1, 1,
    0, 1, 0, 0, 0, 1, 1, 0, 0, 0, 1, 0, 1, 1, 1, 1, 0, 0, 1, 1, 0, 0};

// The table as eight 32-bit words (bit b of word w = entry 32 w + b), computed from it at
// compile time.
struct SimpleBits {
  unsigned w[8];
};
__host__ __device__ constexpr SimpleBits simple_bits() {
  SimpleBits r{};
  for (int i = 0; i < 256; i++)
    if (kSimpleLut[i]) r.w[i >> 5] |= 1u << (i & 31);
  return r;
}
__constant__ SimpleBits c_simple_bits = simple_bits();

// calc_joint's score of label record r for a pixel with neq neighbours of other labels.
__device__ __forceinline__ float joint(float c0, float c1, float c2, int x, int y,
                                       const SweepRec& r, float s2, int neq, float beta) {
  float res = -1000;
  const float x0 = c0 - r.mu_r;
  const float x1 = c1 - r.mu_g;
  const float x2 = c2 - r.mu_b;
  int d0 = x - r.mxi, d1 = y - r.myi;   // == (int)(x - mu_x), see SweepRec
  d0 -= min(max(d0, 0), r.frac & 1);
  d1 -= min(max(d1, 0), (r.frac >> 1) & 1);
  res = res - (x0 * x0 + x1 * x1 + x2 * x2) / s2;
  // (float)(d0 * d0) and so on, by products of the floats (exact below 2^22, so the products
  // round as the integers' conversions do)
  const float f0 = __int_as_float(0x4b400000 + d0) - 12582912.f;
  const float f1 = __int_as_float(0x4b400000 + d1) - 12582912.f;
  res = res - f0 * f0 * r.isx - f1 * f1 * r.isz - 2.f * (f0 * f1) * r.isy;
  res = res - r.logdet;
  // (float)neq for 0 <= neq < 2^23 without a conversion
  res = res - beta * (__uint_as_float(0x4b000000u | (unsigned)neq) - 8388608.f);
  res = res - (r.count <= 10 ? 100.f : 0.f);
  return res;
}

// ---------------------------------------------------------------------------
// Fused sweeps: border pass + the four parity phases of up to NS sweeps in one launch.
// A block owns a TX x TY tile and stages the labels of the tile plus a halo of 4 NS
// pixels.  Sweep s of the ns sweeps of a launch evaluates phase k on the tile grown by
// 4 (ns - s) - 1 - k pixels, so every label a tile pixel depends on is produced inside
// the block exactly as separate launches produce it.  Labels are read from seg_in
// (labels at the launch's start) and the tile is written to seg_out, so neighbouring
// blocks never see each other's updates.
//
// The grid is the list of tiles of every frame of the batch (frame i owns tiles
// [tile_base, tile_base + its tile count)); a block finds its frame by binary
// search, so frames of uneven size cost what their tiles cost.
//
// What bounds it: not bytes (a batch's labels stay in L2) but the instructions and the
// dependent round trips of a tile.  Per launch a tile pays the launch, the slot lookup,
// the staging round trip and the write-back once, however many sweeps it runs, and after
// the first sweep only the pixels next to a change are scored, so four sweeps per launch
// win although the halo is wider (64 x 32 tile: 3 staged labels per tile pixel against
// 4 x 1.41 in four launches, 2.6 scored pixels in the first sweep against 1.15).  In
// between, a phase is a list of its pixels (two barriers), so that the few pixels of a
// late sweep fill warps instead of leaving one active lane per warp.  Measured on batches
// of 8 480x854 frames, the four sweeps of an update: 200-225 us early in a propagated
// frame, 79-95 us late, as four launches of a kernel that scored every border pixel
// within 4 pixels of a change; now 115-170 and 44-50 us (64x32 tiles, 256 threads).  A
// scored pixel takes about 300 instructions of its warp, and a phase of one pixel about
// 2100 cycles (list, 3x3 labels, records, scores, marks: one dependent chain).
constexpr int kReach = 4;             // a sweep's labels depend on labels this far away

// Incremental statistics.  Between two update_params of the BASS loop the labels
// change only in the sweeps, so the statistics of the new labels are those of the old
// ones plus, for every pixel a launch relabels from C to bl, its contribution moved
// from C to bl.  A sweep block collects the moves of its tile's own pixels in a small
// table in shared memory (label -> count and sums, 32-bit fields: colours split into
// 16-bit parts, positions relative to the tile; a tile has at most 3072 pixels to move) and
// adds each touched label's net change to its 64-bit global sums once per launch.  Integer
// sums, so the result is identical to clearing and summing every pixel again.
constexpr int kDeltaTab = 64;         // labels a tile's moves can touch (a power of two)

struct DeltaTab {
  int key[kDeltaTab];                 // label, -1 free
  int v[kDeltaTab][12];               // count, colour lo/hi x 3, sx, sy, sxx, sxy, syy
};

__device__ __forceinline__ int delta_slot(DeltaTab& tb, int k) {
  const unsigned h = ((unsigned)k * 2654435761u) >> 26;
#pragma unroll 1
  for (int p = 0; p < kDeltaTab; p++) {
    const int s = (int)((h + p) & (kDeltaTab - 1));
    const int cur = ((volatile int*)tb.key)[s];
    if (cur == k) return s;
    if (cur == -1) {
      const int old = atomicCAS(&tb.key[s], -1, k);
      if (old == -1 || old == k) return s;
    }
  }
  return -1;
}

// pixel (gx, gy), tile origin (tx0, ty0), moved from label C to label b.
__device__ __forceinline__ void delta_move(DeltaTab& tb, int* count, long long* sums, int C, int b,
                                           int gx, int gy, int tx0, int ty0, float c0, float c1,
                                           float c2) {
  const bool unit = unit_colour(c0) && unit_colour(c1) && unit_colour(c2);
  const int sc = unit ? delta_slot(tb, C) : -1;
  const int sb = unit ? delta_slot(tb, b) : -1;
  if (sc >= 0 && sb >= 0) {
    // colours in [0, 1]: the fixed-point value is one exact conversion, at most 2^28
    const unsigned q0 = fx_unit(c0, kFxAppShift), q1 = fx_unit(c1, kFxAppShift),
                   q2 = fx_unit(c2, kFxAppShift);
    const int x = gx - tx0, y = gy - ty0;
    const int d[12] = {1, (int)(q0 & 0xFFFF), (int)(q0 >> 16), (int)(q1 & 0xFFFF), (int)(q1 >> 16),
                       (int)(q2 & 0xFFFF), (int)(q2 >> 16), x, y, x * x, x * y, y * y};
#pragma unroll
    for (int f = 0; f < 12; f++) {
      atomicAdd(&tb.v[sb][f], d[f]);
      atomicSub(&tb.v[sc][f], d[f]);
    }
    return;
  }
  // other colours, or a full table: the move goes to the global sums at once
  const long long q[3] = {fx_q(c0, kFxAppShift), fx_q(c1, kFxAppShift), fx_q(c2, kFxAppShift)};
  const long long X = gx, Y = gy;
  const long long d[8] = {q[0], q[1], q[2], X, Y, X * X, X * Y, Y * Y};
  unsigned long long* ab = (unsigned long long*)(sums + 8 * (size_t)b);
  unsigned long long* ac = (unsigned long long*)(sums + 8 * (size_t)C);
  atomicAdd(&count[b], 1);
  atomicSub(&count[C], 1);
#pragma unroll
  for (int f = 0; f < 8; f++) {
    atomicAdd(ab + f, (unsigned long long)d[f]);
    atomicAdd(ac + f, (unsigned long long)(-d[f]));
  }
}

// The table's net changes to the global sums (block-wide; after the last phase).
__device__ __forceinline__ void delta_flush(DeltaTab& tb, int* count, long long* sums, int tx0,
                                            int ty0) {
  for (int i = threadIdx.x; i < kDeltaTab; i += blockDim.x) {
    const int k = tb.key[i];
    if (k < 0) continue;
    const int* v = tb.v[i];
    const long long n = v[0], X = tx0, Y = ty0;
    const long long sx = v[7], sy = v[8];
    const long long d[8] = {(long long)v[2] * 65536 + v[1], (long long)v[4] * 65536 + v[3],
                            (long long)v[6] * 65536 + v[5], n * X + sx, n * Y + sy,
                            n * X * X + 2 * X * sx + v[9], n * X * Y + X * sy + Y * sx + v[10],
                            n * Y * Y + 2 * Y * sy + v[11]};
    unsigned long long* acc = (unsigned long long*)(sums + 8 * (size_t)k);
    atomicAdd(&count[k], v[0]);
#pragma unroll
    for (int f = 0; f < 8; f++) atomicAdd(acc + f, (unsigned long long)d[f]);
  }
}

// Bits [0, n) of a 32-bit word (n clamped to 0..32), and bits [a, b) of word w of a row
// of 32-pixel words.
__device__ __forceinline__ unsigned bits32_below(int n) {
  return ~__funnelshift_lc(0u, 0xffffffffu, (unsigned)max(n, 0));
}
__device__ __forceinline__ unsigned range32(int a, int b, int w) {
  return bits32_below(b - 32 * w) & ~bits32_below(a - 32 * w);
}

// Shared memory of a sweep block.  Masks are rows of 32-pixel words over the label
// region (bit x & 31 of word x >> 5 of row y = label-region pixel (x, y)).
template <int TX, int TY, int NS>
struct SweepTile {
  static constexpr int kSH = kReach * NS;                            // label halo
  static constexpr int kG0 = kSH - 1;                                // first sweep's growth
  static constexpr int kLX = TX + 2 * kSH, kLY = TY + 2 * kSH;       // staged labels
  static constexpr int kCK = (kLX + 31) / 32;                        // words per row
  static constexpr int kClass = (TX / 2 + kG0) * (TY / 2 + kG0);     // a phase's pixels
  static constexpr int kMaxList = kClass > TX * TY ? kClass : TX * TY;
  static_assert(kLX < 256 && kLY < 256, "list entries pack (y << 8) | x");
  static_assert(kLX % 8 == 0 && kLY % 8 == 0, "8-pixel groups, rows in whole warp spans");
  static_assert((long long)TX * TY * 65535 < (1LL << 31), "statistics moves fit 32 bits");
  static_assert(kSH % 2 == 0 && TX % 16 == 0 && TY % 2 == 0, "region parity = image parity");
  __align__(16) int L[kLX * kLY];
  unsigned short list[kMaxList];      // pixels of the running phase, (y << 8) | x
  int cnt[2][4];                      // list lengths by phase, alternating between sweeps
  int wcnt;                           // length of the write-back list
  int neg;                            // a staged label is negative (outside the image)
  union {
    struct {
      // label edges: edE bit set when a pixel and its right neighbour differ, edS when a
      // pixel and the one below differ.  Built at staging, kept current by the relabels.
      unsigned edE[kLY][kCK], edS[kLY][kCK];
      unsigned seed[kLY][kCK];        // changed pixels the first sweep starts from
      unsigned dirty[kLY][kCK];       // pixels to score at their next phase (see sweep_tile)
      unsigned bm[kLY][kCK];          // border pixels at the start of the running sweep
    };
    DeltaTab delta;                   // after the sweeps: statistics moves of the tile's pixels
  };
  unsigned sin[kLY][kCK];             // pixels where seg_out differs from seg_in at the start
  unsigned all[kLY][kCK];             // tile pixels relabelled by this launch
};

// The slot fields a sweep reads, loaded together (one round trip; the slot table is read
// from L2 by every block).
struct SweepSlot {
  const int* in;
  int* out;
  const uint16_t* chg_in;
  uint16_t* chg_out;
  const float* img;
  const SweepRec* rec;
  const uint8_t* recchg;
  int* count;
  long long* acc;
  int H, W, cap, tile0;
};
__device__ __forceinline__ SweepSlot sweep_slot(const Slot& S, int parity, int v) {
  SweepSlot r;
  int* a = S.seg;
  int* b = S.seg_alt;
  uint8_t* c0 = S.chg[0];
  uint8_t* c1 = S.chg[1];
  r.img = S.img;
  r.rec = S.sp.rec;
  r.recchg = S.recchg;
  r.count = S.sp.count;
  r.acc = S.sp.acc;
  r.H = S.H; r.W = S.W; r.cap = S.cap;
  r.tile0 = S.tile_base[v];
  r.in = parity ? b : a;
  r.out = parity ? a : b;
  r.chg_in = (const uint16_t*)(parity ? c0 : c1);
  r.chg_out = (uint16_t*)(parity ? c1 : c0);
  return r;
}

// The three 16-byte words of label k's record.
__device__ __forceinline__ SweepRec load_rec(const SweepRec* __restrict__ rec, int k) {
  union { SweepRec r; uint4 q[3]; } u;
  const uint4* p = (const uint4*)(rec + k);
#pragma unroll
  for (int i = 0; i < 3; i++) u.q[i] = __ldg(p + i);
  return u.r;
}

// Scores and relabels the n <= threads / 4 listed pixels of a phase, four lanes to a pixel:
// lane q takes candidate q of N, S, W, E (its simple-point code, record and score), two
// exchanges find the best, and each lane updates its edge.  The result is that of one thread
// per pixel (a repeated candidate scores the same, so the first of the best stands), in a
// third of the dependent instructions: a phase of few pixels lasts one warp's chain, about
// 350 instructions with a thread per pixel.  Up to a quarter of the block's threads in pixels:
// above, one round no longer holds them (half, in two rounds, was 1 to 2 % slower, two lanes
// to a pixel there too, all in rounds 12 %).  With the listing by atomics (below) a launch on
// a 240x320 frame fell from 18.7 to 14.5 us, on 720x1280 from 43.4 to 37.8, on 8 frames of
// 480x854 from 83.4 to 75.4.
template <int TX, int TY, int NS>
__device__ __forceinline__ void sweep_quad(const SweepSlot& S, SweepTile<TX, TY, NS>& sm, int rx0,
                                           int ry0, int n, float s2, float potts,
                                           const unsigned* lut_bits, bool neg) {
  using Tile = SweepTile<TX, TY, NS>;
  constexpr int kSH = Tile::kSH, kLX = Tile::kLX;
  int* L = sm.L;
  const int lane = threadIdx.x & 31, q = lane & 3, j = threadIdx.x >> 2;
  const int W = S.W, cap = S.cap;
  const bool act = j < n;
  const int ent = sm.list[act ? j : 0];
  const int ax = ent & 255, ay = ent >> 8;
  const int gx = rx0 + ax, gy = ry0 + ay;
  const int p = ay * kLX + ax;
  const float* pix = S.img + 3 * ((size_t)gy * W + gx);
  const float c0 = __ldg(pix), c1 = __ldg(pix + 1), c2 = __ldg(pix + 2);
  const int v = L[p + (q < 2 ? (q ? kLX : -kLX) : (q == 2 ? -1 : 1))];
  const int C = L[p];
  const int N = L[p - kLX], So = L[p + kLX], Wl = L[p - 1], E = L[p + 1];
  const int nb[8] = {L[p - kLX - 1], N, L[p - kLX + 1], Wl, E, L[p + kLX - 1], So, L[p + kLX + 1]};
  const bool in = (unsigned)C < (unsigned)cap && max(max(N, So), max(Wl, E)) < cap &&
                  !(N == C && So == C && Wl == C && E == C);
  const SweepRec r = load_rec(S.rec, in ? max(v, 0) : 0);
  const int n_c = __ldg(&S.rec[in ? C : 0].count);
  unsigned d = 0, m1 = 0;
#pragma unroll
  for (int i = 0; i < 8; i++) d |= (unsigned)(nb[i] == v) << i;
  if (neg) {                                        // block-uniform
#pragma unroll
    for (int i = 0; i < 8; i++) m1 |= (unsigned)(nb[i] == -1) << i;
    d |= m1;
  }
  const unsigned simple =
      __ballot_sync(0xffffffffu, ((lut_bits[d >> 5] >> (d & 31)) & 1u) && in && act);
  const float sc = joint(c0, c1, c2, gx, gy, r, s2, 8 - __popc(d), potts);
  const bool cand = v >= 0 && sc > -9999.f;
  float best = cand ? sc : -9999.f;
  int bl = cand ? v : C;
#pragma unroll
  for (int o = 1; o <= 2; o <<= 1) {
    const float ob = __shfl_xor_sync(0xffffffffu, best, o);
    const int ol = __shfl_xor_sync(0xffffffffu, bl, o);
    if (ob > best || (ob == best && (lane & o))) { best = ob; bl = ol; }
  }
  if (((simple >> (lane & 28)) & 15u) != 15u) return;
  if (bl == C && n_c <= 2) bl = N >= 0 ? N : E >= 0 ? E : So >= 0 ? So : Wl >= 0 ? Wl : C;
  if (bl == C) return;
  if (q == 0) {
    L[p] = bl;
    if (ay >= kSH && ay < kSH + TY && ax >= kSH && ax < kSH + TX)
      atomicOr(&sm.all[ay][ax >> 5], 1u << (ax & 31));
  }
  if (q < 3) {                                      // row ay - 1 + q of its 3x3 is dirty
    const unsigned long long three = 7ull << ((ax & 31) + 31);   // bits 31.. = word ax >> 5
    unsigned* row = sm.dirty[ay - 1 + q] + (ax >> 5);
    atomicOr(row, (unsigned)(three >> 32));
    if (!(ax & 31)) atomicOr(row - 1, 0x80000000u);
    if ((ax & 31) == 31) atomicOr(row + 1, 1u);
  }
  // the lane's edge: of N and S rows' edS, of W and E columns' edE (the pixels of a phase
  // are never 4-neighbours, so each edge has one writer; words are shared)
  const int ex = q == 2 ? ax - 1 : ax, ey = q == 0 ? ay - 1 : ay;
  if ((C != v) != (bl != v))
    atomicXor(q < 2 ? &sm.edS[ey][ex >> 5] : &sm.edE[ey][ex >> 5], 1u << (ex & 31));
}

// What a sweep scores.  The parameters are fixed across the sweeps of one update_seg
// call, and a pixel's decision depends only on its 3x3 labels at its phase, its colour
// and the records of its own and its 4-neighbours' labels.  So a pixel whose 3x3 labels
// and records have not changed since it was last scored keeps its label, and only the
// others, the dirty pixels, are scored: a relabelled pixel makes its 3x3 dirty, a phase
// scores the dirty pixels of its class that were border pixels at the start of the sweep
// (the reference's border mask is built once per sweep) and clears their bits; a dirty
// pixel that was no border pixel then stays dirty.  The first sweep of a launch starts
// from
//   mode 0: every border pixel (seg_out holds nothing of use);
//   mode 1: the pixels within 1 of a change of the previous launch of the call (chg_in);
//   mode 2: within 1 of a change of the previous call's last launch, or of a pixel of a
//           label whose record the posterior between the calls changed.
// A pixel of phase k depends, through the phases before it, on labels within Chebyshev
// distance k + 1 <= 4, so the label region holds everything a tile pixel depends on.
// A launch writes the union of its sweeps' changes (chg_out): a superset of the last
// sweep's, and every pixel where seg_out and seg_in differ.  So when a launch in mode 1
// or 2 starts, seg_out (the labels before the previous launch) equals seg_in but at the
// pixels of chg_in, and only those and the launch's own changes are stored.
//
// NT: threads of the block.
template <int TX, int TY, int NS, int NT>
__device__ __forceinline__ void sweep_tile(const SweepSlot& S, int bx, int by, int ns, float s2,
                                           float potts, SweepTile<TX, TY, NS>& sm,
                                           const unsigned* lut_bits, int mode, int deltas) {
  using Tile = SweepTile<TX, TY, NS>;
  constexpr int kSH = Tile::kSH, kLX = Tile::kLX, kLY = Tile::kLY, kCK = Tile::kCK;
  constexpr int kWords = kLY * kCK, kWarps = NT / 32;
  int* L = sm.L;
  const int H = S.H, W = S.W;
  const int* __restrict__ seg_in = S.in;
  int* __restrict__ seg_out = S.out;
  const int tx0 = bx * TX, ty0 = by * TY;
  const int rx0 = tx0 - kSH, ry0 = ty0 - kSH;        // label region origin
  // change flags: one bit per pixel, rows of P16 16-bit words (bit x & 15 of word
  // x >> 4); a tile's x origin is a multiple of 16, so every word has one writer
  const uint16_t* __restrict__ chg_in = S.chg_in;
  uint16_t* __restrict__ chg_out = S.chg_out;
  const int P16 = (W + 15) >> 4;
  const int cap = S.cap;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;

  // --- staging: the label region to shared memory, a span of rows per warp; every load
  // of a thread is issued before the first store (one memory round trip)
  {
    constexpr int kRW = (kLY + kWarps - 1) / kWarps;      // warp w: rows w, w + kWarps, ..
    int lv[kRW][kCK];
    if (rx0 >= 0 && ry0 >= 0 && rx0 + kLX <= W && ry0 + kLY <= H) {
      // inside the frame (most tiles): one row pointer per row
      const int* base = seg_in + (size_t)(ry0 + warp) * W + rx0 + lane;
      const size_t step = (size_t)kWarps * W;
#pragma unroll
      for (int a = 0; a < kRW; a++)
#pragma unroll
        for (int c = 0; c < kCK; c++)
          lv[a][c] = (kLX % 32 == 0 || lane + 32 * c < kLX) &&
                             (kLY % kWarps == 0 || a * kWarps + warp < kLY)
                         ? base[a * step + 32 * c] : -1;
    } else {
#pragma unroll
      for (int a = 0; a < kRW; a++) {
        const int gy = ry0 + a * kWarps + warp;
#pragma unroll
        for (int c = 0; c < kCK; c++) {
          const int x = lane + 32 * c, gx = rx0 + x;
          lv[a][c] = (gy >= 0 && gy < H && a * kWarps + warp < kLY && x < kLX && gx >= 0 && gx < W)
                         ? seg_in[(size_t)gy * W + gx] : -1;
        }
      }
    }
    // the changes of the previous launch, meanwhile
    for (int i = threadIdx.x; i < kWords; i += NT) {
      unsigned w = 0;
      if (mode) {
        const int r = i / kCK, c = i - r * kCK;
        const int gy = ry0 + r, x = rx0 + 32 * c;
        const int w0 = x >> 4, off = x & 15;         // x >= -16: the shift floors
        if (gy >= 0 && gy < H) {
          const uint16_t* row = chg_in + (size_t)gy * P16;
          unsigned long long v = 0;
#pragma unroll
          for (int k = 0; k < (kSH % 16 ? 3 : 2); k++)
            if (w0 + k >= 0 && w0 + k < P16) v |= (unsigned long long)row[w0 + k] << (16 * k);
          w = (unsigned)(v >> off) & range32(0, kLX, c);
        }
      }
      (&sm.sin[0][0])[i] = w;
      (&sm.all[0][0])[i] = 0;
    }
    if (threadIdx.x < 8) (&sm.cnt[0][0])[threadIdx.x] = 0;
    if (threadIdx.x == 8) { sm.wcnt = 0; sm.neg = 0; }
#pragma unroll
    for (int a = 0; a < kRW; a++)
#pragma unroll
      for (int c = 0; c < kCK; c++)
        if ((kLX % 32 == 0 || lane + 32 * c < kLX) &&
            (kLY % kWarps == 0 || a * kWarps + warp < kLY))
          L[(a * kWarps + warp) * kLX + lane + 32 * c] = lv[a][c];
  }
  __syncthreads();
  // --- label edges and seeds, 8 pixels of a row per thread: bytes of the mask rows.
  // A border pixel (find_border_pixels, seg_utils.cu:164-195) is one with an edge to any of
  // its 4 neighbours; labels outside the image are staged as -1, so in-image pixels of the
  // image's edge rows and columns count as border pixels as in the reference.
  bool seed = false;
  {
    constexpr int kGrp = kLX / 8;
    const uint8_t* __restrict__ recchg = S.recchg;
    int sign = 0;
    for (int i = threadIdx.x; i < kGrp * kLY; i += NT) {
      const int r = i / kGrp, g = i - r * kGrp;
      const int* row = L + r * kLX + 8 * g;
      const int* below = r + 1 < kLY ? row + kLX : row;
      const int4 va = *(const int4*)row, vb = *(const int4*)(row + 4);
      const int4 da = *(const int4*)below, db = *(const int4*)(below + 4);
      const int v[9] = {va.x, va.y, va.z, va.w, vb.x, vb.y, vb.z, vb.w,
                        g + 1 < kGrp ? row[8] : vb.w};
      const int d[8] = {da.x, da.y, da.z, da.w, db.x, db.y, db.z, db.w};
      unsigned e = 0, s = 0;
#pragma unroll
      for (int q = 0; q < 8; q++) {
        e |= (unsigned)(v[q] != v[q + 1]) << q;
        s |= (unsigned)(v[q] != d[q]) << q;
        sign |= v[q];
      }
      ((uint8_t*)sm.edE[r])[g] = (uint8_t)e;
      ((uint8_t*)sm.edS[r])[g] = (uint8_t)s;
      if (mode) {
        unsigned q8 = ((const uint8_t*)sm.sin[r])[g];
        if (mode == 2) {
#pragma unroll
          for (int q = 0; q < 8; q++)
            q8 |= (unsigned)((unsigned)v[q] < (unsigned)cap && recchg[v[q]] != 0) << q;
        }
        ((uint8_t*)sm.seed[r])[g] = (uint8_t)q8;
        seed |= q8 != 0;
      }
    }
    if (sign < 0) sm.neg = 1;
    // bytes past the region's columns in a row's last word
    if (kGrp % 4)
      for (int r = threadIdx.x; r < kLY; r += NT)
#pragma unroll
        for (int g = kGrp; g < 4 * kCK; g++) {
          ((uint8_t*)sm.edE[r])[g] = 0;
          ((uint8_t*)sm.edS[r])[g] = 0;
          ((uint8_t*)sm.seed[r])[g] = 0;
        }
  }
  constexpr int kTW = TX / 16;
  if (!__syncthreads_or(seed || mode == 0)) {
    // nothing within reach changed: the tile keeps its labels, which seg_out holds
    for (int i = threadIdx.x; i < TY * kTW; i += NT) {
      const int gy = ty0 + i / kTW, wi = (tx0 >> 4) + i % kTW;
      if (gy < H && wi < P16) chg_out[(size_t)gy * P16 + wi] = 0;
    }
    return;
  }
  // --- the sweeps
  const float* __restrict__ img = S.img;
  const SweepRec* __restrict__ rec = S.rec;
  const bool neg = sm.neg != 0;
  // the grid of a phase: words, or quarters, of the rows of one y parity
  constexpr int kParts = kLY / 2 * 4 * kCK <= NT ? 4 : 1, kPartBits = 32 / kParts;
  constexpr int kRowParts = kParts * kCK, kItems = kLY / 2 * kRowParts;
  for (int s = 0; s < ns; s++) {
    const int cur = s & 1;
    const int G = kReach * (ns - s) - 1;
    // border mask at the sweep's start, inside the image and the tile grown by G; the
    // first sweep's dirty pixels
    bool any = false;
    for (int i = threadIdx.x; i < kWords; i += NT) {
      const int ay = i / kCK, c = i - ay * kCK;
      unsigned m = 0;
      if (ay >= max(kSH - G, -ry0) && ay < min(kSH + TY + G, H - ry0)) {
        const unsigned e = sm.edE[ay][c];
        m = e | (e << 1) | sm.edS[ay][c] | sm.edS[ay - 1][c];
        if (kCK > 1 && c > 0) m |= sm.edE[ay][c - 1] >> 31;
        m &= range32(max(kSH - G, -rx0), min(kSH + TX + G, W - rx0), c);
      }
      sm.bm[ay][c] = m;
      unsigned d = 0xffffffffu;
      if (s > 0) {
        d = sm.dirty[ay][c];
      } else {
        if (mode) {
          unsigned p = 0, w = 0, n = 0;
#pragma unroll
          for (int k = -1; k <= 1; k++) {
            const int r = ay + k;
            if (r < 0 || r >= kLY) continue;
            w |= sm.seed[r][c];
            if (kCK > 1 && c > 0) p |= sm.seed[r][c - 1];
            if (kCK > 1 && c + 1 < kCK) n |= sm.seed[r][c + 1 < kCK ? c + 1 : c];
          }
          d = w | __funnelshift_l(p, w, 1) | __funnelshift_r(w, n, 1);
        }
        sm.dirty[ay][c] = d;
      }
      any |= (m & d) != 0;
    }
    if (threadIdx.x < 4) sm.cnt[cur ^ 1][threadIdx.x] = 0;
    if (!__syncthreads_or(any)) break;   // nothing to score: nor in the later sweeps
    for (int ph = 0; ph < 4; ph++) {
      // the phase's pixels: dirty border pixels of the class ((x parity << 1) | y parity)
      // on the tile grown by G - ph, listed by a shared atomic per word, or quarter of a
      // word where the threads suffice (a warp scan first took 8 % of a launch more on a
      // 240x320 frame, 5 % on larger ones)
      const int g = G - ph;
      for (int i = threadIdx.x; i < kItems; i += NT) {
        const int ay = 2 * (i / kRowParts) + (ph & 1), h = i % kRowParts, w = h / kParts;
        if (ay < kSH - g || ay >= kSH + TY + g) continue;
        unsigned m = sm.dirty[ay][w] & sm.bm[ay][w] &
                     ((0xffffffffu >> (32 - kPartBits)) << (kPartBits * (h % kParts))) &
                     ((ph & 2) ? 0xAAAAAAAAu : 0x55555555u) & range32(kSH - g, kSH + TX + g, w);
        if (m) {
          atomicAnd(&sm.dirty[ay][w], ~m);
          int at = atomicAdd(&sm.cnt[cur][ph], __popc(m));
          for (const int ent = (ay << 8) | (32 * w); m; m &= m - 1)
            sm.list[at++] = (unsigned short)(ent + __ffs(m) - 1);
        }
      }
      __syncthreads();
      const int n = sm.cnt[cur][ph];
      if (!n) continue;                               // block-uniform
      if (n <= NT / 4) {                              // block-uniform
        if (8 * warp < n) sweep_quad<TX, TY, NS>(S, sm, rx0, ry0, n, s2, potts, lut_bits, neg);
        __syncthreads();
        continue;
      }
      for (int j = threadIdx.x; j < n; j += NT) {
        const int ent = sm.list[j];
        const int ax = ent & 255, ay = ent >> 8;
        const int gx = rx0 + ax, gy = ry0 + ay;
        const int p = ay * kLX + ax;
        // the loads first (colour, 3x3 labels, then the records of the first two
        // candidates: most border pixels have two), so their round trips overlap the
        // simple-point tests
        const float* pix = img + 3 * ((size_t)gy * W + gx);
        const float c0 = __ldg(pix), c1 = __ldg(pix + 1), c2 = __ldg(pix + 2);
        const int C = L[p];
        const int N = L[p - kLX], So = L[p + kLX], Wl = L[p - 1], E = L[p + 1];
        const int nb[8] = {L[p - kLX - 1], N, L[p - kLX + 1], Wl, E, L[p + kLX - 1], So,
                           L[p + kLX + 1]};
        // the distinct candidates in the order N, S, W, E (nothing to choose when every
        // neighbour took this pixel's label since the sweep began)
        const bool hS = So != N, hW = Wl != N && Wl != So, hE = E != N && E != So && E != Wl;
        const int nc = 1 + hS + hW + hE;
        if ((unsigned)C >= (unsigned)cap || (nc == 1 && N == C) || N >= cap || So >= cap ||
            Wl >= cap || E >= cap)
          continue;
        const int k1 = hS ? So : hW ? Wl : hE ? E : N;
        const int k2 = hS && hW ? Wl : E;
        const SweepRec r0 = load_rec(rec, max(N, 0));
        const SweepRec r1 = load_rec(rec, max(k1, 0));
        // simple-point codes of the candidates: bit i set when neighbour i
        // (NW,N,NE,W,E,SW,S,SE) carries the candidate or lies outside the image;
        // differing neighbours = 8 - popcount
        unsigned m1 = 0;
        if (neg) {                                    // block-uniform
#pragma unroll
          for (int q = 0; q < 8; q++) m1 |= (unsigned)(nb[q] == -1) << q;
        }
        auto code = [&](int v) {
          unsigned c = m1;
#pragma unroll
          for (int q = 0; q < 8; q++) c |= (unsigned)(nb[q] == v) << q;
          return c;
        };
        auto simple = [&](unsigned c) { return (lut_bits[c >> 5] >> (c & 31)) & 1u; };
        const unsigned d0 = code(N), d1 = code(k1);
        if (!(simple(d0) & simple(d1))) continue;
        unsigned d2 = 0, d3 = 0;
        if (nc > 2) {
          d2 = code(k2);
          if (!simple(d2)) continue;
          if (nc > 3) {
            d3 = code(E);
            if (!simple(d3)) continue;
          }
        }
        // (both scores in one straight line: their chains overlap)
        const float s0 = joint(c0, c1, c2, gx, gy, r0, s2, 8 - __popc(d0), potts);
        const float s1 = joint(c0, c1, c2, gx, gy, r1, s2, 8 - __popc(d1), potts);
        float best = -9999.f;
        int bl = C;
        if (N >= 0 && s0 > best) { best = s0; bl = N; }
        if (nc > 1 && k1 >= 0 && s1 > best) { best = s1; bl = k1; }
        if (nc > 2) {
          if (k2 >= 0) {
            const float t = joint(c0, c1, c2, gx, gy, load_rec(rec, k2), s2, 8 - __popc(d2), potts);
            if (t > best) { best = t; bl = k2; }
          }
          if (nc > 3 && E >= 0) {
            const float t = joint(c0, c1, c2, gx, gy, load_rec(rec, E), s2, 8 - __popc(d3), potts);
            if (t > best) { best = t; bl = E; }
          }
        }
        if (bl == C) {
          const int n_c = N == C ? r0.count : k1 == C ? r1.count : __ldg(&rec[C].count);
          if (n_c <= 2) {
            if (N >= 0) bl = N;
            else if (E >= 0) bl = E;
            else if (So >= 0) bl = So;
            else if (Wl >= 0) bl = Wl;
          }
        }
        if (bl != C) {
          L[p] = bl;
          const int wx = ax >> 5;
          const unsigned bit = 1u << (ax & 31);
          // its 3x3 is dirty
          const unsigned long long three = 7ull << ((ax & 31) + 31);   // bits 31.. = word wx
          const unsigned mid = (unsigned)(three >> 32), lo = (unsigned)three & 0x80000000u;
#pragma unroll
          for (int k = -1; k <= 1; k++) {
            atomicOr(&sm.dirty[ay + k][wx], mid);
            if (lo) atomicOr(&sm.dirty[ay + k][wx - 1], lo);
            if (bit >> 31) atomicOr(&sm.dirty[ay + k][wx + 1], 1u);
          }
          // and its four edges change (the pixels of a phase are never 4-neighbours, so
          // each edge has one writer; words are shared)
          atomicXor(&sm.edE[ay][wx], (C != E) != (bl != E) ? bit : 0u);
          atomicXor(&sm.edE[ay][(ax - 1) >> 5],
                    (C != Wl) != (bl != Wl) ? 1u << ((ax - 1) & 31) : 0u);
          atomicXor(&sm.edS[ay][wx], (C != So) != (bl != So) ? bit : 0u);
          atomicXor(&sm.edS[ay - 1][wx], (C != N) != (bl != N) ? bit : 0u);
          if (ay >= kSH && ay < kSH + TY && ax >= kSH && ax < kSH + TX)
            atomicOr(&sm.all[ay][wx], bit);
        }
      }
      __syncthreads();
    }
  }
  // --- write-back.  The pixels where seg_out is behind (mode 0: every pixel of the tile is
  // stored) are listed like a phase's, and a relabelled one moves its statistics
  // from the label it had at the launch's start to the one it has now.
  // (In one round: 16 rows at a time, three barriers and two memory round trips each, took
  // 4 % of a launch of 64x48 tiles more.)
  __syncthreads();
  if (deltas)
    for (int i = threadIdx.x; i < kDeltaTab * 13; i += NT)
      ((int*)&sm.delta)[i] = i < kDeltaTab ? -1 : 0;
  if (mode == 0)
    for (int i = threadIdx.x; i < TX * TY; i += NT) {
      const int x = i % TX + kSH, y = i / TX + kSH;
      const int gx = rx0 + x, gy = ry0 + y;
      if (gx < W && gy < H) seg_out[(size_t)gy * W + gx] = L[y * kLX + x];
    }
  // change words: word q of a tile row holds label-region columns kSH + 16 q ..
  for (int i = threadIdx.x; i < TY * kTW; i += NT) {
    const int y = i / kTW, q = i % kTW;
    const int gy = ty0 + y, wi = (tx0 >> 4) + q;
    if (gy < H && wi < P16) {
      const int b = kSH + 16 * q, c = b >> 5;
      const unsigned lo = sm.all[y + kSH][c];
      const unsigned hi = c + 1 < kCK ? sm.all[y + kSH][c + 1 < kCK ? c + 1 : c] : 0u;
      chg_out[(size_t)gy * P16 + wi] = (uint16_t)__funnelshift_r(lo, hi, b & 31);
    }
  }
  for (int i = threadIdx.x; i < TY * kCK; i += NT) {
    const int y = i / kCK + kSH, c = i % kCK;
    unsigned m = (sm.sin[y][c] & (mode ? range32(kSH, kSH + TX, c) : 0u)) | sm.all[y][c];
    if (m) {
      int at = atomicAdd(&sm.wcnt, __popc(m));
      for (const int ent = (y << 8) | (32 * c); m; m &= m - 1)
        sm.list[at++] = (unsigned short)(ent + __ffs(m) - 1);
    }
  }
  __syncthreads();
  const int nw = sm.wcnt;
  for (int j = threadIdx.x; j < nw; j += NT) {
    const int ent = sm.list[j];
    const int ax = ent & 255, ay = ent >> 8;
    const int gx = rx0 + ax, gy = ry0 + ay;
    const size_t g = (size_t)gy * W + gx;
    const int b = L[ay * kLX + ax];
    if (mode) seg_out[g] = b;
    if (deltas && ((sm.all[ay][ax >> 5] >> (ax & 31)) & 1u)) {
      const int o = seg_in[g];
      if (o != b) {
        const float* pix = img + 3 * g;
        delta_move(sm.delta, S.count, S.acc, o, b, gx, gy, tx0, ty0, __ldg(pix),
                   __ldg(pix + 1), __ldg(pix + 2));
      }
    }
  }
  if (deltas) {
    __syncthreads();
    delta_flush(sm.delta, S.count, S.acc, tx0, ty0);
  }
}

template <int TX, int TY, int NS, int NT>
__device__ __forceinline__ void sweep_flat(const Slot* __restrict__ slots, int B, int parity,
                                           int ns, float s2, float potts, int mode, int deltas) {
  extern __shared__ __align__(16) unsigned char sweep_smem[];
  SweepTile<TX, TY, NS>& sm = *(SweepTile<TX, TY, NS>*)sweep_smem;
  __shared__ unsigned lut_bits[8];
  if (threadIdx.x < 8) lut_bits[threadIdx.x] = c_simple_bits.w[threadIdx.x];
  constexpr int v = TY == 48 ? 3 : TX == 32 ? 0 : TX == 64 ? 1 : 2;   // the tile size (kGeomW)
  const int t = blockIdx.x;
  int lo = 0, hi = B - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (slots[mid].tile_base[v] <= t) lo = mid; else hi = mid - 1;
  }
  const SweepSlot S = sweep_slot(slots[lo], parity, v);
  const int tl = t - S.tile0;
  const int tiles_x = (S.W + TX - 1) / TX;
  sweep_tile<TX, TY, NS, NT>(S, tl % tiles_x, tl / tiles_x, ns, s2, potts, sm, lut_bits, mode,
                             deltas);
}

// Persistent work-queue form of the single-sweep launch: a resident set of blocks
// (the SM count times the blocks an SM holds, at most the tile count) takes the
// batch's tiles in index order from an atomic counter, queue[0], and sweeps each as
// the one-block-per-tile kernel does (the same labels: a launch reads only the labels
// at its start).  The last block to finish, counted in queue[1], sets both counters
// back to zero for the next launch (stream order and the dependent-launch wait make
// that store visible to it).  No block waits on another.
template <int TX, int TY>
__device__ __forceinline__ void sweep_queue(const Slot* __restrict__ slots, int B, int ntiles,
                                            unsigned* queue, int parity, float s2, float potts,
                                            int mode, int deltas) {
  __shared__ SweepTile<TX, TY, 1> sm;
  __shared__ unsigned lut_bits[8];
  __shared__ int next;
  if (threadIdx.x < 8) lut_bits[threadIdx.x] = c_simple_bits.w[threadIdx.x];
  const int v = TX == 32 ? 0 : TX == 64 ? 1 : 2;   // which tile_base of the slots
  for (;;) {
    if (threadIdx.x == 0) next = (int)atomicAdd(&queue[0], 1u);
    __syncthreads();
    const int t = next;
    if (t >= ntiles) break;
    int lo = 0, hi = B - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (slots[mid].tile_base[v] <= t) lo = mid; else hi = mid - 1;
    }
    const SweepSlot S = sweep_slot(slots[lo], parity, v);
    const int tl = t - S.tile0;
    const int tiles_x = (S.W + TX - 1) / TX;
    sweep_tile<TX, TY, 1, 256>(S, tl % tiles_x, tl / tiles_x, 1, s2, potts, sm, lut_bits, mode,
                               deltas);
    __syncthreads();          // the tile's shared memory and `next` are free again
  }
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&queue[1], 1u) == gridDim.x - 1) {
      queue[0] = 0u;
      queue[1] = 0u;
      __threadfence();
    }
  }
}

#define STSPIX_SWEEPQ_KERNEL(name, TX, MINB)                                                \
  __global__ void __launch_bounds__(256, MINB) name(const Slot* __restrict__ slots, int B,    \
                                                    int ntiles, unsigned* queue, int parity,  \
                                                    float s2, float potts, int mode,          \
                                                    int deltas) {                             \
    pdl_enter();                                                                             \
    sweep_queue<TX, 32>(slots, B, ntiles, queue, parity, s2, potts, mode, deltas);           \
  }
STSPIX_SWEEPQ_KERNEL(kb_sweepq_t32, 32, 4)
STSPIX_SWEEPQ_KERNEL(kb_sweepq_t64, 64, 4)
STSPIX_SWEEPQ_KERNEL(kb_sweepq_t16, 16, 4)
#undef STSPIX_SWEEPQ_KERNEL

// One block per tile of the batch (grid = the batch's total tile count), ns sweeps per
// launch: up to one (kb_sweep_t*), two (kb_sweep2_t*) or four (kb_sweep4_*, see the rule in
// update_seg).  Dynamic shared memory: the SweepTile (kb_sweep*_smem).
// mode: what the first sweep scores (see sweep_tile).  deltas 1: move the statistics of
// every relabelled tile pixel (incremental statistics: the sums of the labels at the
// call's start stay current); 0: not.
#define STSPIX_SWEEP_KERNEL(name, TX, TY, NS, NT, MINB)                                      \
  __global__ void __launch_bounds__(NT, MINB) name(const Slot* __restrict__ slots, int B,    \
                                                   int parity, int ns, float s2,             \
                                                   float potts, int mode, int deltas) {      \
    pdl_enter();                                                                             \
    sweep_flat<TX, TY, NS, NT>(slots, B, parity, ns, s2, potts, mode, deltas);               \
  }                                                                                          \
  int name##_smem() { return (int)sizeof(SweepTile<TX, TY, NS>); }
STSPIX_SWEEP_KERNEL(kb_sweep_t32, 32, 32, 1, 256, 4)
STSPIX_SWEEP_KERNEL(kb_sweep_t64, 64, 32, 1, 256, 4)
STSPIX_SWEEP_KERNEL(kb_sweep_t16, 16, 32, 1, 256, 4)
STSPIX_SWEEP_KERNEL(kb_sweep2_t32, 32, 32, 2, 256, 4)
STSPIX_SWEEP_KERNEL(kb_sweep2_t16, 16, 32, 2, 256, 4)
STSPIX_SWEEP_KERNEL(kb_sweep2_t64, 64, 32, 2, 256, 4)
STSPIX_SWEEP_KERNEL(kb_sweep4_s, 32, 32, 4, 512, 2)
STSPIX_SWEEP_KERNEL(kb_sweep4_t, 32, 32, 4, 256, 4)
STSPIX_SWEEP_KERNEL(kb_sweep4_m, 64, 32, 4, 256, 4)
STSPIX_SWEEP_KERNEL(kb_sweep4_l, 64, 48, 4, 256, 4)
#undef STSPIX_SWEEP_KERNEL

// ---------------------------------------------------------------------------
// Parameter read-out (read_params, sparams_io.cu:190-286) and prior update
// (update_prior_kernel, sparams_io.cu:584-640) into the caller's SoA params.
__global__ void kb_read_params(const Slot* __restrict__ slots) {
  pdl_enter();
  SLOT_Y;
  const SpDev& sp = S.sp;
  const stspix_params& out = S.pout;
  int n = S.sc->nspix;
  FOR_ID(i, min(n, min(out.capacity, sp.cap))) {
    bool upd = sp.count[i] > 0;
    for (int c = 0; c < 3; c++) {
      float m = sp.mu_app[3 * i + c];
      out.mu_app[3 * i + c] = m;
      out.prior_mu_app[3 * i + c] = upd ? m : sp.prior_mu_app[3 * i + c];
      double s = sp.sigma_shape[3 * i + c];
      out.sigma_shape[3 * i + c] = s;
      out.prior_sigma_shape[3 * i + c] = upd ? s : sp.prior_sigma_shape[3 * i + c];
      out.sample_sigma_shape[3 * i + c] = sp.sample_sigma_shape[3 * i + c];
    }
    for (int c = 0; c < 2; c++) {
      double m = sp.mu_shape[2 * i + c];
      out.mu_shape[2 * i + c] = m;
      out.prior_mu_shape[2 * i + c] = upd ? m : sp.prior_mu_shape[2 * i + c];
    }
    out.logdet_sigma_shape[i] = (float)sp.logdet[i];
    out.counts[i] = sp.count[i];
    out.invalid_counts[i] = sp.icount[i];
    out.sm_counts[i] = sp.sm_count[i];
    out.prior_counts[i] = sp.prior_count[i];
    out.ids[i] = i;
  }
}

// Frame start: counters, buffer sizes of the reference.  One thread per slot (the later steps
// of these scalars are done by the kernels beside them: a launch of its own took 2.3 us).
__global__ void kb_scalars(const Slot* __restrict__ slots, int B) {
  pdl_enter();
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= B) return;
  const Slot& S = slots[i];
  Scalars* sc = S.sc;
  sc->status = STSPIX_OK;
  sc->nsplits = sc->nmerges = sc->nrevived = sc->nminted = sc->near_ties = 0;
  sc->fill_iters = 0;
  sc->ninvalid = 0;
  sc->tmp0 = sc->tmp1 = sc->tmp2 = 0;
  sc->nspix = 0;
  if (S.mode) { sc->max_spix = S.n_prev - 1; sc->nbuf_logical = 10 * S.n_prev; }
  else { sc->max_spix = 0; sc->nbuf_logical = 30 * S.nraw; }
}

// flags := 0 (cap + 2 entries) before a presence scan.
__global__ void kb_clear_flags(const Slot* __restrict__ slots) {
  pdl_enter();
  SLOT_Y;
  FOR_ID(k, S.cap + 2) S.flags[k] = 0;
}

// Keep a copy of the finished labels where the slot's video stream resides.
__global__ void kb_save_prev(const Slot* __restrict__ slots) {
  pdl_enter();
  SLOT_Y;
  if (!S.resident_labels) return;
  FOR_PIX(i, S.npix) S.resident_labels[i] = S.seg[i];
}

// The labels back from seg_alt to seg after a launch that read seg: only the pixels that
// launch changed (change plane 0) differ.  A thread takes one 16-pixel change word.
__global__ void kb_copy_labels(const Slot* __restrict__ slots) {
  pdl_enter();
  SLOT_Y;
  const int W = S.W, P16 = (W + 15) >> 4;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= S.H * P16) return;
  unsigned m = ((const uint16_t*)S.chg[0])[i];
  if (!m) return;
  const int y = i / P16;
  const size_t g = (size_t)y * W + 16 * (i - y * P16);
  for (; m; m &= m - 1) {
    const int q = __ffs(m) - 1;
    S.seg[g + q] = S.seg_alt[g + q];
  }
}

__global__ void k_dump_state(SpDev sp, stspix_state_dump d) {
  pdl_enter();
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= sp.cap || k >= d.capacity) return;
  if (d.count) d.count[k] = sp.count[k];
  if (d.valid) d.valid[k] = sp.valid[k];
  if (d.prior_count) d.prior_count[k] = sp.prior_count[k];
  for (int c = 0; c < 3; c++) {
    if (d.mu_app) d.mu_app[3 * k + c] = sp.mu_app[3 * k + c];
    if (d.sigma_shape) d.sigma_shape[3 * k + c] = sp.sigma_shape[3 * k + c];
  }
  for (int c = 0; c < 2; c++)
    if (d.mu_shape) d.mu_shape[2 * k + c] = sp.mu_shape[2 * k + c];
  if (d.logdet) d.logdet[k] = sp.logdet[k];
  if (d.sums)
    for (int c = 0; c < 8; c++) d.sums[8 * (size_t)k + c] = sp.acc[8 * (size_t)k + c];
}

}  // namespace stspix
