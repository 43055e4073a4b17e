// Kernel declarations of the GB300 streaming-BASS engine.
//
// kb_* kernels are batched: they take the device array of slots (one frame each)
// and pick their slot from the launch's y dimension (z for 3-D grids; x for the
// one-block-per-slot kb_scan).  k_* kernels serve the stand-alone
// utility entry points.
#pragma once
#include "engine.h"

namespace stspix {

// k_bass.cu
__global__ void k_init_hex(int* seg, int H, int W, double Hh, double w, int nx, int ny);
__global__ void k_find_border(const int* seg, uint8_t* border, int H, int W);
__global__ void k_find_border_end(const int* seg, uint8_t* border, int H, int W, int nframes);
constexpr int kMarkPix = 1024;            // pixels per block of k_marked (256 threads)
__global__ void k_marked(float* out, const float* vid, const int* spix, const float* color, int H,
                         int W, long long n);
__global__ void k_dump_state(SpDev sp, stspix_state_dump d);

__global__ void kb_scalars(const Slot* slots, int B);
__global__ void kb_init_hex(const Slot* slots);
__global__ void kb_clear_flags(const Slot* slots);
__global__ void kb_mark_present(const Slot* slots, int mode);
__global__ void kb_scan(const Slot* slots, int mode);
__global__ void kb_remap(const Slot* slots, int mode);
__global__ void kb_compact_gather(const Slot* slots);
__global__ void kb_compact_scatter(const Slot* slots);
__global__ void kb_init_bass_params(const Slot* slots);
__global__ void kb_init_prior_mu(const Slot* slots);
__global__ void kb_clear_stats(const Slot* slots, int all);
__global__ void kb_accumulate(const Slot* slots, int B);
__global__ void kb_posterior(const Slot* slots, int incremental, int log64, int merged);
__global__ void kb_accumulate_fp(const Slot* slots, int mode);
__global__ void kb_accumulate_fp_store(const Slot* slots, int mode);
__global__ void kb_accumulate_fp_clear(const Slot* slots);
__global__ void k_label_stats(const float* img, const int* lab, long long npix, int n, int mode,
                              long long* iacc, float* facc, double* dacc);
__global__ void k_label_stats_out(int n, int mode, const long long* iacc, const float* facc,
                                  const double* dacc, double* out);
__global__ void kb_store_sample(const Slot* slots);
__global__ void kb_find_border(const Slot* slots);
// boundary sweeps, one block per tile of the batch, ns sweeps per launch: 1 (kb_sweep_t*:
// 32x32, 64x32 and 16x32 tiles), up to 2 (kb_sweep2_t*), up to 4 (kb_sweep4_*: 32x32 tiles
// of 512 threads, 64x32 and 64x48 tiles of 256); name_smem: dynamic shared memory in bytes
#define STSPIX_DECL_SWEEP(name)                                                             \
  __global__ void name(const Slot* slots, int B, int parity, int ns, float s2, float potts, \
                       int mode, int deltas);                                               \
  int name##_smem();
STSPIX_DECL_SWEEP(kb_sweep_t32)
STSPIX_DECL_SWEEP(kb_sweep_t64)
STSPIX_DECL_SWEEP(kb_sweep_t16)
STSPIX_DECL_SWEEP(kb_sweep2_t32)
STSPIX_DECL_SWEEP(kb_sweep2_t64)
STSPIX_DECL_SWEEP(kb_sweep2_t16)
STSPIX_DECL_SWEEP(kb_sweep4_s)
STSPIX_DECL_SWEEP(kb_sweep4_t)
STSPIX_DECL_SWEEP(kb_sweep4_m)
STSPIX_DECL_SWEEP(kb_sweep4_l)
#undef STSPIX_DECL_SWEEP
// the single sweep as a persistent work-queue kernel (queue: 2 counters, zero between
// launches)
__global__ void kb_sweepq_t32(const Slot* slots, int B, int ntiles, unsigned* queue, int parity,
                              float s2, float potts, int mode, int deltas);
__global__ void kb_sweepq_t64(const Slot* slots, int B, int ntiles, unsigned* queue, int parity,
                              float s2, float potts, int mode, int deltas);
__global__ void kb_sweepq_t16(const Slot* slots, int B, int ntiles, unsigned* queue, int parity,
                              float s2, float potts, int mode, int deltas);
__global__ void kb_copy_labels(const Slot* slots);
__global__ void kb_read_params(const Slot* slots);
__global__ void kb_save_prev(const Slot* slots);

// k_splitmerge.cu
__global__ void kb_split_clear(const Slot* slots);
__global__ void kb_bbox(const Slot* slots);
__global__ void kb_split_bfs(const Slot* slots, int dir_bass, int dir_prop);
__global__ void kb_split_bfs_big(const Slot* slots, int dir_bass, int dir_prop);
__global__ void kb_sm_accumulate(const Slot* slots);
__global__ void kb_sq_accumulate(const Slot* slots);
__global__ void kb_split_decide(const Slot* slots, SmConsts K, float split_alpha);
__global__ void kb_split_commit(const Slot* slots);
__global__ void kb_split_apply(const Slot* slots);
__global__ void kb_merge_clear(const Slot* slots);
__global__ void kb_merge_candidates(const Slot* slots, int dir_bass, int dir_prop, int use_border);
__global__ void kb_merge_single(const Slot* slots, SmConsts K);
__global__ void kb_merge_decide(const Slot* slots, SmConsts K, float merge_alpha);
__global__ void kb_merge_flag(const Slot* slots);
__global__ void kb_merge_remove(const Slot* slots);
__global__ void kb_merge_apply(const Slot* slots, int sums);

// k_prop.cu
__global__ void kb_prop_clear(const Slot* slots);
__global__ void kb_flow_pool(const Slot* slots);
__global__ void kb_flow_mean(const Slot* slots);
__global__ void kb_shift(const Slot* slots);
__global__ void kb_shift_decode(const Slot* slots);
__global__ void kb_count_labels(const Slot* slots, int which);
__global__ void kb_fill(const Slot* slots, int break_iter, cudaGraphConditionalHandle cond);
__global__ void kb_fill_phase(const Slot* slots, int ph, int B, cudaGraphConditionalHandle cond,
                              int break_iter, int* body_iters, unsigned* ctr);
__global__ void kb_cc_local(const Slot* slots);
__global__ void kb_cc_hook(const Slot* slots);
__global__ void kb_cc_compress(const Slot* slots);
__global__ void kb_list_holes(const Slot* slots);
__global__ void kb_cc_best(const Slot* slots);
__global__ void kb_cc_invalidate(const Slot* slots);
__global__ void kb_shift_params(const Slot* slots);
__global__ void kb_write_params(const Slot* slots);
__global__ void kb_mark_active(const Slot* slots);
__global__ void kb_relabel_init(const Slot* slots);
__global__ void kb_living(const Slot* slots);
__global__ void kb_relabel_compare(const Slot* slots);
__global__ void kb_relabel_mark(const Slot* slots, float thresh_replace, float thresh_new);
__global__ void kb_relabel_ids(const Slot* slots);
__global__ void kb_relabel_params(const Slot* slots);
__global__ void kb_relabel_apply(const Slot* slots);

// k_color.cu
__global__ void k_rgb2lab(const float* rgb, float* lab, long long npix, int first_blue,
                          int nan_copy);
__global__ void kb_lab_ingest(const Slot* slots);
__global__ void k_lab2rgb(const float* lab, float* rgb, long long npix);
__global__ void k_rescale_u8(const uint8_t* in, float* out, long long nvals, float mval);

// k_quality.cu
constexpr int kQUesaIds = 4;              // ids per thread of k_q_uesa
__global__ void k_q_range_init(int* mm);
__global__ void k_q_range(const int32_t* a, const int32_t* b, long long n, int* mm);
__global__ void k_q_accum(const float* vid, const int32_t* spix, const int32_t* gt, long long npix,
                          int H, int W, int off, int S, int G1, int* cnt, double* fsum, int* J);
__global__ void k_q_count(const int32_t* spix, long long npix, int H, int W, int off, int S,
                          int* cnt);
__global__ void k_q_id_time(const int* cnt, const double* fsum, int T, int S, long long* ntot,
                            double* std_out, double* vsum);
__global__ void k_q_mean(const int* cnt, const double* fsum, int S, double* mean, double* msum);
__global__ void k_q_resid(const float* vid, const int32_t* spix, int npix, int off, int S,
                          const double* mean, double* sse);
__global__ void k_q_frame_ids(const int* cnt, const double* fsum, const double* mean,
                              const double* vsum, const long long* ntot, const double* msum, int S,
                              int npix, unsigned long long* live, double* pool2, double* cross,
                              double* pool3);
__global__ void k_q_uesa(const int* cnt, const int* J, const long long* ntot, int T, int S, int G1,
                         unsigned long long* ue, unsigned long long* sa, unsigned long long* size,
                         unsigned long long* ue3, unsigned long long* sa3);
__global__ void k_q_down(const int* mm, int S, const int* cnt, const double* fsum, long long TS,
                         float* down);

// k_legacy.cu
__global__ void k_fill_i32(int32_t* p, long long n, int32_t v);
__global__ void k_lshift(const int32_t* spix, const int32_t* flow, int nspix, int H, int W,
                         int32_t* shifted, int32_t* counts);
__global__ void k_lfill_border(const int32_t* seg, const int32_t* missing, int nmissing, int H,
                               int W, uint8_t* border, int* num_neg);
__global__ void k_lfill_phase(int32_t* seg, const float* centers, int ncenters,
                              const int32_t* missing, const uint8_t* border, int nmissing, int H,
                              int W, int xm, int ym);
__global__ void k_vpool_accum(const float* img, const int32_t* seg, int T, long long npix, int F,
                              int nspix, double* sum, unsigned long long* cnt);
__global__ void k_vpool_mean(const double* sum, const unsigned long long* cnt, long long nbs,
                             int F, float* down, float* counts);
__global__ void k_vpool_write(const float* down, const int32_t* seg, int T, long long npix, int F,
                              int nspix, float* pooled);
__global__ void k_q_pool_write(const int* mm, const int32_t* spix, int npix, int S, long long n,
                               const float* down, float* pooled);
__global__ void k_lmark_ids(const int32_t* spix, long long n, int nids, uint8_t* present);
__global__ void k_lupdate_prior(const uint8_t* present, int nids, int prev_nspix, int invert,
                                const float* mu_app, float* prior_mu_app, const double* mu_shape,
                                double* prior_mu_shape, const double* sigma_shape,
                                double* prior_sigma_shape);
__global__ void k_lshift_tensor(const float* in, const int32_t* spix, const int32_t* flow, int H,
                                int W, int F, int nspix, const int32_t* selected, double* acc,
                                int32_t* counts, uint8_t* contributors);
__global__ void k_round_f32(const double* acc, long long n, float* out);
__global__ void k_lshift_order(const uint8_t* contributors, long long npix_all, int nspix,
                               int32_t* selected);
__global__ void k_lsd_init(int32_t* parent, int npix);
__global__ void k_lsd_hook(const int32_t* spix, int H, int W, int32_t* parent, int* status);
__global__ void k_lsd_roots(int32_t* parent, int npix, int32_t* is_root);
__global__ void k_lscan(const int32_t* in, int n, int32_t* out, int32_t* total);
__global__ void k_lsd_regions(const int32_t* spix, const int32_t* root, const int32_t* rank,
                              int npix, int nspix, int32_t* region_of, int32_t* region_spix,
                              int32_t* region_size, int32_t* spix_counts);
__global__ void k_lsd_starts(const int32_t* spix_counts, int nspix, int32_t* split_starts,
                             int32_t* max_nsplits);
__global__ void k_lsd_offsets(const int32_t* region_spix, const int32_t* region_size,
                              int nregions, int nspix, int32_t* region_offset);
__global__ void k_lsd_update(int32_t* spix, const int32_t* region_of,
                             const int32_t* region_offset, const int32_t* split_starts, int npix,
                             int nspix, int max_nchild, int32_t* children);

}  // namespace stspix
