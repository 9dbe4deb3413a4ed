// Internal declarations shared by the host runtime (gwl_capi.cu) and the
// kernel translation units.  Not part of the public ABI (include/gwlnl.h).
#pragma once

#include <cmath>
#include <cstddef>
#include <cstdint>
#include <vector>
#include <string>

#include <cuda_runtime.h>

#include "../../include/gwlnl.h"

namespace gwl {

constexpr int kMaxDet = GWL_MAX_DETECTORS;
constexpr int kPointsPerCta = 128;     // one thread per parameter point
constexpr int kChunkPlain = 256;       // bins per CTA, float64 kernels
constexpr int kChunkMixed = 512;       // bins per CTA, mixed-precision kernels
constexpr int kBinAlign = 16;          // chunk starts are multiples of this many bins
constexpr int kNumBasis = 8;           // TaylorF2 phase basis functions of f
constexpr int kPartStride = 6;         // partial-sum components per (group, detector, point)
constexpr int kAnchorStep = 8;         // bins between TaylorF2 phase anchors in the table
constexpr int kAnchorOrders = 7;       // Taylor orders 0..6 of the phase about an anchor
constexpr int kAnchorFF = 4;           // orders 0..3 kept in float-float
constexpr int kAnchorFloats = 96;      // per anchor: hi[7][8], lo[4][8], padding
constexpr int kChunksPerGroup = 4;     // chunks walked by one split-K CTA of the TaylorF2 mixed kernel
constexpr int kOrderMaxKeys = 4096;    // buckets of the point ordering by band end
constexpr int kDevStatusOk = 0;
constexpr int kDevStatusTimeout = 1;
constexpr int kDevStatusBadInput = 2;
constexpr int kDevStatusIndex = 3;  // checked builds (-DGWL_CHECK): an index check failed, the access was skipped
constexpr uint32_t kWaitLimit = 1u << 22;  // polls of a bulk-copy barrier before giving up
// Refinement of the TaylorF2 mixed-precision result (see LaunchArgs::rf_tol):
// the error bound of a point is kRefineL2 * L2 + kRefineL1 * L1, with L2 the
// Euclidean norm of its per-bin terms |<d|h>_k| and L1 their sum over the
// bins where the data are signal-dominated (whitened power 4 |d|^2 / (T S)
// above kRefineLoudPower).  The coefficients hold with a margin of 2.5 to 4
// over the measured error of the fast kernel on short, loud analyses.
constexpr double kRefineL2 = 1e-6;
constexpr double kRefineL1 = 1e-7;
constexpr double kRefineLoudPower = 10.0;
constexpr double kRefineDefaultTol = 5e-4;
constexpr int kCosTable = 1024;        // angles of the float-float cos / sin table of the accurate kernel
// Mixed TaylorF2: launch_mixed_few up to this many points x chunks x detectors, and
// from kFewMixedLong seconds on up to kFewMixedSpan (at 128 s) points x chunks.
// There its time grows with the work (a chunk costs about as much as four
// detectors' sums in it), the lane per point's hardly, and the less the longer the
// segment: its anchors get further apart.  Measured per call (us), few against one lane per
// point: 128 s at 4096 Hz, 3 detectors, 96 points 222 / 284, 201 points 394 / 318, 1
// detector, 145 points 173 / 181, 290 points 294 / 196; 128 s at 2048 Hz, 1 detector,
// 292 points 197 / 178, 585 points 347 / 189; 256 s at 2048 Hz, 2 detectors, 73 points 165 /
// 173, 146 points 273 / 196; 64 s at 2048 Hz, 1 detector, 585 points 213 / 229, 1170
// points 374 / 239.  Below, few wins up to the first limit with the masses whose inspirals
// fit the segment: 32 s at 4096 Hz, 1 detector, 1161 points 270 / 382; 8 s at 2048 Hz, 3
// detectors, 3072 points 127 / 238; 4 s at 1024 Hz, 2 detectors, 18432 points 302 / 387 (with 30 to
// 60 solar masses in 2 s, a band of some 60 bins, the lane per point wins from some
// 7000 points of three detectors on: 9216 points 180 / 157).
constexpr int64_t kFewMixedWork = 144 << 10;
constexpr double kFewMixedLong = 48.0, kFewMixedSpan = 75e3;
inline bool mixed_few(int64_t points, int64_t chunks, int detectors, double duration) {
  const int64_t n = points * chunks;
  if (points > 65535 || n * detectors > kFewMixedWork) return false;
  return duration < kFewMixedLong || (double)n * (0.8 + 0.2 * detectors) <= kFewMixedSpan * std::cbrt(128.0 / duration);
}
// Float64: one CTA per (chunk, point) up to this many points, or points x chunks.
// Measured: 128 s (1014 chunks), 8 points 95 / 129, 16 points 148 / 130; 32 s (255),
// 8 points 44 / 50, 16 points 55 / 51; 8 s (32), 64 points 51 / 57, 128 points 61 / 57.
constexpr int kFewWidePoints = 12;
constexpr int64_t kFewWideWork = 3200;
__host__ __device__ constexpr bool wide_few(int64_t points, int64_t chunks) {
  return points <= kFewWidePoints || points * chunks <= kFewWideWork;
}
// ... and ordered by band end from this many points x chunks on: the ordering costs
// 10 to 17 us and saves up to a quarter of the bins (8 s, 64 points 47 / 57).
constexpr int64_t kOrderWideWork = 32 << 10;
constexpr int kWideEnd = kNumBasis + 2 + 2 * kMaxDet, kWideWords = kWideEnd + 1;  // words per point of LaunchArgs::wide_c
constexpr int kExpTable = 256;         // entries 2^(-i / 256) of gwl_wide_sg.cu
constexpr int kWideTable = 2048;       // angles of the float-float cosine table of gwl_wide.cuh
constexpr int kRoqSplits = 8;          // node groups of the mixed ROQ time-marginalised matrix products

// Per-point quantities computed once per evaluation by the float64 prologue.
struct PointRec {
  double fp[kMaxDet], fx[kMaxDet], dt[kMaxDet];  // antenna patterns; (t_geo - t_start) + delay
  uint32_t xfix[kMaxDet][2];                     // frac(dt * df) as 0.64 fixed point {lo, hi}
  uint32_t qfix[kMaxDet][2];                     // TaylorF2 real-part kernel: arg(conj(Q_d)) / 2 pi, 0.64 fixed
  double qabs[kMaxDet];                          // |Q_d|, Q_d = Fp (1 + cos^2 i) / 2 - i Fx cos i
  double amp;          // TaylorF2 amplitude prefactor A0 | sine-Gaussian plus factor
  double amp2;         // sine-Gaussian cross factor
  double sg_f0, sg_a;  // sine-Gaussian centre frequency, pi^2 tau^2
  double m_sec, eta, f_isco, cos_i, phase, dist, jitter;
  double a[8], l[8];                 // TaylorF2 phase coefficients
  float c_hi[kNumBasis + 1];         // TaylorF2 phase basis coefficients in cycles (float-float)
  float c_lo[kNumBasis + 1];         // index kNumBasis: frac of the constant term
  int64_t k_start, k_end;            // TaylorF2 band [k_start, k_end) on the analysis grid
  int32_t valid;                     // 0: waveform undefined (lnL = nan_to_num(-inf))
  int32_t refine;                    // TaylorF2 mixed: error bound above the tolerance (LaunchArgs::rf_tol)
  // mixed time-marginalised kernel over the full grid (k_time_marg): per-point
  // scalars from the float64 prologue, so that the kernel runs no float64 per
  // point before its transform nor per time sample
  float tm_coef[2 * kMaxDet];        // detector response coefficients of the integrand
  double tm_hh;                      // TaylorF2 <h|h>
  int64_t tm_j0, tm_j1;              // FFT indices of the first and last time sample inside the prior
  int32_t tm_row_ly, tm_row_in;      // TaylorF2 with the distance table: the spline's row at this <h|h>
  float tm_row_hy[4];                // (SplineRowF: interval, inside the table, basis values)
  float tm_xp, tm_zs;                // the kernel's largest |X| over the window and ||z||_2, for the error bound
};

// Relative binning, per grid index: its bin and the offset of its frequency
// from the bin's centre.
struct RbBinF {
  int32_t bin;
  float x;
};

struct DetGeom {
  double vertex[3];
  double tensor[9];
  double start_time;
};

// Everything a kernel needs, passed by value.
struct LaunchArgs {
  int model, n_det, precision;
  int cplx;                             // TaylorF2 mixed: 1 = complex <d|h> partials, 0 = real part only
  int64_t B;
  int64_t n_bins, k_lo, k_hi, k_base;   // in-band hull [k_lo, k_hi); chunk origin k_base
  int64_t n_chunks;                     // chunks over [k_base, k_hi)
  int64_t n_groups;                     // CTAs along the bin axis; CTA g walks chunks g, g + G, ...
  int chunk;                            // bins per chunk
  double duration, step, fmin;
  int64_t k_fmin;                       // first bin with f >= minimum_frequency
  DetGeom det[kMaxDet];
  const double* freq;                   // [n_pad] float64 frequency array
  const float* freq_f;                  // [n_pad] float32 copy (sine-Gaussian mixed)
  const double* strain[kMaxDet];        // [2*n_pad] masked strain
  const double* inv_psd[kMaxDet];       // [n_pad] mask / S
  const float2* w[kMaxDet];             // [n_pad] mixed data weights (scaled)
  const uint2* wp[kMaxDet];             // [n_pad] TaylorF2: polar weights {float |w| bits, arg(w) 0.32 cycles}
  const uint4* wq[kMaxDet];             // [n_pad / 2] TaylorF2 fast kernel: per bin pair {|w| even, |w| odd,
                                        // tau even, tau odd}, tau = arg(w) at bins k % 8 == 0, else
                                        // arg(w_k) - arg(w_{k-1}) (0.32 cycles, wrapping)
  const float* v[kMaxDet];              // [n_pad] mixed inverse PSD (scaled)
  const float* v_lo[kMaxDet];           // [n_pad] sine-Gaussian: low words of the scaled inverse PSD (v + v_lo)
  const double* hh_prefix[kMaxDet];     // [n_bins + 1] TaylorF2 <h|h> prefix sums
  double w_scale[kMaxDet], v_scale[kMaxDet];
  const float2* basis;                  // [n_pad][kNumBasis] float-float phase basis
  const double4* ftab;                  // [n_pad] {f^(1/3), ln(f) / 3, f^(-5/3), f^(-7/6)} (float64 TaylorF2)
  // float64 TaylorF2 (gwl_wide.cu): the phase basis and the weights f^(-7/6) d / S
  // in fixed point and float-float, and per point the phase coefficients
  const uint4* wide_phi;                // [n_pad][kNumBasis / 2] two basis functions / wide_scale each, 0.58 fixed
                                        // point {low 27 bits, high 31 bits}
  double wide_wscale[kMaxDet];          // scale of wide_w
  double wide_norm;                     // factor of the sums: 4 / T, or 1 where the weights carry it
  int64_t wide_base, wide_chunks;       // first row of the tables and chunks of kChunkPlain rows from it on
  // rows that are not consecutive bins (multi-banding): per 32 rows the grid
  // index of the first and the stride; the bands {first row, rows, grid index,
  // stride}; prefix sums of f^(-7/3) times the quadratic coefficients.  nullptr:
  // row k is bin k
  const int2* wide_sub;
  const int4* wide_band;
  int wide_bands;
  const double* wide_q[kMaxDet];
  double rbw_scale[kMaxDet];            // relative binning: scale of the cross terms' weights (gwl_wide_relbin.cu)
  const float4* wide_tab;               // [kWideTable] {cos hi, lo, -2 pi / kWideTable sin hi, lo}
  const uint4* wide_w[kMaxDet];         // [n_pad] per bin pair {|w| / w_scale of both, hi words then lo (floats)},
                                        // {arg(w) of both, 0.64 cycles {lo, hi} each}
  const uint64_t* wide_v[kMaxDet];      // sine-Gaussian: [n_pad] mask / S, 0.64 fixed point of 2^wide_ve
  const int32_t* wide_ve[kMaxDet];      // ... [n_chunks * kChunkPlain / 32] its exponent per 32 bins from k_base on
  const uint64_t* wide_exp;             // sine-Gaussian: [kExpTable] 2^(-i / kExpTable), 0.64 fixed point
  double wide_scale[kNumBasis];         // powers of two above each basis function's largest value
  double wide_lnref;                    // ln f of the basis functions is ln f - wide_lnref
  double step_lo;                       // step + step_lo: the grid spacing to twice float64's digits
  uint64_t* wide_c;                     // [kWideWords][B]: c_b wide_scale_b 2^(58 - s), the constant, s + 2, per
                                        // detector the shift per bin and the offset (cycles, 64-bit fractions),
                                        // the grid index of f_ISCO, the grid continued;
                                        // sine-Gaussian: f0 in bins, sqrt(y) per bin, its shift with the fractional
                                        // bits of f0, the largest distance, per detector as above with beta
  const float* anchors;                 // [n_anchors][kAnchorFloats] Taylor tables of the basis
  int64_t n_anchors;
  const double* params;                 // [GWL_NPARAM][B]
  PointRec* rec;                        // [B]
  double* part;                         // [n_groups][n_det][kPartStride][B] (point fastest)
  double* out;                          // [B]
  double* dh_out;                       // optional [2B] complex <d|h> totals
  double* hh_out;                       // optional [B] <h|h> totals
  int* status;                          // device status word
  // error control of the TaylorF2 mixed-precision sums: the prologue bounds
  // each point's error from the prefix sums rf_p2 (|w|^2) and rf_p1 (|w| over
  // signal-dominated bins); a point whose bound exceeds rf_tol is marked
  // (PointRec::refine), counted in rf_count and ordered into the first slots,
  // which the accurate variant of the bin-walking kernel evaluates (float-float
  // cosine from cos_tab, TwoSum accumulation per bin).  rf_tol <= 0: off.
  const double* rf_p2[kMaxDet];         // [n_bins + 1]
  const double* rf_p1[kMaxDet];         // [n_bins + 1]
  double rf_tol;
  int* rf_count;                        // marked points of this analysis (zeroed with the ordering histogram)
  int* rf_total;                        // optional: marked points of the whole launch
  const float4* cos_tab;                // [kCosTable] {cos hi, cos lo, sin hi, sin lo} of 2 pi q / kCosTable
  // optional point ordering (TaylorF2 mixed): thread slot s of the bin-walking
  // kernel evaluates point order[s]; points are grouped by the chunk that
  // holds their band end, longest first, so that the 128 points of a CTA stop
  // at nearly the same bin.  nullptr: slot s evaluates point s.
  int32_t* order;                       // [B]
  int32_t* order_hist;                  // [2 * order_keys]: counts (then bases), cursors; zeroed before use
  int order_keys, order_shift;
  int order_half;                       // keys of marked points (PointRec::refine) are offset by this
  // marginalisation
  int time_marg, phase_marg, dist_marg, jitter;
  double t_min, t_max, delta_tc, start_time0;
  double tm_step, tm_inv_step, tm_prob, inv_ref_dist;  // T / L, L / T, 1 / (t_max - t_min), 1 / ref_dist
  int64_t n_fft;                        // time-marginalisation FFT length (n_bins - 1)
  const double* tx; const double* ty; const double* tc;  // distance spline
  const float* tx_f; const float* ty_f; const float* tc_f; // float32 copy (mixed precision)
  float bbox_x_f[2];                    // bbox[0] rounded up and bbox[1] rounded down to float32: the same
                                        // test of a float32 x as against the float64 bounds
  int nx, ny;
  double bbox[4];
  double ref_dist;
  double* tm_work;                      // time-marginalisation work space
  double* tm_series;                    // optional [B][2 n_fft] FFT of the integrand (float64 kernel)
  int tm_first;                         // time of FFT index j: start + (j + tm_first) * duration / n_fft
  int antenna_fixed;                    // antenna patterns at antenna_time instead of geocent_time
  double antenna_time;
  // relative binning: the model at the bin edges, its ratio to the fiducial
  // response, and the per-bin summary data of each detector
  int relbin;
  int rb_edges;
  const int64_t* rb_index;              // [rb_edges] grid index of each edge
  const double* rb_freq;                // [rb_edges] edge frequencies
  const double2* rb_h0inv[kMaxDet];     // [rb_edges] 1 / h0_d(f_e)
  const double* rb_sum[kMaxDet];        // [rb_edges - 1][6]: a0 re, a0 im, a1 re, a1 im, b0, b1
  // relative binning with time marginalisation: the full-grid weights
  // 4/T h0_d(f) conj(d(f)) / S(f) and the bin of each grid index in
  // [rb_index[0], rb_index[rb_edges - 1]]
  const double2* rb_g[kMaxDet];         // [n_bins]
  const int32_t* rb_bin;                // [rb_index[last] - rb_index[0] + 1]
  // ... and for the mixed-precision kernel, in the order it reads them
  // (window_relbin_order): the weights in float32, zero outside that span, and
  // per grid index its bin with f - (f_b + f_b+1) / 2
  const float2* rb_gf[kMaxDet];
  const RbBinF* rb_bx;
  int tw_refine_only;                   // float64 windowed time marginalisation: only the marked points
  float2* tw_scratch;                   // mixed windowed multi-banding: [tw_scratch_slots][mb_points] banded values
  int64_t tw_scratch_slots;
  int32_t* rf_list;                     // windowed mixed kernel: the marked points, [*rf_count]
  double* tw_part;                      // float64 recomputation: [tw_part_units][n_win_max + 1] complex shares
  int* tw_done;                         // ... finished units per marked point, [tw_part_units], zeroed before
  int64_t tw_part_units;
  // multi-banding: the model at the banded frequencies, weighted by the
  // per-detector linear (complex) and quadratic (real) coefficients
  int multiband;
  int64_t mb_points;
  const double* mb_freq;                // [mb_points] banded frequencies
  const double4* mb_pow;                // [mb_points] {f^(1/3), ln(f) / 3, f^(-5/3), f^(-7/6)}
  const double2* mb_lin[kMaxDet];       // [mb_points]
  const double* mb_quad[kMaxDet];       // [mb_points]
  int mb_bands;
  const int64_t* mb_band_start;         // [mb_bands + 1] first banded index of each band (and the end)
  const double* mb_band_df;             // [mb_bands] frequency spacing of each band
  // mixed precision: the float-float phase basis at the banded frequencies, the
  // linear coefficients times f^(-7/6) in float32 (scaled by mb_lw_scale), and
  // prefix sums of f^(-7/3) times the quadratic coefficients
  const float2* mb_basis;               // [mb_points][kNumBasis]
  const float2* mb_lw[kMaxDet];         // [mb_points]
  double mb_lw_scale[kMaxDet];
  // time marginalisation with a prior other than Uniform: its density on the
  // nodes t0 + g h (g < tm_prior_n, h a power of two), read by 4-node Lagrange
  // interpolation; tm_prior == nullptr means the Uniform density tm_prob
  const double* tm_prior;
  const float* tm_prior_f;
  int64_t tm_prior_n;
  double tm_prior_t0, tm_prior_inv_h;
  const double* mb_qprefix[kMaxDet];    // [mb_points + 1]
  const double* mb_l2prefix[kMaxDet];   // [mb_points + 1] prefix sums of |mb_lw|^2 (error bound of the mixed kernel)
  int mb_refine_only;                   // float64 multi-banding kernel: only the points marked by the mixed one
  // multi-banding with time marginalisation: for each full-resolution index
  // k < n_fft the banded points scattered there, mb_tm_src[mb_tm_ptr[k] ..
  // mb_tm_ptr[k + 1]); a code c >= 0 is banded point c, c < 0 is banded point
  // -c - 1 counted in <h|h> only (replaced at its index within its band)
  int mb_tm;
  const int32_t* mb_tm_ptr;             // [n_fft + 1]
  const int32_t* mb_tm_src;             // [mb_points]
  // multi-banding with the IFFT-FFT <h|h> (multiband.py:613-650, 760-779):
  // the odd-bin part of band b >= 1 of detector d at point i,
  // mb_fft_hh[(b * n_det + d) * B + i], written by k_mb_hh_fft before the
  // kernels that add it to <h|h> (band 0 is wholly in mb_quad); null without it
  const double* mb_fft_hh;
  // distance marginalisation without time marginalisation: a bound r_max =
  // d_ref / d_min on the lnL's slope E[d_ref / d] in <d|h> (and r_max^2 / 2 in
  // <h|h>), by which the mixed kernels scale their error bounds; values <= 1
  // (no distance table, or time marginalisation with its own sensitivities)
  // leave them as they are
  double dist_slope;
  // reduced-order quadrature: the model at the linear and quadratic nodes,
  // time-dependent linear weights on the grid (t_start + k) dt, k < n_time
  int roq;
  int roq_nl, roq_nq;
  int64_t roq_time_start, roq_n_time;
  double roq_dt;
  const double* roq_fl;                 // [roq_nl] linear nodes
  const double* roq_fq;                 // [roq_nq] quadratic nodes
  const double4* roq_pl;                // [roq_nl] TaylorF2 powers of the linear nodes
  const double4* roq_pq;                // [roq_nq] and of the quadratic nodes
  const double2* roq_wl[kMaxDet];       // [roq_n_time][roq_nl]
  const double* roq_wq[kMaxDet];        // [roq_nq]
  // ROQ with time marginalisation (roq.py:320-331, 535-541, 604-651): the
  // regular time grid of the marginalisation and the most weight rows one
  // point reads per detector; the prologue then stores in dt[d] the detector's
  // delay at antenna_time alone
  int roq_tm;
  int64_t roq_tm_n, roq_tm_chunk, roq_tm_rows;  // samples, samples per chunk, rows per chunk (at most)
  const double* roq_tm_times;           // [roq_tm_n]
  // ... in mixed precision, over one chunk of points [roq_c0, roq_c0 + roq_cn):
  // conj(h_d) at the linear nodes in float32, complex float32 matrix
  // products per detector over every weight row, the nodes split into
  // kRoqSplits groups of roq_ks (roq_d32[d][s] = roq_wl32 h over group s),
  // then per point the groups' sums in float-float and the per-sample
  // interpolation and marginalisation in float32
  const float2* roq_wl32[kMaxDet];      // [roq_n_time][roq_nl_pad] float32 copy of roq_wl, zero-padded
  float roq_wnorm[kMaxDet][kRoqSplits]; // per node group: largest Euclidean norm of a row of roq_wl
  int roq_nl_pad, roq_ks;               // kRoqSplits * roq_ks nodes (padded), roq_ks per group
  const int2* roq_tm_g;                 // [roq_tm_n] (t_j - start_0 - t_grid0) / dt: {floor, float fraction bits}
  float2* roq_h32;                      // [n_det][roq_cn][roq_nl_pad]
  float2* roq_d32;                      // [n_det][kRoqSplits][roq_cn][roq_n_time]
  double* roq_hh;                       // [roq_cn] <h|h>
  int64_t roq_c0, roq_cn;
  int rf_list_only;                     // float64 ROQ time marginalisation of the listed points alone
  const float4 *wide_tm_tw, *wide_tm_spec;  // time marginalised: TmPlan::tw, spec (gwl_wide_tm.cu)
};

// A batch over several analyses evaluated by one persistent launch: per item
// (one analysis and its points) a LaunchArgs; work units (item, point tile,
// chunk group) are pulled by the persistent CTAs from an atomic counter.
struct MultiArgs {
  const LaunchArgs* args;   // [n_items]
  const int64_t* offsets;   // [n_items + 1] first global point of each item
  int n_items;
  int64_t total_points;
  const int4* units;        // [n_units] {item, tile, group, 0}, grouped by kernel class
  int64_t unit_begin[9];    // units of class q = 2 D + cplx: [unit_begin[q], unit_begin[q + 1])
  int* counter;             // [kMultiCounters], zeroed before the launch: units taken per class by the
                            // fast kernels, then by the accurate kernels, then the marked points
  int ordered;              // items carry a point ordering (LaunchArgs::order)
};

// One compiled prior (gwl_priors_create): device copy of a gwl_prior with
// device table pointers.
struct PriorEntry {
  int kind, target, column, table_n;
  double p[4];
  const double* x;
  const double* y;
};

// A second, high-priority stream on which the accurate kernel runs beside the
// fast one: forked from the launching stream after the ordering and joined
// before the reduction (both capturable in a CUDA graph).
struct SideStream {
  cudaStream_t stream = nullptr;
  cudaEvent_t fork = nullptr, join = nullptr;
};
cudaError_t side_stream_create(SideStream* s);
void side_stream_destroy(SideStream* s);
cudaError_t side_fork(SideStream& side, cudaStream_t s);   // side waits for the work enqueued so far on s
cudaError_t side_join(SideStream& side, cudaStream_t s);   // s waits for the work enqueued so far on side

// Kernel launchers (defined in gwl_kernels.cu / gwl_marg.cu).
constexpr int kMultiMaxDet = 3;
constexpr int kMultiClasses = 2 * (kMultiMaxDet + 1);  // kernel class q = 2 * detectors + cplx
constexpr int kMultiCounters = 2 * kMultiClasses + 1;  // unit counters (fast, accurate), then the marked points
cudaError_t launch_multi(const MultiArgs& m, const int* ctas, const int* ctas_acc, cudaStream_t s, SideStream* side);
int multi_tf2_ctas_per_sm(int q, bool acc);
cudaError_t launch_prologue(const LaunchArgs& a, cudaStream_t s);
// The float64 likelihood (gwl_wide.cu, gwl_wide_sg.cu): partial sums, totals and lnL.
cudaError_t launch_wide(const LaunchArgs& a, cudaStream_t s);
cudaError_t launch_wide_sg(const LaunchArgs& a, cudaStream_t s);
// Relative binning: rows are the bin edges, pairs of wide_w {|w|, m} and {arg w,
// arg of the neighbours' ratio}, wide_q prefix sums over the edges.
cudaError_t launch_wide_relbin(const LaunchArgs& a, cudaStream_t s);
// Their tables: the basis functions of rows [k0, n) of f (zero where f <= 0 and
// outside), the weights z u f^(-7/6) inv_scale of n (even) rows (powers of f from
// ftab, none without it).
cudaError_t launch_wide_basis(const double* f, int64_t k0, int64_t n, int64_t pad, double lnref, const double* scale,
                              uint4* out, cudaStream_t s);
cudaError_t launch_wide_weights(const double2* z, const double* u, const double4* ftab, double inv_scale, int64_t n,
                                uint4* out, cudaStream_t s);
cudaError_t launch_mixed(const LaunchArgs& a, cudaStream_t s);
// Few points of TaylorF2 in mixed precision, totals and lnL included (no ordering).
cudaError_t launch_mixed_few(const LaunchArgs& a, cudaStream_t s);
// The accurate kernel for the marked points (nothing when rf_tol <= 0).
cudaError_t launch_mixed_acc(const LaunchArgs& a, cudaStream_t s);

cudaError_t launch_finalize(const LaunchArgs& a, cudaStream_t s);
cudaError_t launch_sg_refine(const LaunchArgs& a, cudaStream_t s);
cudaError_t launch_order(const LaunchArgs& a, cudaStream_t s);
cudaError_t launch_relbin(const LaunchArgs& a, cudaStream_t s);
cudaError_t launch_multiband(const LaunchArgs& a, cudaStream_t s);
cudaError_t launch_multiband_mixed(const LaunchArgs& a, cudaStream_t s);
cudaError_t launch_roq(const LaunchArgs& a, cudaStream_t s);
cudaError_t launch_roq_time_marginalized(const LaunchArgs& a, cudaStream_t s);
// Mixed ROQ time marginalisation of one chunk: the node values before the
// matrix products, the interpolation and marginalisation after them.
constexpr int64_t kRoqMixedChunk = 1024;  // points per chunk
// whether the mixed kernel's shared memory (rows of every detector, spline knots) fits
bool roq_tm_mixed_fits(const LaunchArgs& a);
cudaError_t launch_roq_nodes32(const LaunchArgs& a, cudaStream_t s);
cudaError_t launch_roq_tm_mixed(const LaunchArgs& a, cudaStream_t s);
void order_layout(int64_t n_chunks, int* keys, int* shift);
// Ordering of a mixed TaylorF2 launch: the band-end keys, doubled when points
// can be marked for the accurate kernel (rf_tol > 0; their keys take the upper
// half); the marked count follows the 2 * order_keys histogram words (zeroed
// with them: 2 * order_keys + 1 words in all).  order_hist, if set, must hold them.
void ordering_with_marks(LaunchArgs& L);
void ordering_by_peak(LaunchArgs& L);
cudaError_t launch_time_marginalized(const LaunchArgs& a, cudaStream_t s);
// ... float64 TaylorF2 over the full grid (gwl_wide_tm.cu), where the prior
// window's samples fit its convolution and no series is requested
bool wide_tm_fits(const LaunchArgs& a);
// ... its tables for the analysis's time prior (LaunchArgs::wide_tm_tw, wide_tm_spec; nullptr where the window
// does not fit), on the device when it returns
cudaError_t wide_tm_tables(const LaunchArgs& a, cudaStream_t s, const float4** tw, const float4** spec);
cudaError_t launch_wide_tm(const LaunchArgs& a, cudaStream_t s);
// The mixed full-grid time-marginalised kernel's error bounds, from what it
// stored in the point records: marks the points over the tolerance.
cudaError_t launch_time_marg_marks(const LaunchArgs& a, cudaStream_t s);
// Relative binning / multi-banding with time marginalisation by the windowed
// four-step transform (gwl_marg_window.cu): whether this launch's shared
// memory fits, and the launch (mixed precision: relative binning only).
bool time_marg_window_fits(const LaunchArgs& a);
// the grid index at each position of the mixed relative-binning tables (-1: none);
// false where that kernel does not take the length
bool window_relbin_order(int64_t n_fft, std::vector<int32_t>* order);
bool time_marg_window_mixed_ready(const LaunchArgs& a);  // the mixed kernel's tables and work space are there
bool time_marg_window_refine_fits(const LaunchArgs& a);  // the float64 recomputation of marked points fits
int64_t time_marg_window_slots();                        // work-space slots of the mixed multi-banding kernel
// bytes per unit of the float64 recomputation's shares (0: the window does not fit)
size_t time_marg_window_share_bytes(const LaunchArgs& a);
cudaError_t launch_time_marg_window(const LaunchArgs& a, cudaStream_t s);
// FFT lengths the time-marginalised kernels take: L = m 2^p with m odd,
// m <= kTmMaxOddFactor and p >= 4 (m and p returned)
constexpr int kTmMaxOddFactor = 127;
bool fft_length_supported(int64_t L, int* m_odd, int* log2N);
size_t time_marg_work_bytes(const LaunchArgs& a);
// Multi-banding with the IFFT-FFT <h|h> (gwl_mb_fft.cu): one band's odd-bin
// transform.  Transforms of at most 2^kMbFftSmemLog2 samples run in shared
// memory, longer ones in a global slot of 2^log2m double2 per CTA.
constexpr int kMbFftSmemLog2 = 13;
struct MbFftBand {
  int band;                      // b >= 1
  int ks;                        // K_s: grid index of the band's first banded point
  int log2m;                     // M = Mbs[b] = 2^log2m samples
  int log2m_max;                 // twiddle table length 2^log2m_max >= M
  int in_smem;                   // 1: the transform in shared memory
  double scale;                  // 4 / That_b
  const double* odd[kMaxDet];    // [M / 2] Re I_(2j+1) of each detector
  const double* sqrtw;           // [mb_points] square roots of the band windows
  const double2* tw;             // [2^(log2m_max + 1)] exp(-i pi k / 2^log2m_max)
  double* out;                   // the mb_fft_hh slab
  // float64 kernel: only the listed points (list_count of them), or all
  const int32_t* list;
  const int32_t* list_count;
  // float32 kernel (TaylorF2, mixed precision): the twiddles in float32, the
  // banded amplitude table sqrt(w_k) f_k^(-7/6) / aw_scale, and the error slab
  // (same layout as out)
  const float2* tw32;
  const float* aw;
  double aw_scale;
  const float2* odd32[kMaxDet];  // [M / 2] float-float Re I_(2j+1) / odd32_scale
  double odd32_scale;            // the band's largest |Re I_(2j+1)|
  double* err;
};
size_t mb_hh_fft_smem(int log2m);  // dynamic shared memory of a float64 transform in shared memory, 0 if it does not fit
bool mb_hh_fft32_in_smem(int log2m);
// one band's transforms: float64 (mixed = false; all points or the listed
// ones) or float32 with the error bound (mixed = true); scratch holds
// scratch_slots slots of 2^log2m complex values of that precision
cudaError_t launch_mb_hh_fft(const LaunchArgs& a, const MbFftBand& band, void* scratch, int64_t scratch_slots,
                             bool mixed, cudaStream_t s);
// the points whose float32 error, summed over bands and detectors, exceeds tol
cudaError_t launch_mb_fft_marks(const LaunchArgs& a, const double* err, double tol, int32_t* list, int32_t* count,
                                cudaStream_t s);
cudaError_t launch_source_polarizations(int model, const double* freq, int64_t n, const double* params,
                                        double fmin, double* plus, double* cross, cudaStream_t s);
cudaError_t launch_detector_response(const DetGeom& g, const double* freq, int64_t n, const double* plus,
                                     const double* cross, const double* params, double* resp, cudaStream_t s);

cudaError_t launch_distance_table(const double* dh_axis, int n_dh, const double* hh_axis, int n_hh,
                                  const double* scaling, const double* scaling2, const double* weight, int n,
                                  double* lni0_work, int phase, double log_norm, double* table);
cudaError_t launch_wait_selftest(uint32_t limit, int* status, int* arrived, cudaStream_t s);
cudaError_t launch_set_status(int* status, int value, cudaStream_t s);

void set_error(const std::string& msg);
int noalloc_launch_args(gwl_analysis* a, int64_t B, LaunchArgs* L, size_t* rec_bytes, size_t* part_bytes);

}  // namespace gwl
