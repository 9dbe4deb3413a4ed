// Float64 TaylorF2 with time marginalisation (bilby/gw/likelihood/base.py:
// 325-330, 794-820, 1027-1035) on the 32-bit pipes.
//
// The samples inside the geocent_time prior are a few hundred of the
// transform's L, and the signal's bins [ks, ke) a few hundred to a few thousand:
//   X[j] = sum_k z_k e^{-2 pi i j k / L},  j = j0 + n,  k = k0 + m,
// is a convolution with a chirp (Bluestein): with n m = (n^2 + m^2 - (n - m)^2) / 2
//   X[j0 + n] = e^{-pi i (2 n k0 + n^2) / L} sum_m Y_m e^{pi i (n - m)^2 / L},
//   Y_m = z_m e^{-pi i (2 j0 (k0 + m) + m^2) / L},
// two transforms of length M >= samples + bins instead of one of length L, in
// shared memory.  Bands longer than the convolution takes go block by block.
// The phases of Y_m are exact fixed-point sums with the waveform's, the
// transforms float-float: {hi.re, hi.im, lo.re, lo.im} per element.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <type_traits>

#include "gwl_device.cuh"
#include "gwl_device_cache.h"
#include "gwl_internal.h"
#include "gwl_marg_common.cuh"
#include "gwl_math.cuh"
#include "gwl_wide.cuh"

namespace gwl {

constexpr int kTmMinLog = 10, kTmMaxLog = 13;

// The convolution's plan: M = 2^log2m, at most cap samples, so bins m with
// n - m in [cap - M, cap): kb = M - cap (even) of them per block.
struct TmPlan {
  int log2m, cap, kb;
  const float4* tw;    // [M] e^{-2 pi i q / M}, {cos hi, cos lo, sin hi, sin lo}
  const float4* spec;  // [M] the chirp's transform / M, in the order the forward passes leave
  uint64_t inv, inv_lo;  // 2^128 / (2 L): cycles per unit of an integer mod 2 L
};

// a complex float-float: h = (re, im) high words, l the low words
struct cff {
  float2 h, l;
};
__device__ __forceinline__ cff as_cff(const float4& v) { return cff{make_float2(v.x, v.y), make_float2(v.z, v.w)}; }
__device__ __forceinline__ float4 as_float4(const cff& v) { return make_float4(v.h.x, v.h.y, v.l.x, v.l.y); }

__device__ __forceinline__ cff operator+(const cff& a, const cff& b) {
  cff r;
  float2 e;
  two_sum2(a.h, b.h, r.h, e);
  r.l = add2(add2(a.l, b.l), e);
  return r;
}
__device__ __forceinline__ cff operator-(const cff& a, const cff& b) {
  cff r;
  r.h = sub2(a.h, b.h);
  const float2 bb = sub2(r.h, a.h);
  const float2 e = sub2(sub2(a.h, sub2(r.h, bb)), add2(b.h, bb));
  r.l = add2(sub2(a.l, b.l), e);
  return r;
}
__device__ __forceinline__ float2 turn(float2 a) { return make_float2(a.y, -a.x); }  // times -i
__device__ __forceinline__ cff turn(const cff& a) { return cff{turn(a.h), turn(a.l)}; }
// a (c + i s), t = {c hi, c lo, s hi, s lo}; CONJ: a (c - i s)
template <bool CONJ>
__device__ __forceinline__ cff twiddle(const cff& a, const float4& t) {
  const float sh = CONJ ? t.z : -t.z, sl = CONJ ? t.w : -t.w;
  // a (c + i s) = c a - s (-i a)
  const cff b = turn(a);
  const float2 p = mul2(a.h, splat2(t.x)), q = mul2(b.h, splat2(sh));
  float2 e = fma2(a.h, splat2(t.x), mul2(p, splat2(-1.f)));
  float2 f = fma2(b.h, splat2(sh), mul2(q, splat2(-1.f)));
  e = fma2(a.h, splat2(t.y), e);
  f = fma2(b.h, splat2(sl), f);
  e = fma2(a.l, splat2(t.x), e);
  f = fma2(b.l, splat2(sh), f);
  cff r;
  float2 g;
  two_sum2(p, q, r.h, g);
  r.l = add2(add2(e, f), g);
  return r;
}
// a / sqrt(2)
__device__ __forceinline__ cff root_half(const cff& a) {
  constexpr float ch = 0.7071067690849304f, cl = 1.2101617485882343e-08f;
  cff r;
  r.h = mul2(a.h, splat2(ch));
  float2 e = fma2(a.h, splat2(ch), mul2(r.h, splat2(-1.f)));
  e = fma2(a.h, splat2(cl), e);
  r.l = fma2(a.l, splat2(ch), e);
  return r;
}
// a e^{-2 pi i k / 8} (INV: the conjugate), k < 4
template <bool INV>
__device__ __forceinline__ cff eighth(const cff& a, int k) {
  if (k == 0) return a;
  const cff b = turn(a);  // -i a
  if (k == 2) return INV ? cff{mul2(b.h, splat2(-1.f)), mul2(b.l, splat2(-1.f))} : b;
  // e^{-i pi / 4} a = (a - i a) / sqrt 2, e^{+i pi / 4} a = (a + i a) / sqrt 2;
  // e^{-3 i pi / 4} a = (-a - i a) / sqrt 2, e^{+3 i pi / 4} a = (-a + i a) / sqrt 2
  if (k == 1) return root_half(INV ? a - b : a + b);
  const cff s = root_half(INV ? a + b : b - a);
  return INV ? cff{mul2(s.h, splat2(-1.f)), mul2(s.l, splat2(-1.f))} : s;
}

// R-point transforms in registers: forward, natural order in and bit-reversed
// out (decimation in frequency), and its mirror image.
template <int R>
__device__ __forceinline__ void forward_points(cff (&x)[R]) {
#pragma unroll
  for (int n = R; n >= 2; n >>= 1)
#pragma unroll
    for (int b = 0; b < R; b += n)
#pragma unroll
      for (int k = 0; k < n / 2; ++k) {
        const cff u = x[b + k], v = x[b + k + n / 2];
        x[b + k] = u + v;
        x[b + k + n / 2] = eighth<false>(u - v, k * (8 / n));
      }
}
template <int R>
__device__ __forceinline__ void inverse_points(cff (&x)[R]) {
#pragma unroll
  for (int n = 2; n <= R; n <<= 1)
#pragma unroll
    for (int b = 0; b < R; b += n)
#pragma unroll
      for (int k = 0; k < n / 2; ++k) {
        const cff u = x[b + k], v = eighth<true>(x[b + k + n / 2], k * (8 / n));
        x[b + k] = u + v;
        x[b + k + n / 2] = u - v;
      }
}
template <int R>
__device__ __forceinline__ constexpr int reversed(int r) {
  return R == 8 ? ((r & 1) << 2) | (r & 2) | (r >> 2) : (R == 4 ? ((r & 1) << 1) | (r >> 1) : r);
}

// the same value with |l| at most half a unit of h's last place (sums and
// products let l grow by a unit each, and with it their dropped terms)
__device__ __forceinline__ float4 settled(const cff& v) {
  const float2 h = add2(v.h, v.l);
  return as_float4(cff{h, sub2(v.l, sub2(h, v.h))});
}

// position of element q: one slot of padding after every 8 (a quarter-warp of
// 16-byte elements at stride 8 covers all banks)
__device__ __forceinline__ int tm_pos(int q) { return q + (q >> 3); }

// One pass over blocks of 2^LEN elements: elements p + m 2^LEN / R
template <int LOGM, int LEN, int R, bool INV>
__device__ __forceinline__ void tm_pass(float4* buf, const float4* tw) {
  constexpr int M = 1 << LOGM, H = (1 << LEN) / R;
  for (int g = threadIdx.x; g < M / R; g += blockDim.x) {
    const int p = g & (H - 1), b0 = (g / H) * (H * R) + p;
    cff x[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      x[r] = as_cff(buf[tm_pos(b0 + r * H)]);
      if (INV && r) x[r] = twiddle<true>(x[r], __ldg(tw + ((p * reversed<R>(r)) << (LOGM - LEN))));
    }
    if (INV) inverse_points(x);
    else forward_points(x);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (!INV && r) x[r] = twiddle<false>(x[r], __ldg(tw + ((p * reversed<R>(r)) << (LOGM - LEN))));
      buf[tm_pos(b0 + r * H)] = settled(x[r]);
    }
  }
  __syncthreads();
}

// The radix of the first forward (last inverse) pass; the others are 8.
template <int LOGM>
struct TmRadix {
  static constexpr int kFirst = LOGM % 3 == 0 ? 8 : (LOGM % 3 == 1 ? 2 : 4);
  static constexpr int kRest = LOGM - (LOGM % 3 == 0 ? 3 : LOGM % 3);  // log2 of the blocks after it, a multiple of 3
};

template <int LOGM, int LEN>
__device__ __forceinline__ void forward_eights(float4* buf, const float4* tw) {
  if constexpr (LEN > 3) {
    tm_pass<LOGM, LEN, 8, false>(buf, tw);
    forward_eights<LOGM, LEN - 3>(buf, tw);
  }
}
template <int LOGM, int LEN>
__device__ __forceinline__ void inverse_eights(float4* buf, const float4* tw) {
  if constexpr (LEN > 3) {
    inverse_eights<LOGM, LEN - 3>(buf, tw);
    tm_pass<LOGM, LEN, 8, true>(buf, tw);
  }
}

template <int LOGM>
__device__ __forceinline__ void forward_all(float4* buf, const float4* tw) {
  tm_pass<LOGM, LOGM, TmRadix<LOGM>::kFirst, false>(buf, tw);
  forward_eights<LOGM, TmRadix<LOGM>::kRest>(buf, tw);
}

// The circular convolution with the chirp: the last forward and the first
// inverse pass (blocks of 8, no twiddles) with the product between them.
template <int LOGM>
__device__ __forceinline__ void tm_convolve(float4* buf, const float4* tw, const float4* spec) {
  constexpr int M = 1 << LOGM;
  forward_all<LOGM>(buf, tw);
  for (int g = threadIdx.x; g < M / 8; g += blockDim.x) {
    cff x[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) x[r] = as_cff(buf[tm_pos(8 * g + r)]);
    forward_points(x);
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const float4 s = __ldg(spec + 8 * g + r);  // {re hi, im hi, re lo, im lo}
      x[r] = twiddle<false>(x[r], make_float4(s.x, s.z, s.y, s.w));
    }
    inverse_points(x);
#pragma unroll
    for (int r = 0; r < 8; ++r) buf[tm_pos(8 * g + r)] = settled(x[r]);
  }
  __syncthreads();
  inverse_eights<LOGM, TmRadix<LOGM>::kRest>(buf, tw);
  tm_pass<LOGM, LOGM, TmRadix<LOGM>::kFirst, true>(buf, tw);
}

// wide_cos2 (gwl_wide.cuh) to about 2e-15: the second-order term, 1.2e-6 at
// most, as an error-free product too.  (The transforms' errors are of that
// order; wide_cos2's 3e-14 would be the largest of this kernel.)
struct FineArg {
  float2 a, b, v, mh, ml;  // u^2 in table steps; mh + ml = -v/2 + v^2/24
};
__device__ __forceinline__ FineArg fine_arg2(uint32_t a0, uint32_t b0, uint32_t a1, uint32_t b1) {
  constexpr float kh = -4.706193976744544e-06f, kl = -1.384599628961175e-13f;  // -(2 pi / 2048)^2 / 2
  FineArg x;
  x.a = add2(make_float2(__uint_as_float(a0), __uint_as_float(a1)), splat2(-1.5f));
  x.b = add2(make_float2(__uint_as_float(b0), __uint_as_float(b1)), splat2(-1.1920928955078125e-07f));  // 2^-23
  x.v = mul2(x.a, x.a);
  float2 e = fma2(x.a, x.a, mul2(x.v, splat2(-1.f)));
  e = fma2(add2(x.a, x.a), x.b, e);
  x.mh = mul2(x.v, splat2(kh));
  x.ml = fma2(x.v, splat2(kh), mul2(x.mh, splat2(-1.f)));
  x.ml = fma2(e, splat2(kh), x.ml);
  x.ml = fma2(x.v, fma2(x.v, splat2(kh * kh / 6.0f), splat2(kl)), x.ml);
  return x;
}
__device__ __forceinline__ void fine_cos2(const float4 t0, const float4 t1, const FineArg& x, float2& ch, float2& cl) {
  constexpr float k6 = -9.41238823040901e-06f / 6.0f;
  const float2 Ch = make_float2(t0.x, t1.x), Cl = make_float2(t0.y, t1.y);
  const float2 Th = make_float2(t0.z, t1.z), Tl = make_float2(t0.w, t1.w);
  const float2 p = mul2(Th, x.a), c = mul2(Ch, x.mh);
  float2 r = fma2(Th, x.a, mul2(p, splat2(-1.f)));
  r = fma2(Th, x.b, r);
  r = fma2(Tl, x.a, r);
  r = fma2(mul2(p, x.v), splat2(k6), r);
  float2 q = fma2(Ch, x.mh, mul2(c, splat2(-1.f)));
  q = fma2(Ch, x.ml, q);
  q = fma2(Cl, x.mh, q);
  const float2 h = add2(Ch, p), e = sub2(p, sub2(h, Ch));  // |C| >= |p| or C = 0
  float2 g;
  two_sum2(h, c, ch, g);
  cl = add2(add2(add2(e, g), add2(r, q)), Cl);
  const float2 w = add2(ch, cl);
  cl = sub2(cl, sub2(w, ch));
  ch = w;
}

// x / (2 L) cycles as 0.64 fixed point
__device__ __forceinline__ uint64_t tm_cycles(const TmPlan& p, uint64_t x) { return x * p.inv + __umul64hi(x, p.inv_lo); }

__host__ __device__ constexpr int tm_threads(int log2m) { return log2m <= 12 ? (1 << log2m) / 8 : 512; }
__host__ __device__ constexpr int tm_slots(int log2m) { return (1 << log2m) + (1 << log2m) / 8; }

// Over the CTA, in a fixed order; red: a double per warp.
__device__ __forceinline__ double block_max(double v, double* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  for (int w = 0; w < (int)blockDim.x / 32; ++w) v = fmax(v, red[w]);
  return v;
}
__device__ __forceinline__ double block_sum(double v, double* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  v = 0.0;
  for (int w = 0; w < (int)blockDim.x / 32; ++w) v += red[w];
  return v;
}

constexpr double kTmBesselMax = 500.0;  // as ln_i0: I0(500) = 2.5e215, and its sum over the samples, are in range

// One CTA per point.  Bound by latency and, at the samples' I0, by the float64
// pipe (the transforms leave it idle).  6 s at 2048 Hz, two detectors, 2047 points,
// phase marginalised: 189 us (231 us with a logarithm and an exponential per sample),
// where the whole float64 transform through global memory (k_time_marg) took 2240 us.
// Seven CTAs per SM instead of six take the call from 267 to 259 us; eight spill more
// and take 281 us.  The error of a sample's <d|h> against 80-bit arithmetic, relative to the largest: 3e-15 rms
// (k_time_marg 6e-15).
template <int LOGM>
__global__ void __launch_bounds__(tm_threads(LOGM), LOGM == 10 ? 7 : 1) k_wide_tm(LaunchArgs a, TmPlan plan) {
  constexpr int M = 1 << LOGM, T = tm_threads(LOGM), kWarps = T / 32;
  extern __shared__ __align__(16) unsigned char smem[];
  float4* buf = reinterpret_cast<float4*>(smem);
  float4* acc = buf + tm_slots(LOGM);  // [cap] the samples' sums, then their lnL
  __shared__ double s_red[kWarps], s_hh[3], s_hy[4];
  __shared__ float s_gh[kMaxDet], s_gl[kMaxDet];
  __shared__ uint64_t s_x[kMaxDet], s_q[kMaxDet];
  __shared__ int64_t s_j0;
  __shared__ int s_n, s_ly;
  const int64_t i = blockIdx.x;
  const PointRec& r = a.rec[i];
  if (!r.valid) {  // uniform over the CTA
    if (threadIdx.x == 0) a.out[i] = neg_huge();
    return;
  }
  const int64_t L = a.n_fft;
  const int D = a.n_det;
  if (threadIdx.x == 0) {
    // candidate window from the real-valued bounds, checked exactly per sample
    const double jl = floor((a.t_min - a.start_time0 - r.jitter) / a.tm_step) - 3.0;
    const double jh = ceil((a.t_max - a.start_time0 - r.jitter) / a.tm_step) + 2.0;
    const int64_t lo = (int64_t)fmax(0.0, jl), hi = (int64_t)fmin((double)(L - 1), jh);
    s_j0 = lo;
    s_n = (int)min(max(hi - lo + 1, (int64_t)0), (int64_t)plan.cap);
  } else if (threadIdx.x == 32) {
    // A0 |Q_d| of the detectors, the largest taken out
    double g[kMaxDet], most = 0.0, all = 0.0;
    for (int d = 0; d < D; ++d) {
      g[d] = r.qabs[d] * a.wide_wscale[d];
      most = fmax(most, g[d]);
      all += g[d];
    }
    for (int d = 0; d < D; ++d) {
      const double q = most > 0.0 ? g[d] / most : 0.0;
      s_gh[d] = (float)q;
      s_gl[d] = (float)(q - (double)s_gh[d]);
      s_x[d] = a.wide_c[(int64_t)(kNumBasis + 2 + d) * a.B + i];
      s_q[d] = a.wide_c[(int64_t)(kNumBasis + 2 + kMaxDet + d) * a.B + i];
    }
    s_hh[2] = 4.0 / a.duration * r.amp * (isfinite(all) ? most : all);
  } else if (threadIdx.x == 64) {
    double hh = 0.0;
    const int64_t k1 = min(r.k_end, a.n_bins), k0 = min(r.k_start, k1);
    for (int d = 0; d < D; ++d) hh += tf2_norm(r, d, 4.0 / a.duration, a.hh_prefix[d][k1] - a.hh_prefix[d][k0]);
    const double ref = hh * r.dist * r.dist / (a.ref_dist * a.ref_dist);
    s_hh[0] = hh;
    s_hh[1] = ref;
    if (a.dist_marg) s_ly = bicubic_row(a.ty, a.ny, a.bbox, ref, s_hy);
  }
  uint64_t c[kNumBasis], c0;
  int shift;
  {
    const uint64_t* w = a.wide_c + i;
#pragma unroll
    for (int b = 0; b < kNumBasis; ++b) c[b] = w[(int64_t)b * a.B];
    c0 = w[(int64_t)kNumBasis * a.B];
    shift = (int)w[(int64_t)(kNumBasis + 1) * a.B];
  }
  __syncthreads();
  const int64_t j0 = s_j0, ks = max(r.k_start, a.k_lo), ke = min(r.k_end, L);  // (no weights below k_lo)
  const int n = s_n;
  for (int t = threadIdx.x; t < n; t += T) acc[t] = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int64_t k0 = ks & ~(int64_t)1; k0 < ke; k0 += plan.kb) {
    // Y_m, a pair of bins at a time
    for (int t = threadIdx.x; t < M / 2; t += T) {
      const int64_t k = k0 + 2 * t;
      const bool on0 = 2 * t < plan.kb && k >= ks && k < ke, on1 = 2 * t + 1 < plan.kb && k + 1 >= ks && k + 1 < ke;
      float2 sr, er, si, ei;  // sums over the detectors of the cosines and sines
      sr = er = si = ei = make_float2(0.f, 0.f);
      if (on0 || on1) {
        uint64_t b[2];
        const uint4* m = a.wide_phi + k * (kNumBasis / 2);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          uint64_t s = 0;
          int64_t cross = 0;
#pragma unroll
          for (int v = 0; v < kNumBasis / 2; ++v) {
            const uint4 e = __ldg(m + u * (kNumBasis / 2) + v);
            wide_mac(s, cross, (int32_t)(c[2 * v] >> 32), (int32_t)c[2 * v], (int32_t)e.x, (int32_t)e.y);
            wide_mac(s, cross, (int32_t)(c[2 * v + 1] >> 32), (int32_t)c[2 * v + 1], (int32_t)e.z, (int32_t)e.w);
          }
          const uint64_t mm = (uint64_t)(2 * t + u);
          b[u] = c0 + wide_fraction(s, cross, shift) + tm_cycles(plan, 2 * (uint64_t)j0 * (uint64_t)(k + u) + mm * mm);
        }
        for (int d = 0; d < D; ++d) {
          const uint64_t sh = (uint64_t)k * s_x[d] + s_q[d];
          const uint4 um = __ldg(a.wide_w[d] + k), ut = __ldg(a.wide_w[d] + k + 1);
          uint32_t q0, q1, ra0, ra1, rb0, rb1;
          wide_remainder(b[0] + sh + (((uint64_t)ut.y << 32) | ut.x), q0, ra0, rb0);
          wide_remainder(b[1] + sh + s_x[d] + (((uint64_t)ut.w << 32) | ut.z), q1, ra1, rb1);
          const FineArg x = fine_arg2(ra0, rb0, ra1, rb1);
          // |w| times the detector's factor
          float2 wh, wl, p, e;
          wide_term2(make_float2(__uint_as_float(um.x), __uint_as_float(um.y)),
                     make_float2(__uint_as_float(um.z), __uint_as_float(um.w)), splat2(s_gh[d]), splat2(s_gl[d]), wh, wl);
          fine_cos2(a.wide_tab[q0], a.wide_tab[q1], x, p, e);
          wide_term2(wh, wl, p, e, p, e);
          wide_add2(sr, er, p, e);
          fine_cos2(a.wide_tab[(q0 - kWideTable / 4) & (kWideTable - 1)],
                    a.wide_tab[(q1 - kWideTable / 4) & (kWideTable - 1)], x, p, e);
          wide_term2(wh, wl, p, e, p, e);
          wide_add2(si, ei, p, e);
        }
      }
      // h conj(d) / S = conj of the sums
      buf[tm_pos(2 * t)] = on0 ? make_float4(sr.x, -si.x, er.x, -ei.x) : make_float4(0.f, 0.f, 0.f, 0.f);
      buf[tm_pos(2 * t + 1)] = on1 ? make_float4(sr.y, -si.y, er.y, -ei.y) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __syncthreads();
    tm_convolve<LOGM>(buf, plan.tw, plan.spec);
    for (int t = threadIdx.x; t < n; t += T) {
      const uint64_t ang = tm_cycles(plan, 2 * (uint64_t)t * (uint64_t)k0 + (uint64_t)t * (uint64_t)t);
      uint32_t q, ra, rb;
      wide_remainder(ang, q, ra, rb);
      const FineArg x = fine_arg2(ra, rb, ra, rb);
      float2 h, l;  // cos and sin of the angle
      fine_cos2(a.wide_tab[q], a.wide_tab[(q - kWideTable / 4) & (kWideTable - 1)], x, h, l);
      acc[t] = as_float4(as_cff(acc[t]) + twiddle<true>(as_cff(buf[tm_pos(t)]), make_float4(h.x, l.x, h.y, l.y)));
    }
    __syncthreads();
  }
  // The samples: with phase marginalisation alone the sum of their I0 itself where
  // the largest argument leaves it in range (168 float64 instructions per sample
  // with a logarithm and an exponential around each I0, 110 without), else their
  // lnL and sum exp(l - max); sums in a fixed order.
  const double hh = s_hh[0], scale = s_hh[2], sr = r.dist / a.ref_dist, jit = r.jitter;
  const bool bessel = a.phase_marg && !a.dist_marg;
  double most = -INFINITY;
  for (int t = threadIdx.x; t < n; t += T) {
    double pw = 1.0, l = -INFINITY;  // l: |X| with phase marginalisation alone
    const double time = tm_sample_time(a, j0 + t, L, a.tm_step, jit);
    if (a.tm_prior) pw = tm_prior_density(a, time);
    if (time >= a.t_min && time <= a.t_max && pw > 0.0) {
      const float4 v = acc[t];
      const double xr = scale * ((double)v.x + (double)v.z), xi = scale * ((double)v.y + (double)v.w);
      if (a.dist_marg) {
        const double dx = a.phase_marg ? sqrt(xr * xr + xi * xi) * sr : xr * sr;
        l = bicubic_at(a.tx, a.nx, a.ny, a.tc, a.bbox, dx, s_ly, s_hy);
      } else {
        l = bessel ? sqrt(xr * xr + xi * xi) : xr - hh / 2;
      }
      if (!bessel && a.tm_prior) l += log(pw);
    }
    most = fmax(most, l);
    *reinterpret_cast<double2*>(acc + t) = make_double2(l, pw);
  }
  most = block_max(most, s_red);
  if (bessel && !(most < kTmBesselMax)) {
    most = -INFINITY;
    for (int t = threadIdx.x; t < n; t += T) {
      double2* v = reinterpret_cast<double2*>(acc + t);
      if (!(v->x >= 0.0)) continue;
      v->x = ln_i0(v->x) - hh / 2;
      if (a.tm_prior) v->x += log(v->y);
      most = fmax(most, v->x);
    }
    most = block_max(most, s_red);
  } else if (bessel) {
    double sum = 0.0;
    for (int t = threadIdx.x; t < n; t += T) {
      const double2 v = *reinterpret_cast<const double2*>(acc + t);
      if (v.x >= 0.0) sum += v.y * cyl_bessel_i0(v.x);
    }
    sum = block_sum(sum, s_red);
    if (threadIdx.x == 0)
      a.out[i] = isfinite(most) ? log(sum * (a.tm_prior ? 1.0 : 1.0 / (a.t_max - a.t_min)) * a.delta_tc) - hh / 2 : most;
    return;
  }
  double sum = 0.0;
  if (isfinite(most))
    for (int t = threadIdx.x; t < n; t += T) {
      const double l = reinterpret_cast<const double2*>(acc + t)->x;
      if (isfinite(l)) sum += exp(l - most);
    }
  sum = block_sum(sum, s_red);
  if (threadIdx.x == 0) {
    const double total = sum * (a.tm_prior ? 1.0 : 1.0 / (a.t_max - a.t_min)) * a.delta_tc;
    a.out[i] = isfinite(most) ? most + log(total) : most;
  }
}

// ---------------------------------------------------------------------------
// tables
// ---------------------------------------------------------------------------
__device__ __forceinline__ float4 split_angle(double half_turns) {
  double s, c;
  sincospi(half_turns, &s, &c);
  const float ch = (float)c, sh = (float)s;
  return make_float4(ch, (float)(c - (double)ch), sh, (float)(s - (double)sh));
}

__global__ void k_tm_twiddles(float4* tw, int m) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q < m) tw[q] = split_angle(-2.0 * (double)q / (double)m);
}

// the chirp e^{pi i l^2 / L}, cap - M <= l < cap, its forward transform / M
template <int LOGM>
__global__ void __launch_bounds__(tm_threads(LOGM)) k_tm_chirp(const float4* tw, float4* spec, int64_t L, int cap) {
  constexpr int M = 1 << LOGM;
  extern __shared__ __align__(16) unsigned char smem[];
  float4* buf = reinterpret_cast<float4*>(smem);
  for (int q = threadIdx.x; q < M; q += blockDim.x) {
    const int64_t l = q < cap ? q : q - M;
    const float4 v = split_angle((double)((l * l) % (2 * L)) / (double)L);
    buf[tm_pos(q)] = make_float4(v.x / M, v.z / M, v.y / M, v.w / M);
  }
  __syncthreads();
  forward_all<LOGM>(buf, tw);
  for (int g = threadIdx.x; g < M / 8; g += blockDim.x) {
    cff x[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) x[r] = as_cff(buf[tm_pos(8 * g + r)]);
    forward_points(x);
#pragma unroll
    for (int r = 0; r < 8; ++r) spec[8 * g + r] = settled(x[r]);
  }
}

namespace {

struct TmTables {
  float4 *tw = nullptr, *spec = nullptr;
};
PerDeviceCache<TmTables> g_tm_tables;  // by (L, log2 M, cap in eighths of M)

template <class F>
cudaError_t with_log2m(int log2m, F f) {
  switch (log2m) {
    case 10: return f(std::integral_constant<int, 10>());
    case 11: return f(std::integral_constant<int, 11>());
    case 12: return f(std::integral_constant<int, 12>());
    default: return f(std::integral_constant<int, 13>());
  }
}

cudaError_t tm_tables(int64_t L, int log2m, int cap, cudaStream_t s, TmTables* out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const int M = 1 << log2m;
  const int64_t key = (L << 8) | ((int64_t)log2m << 4) | (8 * (int64_t)cap / M);
  return (cudaError_t)g_tm_tables.get(dev, key, out, [&](TmTables* t) -> int {
    float4* p = nullptr;
    cudaError_t rc = cudaMalloc(reinterpret_cast<void**>(&p), 2 * (size_t)M * sizeof(float4));
    if (rc != cudaSuccess) return (int)rc;
    t->tw = p;
    t->spec = p + M;
    k_tm_twiddles<<<(M + 127) / 128, 128, 0, s>>>(t->tw, M);
    rc = cudaGetLastError();
    if (rc == cudaSuccess)
      rc = with_log2m(log2m, [&](auto lg) {
        constexpr int LG = decltype(lg)::value;
        const int smem = tm_slots(LG) * (int)sizeof(float4);
        cudaError_t x = cudaFuncSetAttribute(k_tm_chirp<LG>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (x != cudaSuccess) return x;
        k_tm_chirp<LG><<<1, tm_threads(LG), smem, s>>>(t->tw, t->spec, L, cap);
        return cudaGetLastError();
      });
    if (rc == cudaSuccess) rc = cudaStreamSynchronize(s);
    if (rc != cudaSuccess) cudaFree(p);
    return (int)rc;
  });
}

// the most samples a prior window holds, with the margin of the candidate window
int64_t tm_samples(const LaunchArgs& a) {
  const double width = (a.t_max - a.t_min) / a.tm_step;
  return width >= 0.0 && width < 1e6 ? (int64_t)std::ceil(width) + 10 : (int64_t)1 << 30;
}

}  // namespace

// Up to 4096 samples: the longest convolution, 8192 elements of 16 bytes and the
// samples' sums, fills an SM's shared memory.  A longer window (2 s at 4096 Hz)
// is a sizeable part of the segment, where the whole transform (gwl_marg.cu) does
// little that is not needed.
static bool tm_window_fits(const LaunchArgs& a) {
  return a.model == GWL_MODEL_TAYLORF2 && a.n_fft > 0 && a.n_fft < ((int64_t)1 << 40) &&
         tm_samples(a) <= (1 << (kTmMaxLog - 1));
}

// (the tables are there for every window that fits: which kernel runs depends on
// the analysis alone, not on what ran before or whether the stream is captured)
bool wide_tm_fits(const LaunchArgs& a) {
  return tm_window_fits(a) && a.wide_tm_tw && !a.relbin && !a.multiband && !a.roq && !a.tm_series &&
         a.B < ((int64_t)1 << 31);
}

static TmPlan tm_plan(const LaunchArgs& a) {
  const int64_t need = tm_samples(a);
  TmPlan p = {};
  p.log2m = kTmMinLog;
  while ((1 << p.log2m) < 2 * need) ++p.log2m;
  const int M = 1 << p.log2m;
  p.cap = (int)((need + M / 8 - 1) / (M / 8)) * (M / 8);
  p.kb = M - p.cap;
  return p;
}

cudaError_t wide_tm_tables(const LaunchArgs& a, cudaStream_t s, const float4** tw, const float4** spec) {
  *tw = *spec = nullptr;
  if (!tm_window_fits(a)) return cudaSuccess;
  const TmPlan p = tm_plan(a);
  TmTables t;
  const cudaError_t e = tm_tables(a.n_fft, p.log2m, p.cap, s, &t);
  if (e != cudaSuccess) return e;
  *tw = t.tw;
  *spec = t.spec;
  return cudaSuccess;
}

cudaError_t launch_wide_tm(const LaunchArgs& a, cudaStream_t s) {
  TmPlan p = tm_plan(a);
  p.tw = a.wide_tm_tw;
  p.spec = a.wide_tm_spec;
  const unsigned __int128 one = ~(unsigned __int128)0 / (unsigned __int128)(2 * a.n_fft);
  p.inv = (uint64_t)(one >> 64);
  p.inv_lo = (uint64_t)one;
  return with_log2m(p.log2m, [&](auto lg) {
    constexpr int LG = decltype(lg)::value;
    const int smem = (tm_slots(LG) + p.cap) * (int)sizeof(float4);
    cudaError_t x = cudaFuncSetAttribute(k_wide_tm<LG>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (x != cudaSuccess) return x;
    k_wide_tm<LG><<<(unsigned)a.B, tm_threads(LG), smem, s>>>(a, p);
    return cudaGetLastError();
  });
}

}  // namespace gwl
