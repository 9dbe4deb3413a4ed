// The float64 sine-Gaussian likelihood (bilby/gw/source.py:1153-1209 projected
// as in bilby/gw/detector/interferometer.py:303-368, summed as in
// bilby/gw/utils.py:118-138) on the 32-bit pipes (gwl_wide.cuh).
//
// With g1, g2 = exp(-pi^2 tau^2 (f -+ f0)^2), M_d = |(Fp P, Fx X)| and beta_d =
// arg(Fp P + i Fx X) the projection is
//   conj(h_d) = M_d (g1 e^{i beta} + g2 e^{-i beta}) e^{2 pi i f dt},
// so that with w = d / S = |w| e^{2 pi i theta}
//   <d|h>_d = 4/T M sum_k |w_k| (g1 e^{i(phi + beta)} + g2 e^{i(phi - beta)}),
//   phi = 2 pi (k dt_d df + theta_k),
//   <h|h>_d = 4/T M^2 (sum (g1^2 + g2^2) / S + cos 2 beta sum 2 g1 g2 / S).
//
// The Gaussians are 64-bit integers: y = (u s)^2 = pi^2 tau^2 (f -+ f0)^2 log2 e
// in fixed point, 2^-y from a table of 2^(-i/256) and a polynomial, all in
// 64-bit products of 32-bit halves; <h|h> adds integers, <d|h> float-float
// terms.  Inside a sub-block of 32 bins everything is relative to 2^-n0, n0 the
// integer part of the sub-block's smallest y.  Bins whose y is 100 above the
// smallest in-band y (a factor of 2^-100) lie below the rounding of the sum and
// are not visited.
//
// Summation order as in gwl_wide.cu: per sub-block the even and the odd bins in
// order (g1's term before g2's), the sub-blocks in order, then the chunks; the
// integer sums are exact.
#include <cuda_runtime.h>

#include <cstdint>

#include "gwl_device.cuh"
#include "gwl_internal.h"
#include "gwl_marg_common.cuh"
#include "gwl_wide.cuh"

namespace gwl {

constexpr int kSub = 32;                   // bins per sub-block
constexpr int kSubs = kChunkPlain / kSub;  // sub-blocks per chunk
constexpr int kWideThreads = 32 * kSubs;
constexpr float kWideHalf = -0x1.fffffep-24f;  // 2^-47 - 2^-23

// high 64 bits of a b, less up to 2 (the lowest partial product is dropped)
__device__ __forceinline__ uint64_t mulhi(uint64_t a, uint64_t b) {
  const uint32_t ah = (uint32_t)(a >> 32), al = (uint32_t)a, bh = (uint32_t)(b >> 32), bl = (uint32_t)b;
  return (uint64_t)ah * bh + __umulhi(ah, bl) + __umulhi(al, bh);
}

__device__ __forceinline__ uint64_t shift_left(uint64_t x, int s) {  // right for s < 0
  return s >= 0 ? x << s : (s > -64 ? x >> -s : 0ull);
}

// The point's coefficients (LaunchArgs::wide_c, point fastest).
template <int D>
struct SgPoint {
  uint64_t k0, s, top, x[D], beta[D];  // f0 in bins, sqrt(y) per bin, the largest distance, per detector
  int shift, frac;                     // fractional bits of k0, top and the distances
  __device__ __forceinline__ void load(const LaunchArgs& a, int64_t i) {
    const uint64_t* w = a.wide_c + i;
    k0 = w[0];
    s = w[a.B];
    shift = (int)(uint32_t)w[2 * a.B];
    frac = (int)(w[2 * a.B] >> 32);
    top = w[3 * a.B];
#pragma unroll
    for (int d = 0; d < D; ++d) {
      x[d] = w[(int64_t)(kNumBasis + 2 + d) * a.B];
      beta[d] = w[(int64_t)(kNumBasis + 2 + kMaxDet + d) * a.B];
    }
  }
};

// y of the distance u: integer part and fraction
__device__ __forceinline__ int sg_exponent(uint64_t u, int shift, uint64_t s, uint64_t& f) {
  const uint64_t v = mulhi(shift_left(u, shift), s);  // u s with 58 fractional bits, below 64
  const uint32_t vh = (uint32_t)(v >> 32), vl = (uint32_t)v;
  const uint64_t hl = (uint64_t)vh * vl, l0 = hl << 33, lo = l0 + (uint64_t)vl * vl;
  const uint64_t hi = (uint64_t)vh * vh + (hl >> 31) + (lo < l0 ? 1 : 0);  // v^2 with 116 fractional bits
  f = (hi << 12) | (lo >> 52);
  return (int)(hi >> 52);
}

// 2^-f as a 0.64 fraction: the table entry 2^-(i / 256) times e^-z, z = r ln 2 <
// 2^-8.5, e^-z = 1 - z + z^2 (1/2 - z/6 + z^2/24 - z^3/120).  Error below 2^-59.
__device__ __forceinline__ uint64_t sg_power(uint64_t f, const uint64_t* tab) {
  const uint64_t t = tab[f >> 56];
  const uint64_t z = mulhi(f << 8, 0xb17217f7d1cf79acull);  // z 2^72
  const uint64_t zz = mulhi(z, z);                          // z^2 2^80
  const uint32_t zh = (uint32_t)(z >> 32), qh = (uint32_t)(zz >> 32);
  uint64_t c = 0x8000000000000000ull;
  c -= ((uint64_t)zh * 0x2aaaaaabu) >> 8;   // z / 6
  c += ((uint64_t)qh * 0x0aaaaaabu) >> 16;  // z^2 / 24
  c -= ((uint64_t)__umulhi(qh, zh) * 34u) >> 4;  // z^3 / 120 to one percent (1e-18)
  const uint64_t q = (z >> 8) - (mulhi(zz, c) >> 16);
  return t - mulhi(t, q);
}

// a 0.64 fraction as a float pair, 46 bits and half a unit
__device__ __forceinline__ void sg_floats(uint64_t g, uint32_t& a, uint32_t& b) {
  a = 0x3f800000u | (uint32_t)(g >> 41);
  b = 0x34000000u | ((uint32_t)(g >> 18) & 0x7fffffu);
}

// One detector's terms of a pair of bins for one Gaussian (ga, gb: its pair of
// bins as sg_floats' bits): |w| g cos 2 pi (angle + arg w) as p + e, the sine's as
// pi + ei.
template <bool CPLX>
__device__ __forceinline__ void sg_pair(uint64_t a0, uint64_t a1, float2 gh, float2 gl, const uint4& um, const uint4& ut,
                                        const float4* tab, float2& p, float2& e, float2& pi, float2& ei) {
  a0 += ((uint64_t)ut.y << 32) | ut.x;
  a1 += ((uint64_t)ut.w << 32) | ut.z;
  uint32_t q0, q1, ra0, ra1, rb0, rb1;
  wide_remainder(a0, q0, ra0, rb0);
  wide_remainder(a1, q1, ra1, rb1);
  const WideArg x = wide_arg2(ra0, rb0, ra1, rb1);
  const float2 wh = make_float2(__uint_as_float(um.x), __uint_as_float(um.y));
  const float2 wl = make_float2(__uint_as_float(um.z), __uint_as_float(um.w));
  float2 mh, ml, ch, cl;
  wide_term2(wh, wl, gh, gl, mh, ml);
  wide_cos2(tab[q0], tab[q1], x, ch, cl);
  wide_term2(mh, ml, ch, cl, p, e);
  if (CPLX) {
    wide_cos2(tab[(q0 - kWideTable / 4) & (kWideTable - 1)], tab[(q1 - kWideTable / 4) & (kWideTable - 1)], x, ch, cl);
    wide_term2(mh, ml, ch, cl, pi, ei);
  }
}

// The Gaussian at signed distance u (bins; u2 = |u|) relative to 2^-n0.
__device__ __forceinline__ uint64_t sg_gauss(uint64_t u, int shift, uint64_t s, int n0, const uint64_t* tab) {
  uint64_t f;
  const int n = sg_exponent(u, shift, s, f) - n0;
  return n < 64 ? sg_power(f, tab) >> n : 0ull;
}

__device__ __forceinline__ uint64_t abs64(int64_t x) { return (uint64_t)(x < 0 ? -x : x); }

// 2^e as a double (zero below the normal range)
__device__ __forceinline__ double pow2_double(int e) {
  return e < -1022 ? 0.0 : __hiloint2double((1023 + min(e, 1023)) << 20, 0);
}

// The sub-block's bins [j0, j1) of a point, its exponent n0 and whether g2
// reaches the sub-block's last digit.
struct SgBlock {
  int j0, j1, n0;
  bool second;
};
template <int D>
__device__ __forceinline__ SgBlock sg_block(const LaunchArgs& a, int64_t i, bool have, int64_t ks, const SgPoint<D>& pt) {
  SgBlock b{0, 0, 0, false};
  const PointRec& r = a.rec[i];
  if (have && r.valid) {
    const int64_t lo = max(r.k_start, ks), hi = min(r.k_end, ks + kSub);
    if (hi > lo) {
      b.j0 = (int)(lo - ks);
      b.j1 = (int)(hi - ks);
      // the bin nearest to f0 and the one where g2 is largest
      const int64_t kp = (int64_t)(pt.k0 >> pt.frac);
      const int64_t k1 = min(max(kp, lo), hi - 1), k2 = min(k1 + 1, hi - 1);
      const int64_t c0 = (int64_t)pt.k0;
      const uint64_t u1 = abs64((k1 << pt.frac) - c0), u2 = abs64((k2 << pt.frac) - c0);
      uint64_t f;
      b.n0 = sg_exponent(u1 < u2 ? u1 : u2, pt.shift, pt.s, f);
      const uint64_t v = ((uint64_t)lo << pt.frac) + pt.k0;
      b.second = v <= pt.top && sg_exponent(v, pt.shift, pt.s, f) - b.n0 < 64;
    }
  }
  return b;
}

template <int D>
__device__ __forceinline__ void sg_stage(const LaunchArgs& a, int64_t k0, float4* tab, uint64_t* etab, uint4* w, uint64_t* v) {
  for (int q = threadIdx.x; q < kWideTable; q += kWideThreads) tab[q] = a.wide_tab[q];
  for (int q = threadIdx.x; q < kExpTable; q += kWideThreads) etab[q] = a.wide_exp[q];
#pragma unroll
  for (int d = 0; d < D; ++d)
    for (int q = threadIdx.x; q < kChunkPlain; q += kWideThreads) {
      w[d * kChunkPlain + q] = a.wide_w[d][k0 + q];
      v[d * kChunkPlain + q] = a.wide_v[d][k0 + q];
    }
}

// A pair of bins: the Gaussians of both, and the <h|h> products of both with
// every detector's inverse PSD.
struct SgPair {
  uint64_t g1[2], g2[2];
};

template <int D>
__device__ __forceinline__ void sg_hh(const SgPair& g, bool second, const uint64_t* v, int stride, uint64_t* h1, uint64_t* h2) {
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    const uint64_t p1 = (mulhi(g.g1[t], g.g1[t]) >> 1) + (second ? mulhi(g.g2[t], g.g2[t]) >> 1 : 0ull);
#pragma unroll
    for (int d = 0; d < D; ++d) h1[d] += mulhi(p1, v[d * stride + t]) >> 5;
    if (second) {
      const uint64_t p2 = mulhi(g.g1[t], g.g2[t]);
#pragma unroll
      for (int d = 0; d < D; ++d) h2[d] += mulhi(p2, v[d * stride + t]) >> 5;
    }
  }
}

// Batches, as k_wide_tf2: one warp per sub-block, lane = point, the points ordered
// by the number of bins they visit and those bins' middle (unordered by width,
// ordered by f0 alone, 17 of 32 lanes were at work and the kernel took 0.69 ms).
// 10,000 prior draws at 4 s, two detectors: 0.42 ms, 0.60 ms for the call, where
// the kernel in float64 (two exponentials per bin in that pipe) took 10.1 ms.  The
// error against 80-bit arithmetic: <d|h> / sqrt(<h|h>) 5e-13 -> 1.3e-13 rms, <h|h>
// 6e-15 -> 4e-16.
template <int D, bool CPLX>
__global__ void __launch_bounds__(kWideThreads, 2) k_wide_sg(LaunchArgs a, int tiles) {
  constexpr int NC = CPLX ? 4 : 3;
  extern __shared__ __align__(16) unsigned char smem[];
  float4* tab = reinterpret_cast<float4*>(smem);
  uint4* w = reinterpret_cast<uint4*>(tab + kWideTable);
  uint64_t* v = reinterpret_cast<uint64_t*>(w + D * kChunkPlain);
  uint64_t* etab = v + D * kChunkPlain;
  double* sums = reinterpret_cast<double*>(etab + kExpTable);  // [kSubs][D * NC][32]
  const int64_t k0 = a.k_base + (int64_t)blockIdx.x * kChunkPlain;
  sg_stage<D>(a, k0, tab, etab, w, v);
  __syncthreads();
  const int lane = threadIdx.x & 31, sub = threadIdx.x >> 5;
  const int64_t ks = k0 + sub * kSub;
  const int64_t t1 = min((int64_t)(blockIdx.y + 1) * tiles, (a.B + 31) / 32);
  for (int64_t t = (int64_t)blockIdx.y * tiles; t < t1; ++t) {
    const bool have = t * 32 + lane < a.B;
    const int64_t i = have ? (a.order ? (int64_t)a.order[t * 32 + lane] : t * 32 + lane) : 0;
    SgPoint<D> pt;
    pt.load(a, i);
    const SgBlock b = sg_block<D>(a, i, have, ks, pt);
    const bool any2 = __any_sync(0xffffffffu, b.second);
    float2 hr[D], lr[D], hm[D], lm[D];
    uint64_t h1[D], h2[D];
#pragma unroll
    for (int d = 0; d < D; ++d) {
      hr[d] = lr[d] = hm[d] = lm[d] = make_float2(0.f, 0.f);
      h1[d] = h2[d] = 0;
    }
    if (__any_sync(0xffffffffu, b.j1 > 0)) {
      uint64_t sh[D];
#pragma unroll
      for (int d = 0; d < D; ++d) sh[d] = (uint64_t)ks * pt.x[d];
      int64_t u = (ks << pt.frac) - (int64_t)pt.k0;
      const int64_t one = (int64_t)1 << pt.frac;
      const uint4* ws = w + sub * kSub;
      const uint64_t* vs = v + sub * kSub;
#pragma unroll 1
      for (int j = 0; j < kSub; j += 2) {
        if (j + 2 > b.j0 && j < b.j1) {
          const bool on0 = j >= b.j0, on1 = j + 1 < b.j1;
          SgPair g;
          g.g1[0] = on0 ? sg_gauss(abs64(u), pt.shift, pt.s, b.n0, etab) : 0ull;
          g.g1[1] = on1 ? sg_gauss(abs64(u + one), pt.shift, pt.s, b.n0, etab) : 0ull;
          g.g2[0] = g.g2[1] = 0;
          if (any2 && b.second) {
            const uint64_t v0 = (uint64_t)(u + 2 * (int64_t)pt.k0);
            if (on0 && v0 <= pt.top) g.g2[0] = sg_gauss(v0, pt.shift, pt.s, b.n0, etab);
            if (on1 && v0 + (uint64_t)one <= pt.top) g.g2[1] = sg_gauss(v0 + (uint64_t)one, pt.shift, pt.s, b.n0, etab);
          }
          sg_hh<D>(g, any2, vs, kChunkPlain, h1, h2);
#pragma unroll 1
          for (int c = 0; c < (any2 ? 2 : 1); ++c) {
            uint32_t ga0, gb0, ga1, gb1;
            sg_floats(c ? g.g2[0] : g.g1[0], ga0, gb0);
            sg_floats(c ? g.g2[1] : g.g1[1], ga1, gb1);
            const bool z0 = (c ? g.g2[0] : g.g1[0]) != 0, z1 = (c ? g.g2[1] : g.g1[1]) != 0;
            const float2 gh = add2(make_float2(__uint_as_float(ga0), __uint_as_float(ga1)), splat2(-1.f));
            const float2 gl = add2(make_float2(__uint_as_float(gb0), __uint_as_float(gb1)), splat2(kWideHalf));
#pragma unroll
            for (int d = 0; d < D; ++d) {
              const uint64_t be = c ? 0 - pt.beta[d] : pt.beta[d];
              float2 p, e, pi, ei;
              sg_pair<CPLX>(sh[d] + be, sh[d] + pt.x[d] + be, gh, gl, ws[d * kChunkPlain], ws[d * kChunkPlain + 1], tab, p, e,
                            pi, ei);
              if (!(z0 && z1)) {
                if (!z0) p.x = e.x = 0.f;
                if (!z1) p.y = e.y = 0.f;
                if (CPLX && !z0) pi.x = ei.x = 0.f;
                if (CPLX && !z1) pi.y = ei.y = 0.f;
              }
              wide_add2(hr[d], lr[d], p, e);
              if (CPLX) wide_add2(hm[d], lm[d], pi, ei);
            }
          }
        }
#pragma unroll
        for (int d = 0; d < D; ++d) sh[d] += 2 * pt.x[d];
        u += 2 * one;
        ws += 2;
        vs += 2;
      }
    }
    const double sc = pow2_double(-b.n0);
#pragma unroll
    for (int d = 0; d < D; ++d) {
      double* o = sums + (sub * D * NC + d * NC) * 32 + lane;
      o[0] = sc * (((double)hr[d].x + (double)lr[d].x) + ((double)hr[d].y + (double)lr[d].y));
      const double vsc = pow2_double(a.wide_ve[d][(ks - a.k_base) / kSub] - 58 - 2 * b.n0);
      o[32] = vsc * (double)h1[d];
      o[64] = vsc * (double)h2[d];
      if (CPLX) o[96] = sc * (((double)hm[d].x + (double)lm[d].x) + ((double)hm[d].y + (double)lm[d].y));
    }
    __syncthreads();
    for (int c = threadIdx.x; c < 32 * D * NC; c += kWideThreads) {
      const int64_t slot = t * 32 + (c & 31);
      if (slot < a.B) {
        const int64_t ip = a.order ? (int64_t)a.order[slot] : slot;
        double s = sums[c];
#pragma unroll
        for (int q = 1; q < kSubs; ++q) s += sums[q * D * NC * 32 + c];
        a.part[(ip * D * NC + (c >> 5)) * a.n_chunks + blockIdx.x] = s;
      }
    }
    __syncthreads();
  }
}

// Few points, as k_wide_tf2_few: lane = pair of bins, the terms added in
// k_wide_sg's order, the integer sums over the sub-block's 16 lanes (9 us for one
// point; 1.0 ms in the float64 kernel, which had one thread per 256 bins).
constexpr int kPairThreads = kChunkPlain / 2;

template <int D, bool CPLX>
__global__ void __launch_bounds__(kPairThreads) k_wide_sg_few(LaunchArgs a) {
  constexpr int NS = D * (CPLX ? 2 : 1), NC = CPLX ? 4 : 3;
  constexpr int kPer = kSub / 2, kRow = 2 * kPer + 1;  // terms of a parity: g1's and g2's of each bin in turn
  __shared__ float2 term[NS][2][kSubs][kRow];
  __shared__ double part[NS][2][kSubs];
  __shared__ double hpart[2 * D][kSubs];
  __shared__ int s_n0[kSubs];
  const int64_t k0 = a.k_base + (int64_t)blockIdx.x * kChunkPlain;
  const int t = threadIdx.x, sub = t / kPer, pr = t % kPer;
  const int64_t k = k0 + 2 * t, ks = k0 + sub * kSub;
  const int64_t i = blockIdx.y;
  allow_next();
  wait_previous();
  SgPoint<D> pt;
  pt.load(a, i);
  const SgBlock b = sg_block<D>(a, i, true, ks, pt);
  const int j = 2 * pr;
  const bool on0 = j >= b.j0 && j < b.j1, on1 = j + 1 >= b.j0 && j + 1 < b.j1;
  SgPair g;
  g.g1[0] = g.g1[1] = g.g2[0] = g.g2[1] = 0;
  const int64_t one = (int64_t)1 << pt.frac, u = (k << pt.frac) - (int64_t)pt.k0;
  if (on0) g.g1[0] = sg_gauss(abs64(u), pt.shift, pt.s, b.n0, a.wide_exp);
  if (on1) g.g1[1] = sg_gauss(abs64(u + one), pt.shift, pt.s, b.n0, a.wide_exp);
  if (b.second) {
    const uint64_t v0 = (uint64_t)(u + 2 * (int64_t)pt.k0);
    if (on0 && v0 <= pt.top) g.g2[0] = sg_gauss(v0, pt.shift, pt.s, b.n0, a.wide_exp);
    if (on1 && v0 + (uint64_t)one <= pt.top) g.g2[1] = sg_gauss(v0 + (uint64_t)one, pt.shift, pt.s, b.n0, a.wide_exp);
  }
  uint64_t vv[2 * D], h1[D], h2[D];
#pragma unroll
  for (int d = 0; d < D; ++d) {
    vv[2 * d] = a.wide_v[d][k];
    vv[2 * d + 1] = a.wide_v[d][k + 1];
    h1[d] = h2[d] = 0;
  }
  sg_hh<D>(g, b.second, vv, 2, h1, h2);
#pragma unroll
  for (int d = 0; d < D; ++d) {
#pragma unroll
    for (int o = kPer / 2; o > 0; o >>= 1) {
      h1[d] += __shfl_xor_sync(0xffffffffu, h1[d], o);
      h2[d] += __shfl_xor_sync(0xffffffffu, h2[d], o);
    }
    if (pr == 0) {
      const double vsc = pow2_double(a.wide_ve[d][(ks - a.k_base) / kSub] - 58 - 2 * b.n0);
      hpart[2 * d][sub] = vsc * (double)h1[d];
      hpart[2 * d + 1][sub] = vsc * (double)h2[d];
    }
  }
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    const bool z0 = (c ? g.g2[0] : g.g1[0]) != 0, z1 = (c ? g.g2[1] : g.g1[1]) != 0;
    uint32_t ga0, gb0, ga1, gb1;
    sg_floats(c ? g.g2[0] : g.g1[0], ga0, gb0);
    sg_floats(c ? g.g2[1] : g.g1[1], ga1, gb1);
    const float2 gh = add2(make_float2(__uint_as_float(ga0), __uint_as_float(ga1)), splat2(-1.f));
    const float2 gl = add2(make_float2(__uint_as_float(gb0), __uint_as_float(gb1)), splat2(kWideHalf));
#pragma unroll
    for (int d = 0; d < D; ++d) {
      float2 p, e, pi, ei;
      p = e = pi = ei = make_float2(0.f, 0.f);
      if (z0 || z1) {
        const uint64_t sh = (uint64_t)k * pt.x[d] + (c ? 0 - pt.beta[d] : pt.beta[d]);
        sg_pair<CPLX>(sh, sh + pt.x[d], gh, gl, a.wide_w[d][k], a.wide_w[d][k + 1], a.wide_tab, p, e, pi, ei);
      }
      const int s = CPLX ? 2 * d : d;
      term[s][0][sub][2 * pr + c] = z0 ? make_float2(p.x, e.x) : make_float2(0.f, 0.f);
      term[s][1][sub][2 * pr + c] = z1 ? make_float2(p.y, e.y) : make_float2(0.f, 0.f);
      if (CPLX) {
        term[s + 1][0][sub][2 * pr + c] = z0 ? make_float2(pi.x, ei.x) : make_float2(0.f, 0.f);
        term[s + 1][1][sub][2 * pr + c] = z1 ? make_float2(pi.y, ei.y) : make_float2(0.f, 0.f);
      }
    }
  }
  __syncthreads();
  for (int c = t; c < NS * 2 * kSubs; c += kPairThreads) {
    const float2* src = &term[0][0][0][0] + (int64_t)c * kRow;
    float h = 0.f, l = 0.f;
#pragma unroll
    for (int q = 0; q < 2 * kPer; ++q) {
      const float2 v = src[q];
      const float s = __fadd_rn(h, v.x), bb = __fsub_rn(s, h);
      const float err = __fadd_rn(__fsub_rn(h, __fsub_rn(s, bb)), __fsub_rn(v.x, bb));
      h = s;
      l = __fadd_rn(l, __fadd_rn(err, v.y));
    }
    (&part[0][0][0])[c] = (double)h + (double)l;
  }
  if (pr == 0) s_n0[sub] = b.n0;
  __syncthreads();
  if (t < D * NC) {
    const int d = t / NC, c = t % NC;
    double s = 0.0;
#pragma unroll
    for (int q = 0; q < kSubs; ++q) {
      double x;
      if (c == 1 || c == 2) x = hpart[2 * d + c - 1][q];
      else {
        const int n = CPLX ? 2 * d + (c == 3 ? 1 : 0) : d;
        x = pow2_double(-s_n0[q]) * (part[n][0][q] + part[n][1][q]);
      }
      s = q == 0 ? x : s + x;
    }
    a.part[(i * D * NC + t) * a.n_chunks + blockIdx.x] = s;
  }
}

// The chunks' sums in a fixed order, the totals and the lnL.
constexpr int kWideFinThreads = 128;

// (one compiled body, so that both kernels below round alike) p: [n_det][nc]
__device__ __noinline__ void wide_sg_totals(const LaunchArgs& a, int64_t i, const double* p) {
  const PointRec& r = a.rec[i];
  const int nc = a.cplx ? 4 : 3;
  const double norm = 4.0 / a.duration;
  double dr = 0.0, di = 0.0, hh = 0.0;
  for (int d = 0; d < a.n_det; ++d, p += nc) {
    const double A = r.fp[d] * r.amp, C = r.fx[d] * r.amp2, m = norm * a.wide_wscale[d] * hypot(A, C);
    dr += m * p[0];
    if (a.cplx) di += m * p[3];
    // M^2 (S1 + cos 2 beta S2) with M^2 cos 2 beta = A^2 - C^2
    hh += norm * ((A * A + C * C) * p[1] + (A - C) * (A + C) * p[2]);
  }
  if (!r.valid) dr = di = hh = 0.0;  // (nothing was summed, and the factors may be undefined)
  finish_point(a, r, i, dr, di, hh);
}

__global__ void __launch_bounds__(kWideFinThreads) k_wide_sg_finalize(LaunchArgs a) {
  const int lanes = wide_lanes(a.n_chunks), lane = threadIdx.x & (lanes - 1);
  const int64_t slot = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / lanes, i = min(slot, a.B - 1);
  const int n = a.n_det * (a.cplx ? 4 : 3);
  double p[4 * kMaxDet];
  for (int c = 0; c < n; ++c) p[c] = wide_chunk_sum(a.part + (i * n + c) * a.n_chunks, a.n_chunks, lane, lanes);
  if (lane == 0 && slot < a.B) wide_sg_totals(a, i, p);
}

// Few points: a CTA per point and a warp per sum, as k_wide_finalize_few (one
// point at 4 s: 11.9 us to 7.2 us).
__global__ void __launch_bounds__(128 * kMaxDet) k_wide_sg_finalize_few(LaunchArgs a) {
  __shared__ double s_p[4 * kMaxDet];
  const int lanes = wide_lanes(a.n_chunks), lane = threadIdx.x & (lanes - 1), c = threadIdx.x >> 5;
  const int64_t i = blockIdx.x;
  const int n = a.n_det * (a.cplx ? 4 : 3);
  wait_previous();
  const double p = wide_chunk_sum<32>(a.part + (i * n + c) * a.n_chunks, a.n_chunks, lane, lanes);
  if ((threadIdx.x & 31) == 0) s_p[c] = p;
  __syncthreads();
  if (threadIdx.x == 0) wide_sg_totals(a, i, s_p);
}

template <int D, bool CPLX>
static cudaError_t launch_wide_sg_d(const LaunchArgs& a, cudaStream_t s) {
  if (wide_few(a.B, a.n_chunks)) {
    const dim3 grid((unsigned)a.n_chunks, (unsigned)a.B);
    return launch_after(k_wide_sg_few<D, CPLX>, grid, kPairThreads, s, a);
  }
  constexpr int NC = CPLX ? 4 : 3;
  constexpr int smem = kWideTable * 16 + kChunkPlain * D * 24 + kExpTable * 8 + kSubs * D * NC * 32 * 8;
  const cudaError_t set = allow_shared(k_wide_sg<D, CPLX>, smem);
  if (set != cudaSuccess) return set;
  const int64_t tiles = (a.B + 31) / 32;
  const int per = wide_tiles(a.n_chunks, tiles);
  const dim3 grid((unsigned)a.n_chunks, (unsigned)((tiles + per - 1) / per));
  k_wide_sg<D, CPLX><<<grid, kWideThreads, smem, s>>>(a, per);
  return cudaGetLastError();
}

cudaError_t launch_wide_sg(const LaunchArgs& a, cudaStream_t s) {
  cudaError_t e;
  switch (2 * a.n_det + (a.cplx ? 1 : 0)) {
    case 2: e = launch_wide_sg_d<1, false>(a, s); break;
    case 3: e = launch_wide_sg_d<1, true>(a, s); break;
    case 4: e = launch_wide_sg_d<2, false>(a, s); break;
    case 5: e = launch_wide_sg_d<2, true>(a, s); break;
    case 6: e = launch_wide_sg_d<3, false>(a, s); break;
    case 7: e = launch_wide_sg_d<3, true>(a, s); break;
    case 8: e = launch_wide_sg_d<4, false>(a, s); break;
    default: e = launch_wide_sg_d<4, true>(a, s); break;
  }
  if (e != cudaSuccess) return e;
  if (wide_few(a.B, a.n_chunks))
    return launch_after(k_wide_sg_finalize_few, dim3((unsigned)a.B), 32 * a.n_det * (a.cplx ? 4 : 3), s, a);
  k_wide_sg_finalize<<<(unsigned)((a.B * wide_lanes(a.n_chunks) + kWideFinThreads - 1) / kWideFinThreads),
                       kWideFinThreads, 0, s>>>(a);
  return cudaGetLastError();
}

}  // namespace gwl
