// Double precision without the float64 pipe.
//
// GB300 issues float64 at 1/64 of the float32 rate, so kernels that form
// sines and products per (point, bin) in float64 are bound by that pipe
// alone.  The helpers here do the same arithmetic with 32-bit instructions:
//
// * a phase in cycles is a 0.64 fixed-point fraction (modulo one cycle), a
//   sum of integer products of coefficients and table entries whose absolute
//   error stays well below that of a float64 phase;
// * its cosine is a float-float pair (hi + lo) from a table of kWideTable angles
//   rotated by the remainder, with an error of about 3e-14;
// * products with a float-float weight are added by TwoSum.
//
// A float32 instruction pair (f32x2) works on two bins at a time.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "gwl_internal.h"
#include "gwl_phase.cuh"

namespace gwl {

__device__ __forceinline__ float2 splat2(float x) { return make_float2(x, x); }
// a - b, one rounding per lane
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return fma2(b, splat2(-1.f), a); }

// s + e = a + b exactly (Knuth), lane by lane
__device__ __forceinline__ void two_sum2(float2 a, float2 b, float2& s, float2& e) {
  s = add2(a, b);
  const float2 bb = sub2(s, a);
  e = add2(sub2(a, sub2(s, bb)), sub2(b, bb));
}

// One basis function's share of the phase, c phi: the coefficient as the signed
// 59-bit integer c 2^(58 - s) = ch 2^27 + cl, the table entry phi / scale as the
// 58-bit fraction mh 2^-31 + ml 2^-58.  The leading partial product goes to
// acc, the two cross ones to cross (16 of which stay below 2^62), in units of
// 2^(s - 62) and 2^(s - 89) cycles.  acc is meant modulo 2^64, 2^(s + 2) cycles:
// products of nearly 2^62 add up to more (heavy masses, large spins).
__host__ __device__ __forceinline__ void wide_mac(uint64_t& acc, int64_t& cross, int32_t ch, int32_t cl, int32_t ml,
                                                  int32_t mh) {
  acc += (uint64_t)((int64_t)ch * mh);
  cross += (int64_t)ch * ml;
  cross += (int64_t)cl * mh;
}

// The phase in cycles modulo one as 0.64 fixed point (shift = s + 2): an error
// of about 2^(s - 58) cycles, where a float64 phase of up to 2^s cycles has
// several 2^(s - 53).
__host__ __device__ __forceinline__ uint64_t wide_fraction(uint64_t acc, int64_t cross, int shift) {
  return (acc + (uint64_t)(cross >> 27)) << shift;
}

// The remainder of a 0.64 fixed-point angle about the nearest of the table's
// kWideTable = 2^11 angles: q the table index, a + b the remainder in units of
// the table's step, a in [-1/2, 1/2) in multiples of 2^-23 and b in [0, 2^-23)
// of 2^-46, both exact (the angle's lowest 7 bits are dropped: 2^-57 cycle).
static_assert(kWideTable == 2048, "wide_remainder splits the angle as 11 + 53 bits");
__device__ __forceinline__ void wide_remainder(uint64_t angle, uint32_t& q, uint32_t& a, uint32_t& b) {
  const uint32_t hi = (uint32_t)(angle >> 32) + (1u << 20), lo = (uint32_t)angle;
  q = hi >> 21;
  // 1 + a' and 2^-23 (1 + b') as float bits, a' = a + 1/2 and b' in [0, 1) of 23 bits
  a = 0x3f800000u | (__funnelshift_l(lo, hi, 2) & 0x7fffffu);
  b = 0x34000000u | ((lo >> 7) & 0x7fffffu);
}

// cos of the two angles q + a + b from the table entries t0, t1 = {C hi, C lo, T
// hi, T lo} at q, C the cosine and T = -2 pi / kWideTable times the sine:
// with u = a + b and v = (2 pi / kWideTable)^2 u^2,
//   cos = C + T u (1 - v/6) + C (-v/2 + v^2/24)
// (truncation below 3e-18).  T a, the largest correction (1.5e-3 at most), is an
// error-free product; the rest is at most 1.2e-6, in float32: an error of about
// 3e-14 rms.  |C| >= |T a| or C = 0, so three operations add them exactly.
// sin(q + a + b) is the same function at table entry q - kWideTable / 4.
struct WideArg {
  float2 a, b, v, m;  // u^2 (in table steps), -v/2 + v^2/24
};
__device__ __forceinline__ WideArg wide_arg2(uint32_t a0, uint32_t b0, uint32_t a1, uint32_t b1) {
  constexpr float k = 9.41238823040901e-06f;  // (2 pi / 2048)^2
  WideArg x;
  x.a = add2(make_float2(__uint_as_float(a0), __uint_as_float(a1)), splat2(-1.5f));
  x.b = add2(make_float2(__uint_as_float(b0), __uint_as_float(b1)), splat2(-1.1920928955078125e-07f));  // 2^-23
  const float2 u = add2(x.a, x.b);
  x.v = mul2(u, u);
  x.m = mul2(x.v, fma2(x.v, splat2(k * k / 24.0f), splat2(-0.5f * k)));
  return x;
}
__device__ __forceinline__ void wide_cos2(const float4 t0, const float4 t1, const WideArg& x, float2& ch, float2& cl) {
  constexpr float k6 = -9.41238823040901e-06f / 6.0f;
  const float2 Ch = make_float2(t0.x, t1.x), Cl = make_float2(t0.y, t1.y);
  const float2 Th = make_float2(t0.z, t1.z), Tl = make_float2(t0.w, t1.w);
  const float2 p = mul2(Th, x.a);
  float2 r = fma2(Th, x.a, mul2(p, splat2(-1.f)));
  r = fma2(Th, x.b, r);
  r = fma2(Tl, x.a, r);
  r = fma2(Ch, x.m, r);
  r = fma2(mul2(p, x.v), splat2(k6), r);
  ch = add2(Ch, p);
  const float2 e = sub2(p, sub2(ch, Ch));
  cl = add2(e, add2(r, Cl));
}

// p + e = (wh + wl)(ch + cl)
__device__ __forceinline__ void wide_term2(float2 wh, float2 wl, float2 ch, float2 cl, float2& p, float2& e) {
  p = mul2(wh, ch);
  e = fma2(wh, ch, mul2(p, splat2(-1.f)));
  e = fma2(wh, cl, e);
  e = fma2(wl, ch, e);
}

// hi + lo += p + e
__device__ __forceinline__ void wide_add2(float2& hi, float2& lo, float2 p, float2 e) {
  float2 s, err;
  two_sum2(hi, p, s, err);
  hi = s;
  lo = add2(lo, add2(err, e));
}

// The point's coefficients (LaunchArgs::wide_c, point fastest).
template <int D>
struct WidePoint {
  uint64_t c[kNumBasis], c0, x[D], q[D];
  int shift;
  __device__ __forceinline__ void load(const LaunchArgs& a, int64_t i) {
    const uint64_t* w = a.wide_c + i;
#pragma unroll
    for (int b = 0; b < kNumBasis; ++b) c[b] = w[(int64_t)b * a.B];
    c0 = w[(int64_t)kNumBasis * a.B];
    shift = (int)w[(int64_t)(kNumBasis + 1) * a.B];
#pragma unroll
    for (int d = 0; d < D; ++d) {
      x[d] = w[(int64_t)(kNumBasis + 2 + d) * a.B];
      q[d] = w[(int64_t)(kNumBasis + 2 + kMaxDet + d) * a.B];
    }
  }
  // Phi at the bin whose table row is m (kNumBasis entries)
  __device__ __forceinline__ uint64_t phase(const uint4* m) const {
    uint64_t acc = 0;
    int64_t cross = 0;
#pragma unroll
    for (int b = 0; b < kNumBasis / 2; ++b) {
      const uint4 v = m[b];
      wide_mac(acc, cross, (int32_t)(c[2 * b] >> 32), (int32_t)c[2 * b], (int32_t)v.x, (int32_t)v.y);
      wide_mac(acc, cross, (int32_t)(c[2 * b + 1] >> 32), (int32_t)c[2 * b + 1], (int32_t)v.z, (int32_t)v.w);
    }
    return c0 + wide_fraction(acc, cross, shift);
  }
};

// The terms of a pair of bins of one detector, um their weights' magnitudes and
// ut their angles (LaunchArgs::wide_w): |w| cos 2 pi (a + arg w) as p + e, the
// sine's as pi + ei.
template <bool CPLX>
__device__ __forceinline__ void wide_pair(uint64_t a0, uint64_t a1, const uint4& um, const uint4& ut, const float4* tab,
                                          float2& p, float2& e, float2& pi, float2& ei) {
  a0 += ((uint64_t)ut.y << 32) | ut.x;
  a1 += ((uint64_t)ut.w << 32) | ut.z;
  uint32_t q0, q1, ra0, ra1, rb0, rb1;
  wide_remainder(a0, q0, ra0, rb0);
  wide_remainder(a1, q1, ra1, rb1);
  const WideArg x = wide_arg2(ra0, rb0, ra1, rb1);
  const float2 wh = make_float2(__uint_as_float(um.x), __uint_as_float(um.y));
  const float2 wl = make_float2(__uint_as_float(um.z), __uint_as_float(um.w));
  float2 ch, cl;
  wide_cos2(tab[q0], tab[q1], x, ch, cl);
  wide_term2(wh, wl, ch, cl, p, e);
  if (CPLX) {
    wide_cos2(tab[(q0 - kWideTable / 4) & (kWideTable - 1)], tab[(q1 - kWideTable / 4) & (kWideTable - 1)], x, ch, cl);
    wide_term2(wh, wl, ch, cl, pi, ei);
  }
}

// Tiles of 32 points that share a CTA's tables: one, as long as that leaves fewer
// than 16,000 CTAs.  A CTA's work depends on its points' bands, and small ones fill
// the gaps: measured per call, 1 / 2 / 4 / 8 tiles, sine-Gaussian 10,000 points 520 /
// 541 / 574 / 703 us, 20,000 points 923 / 937 / 984 / 1061 us, multi-banding 4001 points
// 613 / 616 / 651 / 678 us; 128 s, 512 points (16,000 CTAs) 1251 / 1247 / 1249 / 1265 us,
// 2048 points 4707 / 4657 / 4661 / 4668 us.
// More than eight where the grid's second axis, which holds 65,535 CTAs, would not
// take the batch (above 16.8 million points).
inline int wide_tiles(int64_t chunks, int64_t tiles) {
  int per = 1;
  while (per < 8 && chunks * (tiles / (2 * per)) >= 8192) per *= 2;
  while ((tiles + per - 1) / per > 65535) per *= 2;
  return per;
}

// The kernel's limit of dynamic shared memory, before each launch that needs more
// than the 48 KB of the default: it belongs to the current device and context,
// so that one setting per process left a second device's launches refused.
template <class K>
inline cudaError_t allow_shared(K kernel, int bytes) {
  return bytes > 48 * 1024 ? cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) : cudaSuccess;
}

// Lanes that add one point's chunks: lane l of them takes chunks l, l + n, ...,
// then a fixed tree.  With 17 chunks (4 s at 2048 Hz) a whole warp per point
// took 81 us for 10,000 points, nearly all of it in the tree's float64 adds.
__host__ __device__ __forceinline__ int wide_lanes(int64_t n_chunks) { return n_chunks > 256 ? 32 : (n_chunks > 32 ? 8 : 4); }

// N: loads in flight per lane
template <int N = 8>
__device__ __forceinline__ double wide_chunk_sum(const double* q, int64_t n, int lane, int lanes) {
  double s = 0.0;
  int64_t g = lane;
  for (; g + (N - 1) * lanes < n; g += N * lanes) {
    double v[N];
#pragma unroll
    for (int u = 0; u < N; ++u) v[u] = q[g + u * lanes];
#pragma unroll
    for (int u = 0; u < N; ++u) s += v[u];
  }
  if (N > 8) {  // the rest by 8, then one by one
    for (; g + 7 * lanes < n; g += 8 * lanes) {
      double v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = q[g + u * lanes];
#pragma unroll
      for (int u = 0; u < 8; ++u) s += v[u];
    }
  }
  for (; g < n; g += lanes) s += q[g];
  for (int o = lanes / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

}  // namespace gwl
