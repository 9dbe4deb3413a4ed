// The float64 TaylorF2 likelihood (bilby/gw/likelihood/base.py:419-477 over
// bilby/gw/detector/interferometer.py:303-368 and bilby/gw/utils.py:118-138)
// on the 32-bit pipes: phases in 0.64 fixed point, float-float sines and
// products (gwl_wide.cuh).
//
// Re <d|h>_d = 4/T A0 |Q_d| sum_k |w_k| cos 2 pi (Phi_k + k dt_d df + alpha_d +
// theta_k), with w = f^(-7/6) d / S = |w| e^{2 pi i theta}, alpha_d = arg(conj
// Q_d); the imaginary part (phase marginalisation, requested inner products)
// takes the sine and leaves alpha_d to the finalize.  Phi_k = sum_b c_b
// phi_b(f_k) over the eight basis functions of the 3.5PN phase.
//
// Summation order, the same for every batch size and launch shape: a chunk of
// kChunkPlain bins is cut into sub-blocks of 32; in a sub-block the even and
// the odd bins are added in order into one float-float sum each; the
// sub-blocks' sums are added in order in float64; the finalize adds the chunks
// (lane l of a warp takes chunks l, l + 32, ..., then a fixed tree).
#include <cuda_runtime.h>

#include <cstdint>

#include "gwl_device.cuh"
#include "gwl_internal.h"
#include "gwl_marg_common.cuh"
#include "gwl_wide.cuh"

namespace gwl {

constexpr int kSub = 32;                       // bins per sub-block
constexpr int kSubs = kChunkPlain / kSub;      // sub-blocks per chunk
constexpr int kWideThreads = 32 * kSubs;       // one warp per sub-block

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
    int64_t acc = 0, cross = 0;
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

// The cosine table, the chunk's phase basis and the chunk's weights.
template <int D>
__device__ __forceinline__ void wide_stage(const LaunchArgs& a, int64_t k0, float4* tab, uint4* phi, uint4* w) {
  for (int q = threadIdx.x; q < kWideTable; q += kWideThreads) tab[q] = a.wide_tab[q];
  const uint4* src = a.wide_phi + k0 * (kNumBasis / 2);
  for (int q = threadIdx.x; q < kChunkPlain * kNumBasis / 2; q += kWideThreads) phi[q] = src[q];
#pragma unroll
  for (int d = 0; d < D; ++d)
    for (int q = threadIdx.x; q < kChunkPlain; q += kWideThreads) w[d * kChunkPlain + q] = a.wide_w[d][k0 + q];
}

// Batches.  CTA (chunk, point slice): one warp per sub-block, lane = point, 32
// points at a time; the chunk's tables stay in shared memory over the slice's
// points.  Bound by the heavier half of the FMA pipe (72% of its cycles: the
// 64-bit multiply-adds of the phase and the packed float pairs), two CTAs per
// SM by registers; three CTAs (80 registers) spill and take 1.41 ms.
// 128 s, three detectors, 512 points: 1.19 ms for this kernel, 1.32 ms for the
// call, where the kernel in float64 (its pipe 88% busy) took 25.7 ms; the error
// of lnL against 80-bit arithmetic went from 7e-10 to 4e-12 rms.
template <int D, bool CPLX>
__global__ void __launch_bounds__(kWideThreads, 2) k_wide_tf2(LaunchArgs a, int tiles) {
  constexpr int NC = CPLX ? 2 : 1;
  extern __shared__ __align__(16) unsigned char smem[];
  float4* tab = reinterpret_cast<float4*>(smem);
  uint4* phi = reinterpret_cast<uint4*>(tab + kWideTable);
  uint4* w = reinterpret_cast<uint4*>(phi + kChunkPlain * kNumBasis / 2);
  double* sums = reinterpret_cast<double*>(w + D * kChunkPlain);  // [kSubs][D * NC][32]
  const int64_t k0 = a.k_base + (int64_t)blockIdx.x * kChunkPlain;
  wide_stage<D>(a, k0, tab, phi, w);
  __syncthreads();
  const int lane = threadIdx.x & 31, sub = threadIdx.x >> 5;
  const int64_t ks = k0 + sub * kSub;
  const int64_t t1 = min((int64_t)(blockIdx.y + 1) * tiles, (a.B + 31) / 32);
  for (int64_t t = (int64_t)blockIdx.y * tiles; t < t1; ++t) {
    const bool have = t * 32 + lane < a.B;
    const int64_t i = have ? (a.order ? (int64_t)a.order[t * 32 + lane] : t * 32 + lane) : 0;
    int64_t lo = 0, hi = 0;
    if (have && a.rec[i].valid) {
      lo = max(a.rec[i].k_start, ks);
      hi = min(a.rec[i].k_end, ks + kSub);
    }
    const int j0 = (int)(lo - ks), j1 = hi > lo ? (int)(hi - ks) : 0;  // this lane's bins [j0, j1) of the sub-block
    float2 hr[D], lr[D], hm[D], lm[D];
#pragma unroll
    for (int d = 0; d < D; ++d) hr[d] = lr[d] = hm[d] = lm[d] = make_float2(0.f, 0.f);
    if (__any_sync(0xffffffffu, j1 > 0)) {
      WidePoint<D> pt;
      pt.load(a, i);
      uint64_t sh[D];
#pragma unroll
      for (int d = 0; d < D; ++d) sh[d] = (uint64_t)ks * pt.x[d] + pt.q[d];
      const uint4* m = phi + sub * kSub * (kNumBasis / 2);
      const uint4* ws = w + sub * kSub;
#pragma unroll 1
      for (int j = 0; j < kSub; j += 2) {
        if (j + 2 > j0 && j < j1) {
          const uint64_t b0 = pt.phase(m), b1 = pt.phase(m + kNumBasis / 2);
          const bool on0 = j >= j0, on1 = j + 1 < j1, edge = !(on0 && on1);  // a pair across the band's edge
#pragma unroll
          for (int d = 0; d < D; ++d) {
            float2 p, e, pi, ei;
            wide_pair<CPLX>(b0 + sh[d], b1 + (sh[d] + pt.x[d]), ws[d * kChunkPlain], ws[d * kChunkPlain + 1], tab, p, e, pi,
                            ei);
            if (edge) {
              if (!on0) p.x = e.x = 0.f;
              if (!on1) p.y = e.y = 0.f;
              if (CPLX && !on0) pi.x = ei.x = 0.f;
              if (CPLX && !on1) pi.y = ei.y = 0.f;
            }
            wide_add2(hr[d], lr[d], p, e);
            if (CPLX) wide_add2(hm[d], lm[d], pi, ei);
          }
        }
#pragma unroll
        for (int d = 0; d < D; ++d) sh[d] += 2 * pt.x[d];
        m += kNumBasis;
        ws += 2;
      }
    }
#pragma unroll
    for (int d = 0; d < D; ++d) {
      sums[(sub * D * NC + d * NC) * 32 + lane] = ((double)hr[d].x + (double)lr[d].x) + ((double)hr[d].y + (double)lr[d].y);
      if (CPLX)
        sums[(sub * D * NC + d * NC + 1) * 32 + lane] =
            ((double)hm[d].x + (double)lm[d].x) + ((double)hm[d].y + (double)lm[d].y);
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

// Few points: lane = pair of bins.  CTA (chunk, point): each of 128 threads
// forms the terms of two bins, then one thread per (sub-block, sum, parity)
// adds its 16 terms in the order of k_wide_tf2.  A lane per point leaves a
// small batch on one warp per sub-block that walks its 32 bins in sequence; one
// point of the 128 s segment takes 15 us here (2 ms in the float64 kernel, which
// had one thread per 256 bins).
constexpr int kPairThreads = kChunkPlain / 2;

template <int D, bool CPLX>
__global__ void __launch_bounds__(kPairThreads) k_wide_tf2_few(LaunchArgs a) {
  constexpr int NC = CPLX ? 2 : 1, NS = D * NC;
  constexpr int kPer = kSub / 2, kRow = kPer + 1;  // pairs per sub-block, padded
  __shared__ float2 term[NS][2][kSubs][kRow];      // (p, e) of one bin
  __shared__ double part[NS][2][kSubs];
  const int64_t k0 = a.k_base + (int64_t)blockIdx.x * kChunkPlain;
  const int t = threadIdx.x, sub = t / kPer, pr = t % kPer;
  const int64_t k = k0 + 2 * t;
  uint4 m[kNumBasis];
#pragma unroll
  for (int b = 0; b < kNumBasis; ++b) m[b] = a.wide_phi[k * (kNumBasis / 2) + b];
  uint4 w0[D], w1[D];
#pragma unroll
  for (int d = 0; d < D; ++d) {
    w0[d] = a.wide_w[d][k];
    w1[d] = a.wide_w[d][k + 1];
  }
  for (int64_t i = blockIdx.y; i < a.B; i += gridDim.y) {
    const PointRec& r = a.rec[i];
    const int64_t lo = r.k_start, hi = r.valid ? r.k_end : 0;
    const bool on0 = k >= lo && k < hi, on1 = k + 1 >= lo && k + 1 < hi;
    WidePoint<D> pt;
    uint64_t b0 = 0, b1 = 0;
    if (on0 || on1) {
      pt.load(a, i);
      b0 = pt.phase(m);
      b1 = pt.phase(m + kNumBasis / 2);
    }
#pragma unroll
    for (int d = 0; d < D; ++d) {
      float2 p, e, pi, ei;
      p = e = pi = ei = make_float2(0.f, 0.f);
      if (on0 || on1) {
        const uint64_t sh = (uint64_t)k * pt.x[d] + pt.q[d];
        wide_pair<CPLX>(b0 + sh, b1 + (sh + pt.x[d]), w0[d], w1[d], a.wide_tab, p, e, pi, ei);
      }
      term[d * NC][0][sub][pr] = on0 ? make_float2(p.x, e.x) : make_float2(0.f, 0.f);
      term[d * NC][1][sub][pr] = on1 ? make_float2(p.y, e.y) : make_float2(0.f, 0.f);
      if (CPLX) {
        term[d * NC + 1][0][sub][pr] = on0 ? make_float2(pi.x, ei.x) : make_float2(0.f, 0.f);
        term[d * NC + 1][1][sub][pr] = on1 ? make_float2(pi.y, ei.y) : make_float2(0.f, 0.f);
      }
    }
    __syncthreads();
    for (int c = t; c < NS * 2 * kSubs; c += kPairThreads) {
      const float2* src = &term[0][0][0][0] + (int64_t)c * kRow;
      float h = 0.f, l = 0.f;
#pragma unroll
      for (int q = 0; q < kPer; ++q) {
        const float2 v = src[q];
        const float s = __fadd_rn(h, v.x), bb = __fsub_rn(s, h);
        const float err = __fadd_rn(__fsub_rn(h, __fsub_rn(s, bb)), __fsub_rn(v.x, bb));
        h = s;
        l = __fadd_rn(l, __fadd_rn(err, v.y));
      }
      (&part[0][0][0])[c] = (double)h + (double)l;
    }
    __syncthreads();
    if (t < NS) {
      double s = part[t][0][0] + part[t][1][0];
#pragma unroll
      for (int q = 1; q < kSubs; ++q) s += part[t][0][q] + part[t][1][q];
      a.part[(i * NS + t) * a.n_chunks + blockIdx.x] = s;
    }
  }
}

// One warp per point: the chunks' sums in a fixed order, the totals and the
// lnL.
constexpr int kWideFinWarps = 4;

__global__ void __launch_bounds__(32 * kWideFinWarps) k_wide_finalize(LaunchArgs a) {
  const int lane = threadIdx.x & 31;
  const int64_t i = (int64_t)blockIdx.x * kWideFinWarps + (threadIdx.x >> 5);
  if (i >= a.B) return;  // uniform over the warp
  const PointRec& r = a.rec[i];
  const int nc = a.cplx ? 2 : 1;
  double p[2 * kMaxDet];
  for (int c = 0; c < a.n_det * nc; ++c) {
    const double* q = a.part + (i * a.n_det * nc + c) * a.n_chunks;
    double s = 0.0;
    for (int64_t g = lane; g < a.n_chunks; g += 32) s += q[g];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    p[c] = s;
  }
  if (lane == 0) {
    double dr = 0.0, di = 0.0, hh = 0.0;
    for (int d = 0; d < a.n_det; ++d) {
      double x, z, h;
      tf2_detector_totals(a, r, d, p + d * nc, &x, &z, &h);
      dr += x;
      di += z;
      hh += h;
    }
    finish_point(a, r, i, dr, di, hh);
  }
}

template <int D, bool CPLX>
static cudaError_t launch_wide_d(const LaunchArgs& a, cudaStream_t s) {
  if (a.B <= kWideFewPoints) {
    const dim3 grid((unsigned)a.n_chunks, (unsigned)a.B);
    k_wide_tf2_few<D, CPLX><<<grid, kPairThreads, 0, s>>>(a);
    return cudaGetLastError();
  }
  constexpr int NC = CPLX ? 2 : 1;
  constexpr int smem = kWideTable * 16 + kChunkPlain * (kNumBasis * 8 + D * 16) + kSubs * D * NC * 32 * 8;
  static const cudaError_t set =
      cudaFuncSetAttribute(k_wide_tf2<D, CPLX>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (set != cudaSuccess) return set;
  const int64_t tiles = (a.B + 31) / 32;
  // up to eight tiles share a CTA's tables while the grid stays at eight CTAs
  // per SM or more
  int per = 1;
  while (per < 8 && a.n_chunks * (tiles / (2 * per)) >= 8 * 152) per *= 2;
  const dim3 grid((unsigned)a.n_chunks, (unsigned)((tiles + per - 1) / per));
  k_wide_tf2<D, CPLX><<<grid, kWideThreads, smem, s>>>(a, per);
  return cudaGetLastError();
}

cudaError_t launch_wide(const LaunchArgs& a, cudaStream_t s) {
  cudaError_t e;
  switch (2 * a.n_det + (a.cplx ? 1 : 0)) {
    case 2: e = launch_wide_d<1, false>(a, s); break;
    case 3: e = launch_wide_d<1, true>(a, s); break;
    case 4: e = launch_wide_d<2, false>(a, s); break;
    case 5: e = launch_wide_d<2, true>(a, s); break;
    case 6: e = launch_wide_d<3, false>(a, s); break;
    case 7: e = launch_wide_d<3, true>(a, s); break;
    case 8: e = launch_wide_d<4, false>(a, s); break;
    default: e = launch_wide_d<4, true>(a, s); break;
  }
  if (e != cudaSuccess) return e;
  k_wide_finalize<<<(unsigned)((a.B + kWideFinWarps - 1) / kWideFinWarps), 32 * kWideFinWarps, 0, s>>>(a);
  return cudaGetLastError();
}

}  // namespace gwl
