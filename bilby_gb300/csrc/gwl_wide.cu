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
// sub-blocks' sums are added in order in float64; the finalize adds the n chunks
// with wide_lanes(n) = 4, 8 or 32 lanes (lane l takes chunks l, l + lanes, ..., then
// a fixed tree over the lanes), a number that depends on the analysis alone.
#include <cuda_runtime.h>

#include <cstdint>

#include "gwl_device.cuh"
#include "gwl_internal.h"
#include "gwl_marg_common.cuh"
#include "gwl_wide.cuh"
#include "gwl_wide_basis.cuh"

namespace gwl {

constexpr int kSub = 32;                       // bins per sub-block
constexpr int kSubs = kChunkPlain / kSub;      // sub-blocks per chunk
constexpr int kWideThreads = 32 * kSubs;       // one warp per sub-block

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

// The sub-block at table row k: its first grid index and stride.
struct WideRows {
  int64_t first, stride;
};
__device__ __forceinline__ WideRows wide_block(const LaunchArgs& a, int64_t k) {
  if (!a.wide_sub) return WideRows{k, 1};
  const int2 s = a.wide_sub[k / kSub];
  return WideRows{s.x, s.y};
}
// The grid index of the point's band end, for a list beyond the grid's last too.
__device__ __forceinline__ int64_t wide_end(const LaunchArgs& a, int64_t i) {
  return a.wide_sub ? (int64_t)a.wide_c[(int64_t)kWideEnd * a.B + i] : a.rec[i].k_end;
}
// Its rows [j0, j1) inside the band [lo, hi) of grid indices (a list's lower end
// is in its weights: its frequencies, not the grid's, are tested on the host).
__device__ __forceinline__ void wide_rows(const WideRows& b, int64_t lo, int64_t hi, int& j0, int& j1) {
  if (b.stride == 1) {
    j0 = (int)min(max(lo - b.first, (int64_t)0), (int64_t)kSub);
    j1 = (int)min(max(hi - b.first, (int64_t)0), (int64_t)kSub);
  } else {
    j0 = 0;
    j1 = hi > b.first ? (int)min((hi - b.first + b.stride - 1) / b.stride, (int64_t)kSub) : 0;
  }
  if (j1 <= j0) j1 = 0;
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
  const int64_t k0 = a.wide_base + (int64_t)blockIdx.x * kChunkPlain;
  wide_stage<D>(a, k0, tab, phi, w);
  __syncthreads();
  const int lane = threadIdx.x & 31, sub = threadIdx.x >> 5;
  const WideRows rows = wide_block(a, k0 + sub * kSub);
  const int64_t t1 = min((int64_t)(blockIdx.y + 1) * tiles, (a.B + 31) / 32);
  for (int64_t t = (int64_t)blockIdx.y * tiles; t < t1; ++t) {
    const bool have = t * 32 + lane < a.B;
    const int64_t i = have ? (a.order ? (int64_t)a.order[t * 32 + lane] : t * 32 + lane) : 0;
    int j0 = 0, j1 = 0;  // this lane's rows [j0, j1) of the sub-block
    if (have && a.rec[i].valid) wide_rows(rows, a.wide_sub ? 0 : a.rec[i].k_start, wide_end(a, i), j0, j1);
    float2 hr[D], lr[D], hm[D], lm[D];
#pragma unroll
    for (int d = 0; d < D; ++d) hr[d] = lr[d] = hm[d] = lm[d] = make_float2(0.f, 0.f);
    if (__any_sync(0xffffffffu, j1 > 0)) {
      WidePoint<D> pt;
      pt.load(a, i);
      uint64_t sh[D];
#pragma unroll
      for (int d = 0; d < D; ++d) {
        sh[d] = (uint64_t)rows.first * pt.x[d] + pt.q[d];
        pt.x[d] *= (uint64_t)rows.stride;
      }
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
        a.part[(ip * D * NC + (c >> 5)) * a.wide_chunks + blockIdx.x] = s;
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
  const int64_t k0 = a.wide_base + (int64_t)blockIdx.x * kChunkPlain;
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
  const int64_t i = blockIdx.y;
  const PointRec& r = a.rec[i];
  const WideRows rows = wide_block(a, k0 + sub * kSub);
  int j0 = 0, j1 = 0;
  allow_next();
  wait_previous();
  if (r.valid) wide_rows(rows, a.wide_sub ? 0 : r.k_start, wide_end(a, i), j0, j1);
  const int j = 2 * pr;
  const bool on0 = j >= j0 && j < j1, on1 = j + 1 >= j0 && j + 1 < j1;
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
      const uint64_t sh = (uint64_t)(rows.first + j * rows.stride) * pt.x[d] + pt.q[d];
      wide_pair<CPLX>(b0 + sh, b1 + (sh + (uint64_t)rows.stride * pt.x[d]), w0[d], w1[d], a.wide_tab, p, e, pi, ei);
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
    a.part[(i * NS + t) * a.wide_chunks + blockIdx.x] = s;
  }
}

// The chunks' sums in a fixed order, the totals and the lnL.
constexpr int kWideFinThreads = 128;

// <h|h>_d per A0^2 |Q|^2 and norm, in every lane of the point's lanes
__device__ __forceinline__ double wide_hh(const LaunchArgs& a, const PointRec& r, int64_t i, int d, int lane, int lanes) {
  if (!a.wide_sub) {
    const int64_t k1 = min(r.k_end, a.n_bins), k0 = min(r.k_start, k1);
    return a.hh_prefix[d][k1] - a.hh_prefix[d][k0];
  }
  const int64_t end = wide_end(a, i);
  double s = 0.0;
  for (int b = lane; b < a.wide_bands; b += lanes) {
    const int4 v = a.wide_band[b];
    const int64_t n = end > v.z ? min((end - v.z + v.w - 1) / v.w, (int64_t)v.y) : 0;
    s += a.wide_q[d][v.x + n] - a.wide_q[d][v.x];
  }
  for (int o = lanes / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// (one compiled body, so that both kernels below round alike)
__device__ __noinline__ void wide_totals(const LaunchArgs& a, int64_t i, const double* p, const double* sum) {
  const PointRec& r = a.rec[i];
  const int nc = a.cplx ? 2 : 1;
  double dr = 0.0, di = 0.0, hh = r.valid ? mb_fft_hh_total(a, i) : 0.0;
  for (int d = 0; d < a.n_det; ++d) {
    double x, z;
    tf2_project(a, r, d, a.wide_norm * a.wide_wscale[d], p + d * nc, &x, &z);
    dr += x;
    di += z;
    hh += tf2_norm(r, d, a.wide_norm, sum[d]);
  }
  if (!r.valid) {  // (nothing was summed, and the factors may be undefined)
    dr = di = 0.0;
    if (a.wide_sub) hh = 0.0;
  }
  finish_point(a, r, i, dr, di, hh);
}

__global__ void __launch_bounds__(kWideFinThreads) k_wide_finalize(LaunchArgs a) {
  const int lanes = wide_lanes(a.wide_chunks), lane = threadIdx.x & (lanes - 1);
  const int64_t slot = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / lanes, i = min(slot, a.B - 1);
  const int nc = a.cplx ? 2 : 1;
  double p[2 * kMaxDet], sum[kMaxDet];
  for (int c = 0; c < a.n_det * nc; ++c)
    p[c] = wide_chunk_sum(a.part + (i * a.n_det * nc + c) * a.wide_chunks, a.wide_chunks, lane, lanes);
  for (int d = 0; d < a.n_det; ++d) sum[d] = wide_hh(a, a.rec[i], i, d, lane, lanes);
  if (lane == 0 && slot < a.B) wide_totals(a, i, p, sum);
}

// Few points: a CTA per point and a warp per sum, 32 loads in flight per lane; the
// additions are those of k_wide_finalize.  Bound by the latency of the chain: one
// point of the 128 s segment (1015 chunks) 21.5 us there, 12.0 us here.
__global__ void __launch_bounds__(64 * kMaxDet) k_wide_finalize_few(LaunchArgs a) {
  __shared__ double s_p[2 * kMaxDet], s_sum[kMaxDet];
  const int lanes = wide_lanes(a.wide_chunks), lane = threadIdx.x & (lanes - 1);
  const int nc = a.cplx ? 2 : 1, c = threadIdx.x >> 5, d = c / nc;
  const int64_t i = blockIdx.x;
  double h = 0.0;
  wait_previous();
  if (c == d * nc) h = wide_hh(a, a.rec[i], i, d, lane, lanes);
  const double p = wide_chunk_sum<32>(a.part + (i * a.n_det * nc + c) * a.wide_chunks, a.wide_chunks, lane, lanes);
  if ((threadIdx.x & 31) == 0) {
    s_p[c] = p;
    if (c == d * nc) s_sum[d] = h;
  }
  __syncthreads();
  if (threadIdx.x == 0) wide_totals(a, i, s_p, s_sum);
}

// ---------------------------------------------------------------------------
// tables
// ---------------------------------------------------------------------------
struct WideScale {
  double inv[kNumBasis];
};

__device__ __forceinline__ uint64_t fraction64(double hi, double lo) {
  return (uint64_t)ldexp(hi, 64) + (uint64_t)__double2ll_rn(ldexp(lo, 64));
}

__global__ void k_wide_basis(const double* f, int64_t k0, int64_t n, int64_t pad, double lnref, WideScale sc, uint4* out) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= pad) return;
  uint64_t v[kNumBasis];
#pragma unroll
  for (int b = 0; b < kNumBasis; ++b) v[b] = 0;
  if (k >= k0 && k < n && f[k] > 0) {
    double hi[kNumBasis], lo[kNumBasis];
    wide_basis(f[k], lnref, hi, lo);
#pragma unroll
    for (int b = 0; b < kNumBasis; ++b)  // rounded to 58 bits (below 1: the scale leaves a margin of 1e-9)
      v[b] = (fraction64(hi[b] * sc.inv[b], lo[b] * sc.inv[b]) + 32) >> 6;
  }
#pragma unroll
  for (int b = 0; b < kNumBasis / 2; ++b)
    out[k * (kNumBasis / 2) + b] =
        make_uint4((uint32_t)(v[2 * b] & 0x7ffffff), (uint32_t)(v[2 * b] >> 27), (uint32_t)(v[2 * b + 1] & 0x7ffffff),
                   (uint32_t)(v[2 * b + 1] >> 27));
}

// thread: a pair of rows
__global__ void k_wide_weights(const double2* z, const double* u, const double4* ftab, double inv_scale, int64_t n,
                               uint4* out) {
  const int64_t k = 2 * ((int64_t)blockIdx.x * blockDim.x + threadIdx.x);
  if (k >= n) return;
  float2 m[2];
  uint64_t t[2];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const double g = (ftab ? ftab[k + q].w : 1.0) * u[k + q] * inv_scale;
    const double x = g == 0.0 ? 0.0 : g * z[k + q].x, y = g == 0.0 ? 0.0 : g * z[k + q].y;
    const double h = hypot(x, y), c = atan2(y, x) / kTwoPi;
    m[q].x = (float)h;
    m[q].y = (float)(h - (double)m[q].x);
    t[q] = fraction64(c < 0.0 ? c + 1.0 : c, 0.0);
  }
  out[k] = make_uint4(__float_as_uint(m[0].x), __float_as_uint(m[1].x), __float_as_uint(m[0].y), __float_as_uint(m[1].y));
  out[k + 1] = make_uint4((uint32_t)t[0], (uint32_t)(t[0] >> 32), (uint32_t)t[1], (uint32_t)(t[1] >> 32));
}

cudaError_t launch_wide_basis(const double* f, int64_t k0, int64_t n, int64_t pad, double lnref, const double* scale,
                              uint4* out, cudaStream_t s) {
  WideScale sc;
  for (int b = 0; b < kNumBasis; ++b) sc.inv[b] = 1.0 / scale[b];
  k_wide_basis<<<(unsigned)((pad + 127) / 128), 128, 0, s>>>(f, k0, n, pad, lnref, sc, out);
  return cudaGetLastError();
}

cudaError_t launch_wide_weights(const double2* z, const double* u, const double4* ftab, double inv_scale, int64_t n,
                                uint4* out, cudaStream_t s) {
  k_wide_weights<<<(unsigned)((n / 2 + 127) / 128), 128, 0, s>>>(z, u, ftab, inv_scale, n, out);
  return cudaGetLastError();
}

template <int D, bool CPLX>
static cudaError_t launch_wide_d(const LaunchArgs& a, cudaStream_t s) {
  if (wide_few(a.B, a.wide_chunks)) {
    const dim3 grid((unsigned)a.wide_chunks, (unsigned)a.B);
    return launch_after(k_wide_tf2_few<D, CPLX>, grid, kPairThreads, s, a);
  }
  constexpr int NC = CPLX ? 2 : 1;
  constexpr int smem = kWideTable * 16 + kChunkPlain * (kNumBasis * 8 + D * 16) + kSubs * D * NC * 32 * 8;
  const cudaError_t set = allow_shared(k_wide_tf2<D, CPLX>, smem);
  if (set != cudaSuccess) return set;
  const int64_t tiles = (a.B + 31) / 32;
  const int per = wide_tiles(a.wide_chunks, tiles);
  const dim3 grid((unsigned)a.wide_chunks, (unsigned)((tiles + per - 1) / per));
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
  if (wide_few(a.B, a.wide_chunks))
    return launch_after(k_wide_finalize_few, dim3((unsigned)a.B), 32 * a.n_det * (a.cplx ? 2 : 1), s, a);
  k_wide_finalize<<<(unsigned)((a.B * wide_lanes(a.wide_chunks) + kWideFinThreads - 1) / kWideFinThreads), kWideFinThreads, 0,
                    s>>>(a);
  return cudaGetLastError();
}

}  // namespace gwl
