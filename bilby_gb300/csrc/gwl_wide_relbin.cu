// Float64 relative binning of TaylorF2 (bilby/gw/likelihood/relative.py:365-402)
// on the 32-bit pipes (gwl_wide.cuh).
//
// With the ratio q_e = h_e g_e at edge e (g = 1 / h0), r0 = (q_{b+1} + q_b) / 2 and
// r1 = (q_{b+1} - q_b) / (f_{b+1} - f_b) are linear in the edges, so that
//   <d|h> = sum_b a0 conj(r0) + a1 conj(r1) = sum_e conj(h_e) w_e,
//   <h|h> = sum_b b0 |r0|^2 + 2 b1 Re(r0 conj r1)
//         = sum_e c_e |h_e|^2 + sum_b m_b |h_b| |h_{b+1}| cos(arg q_{b+1} - arg q_b)
// with w, c and m from the summary data (set up on the host).  |h_e| has no phase,
// so its sum is a difference of prefix sums; what is left per edge and detector
// are two cosines of fixed-point angles, evaluated as one packed pair.
//
// One warp per point, lane l at edge 31 q + l in pass q (the neighbour's phase by
// a shuffle); float-float sums over the lanes in a fixed tree; a second kernel,
// thread = point, adds the detectors in float64.  In float64 the model, three
// sincos and the sums per edge kept that pipe busy for 690 us per 16,384 points
// (128 s, three detectors, 62 edges); here they take 41 us.
#include <cuda_runtime.h>

#include <cstdint>

#include "gwl_device.cuh"
#include "gwl_internal.h"
#include "gwl_marg_common.cuh"
#include "gwl_wide.cuh"

namespace gwl {

constexpr int kRbThreads = 256;

template <int D, bool CPLX>
__global__ void __launch_bounds__(kRbThreads) k_wide_relbin(LaunchArgs a) {
  __shared__ float4 tab[kWideTable];
  for (int q = threadIdx.x; q < kWideTable; q += kRbThreads) tab[q] = a.wide_tab[q];
  __syncthreads();
  constexpr int NC = CPLX ? 6 : 4;  // floats per detector: sums' hi words (re, cross), lo words, im
  const int lane = threadIdx.x & 31, nE = a.rb_edges;
  const int64_t step = (int64_t)gridDim.x * (kRbThreads / 32);
  for (int64_t i = (int64_t)blockIdx.x * (kRbThreads / 32) + (threadIdx.x >> 5); i < a.B; i += step) {
    const PointRec& r = a.rec[i];
    float2 hi[D], lo[D], him[D], lom[D];
#pragma unroll
    for (int d = 0; d < D; ++d) hi[d] = lo[d] = him[d] = lom[d] = make_float2(0.f, 0.f);
    int n_in = 0;  // edges below f_ISCO
    if (r.valid) {
      WidePoint<D> pt;
      pt.load(a, i);
      const int64_t k_end = r.k_end;
      for (int base = 0; base < nE - 1; base += 31) {
        const int e = min(base + lane, nE - 1);
        const int64_t k = a.rb_index[e], kn = a.rb_index[min(e + 1, nE - 1)];
        const bool in = base + lane < nE && k < k_end;
        const bool edge = in && (lane < 31 || e == nE - 1), bin = in && lane < 31 && e + 1 < nE && kn < k_end;
        n_in += __popc(__ballot_sync(0xffffffffu, edge));
        const uint64_t ph = pt.phase(a.wide_phi + (int64_t)e * (kNumBasis / 2));
        const uint64_t diff = __shfl_down_sync(0xffffffffu, ph, 1) - ph;
#pragma unroll
        for (int d = 0; d < D; ++d) {
          const uint4 um = a.wide_w[d][2 * e], ut = a.wide_w[d][2 * e + 1];
          float2 p, e2, pi, ei;
          wide_pair<CPLX>(ph + (uint64_t)k * pt.x[d] + pt.q[d], diff + (uint64_t)(kn - k) * pt.x[d], um, ut, tab, p, e2, pi,
                          ei);
          if (!edge) p.x = e2.x = pi.x = ei.x = 0.f;
          if (!bin) p.y = e2.y = 0.f;
          wide_add2(hi[d], lo[d], p, e2);
          if (CPLX) wide_add2(him[d], lom[d], pi, ei);
        }
      }
    }
#pragma unroll
    for (int d = 0; d < D; ++d) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float2 oh = make_float2(__shfl_xor_sync(0xffffffffu, hi[d].x, o), __shfl_xor_sync(0xffffffffu, hi[d].y, o));
        const float2 ol = make_float2(__shfl_xor_sync(0xffffffffu, lo[d].x, o), __shfl_xor_sync(0xffffffffu, lo[d].y, o));
        wide_add2(hi[d], lo[d], oh, ol);
        if (CPLX) {
          const float2 mh = make_float2(__shfl_xor_sync(0xffffffffu, him[d].x, o), 0.f);
          const float2 ml = make_float2(__shfl_xor_sync(0xffffffffu, lom[d].x, o), 0.f);
          wide_add2(him[d], lom[d], mh, ml);
        }
      }
    }
    if (lane == 0) {
      float* out = reinterpret_cast<float*>(a.part) + i * (D * NC + 1);
#pragma unroll
      for (int d = 0; d < D; ++d) {
        out[d * NC] = hi[d].x;
        out[d * NC + 1] = lo[d].x;
        out[d * NC + 2] = hi[d].y;
        out[d * NC + 3] = lo[d].y;
        if (CPLX) {
          out[d * NC + 4] = him[d].x;
          out[d * NC + 5] = lom[d].x;
        }
      }
      out[D * NC] = __int_as_float(n_in);
    }
  }
}

__global__ void k_wide_relbin_finalize(LaunchArgs a) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.B) return;
  const PointRec& r = a.rec[i];
  const int nc = a.cplx ? 6 : 4;
  const float* p = reinterpret_cast<const float*>(a.part) + i * (a.n_det * nc + 1);
  const int n = __float_as_int(p[a.n_det * nc]);
  double dr = 0.0, di = 0.0, hh = 0.0;
  for (int d = 0; d < a.n_det; ++d) {
    const float* v = p + d * nc;
    const double s[2] = {(double)v[0] + (double)v[1], a.cplx ? (double)v[4] + (double)v[5] : 0.0};
    double x, z;
    tf2_project(a, r, d, a.wide_wscale[d], s, &x, &z);
    dr += x;
    di += z;
    hh += tf2_norm(r, d, 1.0, a.wide_q[d][n] + a.rbw_scale[d] * ((double)v[2] + (double)v[3]));
  }
  if (!r.valid) dr = di = hh = 0.0;  // (nothing was summed, and the factors may be undefined)
  finish_point(a, r, i, dr, di, hh);
}

template <int D, bool CPLX>
static cudaError_t launch_wide_relbin_d(const LaunchArgs& a, cudaStream_t s) {
  const int64_t ctas = (a.B + kRbThreads / 32 - 1) / (kRbThreads / 32);
  k_wide_relbin<D, CPLX><<<(unsigned)(ctas < 152 * 4 ? ctas : 152 * 4), kRbThreads, 0, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_wide_relbin(const LaunchArgs& a, cudaStream_t s) {
  cudaError_t e;
  switch (2 * a.n_det + (a.cplx ? 1 : 0)) {
    case 2: e = launch_wide_relbin_d<1, false>(a, s); break;
    case 3: e = launch_wide_relbin_d<1, true>(a, s); break;
    case 4: e = launch_wide_relbin_d<2, false>(a, s); break;
    case 5: e = launch_wide_relbin_d<2, true>(a, s); break;
    case 6: e = launch_wide_relbin_d<3, false>(a, s); break;
    case 7: e = launch_wide_relbin_d<3, true>(a, s); break;
    case 8: e = launch_wide_relbin_d<4, false>(a, s); break;
    default: e = launch_wide_relbin_d<4, true>(a, s); break;
  }
  if (e != cudaSuccess) return e;
  k_wide_relbin_finalize<<<(unsigned)((a.B + 127) / 128), 128, 0, s>>>(a);
  return cudaGetLastError();
}

}  // namespace gwl
