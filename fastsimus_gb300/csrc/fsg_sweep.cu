// Plain fused FP32 simus and pfield sweeps for GB300 (sm_103a): set-up tables, the geometry
// pre-pass, the reductions and the launch dispatch.  The sweep kernels themselves are templates
// in fsg_sweep_lane.cuh, fsg_sweep_stash.cuh and fsg_sweep_kernels.cuh (pfield).
//
// simus, per chunk of scatterers:
//   geometry           once per (scatterer, source): double-float distance, amplitude
//                      (obliquity x centre-frequency sinc / sqrt(r) / n_sub), recurrence step
//                      (and half_seg sin(theta) with full-frequency directivity), written as
//                      one block per tile into an L2-sized cache (geometry_kernel here for
//                      simus_stash_kernel, lane_geometry_kernel for simus_lane_kernel);
//   sweep              simus_lane_kernel or simus_stash_kernel, one CTA per SM, each sweeping an
//                      even share of the chunk's (band, tile) units into the band's partial slot;
// then simus_reduce sums the slots' partial spectra in a fixed order.  Neither the
// scatterer x element Green's tile nor W ever leaves the SM.
// pfield: pfield_band_kernel computes its geometry in place (one band for large grids) and
// accumulates |pulse probe P|^2; pfield_reduce sums the bands and takes the square root.

#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "fsg_common.cuh"
#include "fsg_internal.h"
#include "fsg_sweep_kernels.cuh"

namespace fsg {

constexpr double kNeperToDb = 8.685889638065035;  // 20 / ln(10)

// Element / sub-element positions (utils/geometry.py:18-88, _pfield_math.py:40-67),
// per-frequency wavenumber / attenuation / spectra, per-anchor delay-apodization factors.
// Bound by the latency of its FP64 chains (sines, roots, a division); with one thread taking all of its
// jobs in turn a 64-element plan took 11.5 us, now 5.8.
__global__ void setup_tables(SetupArgs a) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int n_src = a.E * a.U;
  const bool linear = isinf(a.radius);
  if (i < setup_round(n_src)) {
    if (i >= n_src) return;
    const int e = i / a.U, u = i % a.U;
    const double off = -a.width / 2.0 + a.seg / 2.0 + u * a.seg;
    double sx, sz, co = 1.0, si = 0.0;
    if (linear) {
      // float32 arithmetic, as NumPy 2 evaluates arange(float32) - (N-1)/2 times pitch
      float idx = __fsub_rn((float)e, (float)((a.E - 1) * 0.5));
      sx = (double)__fmul_rn(idx, (float)a.pitch) + off;
      sz = 0.0;
    } else {
      double half = asin(a.pitch / 2.0 / a.radius);
      double total = half * (a.E - 1);
      double chord = 2.0 * a.radius * sin(total);
      double apex = sqrt(a.radius * a.radius - (chord / 2.0) * (chord / 2.0));
      double t0 = atan2(-chord / 2.0, apex), t1 = atan2(chord / 2.0, apex);
      const double te = (a.E > 1) ? ((e == a.E - 1) ? t1 : t0 + e * ((t1 - t0) / (a.E - 1))) : t0;
      sincos(te, &si, &co);
      sx = a.radius * si + off * co;
      sz = a.radius * co - apex - off * si;
    }
    dfl hx = split_double(sx), hz = split_double(sz);
    a.t.src_pos[i] = make_float4(hx.hi, hx.lo, hz.hi, hz.lo);
    if (u == 0) a.t.rot_e[e] = make_float2((float)co, (float)si);
    return;
  }
  i -= setup_round(n_src);
  if (i < setup_round(a.F)) {
    if (i >= a.F) return;
    double f = a.f0 + i * a.df;
    dfl k = split_double(2.0 * kPi * f / a.c);
    a.t.kf[i] = make_float2(k.hi, k.lo);
    a.t.af[i] = (float)(a.att / kNeperToDb * f / 1e6 * 1e2);
    double pr = a.probe[i];
    a.t.pp[i] = make_float2((float)(a.pulse[2 * i] * pr), (float)(a.pulse[2 * i + 1] * pr));
    a.t.probe[i] = (float)pr;
    return;
  }
  i -= setup_round(a.F);
  if (i < setup_round(a.n_anchor * a.E)) {
    if (i >= a.n_anchor * a.E) return;
    const int m = i / a.E, e = i % a.E;
    double tau = a.delays[e];
    double w = a.apod ? a.apod[e] : 1.0;
    if (isnan(tau)) { tau = 0.0; w = 0.0; }
    double f = a.f0 + (double)m * a.anchor_step * a.df;
    double s, c;
    sincos(2.0 * kPi * f * tau, &s, &c);
    a.t.da[i] = make_float2((float)(w * c), (float)(w * s));
    if (a.t.dph) a.t.dph[i] = make_float2((float)c, (float)s);
    if (a.t.wtx && m == 0) a.t.wtx[e] = (float)w;
    return;
  }
  i -= setup_round(a.n_anchor * a.E);
  if (a.n_anchor > 0 && i < a.E) {
    const double tau = isnan(a.delays[i]) ? 0.0 : a.delays[i];
    double s, c;
    sincos(2.0 * kPi * a.df * tau, &s, &c);
    a.t.dstep[i] = make_float2((float)c, (float)s);
  }
}

// Geometry of a chunk's tiles, once per (scatterer, source) for all frequency bands.  A CTA
// takes one tile at a time: its scatterers' coordinates are split into double-float pairs
// once, then thread i handles (source, point) items i, i + 256, ...; consecutive threads take
// consecutive points, so the writes of a warp are contiguous.  Points past the end of the
// scatterer list repeat the tile's first point (their rc is 0 in the sweep).
__global__ void __launch_bounds__(kThreads) geometry_kernel(const BandArgs A, int64_t chunk_tiles) {
  __shared__ float4 xz[kThreads];  // st <= 64 points of the tile
  const SmemLayout L = smem_layout(A.st, A.E, A.U, A.plane_pad, A.C.ffd != 0);
  const int items = A.n_src * A.st;
  for (int64_t tile = blockIdx.x; tile < chunk_tiles; tile += gridDim.x) {
    __syncthreads();
    if (threadIdx.x < A.st) {
      int64_t s = A.chunk_s0 + tile * A.st + threadIdx.x;
      if (s >= A.n_pts) s = A.chunk_s0 + tile * A.st;
      const dfl hx = load_coord(A.pts + 2 * s), hz = load_coord(A.pts + 2 * s + 1);
      xz[threadIdx.x] = make_float4(hx.hi, hx.lo, hz.hi, hz.lo);
    }
    __syncthreads();
    unsigned char* blk = A.geo + tile * A.geo_bytes;
    float* rhi = reinterpret_cast<float*>(blk + L.off_rhi);
    float* rlo = reinterpret_cast<float*>(blk + L.off_rlo);
    float* amp = reinterpret_cast<float*>(blk + L.off_amp);
    float2* stp = reinterpret_cast<float2*>(blk + L.off_step);
    float* dir = A.C.ffd ? reinterpret_cast<float*>(blk + L.off_dir) : nullptr;
    for (int it = threadIdx.x; it < items; it += blockDim.x) {
      const int pt = it % A.st, src = it / A.st;
      const int e = src / A.U, u = src - e * A.U;
      const float4 c = xz[pt];
      store_geometry(rhi, rlo, amp, stp, dir, u * L.plane + e * L.pitch + pt, dfl{c.x, c.y}, dfl{c.z, c.w}, A, src);
    }
  }
}

// out (layout) = probe_f * corr * sum over slots of partial[q][f][e], fixed slot order.
__global__ void simus_reduce(const float2* __restrict__ partial, int n_slices, int F, int E,
                             const float* __restrict__ probe, float corr, int full, int n_rows, int idx0,
                             const int* __restrict__ status, const double* __restrict__ rx_delays, double f0,
                             double df, float2* __restrict__ out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (int64_t)n_rows * E) return;
  if (*status != FSG_OK) {  // a sweep CTA gave up waiting: make the failure visible in the output
    out[i] = make_float2(__int_as_float(0x7fc00000), __int_as_float(0x7fc00000));
    return;
  }
  const int row = (int)(i / E), e = (int)(i % E);
  const int f = full ? row - idx0 : row;
  float2 acc = make_float2(0.f, 0.f);
  if (f >= 0 && f < F) {
#pragma unroll 8
    for (int q = 0; q < n_slices; ++q) acc = cadd(acc, partial[((size_t)q * F + f) * E + e]);
    float s = probe[f] * corr;
    acc = make_float2(acc.x * s, acc.y * s);
    if (rx_delays) {
      double tau = rx_delays[e];
      if (isnan(tau)) tau = 0.0;
      double sn, cs;
      sincos(2.0 * kPi * (f0 + f * df) * tau, &sn, &cs);
      acc = cmul(acc, make_float2((float)cs, (float)-sn));
    }
  }
  out[i] = acc;
}

__global__ void pfield_reduce(const float* __restrict__ partial, int n_bands, int64_t n_pts, float corr,
                              float* __restrict__ out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_pts) return;
  float acc = 0.f;
  for (int b = 0; b < n_bands; ++b) acc += partial[(size_t)b * n_pts + i];
  out[i] = sqrtf(acc * corr);
}

cudaError_t launch_simus_any(int U, const SweepConfig& c, const BandArgs& A, cudaStream_t s) {
  if (c.kind == 2) return launch_simus_lane(U, c, A, s);
  return A.C.ffd ? launch_simus_stash_ffd(U, c, A, s) : launch_simus_stash(U, c, A, s);
}

cudaError_t launch_pfield_band_any(const SweepConfig& c, const BandArgs& A, cudaStream_t s) {
  return A.C.ffd ? launch_pfield_band_ffd(c, A, s) : launch_pfield_band_gn<0>(c, A, s);
}

}  // namespace fsg
