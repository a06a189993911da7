// Device functions of the plain sweep kernels and the pfield kernel's template and launcher, which
// fsg_sweep.cu (without full-frequency directivity) and fsg_sweep_ffd.cu (with it) instantiate.
#pragma once

#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "fsg_common.cuh"
#include "fsg_internal.h"
#include "fsg_tc.cuh"

namespace fsg {

constexpr size_t kBulkPiece = 32 * 1024;            // bytes per TMA bulk copy instruction
constexpr uint32_t kBulkWaitTries = 1u << 26;       // bound on the polls of one copy's mbarrier

__device__ __forceinline__ dfl load_coord(const double* p) {
  return split_double(*p);
}

// Loads the band's per-frequency tables into shared memory.
__device__ __forceinline__ void load_band_tables(const BandArgs& A, const PfieldLayout& L, unsigned char* sm, int f_b0) {
  float2* pp = reinterpret_cast<float2*>(sm + L.off_pp);
  float2* ka = reinterpret_cast<float2*>(sm + L.off_ka);
  float* aa = reinterpret_cast<float*>(sm + L.off_aa);
  float2* da = reinterpret_cast<float2*>(sm + L.off_da);
  const int na = A.fb / kAnchor;
  float* kb = reinterpret_cast<float*>(sm + L.off_kb);
  for (int i = threadIdx.x; i < A.fb; i += blockDim.x) {
    int f = f_b0 + i;
    pp[i] = (f < A.F) ? A.t.pp[f] : make_float2(0.f, 0.f);
    const float k = A.t.kf[min(f, A.F - 1)].x;
    kb[i] = k * k;
  }
  for (int m = threadIdx.x; m < na; m += blockDim.x) {
    int f = min(f_b0 + m * kAnchor, A.F - 1);
    ka[m] = A.t.kf[f];
    aa[m] = A.t.af[f];
  }
  for (int i = threadIdx.x; i < na * A.E; i += blockDim.x) {
    int m = i / A.E, e = i % A.E;
    int ga = min(f_b0 / kAnchor + m, A.n_anchor - 1);
    da[i] = A.t.da[ga * A.E + e];
  }
}

// Geometry of one (point, source) into the geometry arrays at word index idx; with
// full-frequency directivity also half_seg * sin(theta) into dir.
__device__ __forceinline__ void store_geometry(float* rhi, float* rlo, float* amp, float2* stp, float* dir, int idx,
                                               dfl xs, dfl zs, const BandArgs& A, int src) {
  const int e = src / A.U;
  const SrcGeo geo = source_geometry(xs, zs, A.t.src_pos[src], A.t.rot_e[e], A.C);
  rhi[idx] = geo.r_hi;
  rlo[idx] = geo.r_lo;
  amp[idx] = geo.amp;
  stp[idx] = geo.step;
  if (dir) dir[idx] = A.C.half_seg * geo.sth;
}

// TX over one band for one tile, with the tile's geometry computed here first.
// Each thread owns point `sl` of the tile and eight pairs of sources 2 (g + GN p), 2 (g + GN p) + 1;
// the GN threads of a point are GN adjacent lanes of one warp.  Frequencies are processed in blocks
// of GN steps: every lane keeps its partial source sums of the block, then a reduce-scatter across
// the GN lanes (log2 GN shuffle levels, halving the exchanged values each level) leaves lane g with
// the full sum of frequency block + g.  `sink(f_local, psum)` is therefore called by every
// lane, once per block, each for its own frequency.  With DT > 0 every term is weighted by its
// directivity at the step's frequency, sinc(k_f half_seg sin(theta)) (a polynomial of DT terms), folded
// into the packed source sum as a fused multiply-add.
//
// What bounds it: the FP32 pipe and its register read ports (a source step is four packed instructions
// per pair, its sum two).  A thread reads back only the geometry it wrote, so that the arrays are laid
// out by thread and read as 16-byte words; with arrays shared by the tile, their bank padding searched
// on the host and a division by U per source and anchor, the call took 2,978 us for 131,072 points
// and 128 elements x 2 sources, now 2,163, and 283 us (190 of them on the host) for 8,181 points and
// 64 elements, now 87.
template <int GN, int DT, class Sink>
__device__ __forceinline__ void tx_tile(const BandArgs& A, const PfieldLayout& L, unsigned char* sm, int64_t p_idx,
                                        int g, Sink& sink) {
  constexpr int kPairs = kSrcPerThread / 2;
  constexpr bool FFD = DT > 0;
  float4* b_r = reinterpret_cast<float4*>(sm + L.off_r) + threadIdx.x;        // r_hi, r_hi, r_lo, r_lo
  float4* b_st = reinterpret_cast<float4*>(sm + L.off_step) + threadIdx.x;    // step re, re, im, im
  float2* b_amp = reinterpret_cast<float2*>(sm + L.off_amp) + threadIdx.x;
  float2* b_dir = reinterpret_cast<float2*>(sm + L.off_dir) + threadIdx.x;
  const float2* ka = reinterpret_cast<const float2*>(sm + L.off_ka);
  const float* aa = reinterpret_cast<const float*>(sm + L.off_aa);
  const float2* da = reinterpret_cast<const float2*>(sm + L.off_da);
  const float* kb = reinterpret_cast<const float*>(sm + L.off_kb);
  // src / U = src * mag >> 20, exact for src and U up to 512
  const unsigned mag = ((1u << 20) + A.U - 1) / A.U;

  // 1. geometry of my sources, parked in shared memory (rolled loop: one copy of the code)
  {
    const dfl xs = load_coord(A.pts + 2 * p_idx);
    const dfl zs = load_coord(A.pts + 2 * p_idx + 1);
#pragma unroll 1
    for (int p = 0; p < kPairs; ++p) {
      SrcGeo q[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int src = 2 * (g + GN * p) + h;
        q[h] = SrcGeo{0.f, 0.f, 0.f, make_float2(0.f, 0.f), 0.f};
        if (src < A.n_src) {
          const int e = (int)((src * mag) >> 20);
          q[h] = source_geometry(xs, zs, A.t.src_pos[src], A.t.rot_e[e], A.C);
          q[h].step = cmul(q[h].step, A.t.dstep[e]);
        }
      }
      b_r[p * kThreads] = make_float4(q[0].r_hi, q[1].r_hi, q[0].r_lo, q[1].r_lo);
      b_st[p * kThreads] = make_float4(q[0].step.x, q[1].step.x, q[0].step.y, q[1].step.y);
      b_amp[p * kThreads] = make_float2(q[0].amp, q[1].amp);
      if (FFD) b_dir[p * kThreads] = sqr2(make_float2(A.C.half_seg * q[0].sth, A.C.half_seg * q[1].sth));
    }
  }
  // 2. transmit sweep: exact anchor every kTxAnchor steps, FP32 recurrence in between.  The two
  // sources of a pair share one packed FP32x2 lane pair (real and imaginary parts in separate pairs).
  float2 Gr[kPairs], Gi[kPairs], Sr[kPairs], Si[kPairs], Sn[kPairs];
  float2 Dh[FFD ? kPairs : 1];  // FFD: (half_seg sin(theta))^2 of the pair's two sources
#pragma unroll
  for (int p = 0; p < kPairs; ++p) {
    const float4 s = b_st[p * kThreads];
    Sr[p] = make_float2(s.x, s.y);
    Si[p] = make_float2(s.z, s.w);
    Sn[p] = make_float2(-s.z, -s.w);
    if constexpr (FFD) Dh[p] = b_dir[p * kThreads];
  }
  const int n_tx_anchor = (A.fb + kTxAnchor - 1) / kTxAnchor;
  for (int m = 0; m < n_tx_anchor; ++m) {
    const int am = m * (kTxAnchor / kAnchor);  // index into the band's kAnchor-spaced tables
    const float2 k0 = ka[am];
    const float a0 = aa[am];
    const float2* d0 = da + am * A.E;
#pragma unroll
    for (int p = 0; p < kPairs; ++p) {
      const int src = 2 * (g + GN * p);
      const int e0 = min((int)((src * mag) >> 20), A.E - 1), e1 = min((int)(((src + 1) * mag) >> 20), A.E - 1);
      const float4 r = b_r[p * kThreads];
      const float2 am2 = b_amp[p * kThreads];
      const float2 g0 = cmul(anchor_value(r.x, r.z, am2.x, k0, a0), d0[e0]);
      const float2 g1 = cmul(anchor_value(r.y, r.w, am2.y, k0, a0), d0[e1]);
      Gr[p] = make_float2(g0.x, g1.x);
      Gi[p] = make_float2(g0.y, g1.y);
    }
    const int n_steps = min(kTxAnchor, A.fb - m * kTxAnchor);  // a multiple of kAnchor, so of GN
#pragma unroll 1
    for (int jb = 0; jb < n_steps; jb += GN) {
      float vr[GN], vi[GN];
#pragma unroll
      for (int j = 0; j < GN; ++j) {
        float2 ar, ai;
        if constexpr (FFD) {
          const float k = kb[m * kTxAnchor + jb + j];
          const float2 kk = make_float2(k, k);
#pragma unroll
          for (int p = 0; p < kPairs; ++p) {
            const float2 d = sinc_poly2<DT>(__fmul2_rn(Dh[p], kk));
            ar = p ? __ffma2_rn(Gr[p], d, ar) : __fmul2_rn(Gr[p], d);
            ai = p ? __ffma2_rn(Gi[p], d, ai) : __fmul2_rn(Gi[p], d);
            cstep2(Gr[p], Gi[p], Sr[p], Si[p], Sn[p]);
          }
        } else {
          ar = Gr[0];
          ai = Gi[0];
          cstep2(Gr[0], Gi[0], Sr[0], Si[0], Sn[0]);
#pragma unroll
          for (int p = 1; p < kPairs; ++p) {
            ar = __fadd2_rn(ar, Gr[p]);
            ai = __fadd2_rn(ai, Gi[p]);
            cstep2(Gr[p], Gi[p], Sr[p], Si[p], Sn[p]);
          }
        }
        vr[j] = ar.x + ar.y;
        vi[j] = ai.x + ai.y;
      }
      // reduce-scatter: at level h the lane with bit h set keeps the upper half of its values
#pragma unroll
      for (int h = GN / 2; h >= 1; h >>= 1) {
        const bool up = (g & h) != 0;
#pragma unroll
        for (int i = 0; i < h; ++i) {
          const float sr = up ? vr[i] : vr[i + h], si = up ? vi[i] : vi[i + h];
          const float kr = up ? vr[i + h] : vr[i], ki = up ? vi[i + h] : vi[i];
          vr[i] = kr + __shfl_xor_sync(0xffffffffu, sr, h);
          vi[i] = ki + __shfl_xor_sync(0xffffffffu, si, h);
        }
      }
      sink(m * kTxAnchor + jb + g, make_float2(vr[0], vi[0]));
    }
  }
}

struct PfieldSink {
  const float2* pp;
  float acc;
  int fb_valid;
  __device__ __forceinline__ void operator()(int fl, float2 ps) {
    if (fl < fb_valid) {
      float2 v = cmul(pp[fl], ps);
      acc = fmaf(v.x, v.x, fmaf(v.y, v.y, acc));
    }
  }
};

template <int GN, int DT>
__global__ void __launch_bounds__(kThreads, (GN >= 32 || DT) ? 1 : 2) pfield_band_kernel(const BandArgs A) {
  extern __shared__ __align__(16) unsigned char sm[];
  const PfieldLayout L = pfield_layout(A.fb, A.E, DT > 0);
  const int tid = threadIdx.x;
  const int f_b0 = blockIdx.x * A.fb;
  const int64_t p_begin = (int64_t)blockIdx.y * A.per_slice;
  const int64_t p_end = min(A.n_pts, p_begin + A.per_slice);
  load_band_tables(A, L, sm, f_b0);
  __syncthreads();
  const int g = tid % GN;
  const int sl = tid / GN;
  const float2* pp = reinterpret_cast<const float2*>(sm + L.off_pp);
  float* out = reinterpret_cast<float*>(A.partial) + (size_t)blockIdx.x * A.n_pts;
  for (int64_t t0 = p_begin; t0 < p_end; t0 += A.st) {
    int64_t p = t0 + sl;
    bool valid = p < p_end;
    int64_t pi = valid ? p : t0;
    PfieldSink sink{pp, 0.f, min(A.fb, A.F - f_b0)};
    tx_tile<GN, DT>(A, L, sm, pi, g, sink);
    // each lane holds the band's |p|^2 over its own frequencies: sum the GN lanes in a fixed tree
    float acc = sink.acc;
#pragma unroll
    for (int off = 1; off < GN; off <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    if (valid && g == 0) {
      double x = A.pts[2 * pi], z = A.pts[2 * pi + 1];
      bool o = z < 0.0;
      if (A.convex) o = o || (x * x + (z + A.apex) * (z + A.apex) <= A.radius2);
      out[pi] = o ? 0.f : acc;
    }
  }
}

template <int GN, int DT>
static cudaError_t launch_pfield_band(const SweepConfig& c, const BandArgs& A, cudaStream_t s) {
  cudaError_t e =
      cudaFuncSetAttribute(pfield_band_kernel<GN, DT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)c.smem);
  if (e != cudaSuccess) return e;
  pfield_band_kernel<GN, DT><<<dim3(c.n_bands, c.n_slices), kThreads, c.smem, s>>>(A);
  return cudaGetLastError();
}

template <int DT>
static cudaError_t launch_pfield_band_gn(const SweepConfig& c, const BandArgs& A, cudaStream_t s) {
  switch (c.gn) {
    case 4: return launch_pfield_band<4, DT>(c, A, s);
    case 8: return launch_pfield_band<8, DT>(c, A, s);
    case 16: return launch_pfield_band<16, DT>(c, A, s);
    case 32: return launch_pfield_band<32, DT>(c, A, s);
    default: return cudaErrorInvalidValue;
  }
}

// Full-frequency-directivity launcher (fsg_sweep_ffd.cu).
cudaError_t launch_pfield_band_ffd(const SweepConfig& c, const BandArgs& A, cudaStream_t s);

}  // namespace fsg
