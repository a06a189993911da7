// Downstream beamforming of simulated RF: I/Q demodulation (fsg_rf2iq) and delay-and-sum
// (fsg_das matrix-free with compounding, fsg_dasmtx as a CSR matrix).  They restate MUST's
// rf2iq / dasmtx algorithms, which the reference's validation tests call through PyMUST
// (tests/_picmus_phantom_shared.py:407-460).
//
// rf2iq_kernel: one warp per (frame, channel) column, up to eight consecutive columns per CTA.  The IIR
// filter (cascaded second-order sections in FP32; a single high-order recursion loses ~1e-3 in FP32
// at narrow cut-offs, the cascade stays at ~1e-6) is linear in its state, so a segment of a column is
// cut into 32 chunks, one per lane: every lane filters its chunk from a zero state (the first from the
// true one), the chunk-end states are combined by a scan over the lanes with the powers of the chunk's
// state transition M = A^L (computed in FP64 on the host), and every lane filters its chunk again from
// its true state.  The same is done backward.  The down-mixed samples and the forward outputs stay in
// shared memory (records longer than a segment go through the output array between the two passes).
// The down-mixing phasors depend on the sample only: each CTA tabulates them per segment.
// rf2iq_column_kernel: one thread per column, for many short records.
//
// das_kernel: one thread per pixel, looping over groups of firings and, per element, over the
// group's firings.  The transmit delays (times c) and the element frames sit in shared memory;
// the I/Q samples are read channel-major, so the threads of a warp (consecutive pixels of an
// image row) read nearby samples of the same element.

#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <string.h>

#include <type_traits>

#include "../../include/fsgb300.h"
#include "fsg_common.cuh"
#include "fsg_internal.h"

namespace fsg {

constexpr int kDasThreads = 256;      // dasmtx_kernel
constexpr int kDasImgThreads = 128;   // das_kernel: small CTAs spread the pixels evenly over the SMs
constexpr int kDasMaxE = 256;
constexpr int kDasStage = 4;          // groups whose delays sit in shared memory at a time
constexpr int kDasGroup = 8;          // firings whose transmit distances a thread holds at a time
constexpr int kDasImgBlocks = 7;      // das_kernel CTAs per SM the registers are cut for

constexpr int kIqCh = 8;          // channels per CTA, one warp each
constexpr int kIqMaxL = 71;       // samples per lane and segment: eight columns and the phasors fit shared memory
constexpr int kIqScan = 5;        // scan levels: M, M^2, M^4, M^8, M^16
constexpr int kIqColThreads = 64, kIqColMax = 320;  // rf2iq_column_kernel: threads, longest record

struct Rf2IqArgs {
  const float* rf;   // [n_frames][n_samples][n_ch]
  float2* iq;        // [n_frames][n_ch][n_samples]
  int n_frames, n_samples, n_ch, n_sec, pad;
  double cyc_per_sample;  // fc / fs
  double cyc0;            // fc tau
  float sos[FSG_RF2IQ_MAX_SECTIONS][5];  // b0, b1, b2, a1, a2
  float zi[FSG_RF2IQ_MAX_SECTIONS][2];   // steady state for a unit input
  int L;                                 // samples per lane and segment (odd)
  int per_cta;                           // columns per CTA: 1, 2, 4 or 8
  int levels, compensated;               // scan levels whose power is not negligible; bit k: level k's sums compensated
  // A^(L 2^k): state after from state before, FP32 and what it leaves
  float m[kIqScan][2 * FSG_RF2IQ_MAX_SECTIONS][2 * FSG_RF2IQ_MAX_SECTIONS];
  float m_lo[kIqScan][2 * FSG_RF2IQ_MAX_SECTIONS][2 * FSG_RF2IQ_MAX_SECTIONS];
};

// Down-mixing phasor of sample n: exp(-2 pi i (n fc / fs + fc tau)), the phase reduced to
// cycles in FP64.
__device__ __forceinline__ float2 phasor(const Rf2IqArgs& A, int n) {
  const double cyc = fma((double)n, A.cyc_per_sample, A.cyc0);
  const float frac = (float)(cyc - floor(cyc));
  float s, c;
  sincospif(2.0f * frac, &s, &c);
  return make_float2(c, -s);
}

// One sample through the cascade of transposed direct-form-II biquads (real coefficients).
template <int NS>
__device__ __forceinline__ float2 iir_step(const Rf2IqArgs& A, float2 (*z)[2], float2 x) {
#pragma unroll
  for (int s = 0; s < NS; ++s) {
    const float* q = A.sos[s];
    const float2 y = make_float2(fmaf(q[0], x.x, z[s][0].x), fmaf(q[0], x.y, z[s][0].y));
    z[s][0] = make_float2(fmaf(q[1], x.x, fmaf(-q[3], y.x, z[s][1].x)), fmaf(q[1], x.y, fmaf(-q[3], y.y, z[s][1].y)));
    z[s][1] = make_float2(fmaf(q[2], x.x, -q[4] * y.x), fmaf(q[2], x.y, -q[4] * y.y));
    x = y;
  }
  return x;
}

template <int NS>
__device__ __forceinline__ void iir_init(const Rf2IqArgs& A, float2 (*z)[2], float2 x0) {
#pragma unroll
  for (int s = 0; s < NS; ++s)
#pragma unroll
    for (int k = 0; k < 2; ++k) z[s][k] = make_float2(A.zi[s][k] * x0.x, A.zi[s][k] * x0.y);
}

// Adds the state that `from` becomes after A^(L 2^k).  Where little is left of it the sum rounds once; else the
// products and sums are compensated, since the powers of a narrow filter reach 10^6 and cancel.  Error of the
// forward pass with one plain FP32 sum, the serial recursion, and so: 2.1e-5, 1.2e-5, 0.7e-5 at a cut-off
// of 0.01 of Nyquist and 1,015 samples; 7.8e-8, 6.2e-8, 6.2e-8 at 0.5 and 64 samples.
constexpr double kIqPlainMax = 1.0 / 4.0;
template <int NS>
__device__ __forceinline__ void iir_carry(const Rf2IqArgs& A, int k, float2 (*z)[2], const float2 (*from)[2]) {
  if (A.compensated >> k & 1) {
#pragma unroll
    for (int i = 0; i < 2 * NS; ++i) {
      float2 s = z[i >> 1][i & 1], lo = make_float2(0.f, 0.f);
#pragma unroll
      for (int j = 0; j < 2 * NS; ++j) {
        if ((j >> 1) > (i >> 1)) continue;  // a section is driven by the ones before it only
        const float c = A.m[k][i][j], cl = A.m_lo[k][i][j];
        const float2 f = from[j >> 1][j & 1];
        const float2 p = make_float2(__fmul_rn(c, f.x), __fmul_rn(c, f.y));
        const dfl x = two_sum(s.x, p.x), y = two_sum(s.y, p.y);
        s = make_float2(x.hi, y.hi);
        lo.x = __fadd_rn(lo.x, fmaf(cl, f.x, __fadd_rn(x.lo, fmaf(c, f.x, -p.x))));
        lo.y = __fadd_rn(lo.y, fmaf(cl, f.y, __fadd_rn(y.lo, fmaf(c, f.y, -p.y))));
      }
      z[i >> 1][i & 1] = make_float2(__fadd_rn(s.x, lo.x), __fadd_rn(s.y, lo.y));
    }
  } else {
#pragma unroll
    for (int i = 0; i < 2 * NS; ++i) {
      float2 t = make_float2(0.f, 0.f);
#pragma unroll
      for (int j = 0; j < 2 * NS; ++j) {
        if ((j >> 1) > (i >> 1)) continue;
        const float c = A.m[k][i][j];
        t.x = fmaf(c, from[j >> 1][j & 1].x, t.x);
        t.y = fmaf(c, from[j >> 1][j & 1].y, t.y);
      }
      z[i >> 1][i & 1] = cadd(z[i >> 1][i & 1], t);
    }
  }
}

// Filters samples [0, n) of a segment in place (x[i * dir], i < n), the warp's lanes taking L
// consecutive ones each; z holds the state before sample 0 and, on return, after sample n - 1 (in
// every lane).  scale multiplies the outputs.
template <int NS>
__device__ __forceinline__ void iir_segment(const Rf2IqArgs& A, float2* x, int dir, int n, float2 (*z)[2], float scale) {
  const int lane = threadIdx.x & 31, L = A.L;
  const int i0 = lane * L, cnt = max(0, min(L, n - i0));
  float2 s[NS][2];
#pragma unroll
  for (int q = 0; q < 2 * NS; ++q) s[q >> 1][q & 1] = lane == 0 ? z[q >> 1][q & 1] : make_float2(0.f, 0.f);
  for (int i = 0; i < cnt; ++i) iir_step<NS>(A, s, x[(i0 + i) * dir]);
  // inclusive scan of the chunk-end states; one that is not finite reaches every later chunk
  float sum = 0.f;
#pragma unroll
  for (int q = 0; q < 2 * NS; ++q) sum += fabsf(s[q >> 1][q & 1].x) + fabsf(s[q >> 1][q & 1].y);
  const int levels = __any_sync(0xffffffffu, !(sum <= 3.402823466e38f)) ? kIqScan : A.levels;
#pragma unroll 1
  for (int k = 0; k < levels; ++k) {
    float2 f[NS][2];
#pragma unroll
    for (int q = 0; q < 2 * NS; ++q) {
      f[q >> 1][q & 1].x = __shfl_up_sync(0xffffffffu, s[q >> 1][q & 1].x, 1 << k);
      f[q >> 1][q & 1].y = __shfl_up_sync(0xffffffffu, s[q >> 1][q & 1].y, 1 << k);
    }
    if (lane >= (1 << k)) iir_carry<NS>(A, k, s, f);
  }
  // the state before this lane's chunk, and the outputs
#pragma unroll
  for (int q = 0; q < 2 * NS; ++q) {
    const float2 v = s[q >> 1][q & 1];
    const float2 u = make_float2(__shfl_up_sync(0xffffffffu, v.x, 1), __shfl_up_sync(0xffffffffu, v.y, 1));
    if (lane > 0) z[q >> 1][q & 1] = u;
  }
  for (int i = 0; i < cnt; ++i) {
    const float2 o = iir_step<NS>(A, z, x[(i0 + i) * dir]);
    x[(i0 + i) * dir] = make_float2(scale * o.x, scale * o.y);
  }
  const int last = (n - 1) / L;  // the lane that took sample n - 1
#pragma unroll
  for (int q = 0; q < 2 * NS; ++q) {
    z[q >> 1][q & 1].x = __shfl_sync(0xffffffffu, z[q >> 1][q & 1].x, last);
    z[q >> 1][q & 1].y = __shfl_sync(0xffffffffu, z[q >> 1][q & 1].y, last);
  }
  __syncwarp();
}

// What bounds it: the length of a lane's chunk, four filter passes of N / 32 samples, and with many columns
// issue.  Eight columns of the call per CTA, whatever their frames: 153,600 columns of one channel and 1,000
// samples 8,400 us with a CTA per frame, now 1,593 (2,614 with a thread per column and all its host work).
// Calls, a thread per column -> now: 9,600 columns of 1,000 samples 514 -> 118 us (490 of it once on the host),
// 115,200 of 2,400 6,151 -> 2,693.
template <int NS>
__global__ void __launch_bounds__(32 * kIqCh) rf2iq_kernel(const __grid_constant__ Rf2IqArgs A) {
  extern __shared__ __align__(16) float2 iq_sm[];
  __shared__ float2 right[kIqCh][FSG_RF2IQ_MAX_PAD];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int N = A.n_samples, P = A.pad, S = 32 * A.L, pitch = S + 4;  // pitch = 4 mod 16: staging writes conflict-free
  const int64_t cols = (int64_t)A.n_frames * A.n_ch, c0 = (int64_t)blockIdx.x * A.per_cta, cid = c0 + warp;
  const bool active = warp < A.per_cta && cid < cols;
  auto column = [&](int64_t c) { return A.rf + (size_t)(c / A.n_ch) * N * A.n_ch + c % A.n_ch; };
  float2* ph = iq_sm + A.per_cta * pitch;  // the segment's phasors
  float2* col = iq_sm + warp * pitch;      // this warp's samples of the segment
  float2* __restrict__ y = A.iq + cid * N;
  const int n_seg = (N + S - 1) / S;
  // the staging threads: channels side by side, or samples where there are fewer than eight
  const bool by_sample = A.n_ch < kIqCh;
  const int st_c = (by_sample ? warp : threadIdx.x) & (A.per_cta - 1);
  const int st_j = by_sample ? lane + 32 * (warp / A.per_cta) : threadIdx.x / kIqCh;
  const int st_step = 32 * kIqCh / A.per_cta;
  const float* __restrict__ st_rf = c0 + st_c < cols ? column(c0 + st_c) : nullptr;

  float2 z[NS][2];
  // forward pass over [2 x0 - x[P..1], x[0..N-1], 2 x[N-1] - x[N-2..N-1-P]]
  for (int g = 0; g < n_seg; ++g) {
    const int n0 = g * S, n = min(S, N - n0);
    __syncthreads();
    for (int j = threadIdx.x; j < n; j += blockDim.x) ph[j] = phasor(A, n0 + j);
    __syncthreads();
    if (st_rf) {
      const float* src = st_rf + (size_t)n0 * A.n_ch;
#pragma unroll 4
      for (int j = st_j; j < n; j += st_step) {
        const float v = src[(size_t)j * A.n_ch];
        const float2 e = ph[j];
        iq_sm[st_c * pitch + j] = make_float2(v * e.x, v * e.y);
      }
    }
    __syncthreads();
    if (active) {
      if (g == 0) {  // (a segment that is not the last is longer than the pad)
        const float2 x0 = col[0];
        for (int k = 0; k < P; ++k) {
          const float2 v = col[P - k], e = make_float2(2.f * x0.x - v.x, 2.f * x0.y - v.y);
          if (k == 0) iir_init<NS>(A, z, e);
          iir_step<NS>(A, z, e);
        }
        if (P == 0) iir_init<NS>(A, z, x0);
      }
      if (g == n_seg - 1) {
        if (lane < P) {  // the right extension, of samples before they are filtered
          const float2 xn = col[n - 1];
          const int m = N - 2 - lane;
          float2 v;
          if (m >= n0) {
            v = col[m - n0];
          } else {  // in the segment before
            const float r = column(cid)[(size_t)m * A.n_ch];
            const float2 e = phasor(A, m);
            v = make_float2(r * e.x, r * e.y);
          }
          right[warp][lane] = make_float2(2.f * xn.x - v.x, 2.f * xn.y - v.y);
        }
        __syncwarp();
      }
      iir_segment<NS>(A, col, 1, n, z, 1.f);
      if (n_seg > 1)
        for (int j = lane; j < n; j += 32) y[n0 + j] = col[j];
    }
  }
  if (!active) return;
  {
    float2 o = make_float2(0.f, 0.f);
    for (int k = 0; k < P; ++k) {
      o = iir_step<NS>(A, z, right[warp][k]);
      __syncwarp();
      if (lane == 0) right[warp][k] = o;
    }
    __syncwarp();
    // backward pass, started from the last forward output
    iir_init<NS>(A, z, P > 0 ? o : col[(N - 1) - (n_seg - 1) * S]);
    for (int k = P - 1; k >= 0; --k) iir_step<NS>(A, z, right[warp][k]);
  }
  for (int g = n_seg - 1; g >= 0; --g) {
    const int n0 = g * S, n = min(S, N - n0);
    if (n_seg > 1) {
      __syncwarp();
      for (int j = lane; j < n; j += 32) col[j] = y[n0 + j];
      __syncwarp();
    }
    iir_segment<NS>(A, col + n - 1, -1, n, z, 2.f);
    for (int j = lane; j < n; j += 32) y[n0 + j] = col[j];
  }
}

// One thread per column, its recurrence from end to end; the phasors of the whole record in shared memory
// and a chunk's samples requested before they are filtered.  What bounds it: the chain of the recurrence, 0.16 us per
// sample, up to about 100,000 columns (all resident); beyond, the lines of A.iq that a warp's 32 columns touch.
constexpr int kIqColChunk = 16;
template <int NS>
__global__ void __launch_bounds__(kIqColThreads) rf2iq_column_kernel(const __grid_constant__ Rf2IqArgs A) {
  __shared__ float2 ph[kIqColMax];
  const int N = A.n_samples, P = A.pad;
  for (int j = threadIdx.x; j < N; j += blockDim.x) ph[j] = phasor(A, j);
  __syncthreads();
  const int64_t cid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (cid >= (int64_t)A.n_frames * A.n_ch) return;
  const float* __restrict__ col = A.rf + (size_t)(cid / A.n_ch) * N * A.n_ch + cid % A.n_ch;
  float2* __restrict__ y = A.iq + cid * N;
  auto mixed = [&](int n) {
    const float v = col[(size_t)n * A.n_ch];
    return make_float2(v * ph[n].x, v * ph[n].y);
  };
  float2 z[NS][2], right[FSG_RF2IQ_MAX_PAD];
  const float2 x0 = mixed(0), xn = mixed(N - 1);
  iir_init<NS>(A, z, x0);
  for (int k = 0; k < P; ++k) {
    const float2 v = mixed(P - k), e = make_float2(2.f * x0.x - v.x, 2.f * x0.y - v.y);
    if (k == 0) iir_init<NS>(A, z, e);
    iir_step<NS>(A, z, e);
  }
  for (int m0 = 0; m0 < N; m0 += kIqColChunk) {
    float v[kIqColChunk];
#pragma unroll
    for (int j = 0; j < kIqColChunk; ++j) v[j] = m0 + j < N ? col[(size_t)(m0 + j) * A.n_ch] : 0.f;
#pragma unroll
    for (int j = 0; j < kIqColChunk; ++j)
      if (m0 + j < N) {
        const float2 e = ph[m0 + j];
        y[m0 + j] = iir_step<NS>(A, z, make_float2(v[j] * e.x, v[j] * e.y));
      }
  }
  for (int k = 0; k < P; ++k) {
    const float2 v = mixed(N - 2 - k);
    right[k] = iir_step<NS>(A, z, make_float2(2.f * xn.x - v.x, 2.f * xn.y - v.y));
  }
  // backward pass, started from the last forward output
  iir_init<NS>(A, z, P > 0 ? right[P - 1] : y[N - 1]);
  for (int k = P - 1; k >= 0; --k) iir_step<NS>(A, z, right[k]);
  for (int n1 = N - 1; n1 >= 0; n1 -= kIqColChunk) {
    float2 w[kIqColChunk];
#pragma unroll
    for (int j = 0; j < kIqColChunk; ++j) w[j] = n1 - j >= 0 ? y[n1 - j] : make_float2(0.f, 0.f);
#pragma unroll
    for (int j = 0; j < kIqColChunk; ++j)
      if (n1 - j >= 0) {
        const float2 o = iir_step<NS>(A, z, w[j]);
        y[n1 - j] = make_float2(2.f * o.x, 2.f * o.y);
      }
  }
}

struct DasArgs {
  const float2* iq;    // [n_frames][E][n_s]
  const double* txd;   // [n_frames][E]
  const double* pix;   // [n_pix][2]
  float2* out;         // image [n_pix] or CSR values
  int* crow;           // dasmtx only
  int* col;
  int64_t n_pix;
  int n_frames, n_s, E, method, iq_rot;
  double pitch, radius;
  float c, inv_c, fs, two_fc, t0;
  float aperture;      // 1 / (2 f-number), or < 0 for every element
  int slices;          // das_kernel: threads per pixel, each taking every slices-th group of firings
};

// Element centre and frame (sin, cos of its angle): linear arrays along x, convex arrays on
// the arc of the given radius with the apex at z = 0.
__device__ void das_element(const DasArgs& A, int e, float* x, float* z, float* sn, float* cs) {
  if (isinf(A.radius)) {
    *x = (float)(((double)e - 0.5 * (A.E - 1)) * A.pitch);
    *z = 0.f;
    *sn = 0.f;
    *cs = 1.f;
    return;
  }
  const double half = asin(A.pitch / 2.0 / A.radius);
  const double chord = 2.0 * A.radius * sin(half * (A.E - 1));
  const double apex = sqrt(A.radius * A.radius - (chord / 2.0) * (chord / 2.0));
  const double t0 = atan2(-chord / 2.0, apex), t1 = atan2(chord / 2.0, apex);
  const double te = (A.E > 1) ? ((e == A.E - 1) ? t1 : t0 + e * ((t1 - t0) / (A.E - 1))) : t0;
  *x = (float)(A.radius * sin(te));
  *z = (float)(A.radius * cos(te) - apex);
  *sn = (float)sin(te);
  *cs = (float)cos(te);
}

struct DasShared {
  float ex[kDasMaxE], ez[kDasMaxE], es[kDasMaxE], ec[kDasMaxE], ctx[kDasMaxE];
};

__device__ __forceinline__ void das_load_elements(const DasArgs& A, DasShared& S) {
  for (int e = threadIdx.x; e < A.E; e += blockDim.x) das_element(A, e, &S.ex[e], &S.ez[e], &S.es[e], &S.ec[e]);
}

__device__ __forceinline__ void das_load_delays(const DasArgs& A, DasShared& S, int f) {
  for (int e = threadIdx.x; e < A.E; e += blockDim.x) {
    const double v = A.txd[(size_t)f * A.E + e];
    S.ctx[e] = isnan(v) ? INFINITY : (float)(A.c * v);
  }
}

// Transmit distance of pixel (px, pz): the earliest arrival over the firing elements.
__device__ __forceinline__ float das_dtx(const DasArgs& A, const DasShared& S, float px, float pz) {
  float d = INFINITY;
  for (int e = 0; e < A.E; ++e) {
    const float dx = px - S.ex[e], dz = pz - S.ez[e];
    d = fminf(d, S.ctx[e] + sqrtf(fmaf(dx, dx, dz * dz)));
  }
  return d;
}

// Delay, fractional sample and I/Q rotation of element e for pixel (px, pz); false outside
// the receive aperture.
__device__ __forceinline__ bool das_tap(const DasArgs& A, const DasShared& S, int e, float px, float pz, float dtx,
                                        float* s, float2* rot) {
  const float dx = px - S.ex[e], dz = pz - S.ez[e];
  if (A.aperture >= 0.f) {
    const float ax = fmaf(dx, S.es[e], dz * S.ec[e]);
    const float lat = fmaf(dx, S.ec[e], -dz * S.es[e]);
    if (!(ax > 0.f) || fabsf(lat) > ax * A.aperture) return false;
  }
  const float t = (dtx + sqrtf(fmaf(dx, dx, dz * dz))) * A.inv_c;
  *s = (t - A.t0) * A.fs;
  if (A.iq_rot) {
    float sn, cs;
    sincospif(A.two_fc * t, &sn, &cs);
    *rot = make_float2(cs, sn);
  } else {
    *rot = make_float2(1.f, 0.f);
  }
  return true;
}

// floorf(s) and the integer.  Records of up to kDasShort samples do without the conversion unit (a
// quarter of the rate of the others): exact for |s| < 2^22; beyond that, and for infinities and NaN, *i
// is no sample of such a record.
constexpr int kDasShort = 1 << 22;
template <bool kLong>
__device__ __forceinline__ float das_floor(float s, int* i) {
  if constexpr (kLong) {
    const float fi = floorf(s);
    *i = fi >= 0.f && fi < 2147483648.0f ? (int)fi : -1;
    return fi;
  }
  const float t = s + 12582912.0f;  // 1.5 * 2^23: rounds to the nearest integer
  const float r = t - 12582912.0f;
  const int down = r > s ? 1 : 0;
  *i = __float_as_int(t) - 0x4B400000 - down;
  return r - (float)down;
}

// sqrt(d2) from one reciprocal root: s = d2 y plus the residual (d2 - s^2) y / 2, within an ulp.  Images of
// 1 to 25 firings are as far from 64 bits as with correctly rounded roots (2.5e-5 to 1.3e-3, within 0.5%).
__device__ __forceinline__ float das_sqrt(float d2) {
  const float y = rsqrt_normal(fmaxf(d2, 1.17549435e-38f)), s = d2 * y;
  return fmaf(0.5f * y, fmaf(-s, s, d2), s);
}

// Matrix-free compounded delay-and-sum.  The I/Q rotation exp(2 pi i fc (d_tx + d_rx) / c)
// factors into a transmit part per (pixel, firing) and a receive part per (pixel, element), so
// a thread first computes, for a group of firings, the transmit distance and rotation (kept in
// registers), then per element the receive distance, aperture test and rotation
// once, and per firing only the sample gather, the interpolation and one complex multiply-add.
// The group's transmit delays (times c) sit in dynamic shared memory, [element][firing].
//
// What bounds it: instruction issue (60% of the cycles) and the latency of the gathers, two 8-byte loads
// per tap (the host passes neighbouring pixels of a row, whose samples share one or two lines).  The call
// of 75 firings x 64 elements x 131,072 pixels, signal copies and launches included: 1,927 us with the
// firings' values in local memory, a distance per (element, firing) in the transmit search and floor on
// the conversion unit; 1,324 us with groups in registers; 1,124 us with one unsigned test per tap, 32-bit
// offsets, das_sqrt and the delays of four groups staged at a time (barriers per group were 11% of the
// stalls).  Twelve firings 919 -> 373, one 759 -> 254.  Groups of 8 keep the kernel within 72 registers,
// seven CTAs per SM: six took 150 us more, eight 50; groups of 16 (five CTAs) 350, of 12 (five CTAs) 530.
// An image of few pixels leaves SMs idle behind a thread's chain of firings: `slices` threads share a
// pixel's groups, and their sums are added in order.
template <int G, bool kLinear, bool kLong = false, bool kSliced = false>
__global__ void __launch_bounds__(kDasImgThreads, kDasImgBlocks) das_kernel(const __grid_constant__ DasArgs A) {
  __shared__ DasShared S;
  extern __shared__ __align__(16) float ctx_s[];  // [kDasStage][E][G]
  das_load_elements(A, S);
  const int slices = kSliced ? A.slices : 1, px_cta = kDasImgThreads / slices;
  const int slice = kSliced ? threadIdx.x / px_cta : 0;
  const int64_t p = kSliced ? (int64_t)blockIdx.x * px_cta + threadIdx.x % px_cta
                            : (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool valid = p < A.n_pix;
  const float px = valid ? (float)A.pix[2 * p] : 0.f, pz = valid ? (float)A.pix[2 * p + 1] : 0.f;
  const float k_cyc = 0.5f * A.two_fc * A.inv_c;  // cycles per metre of path, fc / c
  const unsigned top = (unsigned)(A.n_s - (kLinear ? 2 : 1));  // the last first sample of a tap
  // linear taps: one rounding for the sample's position instead of three
  const float per_m = A.inv_c * A.fs, s0 = -A.t0 * A.fs;
  using Index = typename std::conditional<kLong, int64_t, unsigned>::type;  // of a sample in the call's I/Q data
  float2 acc = make_float2(0.f, 0.f);
  for (int g0 = 0; g0 < A.n_frames; g0 += G) {
    const int ng = min(G, A.n_frames - g0), stage = g0 / G % kDasStage;
    if (stage == 0) {
      const int left = min(kDasStage * G, A.n_frames - g0);
      __syncthreads();
      for (int i = threadIdx.x; i < kDasStage * G * A.E; i += blockDim.x) {
        const int j = i / (G * A.E) * G + i % G, e = i / G % A.E;
        const double v = j < left ? A.txd[(size_t)(g0 + j) * A.E + e] : NAN;
        ctx_s[i] = isnan(v) ? INFINITY : (float)(A.c * v);
      }
      __syncthreads();
    }
    if (!valid) continue;
    if (kSliced && stage % slices != slice) continue;
    const float* ctx_g = ctx_s + stage * G * A.E;
    float dtx[G];
#pragma unroll
    for (int j = 0; j < G; ++j) dtx[j] = INFINITY;
    for (int e = 0; e < A.E; ++e) {
      const float dx = px - S.ex[e], dz = pz - S.ez[e];
      const float d = das_sqrt(fmaf(dx, dx, dz * dz));
      const float4* cj = reinterpret_cast<const float4*>(ctx_g + e * G);
#pragma unroll
      for (int j = 0; j < G / 4; ++j) {
        const float4 c = cj[j];
        dtx[4 * j] = fminf(dtx[4 * j], c.x + d);
        dtx[4 * j + 1] = fminf(dtx[4 * j + 1], c.y + d);
        dtx[4 * j + 2] = fminf(dtx[4 * j + 2], c.z + d);
        dtx[4 * j + 3] = fminf(dtx[4 * j + 3], c.w + d);
      }
    }
    float2 rtx[G];
#pragma unroll
    for (int j = 0; j < G; ++j) {
      float sn = 0.f, cs = 1.f;
      if (A.iq_rot && dtx[j] < INFINITY) sincospif(2.f * k_cyc * dtx[j], &sn, &cs);
      rtx[j] = make_float2(cs, sn);
    }
    for (int e = 0; e < A.E; ++e) {
      const float dx = px - S.ex[e], dz = pz - S.ez[e];
      if (A.aperture >= 0.f) {
        const float ax = fmaf(dx, S.es[e], dz * S.ec[e]);
        const float lat = fmaf(dx, S.ec[e], -dz * S.es[e]);
        if (!(ax > 0.f) || fabsf(lat) > ax * A.aperture) continue;
      }
      const float dr = das_sqrt(fmaf(dx, dx, dz * dz));
      float2 ae = make_float2(0.f, 0.f);
      // branch-free taps (a tap outside the record reads sample 0 with weight 0; the firings past the
      // last one have no finite delay), unrolled so that the gathers of several firings are in flight
#pragma unroll
      for (int j = 0; j < G; ++j) {
        const float d = dtx[j] + dr;
        const float s = kLinear ? fmaf(d, per_m, s0) : (d * A.inv_c - A.t0) * A.fs;
        int i;
        const float fi = das_floor<kLong>(kLinear ? s : s + 0.5f, &i);
        const bool ok = (unsigned)i <= top;
        const Index col = ((Index)(g0 + (j < ng ? j : 0)) * A.E + e) * A.n_s;
        const float2* cj = A.iq + (Index)(col + (ok ? i : 0));
        float2 v = cj[0];
        if constexpr (kLinear) {
          const float2 b = cj[1];
          const float w = s - fi;
          v = make_float2(fmaf(w, b.x - v.x, v.x), fmaf(w, b.y - v.y, v.y));
        }
        v = ok ? v : make_float2(0.f, 0.f);
        ae.x = fmaf(v.x, rtx[j].x, fmaf(-v.y, rtx[j].y, ae.x));
        ae.y = fmaf(v.x, rtx[j].y, fmaf(v.y, rtx[j].x, ae.y));
      }
      float sn = 0.f, cs = 1.f;
      if (A.iq_rot) sincospif(2.f * k_cyc * dr, &sn, &cs);
      acc.x = fmaf(ae.x, cs, fmaf(-ae.y, sn, acc.x));
      acc.y = fmaf(ae.x, sn, fmaf(ae.y, cs, acc.y));
    }
  }
  if constexpr (kSliced) {  // the slices' sums, in order
    __syncthreads();
    float2* part = reinterpret_cast<float2*>(ctx_s);
    part[threadIdx.x] = acc;
    __syncthreads();
    if (slice > 0) return;
    for (int q = 1; q < slices; ++q) {
      const float2 v = part[q * px_cta + threadIdx.x];
      acc.x += v.x;
      acc.y += v.y;
    }
  }
  if (valid) A.out[p] = acc;
}

__global__ void __launch_bounds__(kDasThreads) dasmtx_kernel(const __grid_constant__ DasArgs A) {
  __shared__ DasShared S;
  das_load_elements(A, S);
  das_load_delays(A, S, 0);
  __syncthreads();
  const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= A.n_pix) return;
  const int per = A.method == FSG_DAS_LINEAR ? 2 * A.E : A.E;
  A.crow[p] = (int)(p * per);
  if (p == A.n_pix - 1) A.crow[A.n_pix] = (int)(A.n_pix * per);
  const float px = (float)A.pix[2 * p], pz = (float)A.pix[2 * p + 1];
  const float dtx = das_dtx(A, S, px, pz);
  int* cl = A.col + p * per;
  float2* vl = A.out + p * per;
  for (int e = 0; e < A.E; ++e) {
    float s = 0.f;
    float2 rot = make_float2(0.f, 0.f);
    const bool on = dtx < INFINITY && das_tap(A, S, e, px, pz, dtx, &s, &rot);
    const int base = e * A.n_s;
    if (A.method == FSG_DAS_LINEAR) {
      const float fi = floorf(s);
      const bool in = on && fi >= 0.f && fi + 1.f <= (float)(A.n_s - 1);
      const int i0 = in ? (int)fi : 0;
      const float w = in ? s - fi : 0.f;
      const float g0 = in ? 1.f - w : 0.f;
      cl[2 * e] = base + i0;
      cl[2 * e + 1] = base + i0 + 1;
      vl[2 * e] = make_float2(g0 * rot.x, g0 * rot.y);
      vl[2 * e + 1] = make_float2(w * rot.x, w * rot.y);
    } else {
      const float fi = floorf(s + 0.5f);
      const bool in = on && fi >= 0.f && fi <= (float)(A.n_s - 1);
      cl[e] = base + (in ? (int)fi : 0);
      vl[e] = in ? rot : make_float2(0.f, 0.f);
    }
  }
}

}  // namespace fsg

using namespace fsg;

// Whether the columns of a call are many and short enough for a thread each: the recurrence takes
// 0.16 us a sample however many columns run beside it, the scan of short chunks about 0.005 us a column.
// Calls (scan, thread each): 38,400 columns of 64 samples 164 us, 45; of 300 samples 213, 155; 9,600 of 300
// 61, 52; 307,200 of 300 1,577, 1,408.  From 384 samples on the scan is ahead (38,400 columns 225, 261;
// 115,200 639, 1,212).
static bool rf2iq_by_column(int n_samples, int64_t cols) {
  return n_samples <= kIqColMax && cols >= 28 * (int64_t)n_samples;
}

extern "C" int32_t fsg_rf2iq(const float* rf, int32_t n_frames, int32_t n_samples, int32_t n_channels, double fs,
                             double fc, double tau, int32_t n_sections, const double* sos, const double* zi,
                             int32_t pad, void* iq_out, void* stream) {
  if (!rf || !iq_out || !sos || !zi) return set_error(FSG_EINVAL, "rf, iq_out, sos and zi must be non-NULL");
  if (n_frames < 1 || n_channels < 1 || n_samples < 1)
    return set_error(FSG_EINVAL, "n_frames, n_samples and n_channels must be >= 1");
  if (n_sections < 1 || n_sections > FSG_RF2IQ_MAX_SECTIONS)
    return set_error(FSG_EUNSUPPORTED, "%d filter sections outside [1, %d]", n_sections, FSG_RF2IQ_MAX_SECTIONS);
  if (pad < 0 || pad > FSG_RF2IQ_MAX_PAD || pad >= n_samples)
    return set_error(FSG_EINVAL, "pad %d must be in [0, min(%d, n_samples - 1)]", pad, FSG_RF2IQ_MAX_PAD);
  if (!(fs > 0) || !(fc >= 0)) return set_error(FSG_EINVAL, "fs must be > 0 and fc >= 0");
  Rf2IqArgs A;
  A.rf = rf;
  A.iq = static_cast<float2*>(iq_out);
  A.n_frames = n_frames;
  A.n_samples = n_samples;
  A.n_ch = n_channels;
  A.n_sec = n_sections;
  A.pad = pad;
  A.cyc_per_sample = fc / fs;
  A.cyc0 = fc * tau;
  for (int sct = 0; sct < FSG_RF2IQ_MAX_SECTIONS; ++sct) {
    const bool on = sct < n_sections;
    if (on && sos[6 * sct + 3] != 1.0) return set_error(FSG_EINVAL, "section %d: a0 must be 1", sct);
    const int take[5] = {0, 1, 2, 4, 5};
    for (int k = 0; k < 5; ++k) A.sos[sct][k] = on ? (float)sos[6 * sct + take[k]] : 0.f;
    for (int k = 0; k < 2; ++k) A.zi[sct][k] = on ? (float)zi[2 * sct + k] : 0.f;
  }
  // segments of at most 32 kIqMaxL samples, the chunk length odd (the lanes' strided shared-memory
  // accesses then use every bank)
  const int n_seg = (n_samples + 32 * kIqMaxL - 1) / (32 * kIqMaxL);
  A.L = ((n_samples + 32 * n_seg - 1) / (32 * n_seg)) | 1;
  {
    // state transition of the cascade over L samples of zero input, and its squares, in FP64
    double m[2 * FSG_RF2IQ_MAX_SECTIONS][2 * FSG_RF2IQ_MAX_SECTIONS], sq[2 * FSG_RF2IQ_MAX_SECTIONS][2 * FSG_RF2IQ_MAX_SECTIONS];
    const int ns2 = 2 * n_sections;
    for (int j = 0; j < ns2; ++j) {
      double z[FSG_RF2IQ_MAX_SECTIONS][2] = {};
      z[j / 2][j % 2] = 1.0;
      for (int n = 0; n < A.L; ++n) {
        double x = 0.0;
        for (int q = 0; q < n_sections; ++q) {
          const float* c = A.sos[q];
          const double o = c[0] * x + z[q][0];
          z[q][0] = c[1] * x - c[3] * o + z[q][1];
          z[q][1] = c[2] * x - c[4] * o;
          x = o;
        }
      }
      for (int i = 0; i < ns2; ++i) m[i][j] = z[i / 2][i % 2];
    }
    memset(A.m, 0, sizeof(A.m));
    memset(A.m_lo, 0, sizeof(A.m_lo));
    A.levels = kIqScan;
    A.compensated = 0;
    for (int k = 0; k < kIqScan; ++k) {
      double top = 0.0;
      for (int i = 0; i < ns2; ++i)
        for (int j = 0; j < ns2; ++j) {
          A.m[k][i][j] = (float)m[i][j];
          A.m_lo[k][i][j] = (float)(m[i][j] - (double)A.m[k][i][j]);
          if (!(fabs(m[i][j]) <= top)) top = fabs(m[i][j]);
        }
      if (top < 1e-16) {  // nothing of a state is left after the chunks of this level
        A.levels = k;
        break;
      }
      if (!(top <= kIqPlainMax)) A.compensated |= 1 << k;
      for (int i = 0; i < ns2; ++i)
        for (int j = 0; j < ns2; ++j) {
          double s = 0.0;
          for (int q = 0; q < ns2; ++q) s += m[i][q] * m[q][j];
          sq[i][j] = s;
        }
      memcpy(m, sq, sizeof(m));
    }
  }
  const int64_t cols = (int64_t)n_frames * n_channels;
  const bool by_column = rf2iq_by_column(n_samples, cols);
  // few columns of fewer than eight channels are spread over the SMs (20 columns of 30,000 samples: on three
  // SMs 390 us, on twenty 244; 200 of 5,000: on 25 73, on 100 49)
  int sms = 0;
  const int st = device_sm_count(&sms);
  if (st != FSG_OK) return st;
  A.per_cta = kIqCh;
  while (n_channels < kIqCh && A.per_cta > 1 && cols <= (int64_t)sms * (A.per_cta / 2)) A.per_cta /= 2;
  const int per_cta = by_column ? kIqColThreads : A.per_cta, threads = by_column ? kIqColThreads : 32 * kIqCh;
  const int64_t grid64 = (cols + per_cta - 1) / per_cta;
  if (grid64 > INT32_MAX) return set_error(FSG_EUNSUPPORTED, "%lld channel groups exceed the grid", (long long)grid64);
  const unsigned grid = (unsigned)grid64;
  const size_t smem = by_column ? 0 : ((size_t)A.per_cta * (32 * A.L + 4) + 32 * A.L) * sizeof(float2);
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  auto launch = [&](auto kernel) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    kernel<<<grid, threads, smem, s>>>(A);
    return cudaGetLastError();
  };
  cudaError_t e;
  switch (n_sections) {
    case 1: e = by_column ? launch(rf2iq_column_kernel<1>) : launch(rf2iq_kernel<1>); break;
    case 2: e = by_column ? launch(rf2iq_column_kernel<2>) : launch(rf2iq_kernel<2>); break;
    case 3: e = by_column ? launch(rf2iq_column_kernel<3>) : launch(rf2iq_kernel<3>); break;
    default: e = by_column ? launch(rf2iq_column_kernel<4>) : launch(rf2iq_kernel<4>); break;
  }
  return check_cuda(e, "rf2iq_kernel launch");
}

static int das_args(const FsgProbe* probe, const FsgDasParams* p, int n_frames, int n_samples, const double* txd,
                    const double* pixels, int64_t n_pixels, DasArgs* A) {
  if (!probe || !p || !txd || (n_pixels > 0 && !pixels))
    return set_error(FSG_EINVAL, "probe, params, tx_delays and pixels must be non-NULL");
  if (probe->n_elements < 1 || probe->n_elements > kDasMaxE)
    return set_error(FSG_EUNSUPPORTED, "n_elements %d outside [1, %d]", probe->n_elements, kDasMaxE);
  if (!(probe->pitch > 0) || !(probe->radius > 0)) return set_error(FSG_EINVAL, "pitch and radius must be > 0");
  if (n_frames < 1 || n_samples < 2 || n_pixels < 0)
    return set_error(FSG_EINVAL, "n_frames >= 1, n_samples >= 2 and n_pixels >= 0 are required");
  if (!(p->speed_of_sound > 0) || !(p->fs > 0)) return set_error(FSG_EINVAL, "speed_of_sound and fs must be > 0");
  if (p->method != FSG_DAS_LINEAR && p->method != FSG_DAS_NEAREST)
    return set_error(FSG_EINVAL, "unknown interpolation method %d", p->method);
  A->txd = txd;
  A->pix = pixels;
  A->n_pix = n_pixels;
  A->n_frames = n_frames;
  A->n_s = n_samples;
  A->E = probe->n_elements;
  A->method = p->method;
  A->iq_rot = p->iq != 0;
  A->pitch = probe->pitch;
  A->radius = probe->radius;
  A->c = (float)p->speed_of_sound;
  A->inv_c = (float)(1.0 / p->speed_of_sound);
  A->fs = (float)p->fs;
  A->two_fc = (float)(2.0 * p->fc);
  A->t0 = (float)p->t0;
  A->aperture = p->fnumber > 0 ? (float)(0.5 / p->fnumber) : -1.f;
  A->slices = 1;
  A->crow = nullptr;
  A->col = nullptr;
  return FSG_OK;
}

template <int G, bool kLong, bool kSliced>
static void launch_das(const DasArgs& A, bool linear, unsigned grid, size_t smem, cudaStream_t s) {
  if (linear) das_kernel<G, true, kLong, kSliced><<<grid, kDasImgThreads, smem, s>>>(A);
  else das_kernel<G, false, kLong, kSliced><<<grid, kDasImgThreads, smem, s>>>(A);
}

extern "C" int32_t fsg_das(const FsgProbe* probe, const FsgDasParams* params, const void* iq, int32_t n_frames,
                           int32_t n_samples, const double* tx_delays, const double* pixels, int64_t n_pixels,
                           void* image_out, void* stream) {
  if (!iq || !image_out) return set_error(FSG_EINVAL, "iq and image_out must be non-NULL");
  DasArgs A;
  int st = das_args(probe, params, n_frames, n_samples, tx_delays, pixels, n_pixels, &A);
  if (st != FSG_OK) return st;
  if (n_pixels == 0) return FSG_OK;
  A.iq = static_cast<const float2*>(iq);
  A.out = static_cast<float2*>(image_out);
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  // up to four firings in one group of four: 259 us against 299 for one firing, 268 against 313 for four
  // (131,072 pixels, 64 elements); at five and more the groups of eight are as fast (311 / 312).  Records
  // or calls beyond 32-bit offsets take 64-bit ones.
  const bool linear = A.method == FSG_DAS_LINEAR,
             lng = n_samples > kDasShort || (int64_t)n_frames * probe->n_elements * n_samples > INT32_MAX,
             few = n_frames <= 4 || lng;
  // few pixels: up to four threads per pixel, as long as the CTAs still fit the SMs at once (75 firings, call:
  // 3,600 pixels 1,111 us with one thread each and 488 with four, 22,372 pixels 1,098 and 502, 65,536 pixels
  // 976 and, with two, 710; 18 firings 401 and 311, 382 and 343)
  int sms = 0;
  if ((st = device_sm_count(&sms)) != FSG_OK) return st;
  const int group = few ? 4 : kDasGroup, groups = (n_frames + group - 1) / group;
  const int64_t ctas = (n_pixels + kDasImgThreads - 1) / kDasImgThreads;
  while (A.slices < kDasStage && 2 * A.slices <= groups && 2 * A.slices * ctas <= (int64_t)sms * kDasImgBlocks)
    A.slices *= 2;
  const unsigned grid = (unsigned)((n_pixels * A.slices + kDasImgThreads - 1) / kDasImgThreads);
  size_t smem = (size_t)group * kDasStage * A.E * sizeof(float);
  if (smem < kDasImgThreads * sizeof(float2)) smem = kDasImgThreads * sizeof(float2);
  // (their own instantiations: with the slices in every kernel 75 firings of 131,072 pixels take 4% more)
  if (A.slices == 1) {
    if (lng) launch_das<4, true, false>(A, linear, grid, smem, s);
    else if (few) launch_das<4, false, false>(A, linear, grid, smem, s);
    else launch_das<kDasGroup, false, false>(A, linear, grid, smem, s);
  } else {
    if (lng) launch_das<4, true, true>(A, linear, grid, smem, s);
    else if (few) launch_das<4, false, true>(A, linear, grid, smem, s);
    else launch_das<kDasGroup, false, true>(A, linear, grid, smem, s);
  }
  return check_cuda(cudaGetLastError(), "das_kernel launch");
}

extern "C" int32_t fsg_dasmtx_nnz_per_row(int32_t method, int32_t n_elements) {
  return method == FSG_DAS_NEAREST ? n_elements : 2 * n_elements;
}

extern "C" int32_t fsg_dasmtx(const FsgProbe* probe, const FsgDasParams* params, int32_t n_samples,
                              const double* tx_delays, const double* pixels, int64_t n_pixels, int32_t* crow,
                              int32_t* col, void* val, void* stream) {
  if (!crow || !col || !val) return set_error(FSG_EINVAL, "crow, col and val must be non-NULL");
  DasArgs A;
  int st = das_args(probe, params, 1, n_samples, tx_delays, pixels, n_pixels, &A);
  if (st != FSG_OK) return st;
  const int64_t per = fsg_dasmtx_nnz_per_row(params->method, probe->n_elements);
  if (n_pixels * per > INT32_MAX || (int64_t)n_samples * probe->n_elements > INT32_MAX)
    return set_error(FSG_EUNSUPPORTED, "matrix of %lld non-zeros exceeds 32-bit CSR indices", (long long)(n_pixels * per));
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (n_pixels == 0) return check_cuda(cudaMemsetAsync(crow, 0, sizeof(int32_t), s), "crow reset");
  A.iq = nullptr;
  A.out = static_cast<float2*>(val);
  A.crow = crow;
  A.col = col;
  dasmtx_kernel<<<(unsigned)((n_pixels + kDasThreads - 1) / kDasThreads), kDasThreads, 0, s>>>(A);
  return check_cuda(cudaGetLastError(), "dasmtx_kernel launch");
}
