// Spectrum -> RF epilogue: irfft of the conjugated spectrum over its nonzero band, plus the
// smooth -100 dB gate (simus.py:336-367), in three kernels.
//
// rf[n][e] = (1/N) sum_k w_k Re(conj(S[k][e]) exp(i 2 pi k n / N)),  n < (N + 1) / 2,
// w_k = 1 for k = 0 and k = N/2, 2 otherwise, k <= N/2 (the Hermitian half that a C2R
// transform reads; the imaginary parts of the DC and Nyquist bins drop out because
// sin(0) = sin(pi n) = 0).  Only the selected band [k_first, k_first + k_count) of the
// simus spectrum is nonzero, so the sum runs over it alone.  The transform is a real GEMM
// [cos | sin](n, k) x [Re S ; Im S](k, e) with the twiddles looked up by the exact integer
// index (k n) mod N in a table of N entries, FP32 accumulation.
//
// A CTA takes 64 samples x 64 elements of one frame, 4 x 4 outputs per thread (elements 16 apart, so
// that a warp's loads of one are contiguous): 32 multiply-adds per two 16-byte broadcasts and four
// 8-byte loads, about where the FP32 pipe and the shared-memory pipe balance.  A
// single frame has too few such tiles for 152 SMs (16 at 1,015 samples x 64 elements), so the
// frequencies are split over the CTAs of a cluster, whose partial tiles are summed in rank order
// through distributed shared memory.  The table sits in shared memory (the lookups scatter), the
// index advances by n per frequency without a division.  Measured: 1,015 samples x 64 elements x 637
// frequencies 121 -> 24 us, 2,290 x 192 x 1,430 359 -> 100 us, 75 frames of 1,080 x 64 x 678 1,028 ->
// 445 us.
//
// The gate multiplies by 0.5 (1 + tanh((|rf| / max|rf| - 1e-5) / 1e-6)) with each frame's own
// peak; the first kernel folds its output tile's peak into a per-frame word with an integer
// atomicMax on the float bits (|rf| >= 0, so the order of the bits is the order of the
// values and the result does not depend on the order of the atomics).

#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "../../include/fsgb300.h"
#include "fsg_internal.h"

namespace cg = cooperative_groups;

namespace fsg {

constexpr int kRfTile = 64;               // samples and elements per CTA tile
constexpr int kRfK = 32;                  // frequencies per shared-memory chunk
constexpr size_t kRfChunk = (size_t)kRfK * kRfTile * sizeof(float2);  // 16 KB; two chunks also hold a partial tile
constexpr size_t kRfMaxTable = 96 * 1024; // longer twiddle tables are gathered from global memory
constexpr int kRfMaxSplit = 8;

// tw[j] = exp(2 pi i j / N), the angle's rounding error to FP32 corrected to first order; also
// resets the frames' peaks.
__global__ void twiddle_kernel(float2* tw, int N, unsigned int* peak, int n_batch) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j < n_batch) peak[j] = 0u;
  if (j >= N) return;
  const double q = 2.0 * (double)j * (1.0 / (double)N);
  const float hi = (float)q, lo = (float)kPi * (float)(q - (double)hi);
  float s, c;
  sincospif(hi, &s, &c);
  tw[j] = make_float2(fmaf(-lo, s, c), fmaf(lo, c, s));
}

__global__ void __launch_bounds__(256) irfft_kernel(const float2* __restrict__ S, int64_t bstride, int E, int N,
                                                    int k0, int kc, int table, const float2* __restrict__ tw,
                                                    int n_samples, float* __restrict__ rf,
                                                    unsigned int* __restrict__ peak) {
  extern __shared__ __align__(16) unsigned char rf_sm[];
  float2(*Ssh)[kRfTile] = reinterpret_cast<float2(*)[kRfTile]>(rf_sm);
  float2(*Tsh)[kRfTile] = reinterpret_cast<float2(*)[kRfTile]>(rf_sm + kRfChunk);
  float2* tws = reinterpret_cast<float2*>(rf_sm + 2 * kRfChunk);
  __shared__ unsigned int s_peak;
  cg::cluster_group cluster = cg::this_cluster();
  const int split = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const int b = blockIdx.z;
  const int n0 = (blockIdx.x / split) * kRfTile, e0 = blockIdx.y * kRfTile;
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;  // samples n0 + 4 ty + i, elements e0 + tx + 16 j
  const float2* Sb = S + (size_t)b * bstride;
  const float inv_n = 1.0f / (float)N;
  // this rank's frequencies, whole chunks of kRfK
  const int chunks = (kc + kRfK - 1) / kRfK;
  const int c_lo = (int)((int64_t)rank * chunks / split) * kRfK;
  const int c_hi = min(kc, (int)((int64_t)(rank + 1) * chunks / split) * kRfK);
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  if (tid == 0) s_peak = 0u;
  const float2* lut = tw;
  if (table) {
    for (int i = tid; i < N; i += blockDim.x) tws[i] = tw[i];
    lut = tws;
  }
  // the table indices of this thread's twiddles: sample n0 + tid % 64, frequencies tid / 64 + 4 i
  const int tn = tid & (kRfTile - 1), tk = tid / kRfTile;
  const unsigned int un = (unsigned int)N;
  unsigned int at = (unsigned int)((long long)(k0 + c_lo + tk) * (n0 + tn) % N);
  const unsigned int adv = (unsigned int)(4LL * (n0 + tn) % N);
  for (int c0 = c_lo; c0 < c_hi; c0 += kRfK) {
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kRfK / 4; ++q) {
      const int kk = tk + 4 * q, k = k0 + c0 + kk, e = e0 + tn;
      float2 v = make_float2(0.f, 0.f);
      if (c0 + kk < c_hi && e < E) {
        v = Sb[(size_t)k * E + e];
        const float w = (k == 0 || 2 * (int64_t)k == N) ? inv_n : 2.0f * inv_n;
        v.x *= w;
        v.y *= w;
      }
      Ssh[kk][tn] = v;
      Tsh[kk][tn] = lut[at];
      at += adv;
      if (at >= un) at -= un;
    }
    __syncthreads();
#pragma unroll 4
    for (int kk = 0; kk < kRfK; ++kk) {
      const float4 ta = *reinterpret_cast<const float4*>(&Tsh[kk][4 * ty]);
      const float4 tb = *reinterpret_cast<const float4*>(&Tsh[kk][4 * ty + 2]);
      const float tr[4] = {ta.x, ta.z, tb.x, tb.z}, ti[4] = {ta.y, ta.w, tb.y, tb.w};
      float sr[4], si[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 v = Ssh[kk][tx + 16 * j];
        sr[j] = v.x;
        si[j] = v.y;
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(sr[j], tr[i], acc[i][j]);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(si[j], ti[i], acc[i][j]);
    }
  }
  float m = 0.f;
  if (split == 1) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int n = n0 + 4 * ty + i;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int e = e0 + tx + 16 * j;
        if (n < n_samples && e < E) {
          rf[((size_t)b * n_samples + n) * E + e] = acc[i][j];
          m = fmaxf(m, fabsf(acc[i][j]));
        }
      }
    }
  } else {
    // every rank leaves its partial tile in its shared memory and sums 64 / split rows of all of them
    __syncthreads();
    float* mine = reinterpret_cast<float*>(rf_sm);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) mine[(4 * ty + i) * kRfTile + tx + 16 * j] = acc[i][j];
    cluster.sync();
    const int rows = kRfTile / split;
    for (int i = tid; i < rows * kRfTile; i += blockDim.x) {
      const int r = rank * rows + i / kRfTile, c = i % kRfTile, n = n0 + r, e = e0 + c;
      float v = 0.f;
      for (int q = 0; q < split; ++q) v += cluster.map_shared_rank(mine, q)[r * kRfTile + c];
      if (n < n_samples && e < E) {
        rf[((size_t)b * n_samples + n) * E + e] = v;
        m = fmaxf(m, fabsf(v));
      }
    }
    cluster.sync();  // no CTA leaves while its tile is being read
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
  __syncthreads();
  if ((tid & 31) == 0) atomicMax(&s_peak, __float_as_uint(m));
  __syncthreads();
  if (tid == 0) atomicMax(&peak[b], s_peak);
}

__global__ void gate_kernel(float* __restrict__ rf, int64_t per_frame, int n_batch, const unsigned int* __restrict__ peak) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= per_frame * n_batch) return;
  const float m = __uint_as_float(peak[i / per_frame]);
  const float v = rf[i];
  const float rel = fabsf(v) / (m + 1e-30f);
  rf[i] = v * (0.5f * (1.0f + tanhf((rel - 1e-5f) / 1e-6f)));
}

static size_t rf_a256(size_t v) { return (v + 255) & ~size_t(255); }

}  // namespace fsg

using namespace fsg;

extern "C" size_t fsg_rf_workspace_size(int32_t n_fft, int32_t n_batch) {
  if (n_fft < 1 || n_batch < 1) return 0;
  return rf_a256((size_t)n_fft * 8) + rf_a256((size_t)n_batch * 4);
}

extern "C" int32_t fsg_irfft_gate(const void* spectrum, int32_t n_batch, int64_t batch_stride, int32_t n_freq_full,
                                  int32_t n_elements, int32_t n_fft, int32_t k_first, int32_t k_count, int32_t gate,
                                  float* rf_out, void* workspace, size_t workspace_bytes, void* stream_ptr) {
  if (!spectrum || !rf_out) return set_error(FSG_EINVAL, "spectrum and rf_out must be non-NULL");
  if (n_batch < 1 || n_elements < 1 || n_fft < 1 || n_freq_full < 1)
    return set_error(FSG_EINVAL, "n_batch, n_elements, n_fft and n_freq_full must be >= 1");
  if (k_first < 0 || k_count < 0 || k_first + k_count > n_freq_full)
    return set_error(FSG_EINVAL, "band [%d, %d) does not fit in n_freq_full = %d", k_first, k_first + k_count,
                     n_freq_full);
  if (batch_stride < (int64_t)n_freq_full * n_elements)
    return set_error(FSG_EINVAL, "batch_stride %lld is smaller than one spectrum", (long long)batch_stride);
  const size_t need = fsg_rf_workspace_size(n_fft, n_batch);
  if (!workspace || workspace_bytes < need)
    return set_error(FSG_EWORKSPACE, "workspace of %zu bytes is smaller than the %zu bytes required", workspace_bytes,
                     need);
  // a C2R transform of length N reads bins 0 .. N/2 only
  int kc = k_count;
  if (k_first > n_fft / 2) kc = 0;
  else if (k_first + kc > n_fft / 2 + 1) kc = n_fft / 2 + 1 - k_first;
  const int n_samples = (n_fft + 1) / 2;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream_ptr);
  unsigned char* ws = static_cast<unsigned char*>(workspace);
  float2* tw = reinterpret_cast<float2*>(ws);
  unsigned int* peak = reinterpret_cast<unsigned int*>(ws + rf_a256((size_t)n_fft * 8));
  int st;
  const int setup = n_fft > n_batch ? n_fft : n_batch;
  twiddle_kernel<<<(setup + 255) / 256, 256, 0, s>>>(tw, n_fft, peak, n_batch);
  if ((st = check_cuda(cudaGetLastError(), "twiddle_kernel launch")) != FSG_OK) return st;
  int sms = 0;
  if ((st = device_sm_count(&sms)) != FSG_OK) return st;
  // split the frequencies while the tiles leave SMs idle (four CTAs fit one) and a rank keeps two chunks
  const int nt = (n_samples + kRfTile - 1) / kRfTile, et = (n_elements + kRfTile - 1) / kRfTile;
  int split = 1;
  while (split < kRfMaxSplit && (int64_t)nt * et * n_batch * split * 2 <= 4 * (int64_t)sms &&
         kc >= 2 * kRfK * split * 2)
    split *= 2;
  const int table = (size_t)n_fft * 8 <= kRfMaxTable ? 1 : 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(nt * split), (unsigned)et, (unsigned)n_batch);
  cfg.blockDim = dim3(256);
  cfg.dynamicSmemBytes = 2 * kRfChunk + (table ? (size_t)n_fft * 8 : 0);
  cfg.stream = s;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim = {(unsigned)split, 1, 1};
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  if ((st = check_cuda(cudaFuncSetAttribute(irfft_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            (int)(2 * kRfChunk + kRfMaxTable)),
                       "cudaFuncSetAttribute(irfft_kernel)")) != FSG_OK)
    return st;
  if ((st = check_cuda(cudaLaunchKernelEx(&cfg, irfft_kernel, static_cast<const float2*>(spectrum), batch_stride,
                                          (int)n_elements, (int)n_fft, (int)k_first, kc, table, (const float2*)tw,
                                          n_samples, rf_out, peak),
                       "irfft_kernel launch")) != FSG_OK)
    return st;
  if (gate) {
    const int64_t per = (int64_t)n_samples * n_elements;
    gate_kernel<<<(unsigned)((per * n_batch + 255) / 256), 256, 0, s>>>(rf_out, per, n_batch, peak);
    if ((st = check_cuda(cudaGetLastError(), "gate_kernel launch")) != FSG_OK) return st;
  }
  return FSG_OK;
}
