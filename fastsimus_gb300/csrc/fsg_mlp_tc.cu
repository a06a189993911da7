// Fused tcgen05 forward pass of the transmit-field surrogate network (inference).
//
// Network: 64 random Fourier features [sin(2 pi B u), cos(2 pi B u)] of the normalised
// inputs, four hidden layers of 256 with SiLU, a linear head of n_out <= 10 outputs (the same
// network that the training kernels of fsg_mlp_train.cu train, with the same SiLU).  A persistent CTA
// takes 128 queries at a time and keeps everything on chip:
//   features -> A (shared memory, BF16 hi + lo, K-major core matrices)
//   per hidden layer: D (TMEM, 128 x 256 FP32) = A_hi W^T + A_lo W^T, two tcgen05.mma
//   kind::f16 per K step of 16, the layer's BF16 weights streamed through four 16 KB
//   shared-memory buffers by TMA bulk copies (32 input columns per copy);
//   epilogue: D + bias -> SiLU -> next layer's A (hi + lo), or, after the last hidden layer,
//   the 256 -> n_out head on the CUDA cores.
// Sixteen worker warps run the features and epilogues, 64 columns at a time; one more streams the weights
// and one issues the MMAs of a layer's 64 input columns as soon as the workers have written them, so the
// products run under the epilogue that feeds them (D alternates between two halves of TMEM).  The
// next tile's features are formed while the last layer's products run.
//
// What bounds it: the chain of a tile, epilogue after epilogue, each waiting for the tail of its products
// (issue 53%, tensor pipe 33% and MUFU 32% of the cycles before the last two steps below).  A layer takes
// 4,200 cycles of MMAs (131 each at N = 256) and the issue of 32,768 SiLUs.  1,048,576 queries: 1,680 us
// with products and epilogues in turn on 8 warps, 1,312 with the products under the epilogues, 1,290 with
// 16 worker warps, 1,191 with four 16 KB weight buffers and their own warp instead of two of 32 KB, 1,130
// with a layer's last inputs multiplied in two halves of the outputs (the epilogue starts on the first),
// 1,016 with the features formed while waiting and packed FP32x2 arithmetic.
//
// The weights are BF16 (as in training) and multiply exactly; splitting the activations into
// hi + lo BF16 keeps them at FP32-class precision (~1e-5 relative), as in the training forward
// pass.  Every mbarrier wait is bounded: on timeout the CTA
// records FSG_ETIMEOUT in the status word, frees its TMEM and returns.

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "../../include/fsgb300.h"
#include "fsg_internal.h"
#include "fsg_tc.cuh"

namespace fsg {

constexpr int kMlpRows = 128;      // queries per tile (MMA M)
constexpr int kMlpWidth = 256;     // hidden width (MMA N)
constexpr int kMlpFeat = 128;      // 2 x 64 Fourier features
constexpr int kMlpChunkK = 64;     // input columns per packed chunk, and per step of the epilogue
constexpr uint32_t kMlpChunkBytes = kMlpWidth * kMlpChunkK * 2;  // 32 KB
constexpr uint32_t kMlpKGroups = kMlpWidth / 8;                 // A operand: 32 core matrices along K
constexpr uint32_t kMlpABytes = kMlpRows * kMlpWidth * 2;       // 64 KB per hi / lo
constexpr uint32_t kOffAHi = 0;
constexpr uint32_t kOffALo = kMlpABytes;
constexpr uint32_t kOffB = 2 * kMlpABytes;
constexpr int kMlpPieceK = 32, kMlpBufs = 4;         // weights are streamed in half chunks of 32 input columns
constexpr uint32_t kMlpPieceBytes = kMlpWidth * kMlpPieceK * 2;  // 16 KB
constexpr uint32_t kMlpSmem = kOffB + kMlpBufs * kMlpPieceBytes;
constexpr uint32_t kMlpWaitTries = 1u << 26;
constexpr uint64_t kMlpDrainNs = 1000000;  // a copy or a layer's products take microseconds
constexpr int kMlpMaxOut = 10;

// SiLU z * sigmoid(z) of two values, evaluated exactly as the training kernels evaluate it.
__device__ __forceinline__ float2 mlp_silu2(float2 z) { return __fmul2_rn(z, tc::sigmoid2(z)); }

// Writes 8 consecutive activations (row r, columns k..k+7) as hi and lo BF16 into the K-major
// A operand.
__device__ __forceinline__ void store_a8(unsigned char* sm, int r, int k, const float* v) {
  uint4 hi, lo;
  tc::split8(v, hi, lo);
  const uint32_t off = tc::kmajor_off(r, k, kMlpKGroups);
  *reinterpret_cast<uint4*>(sm + kOffAHi + off) = hi;
  *reinterpret_cast<uint4*>(sm + kOffALo + off) = lo;
}

constexpr int kMlpWorkers = 512, kMlpBlock = kMlpWorkers + 64;
constexpr int kMlpPiecesPerTile = (kMlpFeat + 3 * kMlpWidth) / kMlpPieceK;

// kWide: the queries start on a 16-byte boundary and are read as such words; else float by float.
template <bool kWide>
__global__ void __launch_bounds__(kMlpBlock, 1) mlp_tc_forward_kernel(const __grid_constant__ FsgMlpWeights W,
                                                                       const float* __restrict__ u, int64_t n,
                                                                       float* __restrict__ out, int* status) {
  extern __shared__ __align__(1024) unsigned char sm[];
  __shared__ uint64_t mbar_full[kMlpBufs], mbar_free[kMlpBufs];  // weight buffers: copied in, released by their MMAs
  __shared__ uint64_t mbar_a[4];                   // 64 columns of A written, one arrival per worker warp
  __shared__ uint64_t mbar_half[2];                // a layer's products done, columns [128 h, 128 h + 128)
  __shared__ uint32_t tmem_holder;
  __shared__ int s_fail;
  __shared__ float bmat[64 * 4];
  __shared__ __align__(16) float whead[kMlpMaxOut][kMlpWidth];
  __shared__ __align__(16) float bias_s[4][kMlpWidth];
  __shared__ float hsum[3][kMlpRows][kMlpMaxOut];

  const int tid = threadIdx.x, warp = tc::warp_uniform(tid >> 5), lane = tid & 31;
  const int nout = W.n_out;
  for (int i = tid; i < 64 * 4; i += blockDim.x) bmat[i] = W.bmat[i];
  for (int i = tid; i < kMlpMaxOut * kMlpWidth; i += blockDim.x)
    whead[i / kMlpWidth][i % kMlpWidth] = (i / kMlpWidth < nout) ? W.w_head[i] : 0.f;
  for (int i = tid; i < 4 * kMlpWidth; i += blockDim.x) bias_s[i / kMlpWidth][i % kMlpWidth] = W.bias[i / kMlpWidth][i % kMlpWidth];
  if (tid == 0) {
    for (int b = 0; b < kMlpBufs; ++b) {
      tc::mbar_init(&mbar_full[b], 1);
      tc::mbar_init(&mbar_free[b], 1);
    }
    for (int c = 0; c < 4; ++c) tc::mbar_init(&mbar_a[c], kMlpWorkers / 32);
    for (int h = 0; h < 2; ++h) tc::mbar_init(&mbar_half[h], 1);
    tc::fence_mbar_init();
    s_fail = 0;
  }
  if (warp == 0) tc::tmem_alloc(&tmem_holder, 2 * kMlpWidth);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = tmem_holder;
  const uint32_t sbase = tc::smem_u32(sm);
  const int64_t n_tiles = (n + kMlpRows - 1) / kMlpRows;
  const int my_tiles = (int)((n_tiles - blockIdx.x + gridDim.x - 1) / gridDim.x);
  // a bounded wait of a whole warp; after one has given up nothing waits any more
  auto wait = [&](uint64_t* mb, uint32_t parity) {
    if (!tc::mbar_test(mb, parity) && !s_fail && !tc::mbar_wait_bounded(mb, parity, kMlpWaitTries)) s_fail = 1;
    __syncwarp();
  };

  const int total = my_tiles * kMlpPiecesPerTile;  // the weights of a tile are one sequence of 16 KB pieces
  if (warp == kMlpWorkers / 32 + 1) {
    // =============================== weights ===============================
    const bool leader = tc::elect_one();
    int j = 0;
    for (int g = 0; g < total && !tc::warp_uniform(s_fail); ++g) {
      const int b = g % kMlpBufs;
      if (g >= kMlpBufs) wait(&mbar_free[b], (g / kMlpBufs - 1) & 1);  // the MMAs of piece g - kMlpBufs
      constexpr int kP0 = kMlpFeat / kMlpPieceK, kP1 = kMlpWidth / kMlpPieceK;
      const int layer = j < kP0 ? 0 : 1 + (j - kP0) / kP1, c = j < kP0 ? j : (j - kP0) % kP1;
      if (leader) {
        tc::mbar_arrive_expect_tx(&mbar_full[b], kMlpPieceBytes);
        tc::bulk_g2s(sm + kOffB + b * kMlpPieceBytes,
                     static_cast<const unsigned char*>(W.packed[layer]) + (size_t)c * kMlpPieceBytes, kMlpPieceBytes,
                     &mbar_full[b]);
      }
      j = j + 1 == kMlpPiecesPerTile ? 0 : j + 1;
    }
  } else if (warp == kMlpWorkers / 32) {
    // =============================== MMAs ===============================
    constexpr uint32_t id_full = tc::idesc_bf16(kMlpRows, kMlpWidth, 0, 0);
    constexpr uint32_t id_half = tc::idesc_bf16(kMlpRows, kMlpWidth / 2, 0, 0);
    const bool leader = tc::elect_one();
    uint32_t ph_a = 0;  // bit c: parity of mbar_a[c]
    int g = 0;
    for (int tile = 0; tile < my_tiles; ++tile) {
      for (int layer = 0; layer < 4; ++layer) {
        const int np = (layer == 0 ? kMlpFeat : kMlpWidth) / kMlpPieceK;
        const uint32_t d = tmem + (layer & 1) * kMlpWidth;
        // piece g (input columns [32 c, 32 c + 32)) times columns [n0, n0 + the descriptor's N) of the weights
        auto products = [&](int c, int b, uint32_t n0, uint32_t idesc) {
          const uint32_t bb = sbase + kOffB + b * kMlpPieceBytes + (n0 >> 3) * 128;
#pragma unroll
          for (int ks = 0; ks < kMlpPieceK / 16; ++ks) {
            const int kk = c * (kMlpPieceK / 16) + ks;  // K step of 16 within the layer
            const uint64_t ah = tc::sdesc(sbase + kOffAHi + kk * 256, 128, kMlpKGroups * 128);
            const uint64_t al = tc::sdesc(sbase + kOffALo + kk * 256, 128, kMlpKGroups * 128);
            // k-group-major packed piece: K stride 4096 bytes, N stride 128
            const uint64_t bd = tc::sdesc(bb + ks * 2 * 4096, 4096, 128);
            tc::mma_bf16(d + n0, ah, bd, idesc, kk > 0);
            tc::mma_bf16(d + n0, al, bd, idesc, 1);
          }
        };
        for (int c = 0; c < np; c += 2, g += 2) {
          const int b0 = g % kMlpBufs, b1 = (g + 1) % kMlpBufs;
          wait(&mbar_a[c >> 1], (ph_a >> (c >> 1)) & 1);
          ph_a ^= 1u << (c >> 1);
          wait(&mbar_full[b0], (g / kMlpBufs) & 1);
          tc::fence_after_sync();
          if (c + 2 < np) {
            if (leader && !s_fail) {
              products(c, b0, 0, id_full);
              tc::commit(&mbar_free[b0]);
            }
            wait(&mbar_full[b1], ((g + 1) / kMlpBufs) & 1);
            tc::fence_after_sync();
            if (leader && !s_fail) {
              products(c + 1, b1, 0, id_full);
              tc::commit(&mbar_free[b1]);
            }
          } else {
            // the last inputs in two halves of the outputs: the epilogue starts on the first
            wait(&mbar_full[b1], ((g + 1) / kMlpBufs) & 1);
            tc::fence_after_sync();
            if (leader && !s_fail) {
#pragma unroll
              for (uint32_t h = 0; h < 2; ++h) {
                products(c, b0, 128 * h, id_half);
                if (h == 1) tc::commit(&mbar_free[b0]);
                products(c + 1, b1, 128 * h, id_half);
                if (h == 1) tc::commit(&mbar_free[b1]);
                tc::commit(&mbar_half[h]);
              }
            }
          }
        }
      }
    }
  } else {
    // =============================== workers ===============================
    // TMEM row of this thread, and its 16 columns of each 64
    const int row = 32 * (warp & 3) + lane, part = warp >> 2;
    const uint32_t trow = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
    auto ready = [&](int c) {  // this warp's part of A columns [64 c, 64 c + 64) is written, its D reads done
      tc::fence_proxy_async_smem();
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&mbar_a[c]);
    };
    // this thread's 16 features of a tile's queries, eight at a time, as hi and lo BF16: sines, cosines
    uint4 f_hi[2][2], f_lo[2][2];
    auto features = [&](int64_t tile, int blk) {
      const int64_t q = tile * kMlpRows + row;
      float4 uv = make_float4(0.f, 0.f, 0.f, 0.f);
      if (q < n) {
        if constexpr (kWide) uv = *reinterpret_cast<const float4*>(u + 4 * q);
        else uv = make_float4(u[4 * q], u[4 * q + 1], u[4 * q + 2], u[4 * q + 3]);
      }
      float sv[8], cv[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float* b = bmat + 4 * (16 * part + 8 * blk + i);
        const float t = b[0] * uv.x + b[1] * uv.y + b[2] * uv.z + b[3] * uv.w;
        sincospif(2.0f * t, &sv[i], &cv[i]);
      }
      tc::split8(sv, f_hi[blk][0], f_lo[blk][0]);
      tc::split8(cv, f_hi[blk][1], f_lo[blk][1]);
    };
    auto store_features = [&]() {  // -> A (K = 128): sines, then cosines
#pragma unroll
      for (int blk = 0; blk < 2; ++blk)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint32_t o = tc::kmajor_off(row, 64 * h + 16 * part + 8 * blk, kMlpKGroups);
          *reinterpret_cast<uint4*>(sm + kOffAHi + o) = f_hi[blk][h];
          *reinterpret_cast<uint4*>(sm + kOffALo + o) = f_lo[blk][h];
        }
    };
    uint32_t ph_layer = 0;
    if (my_tiles > 0) {
      features(blockIdx.x, 0);
      features(blockIdx.x, 1);
      store_features();
      ready(0);
      ready(1);
    }
    for (int it = 0; it < my_tiles; ++it) {
      const int64_t tile = blockIdx.x + (int64_t)it * gridDim.x;
      float head[kMlpMaxOut];
#pragma unroll
      for (int j = 0; j < kMlpMaxOut; ++j) head[j] = 0.f;
      for (int layer = 0; layer < 4; ++layer) {
        // the next tile's features are formed while the last layer's products run
        const bool more = it + 1 < my_tiles;
        if (more && layer == 3) {
          features(tile + gridDim.x, 0);
          features(tile + gridDim.x, 1);
        }
        wait(&mbar_half[0], ph_layer);
        tc::fence_after_sync();
        if (more && layer == 3) {
          store_features();
          ready(0);
        }
        const float* bias = bias_s[layer];
        const uint32_t d = trow + (layer & 1) * kMlpWidth + 16 * part;
        uint32_t next[16];
        tc::tmem_ld16_async(d, next);
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
          const int col0 = 64 * c + 16 * part;
          float v[16];
          if (c == 1) {  // before the second half is read, and before A columns its products read are written
            wait(&mbar_half[1], ph_layer);
            tc::fence_after_sync();
            // only now may the next tile's first layer finish, which completes mbar_half[1] again
            if (more && layer == 3) ready(1);
          }
          tc::tmem_wait_ld16(next);
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(next[i]);
          if (c < 3) tc::tmem_ld16_async(d + 64 * (c + 1), next);  // lands under this chunk's SiLUs
#pragma unroll
          for (int i = 0; i < 16; i += 2) {
            const float2 z = __fadd2_rn(make_float2(v[i], v[i + 1]), *reinterpret_cast<const float2*>(bias + col0 + i));
            const float2 y = mlp_silu2(z);
            v[i] = y.x;
            v[i + 1] = y.y;
          }
          if (layer < 3) {
#pragma unroll
            for (int g8 = 0; g8 < 2; ++g8) store_a8(sm, row, col0 + 8 * g8, v + 8 * g8);
            ready(c);
          } else {
#pragma unroll
            for (int j = 0; j < kMlpMaxOut; ++j) {
              float acc = head[j];
#pragma unroll
              for (int i = 0; i < 16; ++i) acc = fmaf(v[i], whead[j][col0 + i], acc);
              head[j] = acc;
            }
          }
        }
        ph_layer ^= 1u;
      }
      // ---- head: combine the four column sets of each row ----
      tc::fence_before_sync();
      if (part > 0) {
#pragma unroll
        for (int j = 0; j < kMlpMaxOut; ++j) hsum[part - 1][row][j] = head[j];
      }
      tc::bar_sync(1, kMlpWorkers);
      if (part == 0) {
        const int64_t q = tile * kMlpRows + row;
        if (q < n && !s_fail) {
          for (int j = 0; j < nout; ++j)
            out[q * nout + j] = head[j] + hsum[0][row][j] + hsum[1][row][j] + hsum[2][row][j] + W.b_head[j];
        }
      }
      tc::bar_sync(1, kMlpWorkers);
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (s_fail && tid == 0) {
    // a wait gave up: what is still in flight gets its bounded time before the memory goes away
    const uint64_t t0 = tc::global_ns();
    while (tc::global_ns() - t0 < kMlpDrainNs) __nanosleep(1000);
    atomicExch(status, FSG_ETIMEOUT);
  }
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem, 2 * kMlpWidth);
}

// Packs a row-major [256][K] BF16 weight matrix into K/64 chunks of the K-major no-swizzle
// core-matrix layout that the forward kernel copies into shared memory as the B operand.
__global__ void mlp_pack_kernel(const __nv_bfloat16* __restrict__ w, int K, __nv_bfloat16* __restrict__ packed) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= kMlpWidth * K) return;
  const int n = i / K, k = i % K;
  const int c = k / kMlpChunkK, kk = k % kMlpChunkK;
  // bytes within the chunk: core (kk / 8, n / 8) at ((kk / 8) * 32 + n / 8) * 128 (k-group-major)
  const uint32_t off = ((uint32_t)(((kk >> 3) << 5) + (n >> 3)) << 7) + ((uint32_t)(n & 7) << 4) + ((uint32_t)(kk & 7) << 1);
  packed[(size_t)c * (kMlpChunkBytes / 2) + off / 2] = w[i];
}

}  // namespace fsg

using namespace fsg;

extern "C" size_t fsg_mlp_tc_packed_bytes(int32_t n_in) {
  if (n_in < kMlpChunkK || n_in % kMlpChunkK) return 0;
  return (size_t)kMlpWidth * n_in * 2;
}

extern "C" int32_t fsg_mlp_tc_pack(const void* w_bf16, int32_t n_out, int32_t n_in, void* packed, void* stream) {
  if (!w_bf16 || !packed) return set_error(FSG_EINVAL, "NULL argument");
  if (n_out != kMlpWidth || n_in < kMlpChunkK || n_in % kMlpChunkK)
    return set_error(FSG_EUNSUPPORTED, "tensor-core MLP layers are %d x K with K a multiple of %d (got %d x %d)",
                     kMlpWidth, kMlpChunkK, n_out, n_in);
  const int total = n_out * n_in;
  mlp_pack_kernel<<<(total + 255) / 256, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(w_bf16), n_in, static_cast<__nv_bfloat16*>(packed));
  return check_cuda(cudaGetLastError(), "mlp_pack_kernel launch");
}

extern "C" int32_t fsg_mlp_tc_forward(const FsgMlpWeights* weights, const float* u, int64_t n, float* out, int32_t* status,
                                      void* stream_ptr) {
  if (!weights || !u || !out || !status || n < 0) return set_error(FSG_EINVAL, "NULL argument or n < 0");
  for (int l = 0; l < 4; ++l)
    if (!weights->packed[l] || !weights->bias[l]) return set_error(FSG_EINVAL, "layer %d weights or bias missing", l);
  if (!weights->w_head || !weights->b_head || !weights->bmat) return set_error(FSG_EINVAL, "head or features missing");
  if (weights->n_out < 1 || weights->n_out > kMlpMaxOut)
    return set_error(FSG_EUNSUPPORTED, "n_out must be in [1, %d] (got %d)", kMlpMaxOut, weights->n_out);
  if (n == 0) return FSG_OK;
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return check_cuda(e, "device query");
  const auto kernel = (reinterpret_cast<uintptr_t>(u) & 15) == 0 ? mlp_tc_forward_kernel<true> : mlp_tc_forward_kernel<false>;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMlpSmem);
  if (e != cudaSuccess) return check_cuda(e, "cudaFuncSetAttribute(mlp_tc_forward_kernel)");
  const int64_t tiles = (n + kMlpRows - 1) / kMlpRows;
  const int grid = (int)(tiles < sms ? tiles : sms);
  kernel<<<grid, kMlpBlock, kMlpSmem, reinterpret_cast<cudaStream_t>(stream_ptr)>>>(*weights, u, n, out, status);
  return check_cuda(cudaGetLastError(), "mlp_tc_forward_kernel launch");
}
