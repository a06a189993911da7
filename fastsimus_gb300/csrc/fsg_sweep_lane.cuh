// The plain simus sweep for probes of more than 32 elements (1 to 4 sub-elements):
// simus_lane_kernel.  Instantiated by fsg_sweep_lane.cu (without full-frequency directivity) and
// fsg_sweep_lane_ffd.cu (with it), compiled in parallel.
//
// One thread owns two elements (lane and lane + 32 of its warp's 64) of PPT scatterers and runs
// the recurrences of all their sub-elements; NW warps (64 elements each) form a group that takes
// PPT scatterers of a tile, and a CTA holds as many groups as its warps give.  Per
// sub-block of FS frequencies (PPT FS = 16 (scatterer, frequency) pairs):
//
//   generate   m(e, s, f) = sum_u G(s, e, u, f) exp(i 2 pi f tau_e) for the thread's two elements,
//              packed FP32x2 over the elements, kept in registers;
//   transmit   sum_e apod_e m(e, s, f): two elements in the thread, then a reduce-scatter of the
//              16 values over the warp's lanes, and for NW > 1 the warps' sums through shared
//              memory and one named barrier of the group; W = rc pulse probe P, written once per
//              warp and read back as broadcasts;
//   receive    Y'(e, f) += sum_s m(e, s, f) W(s, f) from the registers, added to the group's
//              running spectrum in shared memory once per sub-block (one thread owns each entry).
//
// What bounds it: instruction issue and the FP32 pipe (60% and 59% of the cycles of a 9,000-scatterer,
// 128-element chunk; a packed FP32x2 instruction issues once and holds the pipe for two cycles, and
// a fused multiply-add of three distinct registers sustains 0.62 of the pipe's rate on this part, a
// recurrence step 0.8: the register file's read ports).  Per (scatterer, element, frequency) at two
// sub-elements it takes 8 lane operations for the recurrences, 2 for the sub-element sum, 2 for the
// transmit sum and 4 for the receive products.
//
// The kernels that this one replaced kept the Green's terms of a tile in a shared-memory stash
// between transmit and receive: 16 bytes of shared traffic per term and a CTA-wide hand-over per 8
// frequencies.  Here a term never leaves its thread.  40,000 scatterers, one firing (spectrum
// call): 64 elements x 2 sub-elements 1,583 -> 1,353 us, 64 x 1 2,453 -> 1,081 us, 128 x 2 5,367 ->
// 5,207 us, 128 x 2 with full-frequency directivity 11,850 -> 10,100 us with 14 directivity terms (8 terms:
// 4,570 -> 3,526 us for the convex probe below); 192 x 2, 8,000
// scatterers, 3,547 -> 2,120 us.
//
// Block size: 384 threads (168 registers, three warps per scheduler) beat 256 (232 registers) by
// 0 to 9% without full-frequency directivity; with it the extra state spills, and 256 win by 19%
// (3,526 against 4,326 us for a 128-element convex probe, 15,001 scatterers).  Groups of three warps (129 to 192
// elements) take 384 in either case, which they divide.
//
// The receive sums carry the transmit delay phase exp(i 2 pi f tau_e) of every term; simus_reduce
// multiplies it out, once per (f, e).
#pragma once

#include "fsg_sweep_kernels.cuh"

namespace fsg {

// Geometry block of a tile, from geo + tile * geo_bytes: per group, pair p = u PPT + s and thread,
// the two elements' (r_hi, r_lo), (amp, step re), step im and with FFD (half_seg sin(theta))^2; then
// the tile's reflectivities (0 for padding and out of field).
struct LaneBlock {
  float4* a;   // r_hi0, r_hi1, r_lo0, r_lo1
  float4* b;   // amp0, amp1, step.x0, step.x1
  float2* c;   // step.y0, step.y1
  float2* d;   // dir0^2, dir1^2 (FFD)
  float* w;    // [tile points]
};

__host__ __device__ inline LaneBlock lane_block(unsigned char* base, int slots, bool ffd) {
  LaneBlock B;
  size_t o = 0;
  B.a = reinterpret_cast<float4*>(base); o += (size_t)slots * 16;
  B.b = reinterpret_cast<float4*>(base + o); o += (size_t)slots * 16;
  B.c = reinterpret_cast<float2*>(base + o); o += (size_t)slots * 8;
  B.d = reinterpret_cast<float2*>(base + o); o += ffd ? (size_t)slots * 8 : 0;
  B.w = reinterpret_cast<float*>(base + o);
  return B;
}

// DT: terms of the directivity polynomial with full-frequency directivity (FFD), else 0.
// MAXT: the block's threads, a multiple of the group's 32 NW.
template <int U, int DT, int MAXT>
__global__ void __launch_bounds__(MAXT, 1) simus_lane_kernel(const BandArgs A) {
  constexpr int PPT = lane_points(U), FS = 16 / PPT, NP = U * PPT;
  constexpr bool FFD = DT > 0;
  extern __shared__ __align__(16) unsigned char sm[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int NW = A.nw, T = 32 * NW, FB = A.fb;
  const int n_grp = MAXT / T;
  const int grp = tid / T, tg = tid - grp * T, wg = tg >> 5;
  const LaneLayout L = lane_layout(NW, FB, MAXT, FFD);
  float4* Y = reinterpret_cast<float4*>(sm) + (size_t)grp * FB * T + tg;  // [f] stride T: re0, re1, im0, im1
  float2* pp = reinterpret_cast<float2*>(sm + L.off_pp);
  float* kb = reinterpret_cast<float*>(sm + L.off_kb);
  float2* part = reinterpret_cast<float2*>(sm + L.off_part) + grp * 2 * NW * 16;  // [2][NW][16]
  float2* Wb = reinterpret_cast<float2*>(sm + L.off_w) + warp * 32;                // [2][16]
  float4* tr = reinterpret_cast<float4*>(sm + L.off_tr) + warp * 16 * kLaneTrPitch; // [32][pitch] float2

  const int e0 = wg * 64 + lane, e1 = e0 + 32;
  const int c0 = min(e0, A.E - 1), c1 = min(e1, A.E - 1);
  const float w0 = e0 < A.E ? A.t.wtx[c0] : 0.f, w1 = e1 < A.E ? A.t.wtx[c1] : 0.f;
  const float2 ds0 = A.t.dstep[c0], ds1 = A.t.dstep[c1];
  const int idx = lane & 15, my_s = idx / FS, my_f = idx % FS;  // the (scatterer, frequency) this lane ends up with
  const int slots = n_grp * NP * T;

  const int64_t units = (int64_t)A.n_bands * A.chunk_tiles;
  const int64_t u_end = (int64_t)(blockIdx.x + 1) * units / A.grid;
  int par = 0;
  for (int64_t un = (int64_t)blockIdx.x * units / A.grid; un < u_end;) {
    const int band = (int)(un / A.chunk_tiles);
    const int64_t t_lo = un - (int64_t)band * A.chunk_tiles;
    const int64_t t_hi = min(A.chunk_tiles, t_lo + (u_end - un));
    un += t_hi - t_lo;
    const int slot = (int)blockIdx.x - cta_of_unit((int64_t)band * A.chunk_tiles, units, A.grid);
    const int f_b0 = band * FB;
    __syncthreads();  // the previous segment's sums have been read
    for (int i = tid; i < FB; i += MAXT) {
      const int f = f_b0 + i;
      pp[i] = (f < A.F) ? A.t.pp[f] : make_float2(0.f, 0.f);
      if (FFD) {
        const float k = A.t.kf[min(f, A.F - 1)].x;
        kb[i] = k * k;
      }
    }
    for (int f = 0; f < FB; ++f) Y[f * T] = make_float4(0.f, 0.f, 0.f, 0.f);
    __syncthreads();
    const float2 k0 = A.t.kf[f_b0];
    const float a0 = A.t.af[f_b0];
    const float2 ph0 = A.t.dph[(size_t)band * A.E + c0], ph1 = A.t.dph[(size_t)band * A.E + c1];

    for (int64_t tile = t_lo; tile < t_hi; ++tile) {
      const LaneBlock B = lane_block(A.geo + tile * A.geo_bytes, slots, FFD);
      const float w = B.w[grp * PPT + my_s];
      // exact anchors at the band's first frequency, times the elements' delay phases
      float2 Gr[NP], Gi[NP], Sr[NP], Si[NP], Sn[NP];
      float2 Dh[FFD ? NP : 1];
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        const int i = (grp * NP + p) * T + tg;
        const float4 ga = B.a[i], gb = B.b[i];
        const float2 gc = B.c[i];
        if constexpr (FFD) Dh[p] = B.d[i];
        const float2 g0 = cmul(anchor_value(ga.x, ga.z, gb.x, k0, a0), ph0);
        const float2 g1 = cmul(anchor_value(ga.y, ga.w, gb.y, k0, a0), ph1);
        const float2 s0 = cmul(make_float2(gb.z, gc.x), ds0), s1 = cmul(make_float2(gb.w, gc.y), ds1);
        Gr[p] = make_float2(g0.x, g1.x);
        Gi[p] = make_float2(g0.y, g1.y);
        Sr[p] = make_float2(s0.x, s1.x);
        Si[p] = make_float2(s0.y, s1.y);
        Sn[p] = make_float2(-s0.y, -s1.y);
      }
#pragma unroll 1
      for (int sb = 0; sb < FB; sb += FS) {
        // ---- generate: FS steps; m of every (scatterer, frequency) and its two-element sum ----
        float2 mr[16], mi[16], v[16];
#pragma unroll
        for (int j = 0; j < FS; ++j) {
          float2 kk = make_float2(0.f, 0.f);
          if constexpr (FFD) {
            const float k = kb[sb + j];
            kk = make_float2(k, k);
          }
#pragma unroll
          for (int s = 0; s < PPT; ++s) {
            float2 r, q;
            if constexpr (FFD) {
              const float2 d = sinc_poly2<DT>(__fmul2_rn(Dh[s], kk));
              r = __fmul2_rn(Gr[s], d);
              q = __fmul2_rn(Gi[s], d);
#pragma unroll
              for (int u = 1; u < U; ++u) {
                const float2 du = sinc_poly2<DT>(__fmul2_rn(Dh[u * PPT + s], kk));
                r = __ffma2_rn(Gr[u * PPT + s], du, r);
                q = __ffma2_rn(Gi[u * PPT + s], du, q);
              }
            } else {
              r = Gr[s];
              q = Gi[s];
#pragma unroll
              for (int u = 1; u < U; ++u) {
                r = __fadd2_rn(r, Gr[u * PPT + s]);
                q = __fadd2_rn(q, Gi[u * PPT + s]);
              }
            }
            const int i = s * FS + j;
            mr[i] = r;
            mi[i] = q;
            v[i] = make_float2(fmaf(w1, r.y, w0 * r.x), fmaf(w1, q.y, w0 * q.x));
          }
#pragma unroll
          for (int p = 0; p < NP; ++p) cstep2(Gr[p], Gi[p], Sr[p], Si[p], Sn[p]);
        }
        // ---- transmit: sum over the lanes through the warp's transpose buffer (lane l and l + 16
        // add up value l % 16 of 16 lanes each), then over the warps ----
        float4* tb = tr + lane * (kLaneTrPitch / 2);
#pragma unroll
        for (int i = 0; i < 8; ++i) tb[i] = make_float4(v[2 * i].x, v[2 * i].y, v[2 * i + 1].x, v[2 * i + 1].y);
        __syncwarp();
        float2 P = make_float2(0.f, 0.f);
        {
          const float2* tq = reinterpret_cast<const float2*>(tr) + (lane & 16) * kLaneTrPitch + idx;
          float2 Q = P;
#pragma unroll
          for (int q = 0; q < 16; q += 2) {
            P = __fadd2_rn(P, tq[q * kLaneTrPitch]);
            Q = __fadd2_rn(Q, tq[(q + 1) * kLaneTrPitch]);
          }
          P = __fadd2_rn(P, Q);
        }
        P.x += __shfl_xor_sync(0xffffffffu, P.x, 16);
        P.y += __shfl_xor_sync(0xffffffffu, P.y, 16);
        if (NW > 1) {
          float2* pb = part + par * NW * 16 + idx;
          if (lane < 16) pb[wg * 16] = P;
          tc::bar_sync(1 + grp, T);
          P = pb[0];
          for (int q = 1; q < NW; ++q) P = cadd(P, pb[q * 16]);
        }
        {
          const float2 pv = cmul(pp[sb + my_f], P);
          if (lane < 16) Wb[par * 16 + (FFD ? idx : my_f * PPT + my_s)] = make_float2(w * pv.x, w * pv.y);
        }
        __syncwarp();
        // ---- receive ----
        // two W per read without FFD (200,000 scatterers x 128 elements 24.42 -> 24.05 ms); with it the
        // registers are short, and single reads win (3,527 against 3,580 us)
        const float2* wb = Wb + par * 16;
        const float4* wb2 = reinterpret_cast<const float4*>(wb);  // [frequency][scatterer], without FFD
#pragma unroll
        for (int j = 0; j < FS; ++j) {
          float2 yr = make_float2(0.f, 0.f), yi = yr;
#pragma unroll
          for (int s = 0; s < PPT; ++s) {
            const int i = s * FS + j;
            const float4 w2 = wb2[(j * PPT + s) / 2];
            const float2 q = FFD ? wb[i] : (s & 1 ? make_float2(w2.z, w2.w) : make_float2(w2.x, w2.y));
            yr.x = fmaf(mr[i].x, q.x, yr.x);
            yr.y = fmaf(mr[i].y, q.x, yr.y);
            yi.x = fmaf(mi[i].x, q.x, yi.x);
            yi.y = fmaf(mi[i].y, q.x, yi.y);
            yr.x = fmaf(-mi[i].x, q.y, yr.x);
            yr.y = fmaf(-mi[i].y, q.y, yr.y);
            yi.x = fmaf(mr[i].x, q.y, yi.x);
            yi.y = fmaf(mr[i].y, q.y, yi.y);
          }
          float4 y = Y[(sb + j) * T];
          y.x += yr.x;
          y.y += yr.y;
          y.z += yi.x;
          y.w += yi.y;
          Y[(sb + j) * T] = y;
        }
        par ^= 1;
      }
    }
    // ---- the band's sums over the CTA's groups into its slot ----
    __syncthreads();
    if (slot >= A.n_slots) {  // cannot happen for the host's slot count; fail loudly if it does
      if (tid == 0) atomicExch(A.status, FSG_EINVAL);
      break;
    }
    const float4* Y0 = reinterpret_cast<const float4*>(sm);
    float2* out = reinterpret_cast<float2*>(A.partial) + (size_t)slot * A.F * A.E;
    for (int i = tid; i < FB * T; i += MAXT) {
      const int f = f_b0 + i / T, t = i % T, e = (t >> 5) * 64 + (t & 31);
      if (f >= A.F) continue;
      float4 y = Y0[i];
      for (int q = 1; q < n_grp; ++q) {
        const float4 x = Y0[(size_t)q * FB * T + i];
        y = make_float4(y.x + x.x, y.y + x.y, y.z + x.z, y.w + x.w);
      }
      float2* o = out + (size_t)f * A.E + e;
      if (e < A.E) o[0] = cadd(o[0], make_float2(y.x, y.z));
      if (e + 32 < A.E) o[32] = cadd(o[32], make_float2(y.y, y.w));
    }
  }
}

template <int U, int DT, int MAXT>
static cudaError_t launch_lane_t(const SweepConfig& c, const BandArgs& A, cudaStream_t s) {
  cudaError_t e = cudaFuncSetAttribute(simus_lane_kernel<U, DT, MAXT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)c.smem);
  if (e != cudaSuccess) return e;
  simus_lane_kernel<U, DT, MAXT><<<A.grid, MAXT, c.smem, s>>>(A);
  return cudaGetLastError();
}

template <int DT>
static cudaError_t launch_lane_any(int U, const SweepConfig& c, const BandArgs& A, cudaStream_t s) {
  if constexpr (DT > 0) {
    if (c.nw != 3) switch (U) {
        case 1: return launch_lane_t<1, DT, 256>(c, A, s);
        case 2: return launch_lane_t<2, DT, 256>(c, A, s);
        case 3: return launch_lane_t<3, DT, 256>(c, A, s);
        case 4: return launch_lane_t<4, DT, 256>(c, A, s);
        default: return cudaErrorInvalidValue;
      }
  }
  switch (U) {
    case 1: return launch_lane_t<1, DT, 384>(c, A, s);
    case 2: return launch_lane_t<2, DT, 384>(c, A, s);
    case 3: return launch_lane_t<3, DT, 384>(c, A, s);
    case 4:
      if constexpr (DT == 0) return launch_lane_t<4, DT, 384>(c, A, s);  // 129 or more elements hold at most three
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace fsg
