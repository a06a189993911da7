// simus_lane_kernel instantiations without full-frequency directivity, and its geometry pre-pass.
#include "fsg_sweep_lane.cuh"

namespace fsg {

cudaError_t launch_simus_lane(int U, const SweepConfig& c, const BandArgs& A, cudaStream_t s) {
  return A.C.ffd ? launch_simus_lane_ffd(U, c, A, s) : launch_lane_any<0>(U, c, A, s);
}

// Geometry of a chunk's tiles, once per (scatterer, source) for all frequency bands, in
// lane_block order: a block's threads take consecutive (group, pair, thread) slots of one tile, two
// elements each, so every store of a warp is contiguous.  gridDim.y CTAs share a tile's slots.
__global__ void __launch_bounds__(kThreads) lane_geometry_kernel(const BandArgs A, int64_t chunk_tiles) {
  __shared__ float4 xz[kThreads];  // st <= 48 points of the tile
  const int T = 32 * A.nw, PPT = lane_points(A.U), NP = A.U * PPT;
  const int n_grp = A.st / PPT, slots = n_grp * NP * T;
  for (int64_t tile = blockIdx.x; tile < chunk_tiles; tile += gridDim.x) {
    const LaneBlock B = lane_block(A.geo + tile * A.geo_bytes, slots, A.C.ffd != 0);
    __syncthreads();
    if (threadIdx.x < A.st) {
      const int64_t s = A.chunk_s0 + tile * A.st + threadIdx.x;
      const bool on = s < A.n_pts;
      const int64_t si = on ? s : A.chunk_s0 + tile * A.st;
      const double x = A.pts[2 * si], z = A.pts[2 * si + 1];
      bool out = !on || z < 0.0;
      if (A.convex) out = out || (x * x + (z + A.apex) * (z + A.apex) <= A.radius2);
      if (blockIdx.y == 0) B.w[threadIdx.x] = out ? 0.f : (float)A.rc[si];
      const dfl hx = split_double(x), hz = split_double(z);
      xz[threadIdx.x] = make_float4(hx.hi, hx.lo, hz.hi, hz.lo);
    }
    __syncthreads();
    for (int i = blockIdx.y * blockDim.x + threadIdx.x; i < slots; i += gridDim.y * blockDim.x) {
      const int t = i % T, gp = i / T, p = gp % NP, g = gp / NP;
      const int u = p / PPT, pt = g * PPT + p % PPT, e = (t >> 5) * 64 + (t & 31);
      const float4 c = xz[pt];
      SrcGeo q[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int eh = e + 32 * h, ec = min(eh, A.E - 1);
        q[h] = source_geometry(dfl{c.x, c.y}, dfl{c.z, c.w}, A.t.src_pos[ec * A.U + u], A.t.rot_e[ec], A.C);
        if (eh >= A.E) {  // a padded element: no contribution
          q[h].amp = 0.f;
          q[h].step = make_float2(0.f, 0.f);
        }
      }
      B.a[i] = make_float4(q[0].r_hi, q[1].r_hi, q[0].r_lo, q[1].r_lo);
      B.b[i] = make_float4(q[0].amp, q[1].amp, q[0].step.x, q[1].step.x);
      B.c[i] = make_float2(q[0].step.y, q[1].step.y);
      if (A.C.ffd) B.d[i] = sqr2(make_float2(A.C.half_seg * q[0].sth, A.C.half_seg * q[1].sth));
    }
  }
}

}  // namespace fsg
