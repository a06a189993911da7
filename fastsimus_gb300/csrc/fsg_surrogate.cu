// Transmit-field surrogate support: the exact transmit field at arbitrary (x, z, f, theta)
// samples, and the inputs and outputs of the surrogate network.
//
// Exact field (the training target and the check of the network's error).  For a plane wave
// of steering angle theta on a linear array, delays tau_e = x_e sin(theta) / c - min_e(...)
// (tx_delay.py:116-189); the complex transmit pressure at (x, z) and frequency f is
//     p = pulse(f) probe(f) sum_{e,u} apod_e exp(i 2 pi f tau_e) G(x, z, e, u, f)
// with G as in _init_exponentials (_pfield_math.py:202-247) and the 1/n_sub of pfield.py:159-170
// -- the quantity inside _pfield_strategies.py:48 before |.|^2, evaluated in closed form (no
// recurrence: every sample has its own f and theta).
//
// Network inputs and outputs.  The network (trained by fsg_mlp_train.cu, evaluated by
// fsg_mlp_tc.cu) predicts the complex amplitudes of a few analytic carriers whose phases carry
// the fast oscillation of the field: the ideal plane wave of the firing, the waves from the
// two ends of the aperture and the two first grating lobes of the element pitch.  fsg_surrogate_inputs normalises the samples and evaluates the
// carriers (FP64 phases) for training; fsg_surrogate_combine multiplies the predicted amplitudes back
// onto the carriers (double-float phases).

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "../../include/fsgb300.h"
#include "fsg_common.cuh"
#include "fsg_internal.h"

namespace fsg {

struct TxFieldArgs {
  const double* samples;  // [n][4]: x, z, f (Hz), theta (rad)
  int64_t n;
  float2* out;            // [n] complex transmit pressure
  const float4* src_pos;  // [E*U], z = 0
  float pitch;            // element x = (e - (E-1)/2) * pitch in float32 (utils/geometry.py:33-37)
  int E, U;
  double fc, c, cyc_fc;   // centre frequency, speed of sound, tx_n_wavelengths / fc (cycles of the pulse per Hz)
  double alpha_hz;        // attenuation, Np/m per Hz
  double inv_sigma, shape; // probe response sqrt(exp(-(|f - fc| inv_sigma)^shape))
  SweepConst C;           // geometry constants (dk/dalpha unused)
};

__device__ __forceinline__ float element_x(int e, int E, float pitch) {
  return __fmul_rn(__fsub_rn((float)e, (float)((E - 1) * 0.5)), pitch);
}

// a b for an FP32 number and a double-float one.
__device__ __forceinline__ dfl df_scale(float a, dfl b) {
  const float p = __fmul_rn(a, b.hi);
  return fast_two_sum(p, fmaf(a, b.lo, fmaf(a, b.hi, -p)));
}

__device__ __forceinline__ dfl df_mul(dfl a, dfl b) {
  const float p = __fmul_rn(a.hi, b.hi);
  float e = fmaf(a.hi, b.hi, -p);
  e = fmaf(a.hi, b.lo, e);
  e = fmaf(a.lo, b.hi, e);
  return fast_two_sum(p, e);
}

__device__ __forceinline__ dfl df_neg(dfl a) { return {-a.hi, -a.lo}; }

// sin(pi x) / (pi x) (numpy.sinc)
__device__ __forceinline__ double sinc_pi(double x) { return x == 0.0 ? 1.0 : sinpi(x) / (kPi * x); }

// One thread per sample, one loop over the sources.  The array is linear, so a source differs by its x
// alone and its angle's sine is dx / r.  What a training target must not lose stays as exact as FP64
// gives it: the pulse and the probe response are FP64, once per sample, and the delay's phase,
// x_e k sin(theta), is reduced to a fraction of a cycle in double-float and rounded to FP32 once.  The
// distance is double-float from one y = rsqrt(r^2): s = r^2 y plus the residual (r^2 - s^2) y / 2.
//
// What bounds it: issue, and the FP64 pipe (1/64 of the FP32 rate) beside it.  1,048,576 samples of the
// 64-element probe (two sources per element): 3.2 ms with the delay of every element in FP64, 678 us now.
// With the pulse, the probe response and the angles in double-float and FP32 it took 491 us and moved 0.99 of
// the results by an FP32 ulp, and the gradients of a training step on them by 1e-5 to 1e-4 of their norm.
template <int kBaffle>
__global__ void __launch_bounds__(128) txfield_kernel(const __grid_constant__ TxFieldArgs a) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.n) return;
  const double z = a.samples[4 * i + 1], f = a.samples[4 * i + 2];
  // pulse (times -i) * probe at f (spectrum.py:24-107)
  const double pulse_im = sinc_pi(a.cyc_fc * (f - a.fc)) - sinc_pi(a.cyc_fc * (f + a.fc));
  const double probe = exp(-0.5 * pow(fabs(f - a.fc) * a.inv_sigma, a.shape));
  const float scale = (float)(pulse_im * probe);
  const dfl xs = split_double(a.samples[4 * i]), zs = split_double(z);
  const dfl kf = split_double(2.0 * kPi * f / a.c);
  // cycles of the plane-wave delays, x_e k sin(theta) - min_e(...) (the minimum is at an end)
  const dfl ks = split_double(f / a.c * sin(a.samples[4 * i + 3]));
  const dfl first = df_scale(element_x(a.E - 1, a.E, a.pitch), ks.hi < 0.f ? df_neg(ks) : ks);
  const float first_r = __fsub_rn(first.hi, rintf(first.hi));
  const dfl z2 = df_sqr(zs);
  const float alpha = (float)(a.alpha_hz * f);
  const float half = (float)((a.E - 1) * 0.5);
  float2 acc = make_float2(0.f, 0.f);
  for (int e = 0; e < a.E; ++e) {
    float2 es = make_float2(0.f, 0.f);
    for (int u = 0; u < a.U; ++u) {
      const float2 sp = *reinterpret_cast<const float2*>(a.src_pos + e * a.U + u);
      const dfl dx = df_add(xs, dfl{-sp.x, -sp.y});
      const dfl r2 = df_add(df_sqr(dx), z2);
      // a point on the source (or no number) is seen under 90 degrees, from the clipped distance
      const bool apart = r2.hi > 0.f;
      const float y = rsqrt_normal(fmaxf(r2.hi, 1.17549435e-38f)), s = __fmul_rn(r2.hi, y);
      dfl r = fast_two_sum(s, __fmul_rn(0.5f * y, __fadd_rn(fmaf(-s, s, r2.hi), r2.lo)));
      const float sth = apart ? fminf(1.0f, fmaxf(-1.0f, __fdiv_rn(dx.hi, r.hi))) : 1.0f;
      const float cth = sqrtf((1.0f - sth) * (1.0f + sth));
      if (!apart || r.hi < a.C.min_dist.x || (r.hi == a.C.min_dist.x && r.lo < a.C.min_dist.y))
        r = dfl{a.C.min_dist.x, a.C.min_dist.y};
      float ob = kBaffle == 0 ? cth : (kBaffle == 1 ? 1.0f : __fdiv_rn(cth, cth + a.C.baffle_val));
      if (cth <= 0.0f) ob = 1e-16f;
      const float amp = ob * sinc_rad(a.C.dir_coef * sth) * rsqrt_normal(r.hi) * a.C.inv_nsub;
      es = cadd(es, anchor_value(r.hi, r.lo, amp, make_float2(kf.hi, kf.lo), alpha));
    }
    // the delay's phase in cycles: the whole ones drop out exactly
    const float xe = __fmul_rn(__fsub_rn((float)e, half), a.pitch);
    const float p = __fmul_rn(xe, ks.hi);
    const dfl lead = two_sum(__fsub_rn(p, rintf(p)), first_r);
    const float lead_lo = __fadd_rn(lead.lo, __fadd_rn(fmaf(xe, ks.lo, fmaf(xe, ks.hi, -p)), first.lo));
    float sd, cd;
    sincospif(2.0f * __fadd_rn(__fsub_rn(lead.hi, rintf(lead.hi)), lead_lo), &sd, &cd);
    acc = cfma(es, make_float2(cd, sd), acc);
  }
  const bool out_field = z < 0.0;
  a.out[i] = out_field ? make_float2(0.f, 0.f) : make_float2(-acc.y * scale, acc.x * scale);
}

// ------------------------------------------------------------------------------------------
// Surrogate carriers
// ------------------------------------------------------------------------------------------
constexpr int kMaxCarriers = 5;
constexpr int kAux = 12;  // floats per training row: carriers c_0..c_4, target y (complex)

struct Carriers {
  float2 c[kMaxCarriers], lo[kMaxCarriers];  // (re, im) and what FP32 leaves of them
};

// exp(2 pi i k path), k in cycles per metre, both double-float: the whole cycles drop out exactly, and
// the rest is taken to the nearest quarter cycle, |theta| <= pi / 4, for the Taylor series of sine and
// cosine, whose leading terms are kept double-float; the angle's FP32 remainder tl (below 1e-4) enters to
// first order.  Error about 1e-8.
__device__ __forceinline__ void df_cis_cycles(dfl k, dfl path, float2* c, float2* lo) {
  const float p = __fmul_rn(k.hi, path.hi);
  float e = fmaf(k.hi, path.hi, -p);
  e = fmaf(k.hi, path.lo, e);
  e = fmaf(k.lo, path.hi, e);
  const float x = __fsub_rn(p, rintf(p)), q = rintf(4.0f * x);
  const float t = fmaf(-0.25f, q, x);  // exact
  const float th = __fmul_rn(kTwoPiHi, t);
  const float tl = fmaf(kTwoPiHi, e, fmaf(kTwoPiLo, t, fmaf(kTwoPiHi, t, -th)));
  const float u = __fmul_rn(th, th), ul = fmaf(th, th, -u);
  float ps = fmaf(u, -1.0f / 39916800.0f, 1.0f / 362880.0f);
  ps = fmaf(u, ps, -1.0f / 5040.0f);
  ps = fmaf(u, ps, 1.0f / 120.0f);
  ps = fmaf(u, ps, -1.0f / 6.0f);
  float pc = fmaf(u, 1.0f / 479001600.0f, -1.0f / 3628800.0f);
  pc = fmaf(u, pc, 1.0f / 40320.0f);
  pc = fmaf(u, pc, -1.0f / 720.0f);
  pc = fmaf(u, pc, 1.0f / 24.0f);
  const float ds = __fmul_rn(__fmul_rn(th, u), ps), dc = fmaf(__fmul_rn(u, u), pc, -0.5f * ul), cu = -0.5f * u;
  const float s0 = __fadd_rn(th, ds), c0 = __fadd_rn(1.0f, __fadd_rn(cu, dc));
  const dfl sn = two_sum(th, fmaf(c0, tl, ds));
  dfl cs = fast_two_sum(1.0f, cu);
  cs = fast_two_sum(cs.hi, __fadd_rn(cs.lo, fmaf(-s0, tl, dc)));
  const int quarter = (int)q & 3;
  const bool swap = quarter & 1;
  const float sr = quarter == 1 || quarter == 2 ? -1.0f : 1.0f, si = quarter >= 2 ? -1.0f : 1.0f;
  *c = make_float2(sr * (swap ? sn.hi : cs.hi), si * (swap ? cs.hi : sn.hi));
  *lo = make_float2(sr * (swap ? sn.lo : cs.lo), si * (swap ? cs.lo : sn.lo));
}

// What a thread needs of the domain beside its fields: reciprocals, formed in FP64 on the host.
struct DomainArgs {
  FsgSurrogateDomain d;
  double mul[4], add[4];  // u_k = mul_k sample_k + add_k
  dfl inv_c, c_over_pitch;  // cycles per metre and Hz, lambda / pitch times Hz
  dfl x_end, x_edge;        // x of the last element and of its outer edge
};

// sqrt(a) for a > 0 and 0 else, from y = rsqrt(a): s = a y plus the residual (a - s^2) y / 2.
__device__ __forceinline__ dfl df_sqrt_fast(dfl a) {
  const float y = rsqrt_normal(fmaxf(a.hi, 1.17549435e-38f));
  const float s = __fmul_rn(a.hi, y);
  const dfl r = fast_two_sum(s, __fmul_rn(0.5f * y, __fadd_rn(fmaf(-s, s, a.hi), a.lo)));
  return a.hi > 0.f ? r : dfl{0.f, 0.f};
}

// sqrt((x - xe)^2 + z2)
__device__ __forceinline__ dfl df_distance(dfl x, dfl z2, dfl xe) {
  return df_sqrt_fast(df_add(df_sqr(df_add(x, df_neg(xe))), z2));
}

// a / b
__device__ __forceinline__ dfl df_div(dfl a, dfl b) {
  const float q = __fdividef(a.hi, b.hi);
  const float e = fmaf(-q, b.lo, __fadd_rn(fmaf(-q, b.hi, a.hi), a.lo));
  return fast_two_sum(q, __fdividef(e, b.hi));
}

// c_0: the plane wave exp(i k (x sin th + z cos th - xmin)); c_1, c_2: the waves from the two
// ends of the aperture, exp(i k (r_edge + x_edge sin th - xmin)); c_3, c_4: the grating lobes
// m = -1, +1 of the pitch, exp(i k (x sin th_m + z cos th_m - xmin)) with
// sin th_m = sin th + m lambda / pitch, zero where |sin th_m| >= 1 (evanescent).  Everything but sin and
// cos of theta is double-float: 1,048,576 samples of the combine kernel took 628 us with all of it in
// FP64, 225 us with the edges, lambda / pitch and sin th_m in FP64, 110 us now.
__device__ __forceinline__ Carriers surrogate_carriers(const DomainArgs& D, double x, double z, double f, double th) {
  const FsgSurrogateDomain& d = D.d;
  double st, ct;
  sincos(th, &st, &ct);
  const dfl xs = split_double(x), zs = split_double(z), fs = split_double(f), sd = split_double(st);
  const dfl kc = df_mul(fs, D.inv_c);  // cycles per metre
  const dfl lp = df_div(D.c_over_pitch, fs);
  const dfl z2 = df_sqr(zs);
  // -xmin: the delays' minimum is at an end of the array
  const dfl xe_s = df_mul(D.x_end, sd), first = xe_s.hi < 0.f ? df_neg(xe_s) : xe_s;
  const dfl edge_s = df_mul(D.x_edge, sd);
  dfl path[kMaxCarriers];
  bool on[kMaxCarriers];
  path[0] = df_add(df_mul(xs, sd), df_mul(zs, split_double(ct)));
  path[1] = df_add(df_distance(xs, z2, df_neg(D.x_edge)), df_neg(edge_s));
  path[2] = df_add(df_distance(xs, z2, D.x_edge), edge_s);
  on[0] = on[1] = on[2] = true;
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    const dfl sm = df_add(sd, m ? lp : df_neg(lp));
    const dfl c2 = df_add(dfl{1.f, 0.f}, df_neg(df_sqr(sm)));
    on[3 + m] = c2.hi > 0.f;
    path[3 + m] = df_add(df_mul(xs, sm), df_mul(zs, df_sqrt_fast(c2)));
  }
  Carriers out;
#pragma unroll
  for (int j = 0; j < kMaxCarriers; ++j) {
    df_cis_cycles(kc, df_add(path[j], first), &out.c[j], &out.lo[j]);
    if (!on[j] || j >= d.n_carriers) out.c[j] = out.lo[j] = make_float2(0.f, 0.f);
  }
  return out;
}

// The same in FP64, for training: the carriers are rounded to FP32 once, and their last bits count there
// (the backward pass rounds their products with the residual to BF16).
__device__ void training_carriers(const FsgSurrogateDomain& d, double x, double z, double f, double th, float* out) {
  const double st = sin(th), ct = cos(th);
  const double x0 = -0.5 * (d.n_elements - 1) * d.pitch, x1 = -x0;
  const double xmin = fmin(x0 * st, x1 * st);
  const double kc = f / d.speed_of_sound;  // cycles per metre
  const double lp = d.speed_of_sound / f / d.pitch;  // lambda / pitch
  double path[kMaxCarriers];
  bool on[kMaxCarriers];
  path[0] = x * st + z * ct - xmin;
  const double xl = x0 - 0.5 * d.pitch, xr = x1 + 0.5 * d.pitch;
  path[1] = sqrt((x - xl) * (x - xl) + z * z) + xl * st - xmin;
  path[2] = sqrt((x - xr) * (x - xr) + z * z) + xr * st - xmin;
  on[0] = on[1] = on[2] = true;
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    const double sm = st + (m ? lp : -lp);
    on[3 + m] = fabs(sm) < 1.0;
    path[3 + m] = x * sm + z * sqrt(fmax(0.0, 1.0 - sm * sm)) - xmin;
  }
#pragma unroll
  for (int j = 0; j < kMaxCarriers; ++j) {
    const double cyc = kc * path[j];
    double s, c;
    sincospi(2.0 * (cyc - rint(cyc)), &s, &c);
    const bool use = on[j] && j < d.n_carriers;
    out[2 * j] = use ? (float)c : 0.0f;
    out[2 * j + 1] = use ? (float)s : 0.0f;
  }
}

__global__ void surrogate_inputs_kernel(const __grid_constant__ DomainArgs D, const double* __restrict__ samples,
                                        int64_t n, const float2* __restrict__ field, double inv_scale,
                                        float4* __restrict__ u, float* __restrict__ aux) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double x = samples[4 * i], z = samples[4 * i + 1], f = samples[4 * i + 2], th = samples[4 * i + 3];
  u[i] = make_float4((float)fma(x, D.mul[0], D.add[0]), (float)fma(z, D.mul[1], D.add[1]),
                     (float)fma(f, D.mul[2], D.add[2]), (float)fma(th, D.mul[3], D.add[3]));
  if (!aux) return;
  float* o = aux + kAux * i;
  training_carriers(D.d, x, z, f, th, o);
  const float2 y = field ? field[i] : make_float2(0.f, 0.f);
  o[kAux - 2] = (float)(y.x * inv_scale);
  o[kAux - 1] = (float)(y.y * inv_scale);
}

__global__ void surrogate_combine_kernel(const __grid_constant__ DomainArgs D, const double* __restrict__ samples,
                                         int64_t n, const float* __restrict__ net, double scale,
                                         float2* __restrict__ out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const Carriers c =
      surrogate_carriers(D, samples[4 * i], samples[4 * i + 1], samples[4 * i + 2], samples[4 * i + 3]);
  const float* o = net + (size_t)i * 2 * D.d.n_carriers;
  // FP32 products with their errors carried along: the sum rounds once
  dfl re = {0.f, 0.f}, im = {0.f, 0.f};
  auto add = [](dfl& s, float a, float b, float b_lo) {
    const float p = __fmul_rn(a, b);
    const dfl t = two_sum(s.hi, p);
    s = dfl{t.hi, __fadd_rn(s.lo, __fadd_rn(t.lo, fmaf(a, b_lo, fmaf(a, b, -p))))};
  };
#pragma unroll
  for (int j = 0; j < kMaxCarriers; ++j) {
    if (j < D.d.n_carriers) {
      const float ar = o[2 * j], ai = o[2 * j + 1];
      add(re, ar, c.c[j].x, c.lo[j].x);
      add(re, -ai, c.c[j].y, c.lo[j].y);
      add(im, ar, c.c[j].y, c.lo[j].y);
      add(im, ai, c.c[j].x, c.lo[j].x);
    }
  }
  out[i] = make_float2((float)(((double)re.hi + (double)re.lo) * scale), (float)(((double)im.hi + (double)im.lo) * scale));
}

static DomainArgs domain_args(const FsgSurrogateDomain& d) {
  DomainArgs D;
  D.d = d;
  const double lo[4] = {d.x_lo, d.z_lo, d.f_lo, -d.max_angle}, hi[4] = {d.x_hi, d.z_hi, d.f_hi, d.max_angle};
  for (int k = 0; k < 4; ++k) {
    D.mul[k] = 2.0 / (hi[k] - lo[k]);
    D.add[k] = -(lo[k] + hi[k]) / (hi[k] - lo[k]);
  }
  D.inv_c = split_double(1.0 / d.speed_of_sound);
  D.c_over_pitch = split_double(d.speed_of_sound / d.pitch);
  D.x_end = split_double(0.5 * (d.n_elements - 1) * d.pitch);
  D.x_edge = split_double(0.5 * d.n_elements * d.pitch);
  return D;
}

}  // namespace fsg

using namespace fsg;

extern "C" int32_t fsg_txfield(const FsgProbe* probe, const FsgMedium* medium, double tx_n_wavelengths,
                               double bandwidth, const double* samples, int64_t n, void* out, void* workspace,
                               size_t workspace_bytes, void* stream_ptr) {
  if (!probe || !medium || !samples || !out) return set_error(FSG_EINVAL, "NULL argument");
  if (!isinf(probe->radius)) return set_error(FSG_EUNSUPPORTED, "transmit-field samples need a linear array");
  if (probe->n_elements < 1 || probe->n_sub < 1) return set_error(FSG_EINVAL, "bad probe");
  const int E = probe->n_elements, U = probe->n_sub;
  const size_t need = (size_t)E * U * 16 + (size_t)E * 8 + 1024;
  if (!workspace || workspace_bytes < need) return set_error(FSG_EWORKSPACE, "workspace too small (%zu < %zu)",
                                                             workspace_bytes, need);
  if (n <= 0) return FSG_OK;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream_ptr);
  unsigned char* ws = static_cast<unsigned char*>(workspace);
  SetupArgs sa;
  memset(&sa, 0, sizeof(sa));
  sa.E = E;
  sa.U = U;
  sa.pitch = probe->pitch;
  sa.width = probe->element_width;
  sa.radius = probe->radius;
  sa.c = medium->speed_of_sound;
  sa.seg = probe->element_width / U;
  sa.t.src_pos = reinterpret_cast<float4*>(ws);
  sa.t.rot_e = reinterpret_cast<float2*>(ws + (size_t)E * U * 16);
  setup_tables<<<(E * U + 127) / 128, 128, 0, s>>>(sa);
  int st = check_cuda(cudaGetLastError(), "setup_tables launch");
  if (st != FSG_OK) return st;
  TxFieldArgs a;
  a.samples = samples;
  a.n = n;
  a.out = static_cast<float2*>(out);
  a.src_pos = sa.t.src_pos;
  a.pitch = (float)probe->pitch;
  a.E = E;
  a.U = U;
  a.fc = probe->freq_center;
  a.c = medium->speed_of_sound;
  a.cyc_fc = tx_n_wavelengths / probe->freq_center;
  a.alpha_hz = medium->attenuation / 8.685889638065035 / 1e6 * 1e2;
  {
    // spectrum.py:53-107, in Hz
    const double sigma = bandwidth * probe->freq_center / 2.0;
    a.shape = log(126.0) / log(2.0 / bandwidth);
    a.inv_sigma = pow(log(2.0), 1.0 / a.shape) / sigma;
  }
  FsgFreqPlan dummy;
  memset(&dummy, 0, sizeof(dummy));
  dummy.seg_length = probe->element_width / U;
  a.C = make_sweep_const(probe, medium, &dummy, 0);
  const unsigned grid = (unsigned)((n + 127) / 128);
  if (a.C.baffle == 0) txfield_kernel<0><<<grid, 128, 0, s>>>(a);
  else if (a.C.baffle == 1) txfield_kernel<1><<<grid, 128, 0, s>>>(a);
  else txfield_kernel<2><<<grid, 128, 0, s>>>(a);
  return check_cuda(cudaGetLastError(), "txfield_kernel launch");
}

static int validate_domain(const FsgSurrogateDomain* d) {
  if (!d) return set_error(FSG_EINVAL, "NULL domain");
  if (d->n_carriers < 1 || d->n_carriers > kMaxCarriers) return set_error(FSG_EINVAL, "n_carriers must be 1..5");
  if (!(d->x_hi > d->x_lo) || !(d->z_hi > d->z_lo) || !(d->f_hi > d->f_lo) || !(d->max_angle > 0) ||
      !(d->pitch > 0) || !(d->speed_of_sound > 0) || d->n_elements < 1)
    return set_error(FSG_EINVAL, "bad surrogate domain");
  return FSG_OK;
}

extern "C" int32_t fsg_surrogate_inputs(const FsgSurrogateDomain* dom, const double* samples, int64_t n,
                                        const void* field, double inv_scale, float* u, float* aux, void* stream) {
  int st = validate_domain(dom);
  if (st != FSG_OK) return st;
  if (n < 0 || (n > 0 && (!samples || !u))) return set_error(FSG_EINVAL, "bad surrogate input arguments");
  if (reinterpret_cast<uintptr_t>(u) & 15) return set_error(FSG_EINVAL, "u must start on a 16-byte boundary");
  if (n == 0) return FSG_OK;
  surrogate_inputs_kernel<<<(unsigned)((n + 255) / 256), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      domain_args(*dom), samples, n, static_cast<const float2*>(field), inv_scale, reinterpret_cast<float4*>(u), aux);
  return check_cuda(cudaGetLastError(), "surrogate_inputs_kernel launch");
}

extern "C" int32_t fsg_surrogate_combine(const FsgSurrogateDomain* dom, const double* samples, int64_t n,
                                         const float* net, double scale, void* out, void* stream) {
  int st = validate_domain(dom);
  if (st != FSG_OK) return st;
  if (n < 0 || (n > 0 && (!samples || !net || !out))) return set_error(FSG_EINVAL, "bad surrogate combine arguments");
  if (n == 0) return FSG_OK;
  surrogate_combine_kernel<<<(unsigned)((n + 255) / 256), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      domain_args(*dom), samples, n, net, scale, static_cast<float2*>(out));
  return check_cuda(cudaGetLastError(), "surrogate_combine_kernel launch");
}
