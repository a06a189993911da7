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
// carriers (double-float phases) for training; fsg_surrogate_combine multiplies the predicted
// amplitudes back onto the carriers.

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
  dfl fc, inv_c, cyc_fc;  // centre frequency, 1 / c, tx_n_wavelengths / fc (cycles of the pulse per Hz)
  float alpha_hz;         // attenuation, Np/m per Hz
  float inv_sigma, shape; // probe response sqrt(exp(-(|f - fc| inv_sigma)^shape))
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

// exp(2 pi i k path), k in cycles per metre, both double-float: the whole cycles drop out exactly.
__device__ __forceinline__ float2 df_cis_cycles(dfl k, dfl path) {
  const float p = __fmul_rn(k.hi, path.hi);
  float e = fmaf(k.hi, path.hi, -p);
  e = fmaf(k.hi, path.lo, e);
  e = fmaf(k.lo, path.hi, e);
  const float x = __fadd_rn(__fsub_rn(p, rintf(p)), e);
  float s, c;
  sincospif(2.0f * x, &s, &c);
  return make_float2(c, s);
}

// sin(pi x) / (pi x), the rounding of x to FP32 corrected to first order.
__device__ __forceinline__ float sinc_pi(dfl x) {
  if (x.hi == 0.0f) return 1.0f;
  const dfl px = df_mul(split_double(kPi), x);
  float s, c;
  sincospif(x.hi, &s, &c);
  return __fdiv_rn(fmaf((float)kPi * x.lo, c, s), px.hi);
}

// One thread per sample, one loop over the sources.  The array is linear, so a source differs by its x
// alone and sin and cos of the angle are dx / r and z / r.  Paths and phases are double-float: the
// distance is s = r^2 y, y = rsqrt(r^2), plus the residual (r^2 - s^2) y / 2, the delay's phase
// x_e k sin(theta) is reduced to a fraction of a cycle per element and the distance's per source (their
// sum is exact: both are multiples of 2^-20 or so below one), and the amplitudes are FP32 from y after
// one Newton step.  FP64 is left to sin(theta) and the splits of the sample.
//
// What bounds it: issue, about 90 instructions per source (a third of them sincospi).  1,048,576 samples
// of the 64-element probe (two sources per element): 3.2 ms with delays, phases and spectra in FP64,
// which the part runs at 1/64 of the FP32 rate; 883 us with the sweeps' double-float geometry per
// source (two correctly rounded divisions, two square roots); 491 us now.
template <int kBaffle>
__global__ void __launch_bounds__(128) txfield_kernel(const __grid_constant__ TxFieldArgs a) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.n) return;
  const dfl xs = split_double(a.samples[4 * i]), zs = split_double(a.samples[4 * i + 1]);
  const dfl fs = split_double(a.samples[4 * i + 2]);
  const dfl st = split_double(sin(a.samples[4 * i + 3]));
  // pulse (times -i) * probe at f (spectrum.py:24-107)
  const dfl df = df_add(fs, df_neg(a.fc));
  const float pulse_im = sinc_pi(df_mul(a.cyc_fc, df)) - sinc_pi(df_mul(a.cyc_fc, df_add(fs, a.fc)));
  const float probe = expf(-0.5f * powf(fabsf(df.hi) * a.inv_sigma, a.shape));
  const dfl kc = df_mul(fs, a.inv_c);  // cycles per metre
  // cycles of the plane-wave delays, x_e k sin(theta) - min_e(...) (the minimum is at an end)
  const dfl ks = df_mul(kc, st);
  const dfl first = df_scale(element_x(a.E - 1, a.E, a.pitch), ks.hi < 0.f ? df_neg(ks) : ks);
  const float first_r = __fsub_rn(first.hi, rintf(first.hi));
  const dfl z2 = df_sqr(zs);
  const float alpha = a.alpha_hz * fs.hi;
  const float half = (float)((a.E - 1) * 0.5);
  float2 acc = make_float2(0.f, 0.f);
  for (int e = 0; e < a.E; ++e) {
    const float xe = __fmul_rn(__fsub_rn((float)e, half), a.pitch);
    const float p = __fmul_rn(xe, ks.hi);
    const float lead_lo = fmaf(xe, ks.lo, fmaf(xe, ks.hi, -p)) + first.lo;
    const float lead_r = __fadd_rn(__fsub_rn(p, rintf(p)), first_r);
    for (int u = 0; u < a.U; ++u) {
      const float2 sp = *reinterpret_cast<const float2*>(a.src_pos + e * a.U + u);
      dfl dx = two_sum(xs.hi, -sp.x);
      dx.lo = __fadd_rn(dx.lo, __fsub_rn(xs.lo, sp.y));
      const float d2 = __fmul_rn(dx.hi, dx.hi);
      const float d2_lo = fmaf(2.0f * dx.hi, dx.lo, fmaf(dx.hi, dx.hi, -d2));
      dfl r2 = two_sum(d2, z2.hi);
      r2.lo = __fadd_rn(r2.lo, __fadd_rn(d2_lo, z2.lo));
      const bool apart = r2.hi > 0.f && r2.hi <= 3.402823466e38f;
      float y = rsqrt_normal(fmaxf(r2.hi, 1.17549435e-38f));
      float s = __fmul_rn(r2.hi, y);
      float lo = __fmul_rn(0.5f * y, __fadd_rn(fmaf(-s, s, r2.hi), r2.lo));
      y = fmaf(0.5f * y, fmaf(-s, y, 1.0f), y);
      // a point on the source (or no number) is seen under 90 degrees
      const float sth = apart ? dx.hi * y : 1.0f, cth = apart ? zs.hi * y : 0.0f;
      if (!(s > a.C.min_dist.x || (s == a.C.min_dist.x && lo >= a.C.min_dist.y))) {
        s = a.C.min_dist.x;
        lo = a.C.min_dist.y;
      }
      const float r = __fadd_rn(s, lo);
      float m = kBaffle == 0 ? cth : (kBaffle == 1 ? 1.0f : __fdiv_rn(cth, cth + a.C.baffle_val));
      if (cth <= 0.0f) m = 1e-16f;
      m *= sinc_rad(a.C.dir_coef * sth) * rsqrt_normal(r);
      if (alpha != 0.f) m *= expf(-alpha * r);
      const float q = __fmul_rn(kc.hi, s);
      const float q_lo = fmaf(kc.lo, s, fmaf(kc.hi, lo, fmaf(kc.hi, s, -q)));
      float c = __fadd_rn(__fsub_rn(q, rintf(q)), lead_r);
      c = __fadd_rn(__fsub_rn(c, rintf(c)), __fadd_rn(q_lo, lead_lo));
      float sn, cs;
      sincospif(2.0f * c, &sn, &cs);
      acc.x = fmaf(m, cs, acc.x);
      acc.y = fmaf(m, sn, acc.y);
    }
  }
  // times pulse (= i * pulse_im) * probe, mean over the sub-elements
  const float s = pulse_im * probe * a.C.inv_nsub;
  const bool out_field = a.samples[4 * i + 1] < 0.0;
  a.out[i] = out_field ? make_float2(0.f, 0.f) : make_float2(-acc.y * s, acc.x * s);
}

// ------------------------------------------------------------------------------------------
// Surrogate carriers
// ------------------------------------------------------------------------------------------
constexpr int kMaxCarriers = 5;
constexpr int kAux = 12;  // floats per training row: carriers c_0..c_4, target y (complex)

struct Carriers {
  float2 c[kMaxCarriers];
};

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
// FP64, 225 us with the edges, lambda / pitch and sin th_m in FP64, 108 us now.
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
  for (int j = 0; j < kMaxCarriers; ++j)
    out.c[j] = (on[j] && j < d.n_carriers) ? df_cis_cycles(kc, df_add(path[j], first)) : make_float2(0.f, 0.f);
  return out;
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
  const Carriers c = surrogate_carriers(D, x, z, f, th);
  float* o = aux + kAux * i;
#pragma unroll
  for (int j = 0; j < kMaxCarriers; ++j) {
    o[2 * j] = c.c[j].x;
    o[2 * j + 1] = c.c[j].y;
  }
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
  auto add = [](dfl& s, float a, float b) {
    const float p = __fmul_rn(a, b);
    const dfl t = two_sum(s.hi, p);
    s = dfl{t.hi, __fadd_rn(s.lo, __fadd_rn(t.lo, fmaf(a, b, -p)))};
  };
#pragma unroll
  for (int j = 0; j < kMaxCarriers; ++j) {
    if (j < D.d.n_carriers) {
      const float ar = o[2 * j], ai = o[2 * j + 1];
      add(re, ar, c.c[j].x);
      add(re, -ai, c.c[j].y);
      add(im, ar, c.c[j].y);
      add(im, ai, c.c[j].x);
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
  a.fc = split_double(probe->freq_center);
  a.inv_c = split_double(1.0 / medium->speed_of_sound);
  a.cyc_fc = split_double(tx_n_wavelengths / probe->freq_center);
  a.alpha_hz = (float)(medium->attenuation / 8.685889638065035 / 1e6 * 1e2);
  {
    // spectrum.py:53-107, in Hz
    const double shape = log(126.0) / log(2.0 / bandwidth);
    const double sigma = bandwidth * probe->freq_center / 2.0 / pow(log(2.0), 1.0 / shape);
    a.shape = (float)shape;
    a.inv_sigma = (float)(1.0 / sigma);
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
