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
  const float4* src_pos;  // [E*U]
  const float2* rot_e;    // [E]
  float pitch;            // element x = (e - (E-1)/2) * pitch in float32 (utils/geometry.py:33-37)
  int E, U;
  double fc, inv_c, cyc_fc;  // centre frequency, 1 / c, tx_n_wavelengths / fc (cycles of the pulse per Hz)
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
__device__ __forceinline__ float sinc_pi(double x) {
  if (x == 0.0) return 1.0f;
  const float hi = (float)x, lo = (float)kPi * (float)(x - (double)hi);
  float s, c;
  sincospif(hi, &s, &c);
  return __fdiv_rn(fmaf(lo, c, s), (float)(kPi * x));
}

// One thread per sample.  The path of a source, r + x_e sin(theta) - min_e(...), and its phase are
// double-float, the amplitudes FP32; FP64 is left to sin(theta) and a few products per sample (the
// part runs it at 1/64 of the FP32 rate: with the delays, phases and spectra in FP64 the kernel took
// 3.2 ms for 1,048,576 samples of the 64-element probe, all of it FP64).
__global__ void __launch_bounds__(128) txfield_kernel(const __grid_constant__ TxFieldArgs a) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.n) return;
  const double x = a.samples[4 * i], z = a.samples[4 * i + 1], f = a.samples[4 * i + 2], th = a.samples[4 * i + 3];
  // pulse (times -i) * probe at f (spectrum.py:24-107)
  const float pulse_im = sinc_pi(a.cyc_fc * (f - a.fc)) - sinc_pi(a.cyc_fc * (f + a.fc));
  const float probe = expf(-0.5f * powf((float)fabs(f - a.fc) * a.inv_sigma, a.shape));
  // plane-wave delays: c tau_e = x_e sin(theta) - min_e
  const double st = sin(th);
  const float x_end = element_x(a.E - 1, a.E, a.pitch), x_0 = element_x(0, a.E, a.pitch);
  const dfl std_ = split_double(st), first = split_double(-fmin((double)x_0 * st, (double)x_end * st));
  const dfl xs = split_double(x), zs = split_double(z), kc = split_double(f * a.inv_c);
  const float alpha = a.alpha_hz * (float)f;
  float2 acc = make_float2(0.f, 0.f);
  for (int e = 0; e < a.E; ++e) {
    const dfl lead = df_add(df_scale(element_x(e, a.E, a.pitch), std_), first);
    const float2 rot = a.rot_e[e];
    for (int u = 0; u < a.U; ++u) {
      const SrcGeo geo = source_geometry(xs, zs, a.src_pos[e * a.U + u], rot, a.C);
      const float2 cis = df_cis_cycles(kc, df_add(dfl{geo.r_hi, geo.r_lo}, lead));
      const float m = alpha != 0.f ? geo.amp * expf(-alpha * geo.r_hi) : geo.amp;
      acc.x = fmaf(m, cis.x, acc.x);
      acc.y = fmaf(m, cis.y, acc.y);
    }
  }
  // times pulse (= i * pulse_im) * probe
  const float s = pulse_im * probe;
  const bool out_field = z < 0.0;
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
  double inv_c, c_over_pitch;
};

// sqrt((x - xe)^2 + z^2) in double-float.
__device__ __forceinline__ dfl df_distance(dfl x, dfl z, double xe) {
  const dfl dx = df_add(x, split_double(-xe));
  return df_sqrt(df_add(df_sqr(dx), df_sqr(z)));
}

__device__ __forceinline__ dfl df_mul(dfl a, dfl b) {
  const float p = __fmul_rn(a.hi, b.hi);
  float e = fmaf(a.hi, b.hi, -p);
  e = fmaf(a.hi, b.lo, e);
  e = fmaf(a.lo, b.hi, e);
  return fast_two_sum(p, e);
}

// c_0: the plane wave exp(i k (x sin th + z cos th - xmin)); c_1, c_2: the waves from the two
// ends of the aperture, exp(i k (r_edge + x_edge sin th - xmin)); c_3, c_4: the grating lobes
// m = -1, +1 of the pitch, exp(i k (x sin th_m + z cos th_m - xmin)) with
// sin th_m = sin th + m lambda / pitch, zero where |sin th_m| >= 1 (evanescent).  Paths and phases are
// double-float; FP64 is left to sin and cos of theta and lambda / pitch (1,048,576 samples of the
// combine kernel: 628 us with all of it in FP64).
__device__ __forceinline__ Carriers surrogate_carriers(const DomainArgs& D, double x, double z, double f, double th) {
  const FsgSurrogateDomain& d = D.d;
  double st, ct;
  sincos(th, &st, &ct);
  const double x0 = -0.5 * (d.n_elements - 1) * d.pitch, x1 = -x0;
  const dfl first = split_double(-fmin(x0 * st, x1 * st));
  const dfl kc = split_double(f * D.inv_c);  // cycles per metre
  const double lp = D.c_over_pitch / f;      // lambda / pitch
  const dfl xs = split_double(x), zs = split_double(z), sd = split_double(st);
  dfl path[kMaxCarriers];
  bool on[kMaxCarriers];
  path[0] = df_add(df_mul(xs, sd), df_mul(zs, split_double(ct)));
  const double xl = x0 - 0.5 * d.pitch, xr = x1 + 0.5 * d.pitch;
  path[1] = df_add(df_distance(xs, zs, xl), df_mul(split_double(xl), sd));
  path[2] = df_add(df_distance(xs, zs, xr), df_mul(split_double(xr), sd));
  on[0] = on[1] = on[2] = true;
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    const double sm = st + (m ? lp : -lp);
    on[3 + m] = fabs(sm) < 1.0;
    const dfl smd = split_double(sm), cm = df_sqrt(split_double(fmax(0.0, 1.0 - sm * sm)));
    path[3 + m] = df_add(df_mul(xs, smd), df_mul(zs, cm));
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
  D.inv_c = 1.0 / d.speed_of_sound;
  D.c_over_pitch = d.speed_of_sound / d.pitch;
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
  a.rot_e = sa.t.rot_e;
  a.pitch = (float)probe->pitch;
  a.E = E;
  a.U = U;
  a.fc = probe->freq_center;
  a.inv_c = 1.0 / medium->speed_of_sound;
  a.cyc_fc = tx_n_wavelengths / probe->freq_center;
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
  txfield_kernel<<<(unsigned)((n + 127) / 128), 128, 0, s>>>(a);
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
