// pp_device.cuh -- device-side step functions of the photon-transport kernel.
//
// Each function states the PhotonPropagation.jl v0.9.3 function it stands in
// for (paths inside that project).  Every function comes in two precisions of
// the transcendental functions: kPrecise = true uses the IEEE-accurate CUDA
// math library (used by the replay tests), kPrecise = false uses the SFU
// approximations (lg2/ex2/sin/cos/rcp/sqrt .approx), whose absolute error is
// below 1e-6 on the argument ranges used here.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "pp_internal.h"

namespace ppdev {

constexpr uint32_t kPhiloxM0 = 0xD2511F53u;
constexpr uint32_t kPhiloxM1 = 0xCD9E8D57u;
constexpr uint32_t kPhiloxW0 = 0x9E3779B9u;
constexpr uint32_t kPhiloxW1 = 0xBB67AE85u;
constexpr uint32_t kExtraCall = 0x80000000u;  // first call of the emitter stream
constexpr int kGammaMaxTries = 64;
constexpr float kTwoPi = 6.2831855f;           // Float32(2*pi)
constexpr float kPi = 3.14159274f;
constexpr float kCVac = 0.299792458f;          // m/ns

// ---- Philox4x32-10 (Salmon et al., SC'11) --------------------------------
// Counter = (photon lo, photon hi, call, source), key = seed (lo, hi).
__device__ __forceinline__ uint4 philox(uint4 c, uint32_t k0, uint32_t k1) {
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    if (r > 0) {
      k0 += kPhiloxW0;
      k1 += kPhiloxW1;
    }
    const unsigned long long p0 = (unsigned long long)kPhiloxM0 * c.x;
    const unsigned long long p1 = (unsigned long long)kPhiloxM1 * c.z;
    c = make_uint4((uint32_t)(p1 >> 32) ^ c.y ^ k0, (uint32_t)p1, (uint32_t)(p0 >> 32) ^ c.w ^ k1,
                   (uint32_t)p0);
  }
  return c;
}

// The same with the ten rounds' keys given (key + r * (W0, W1), r = 0..9).
__device__ __forceinline__ uint4 philox(uint4 c, const uint32_t* __restrict__ rk) {
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const unsigned long long p0 = (unsigned long long)kPhiloxM0 * c.x;
    const unsigned long long p1 = (unsigned long long)kPhiloxM1 * c.z;
    c = make_uint4((uint32_t)(p1 >> 32) ^ c.y ^ rk[2 * r], (uint32_t)p1,
                   (uint32_t)(p0 >> 32) ^ c.w ^ rk[2 * r + 1], (uint32_t)p0);
  }
  return c;
}

// The steps of one photon share most of rounds 1 and 2: with counter (plo,
// phi, k, s), the products with plo and s-mixed words do not depend on the
// step k, and those with k and phi not on the photon's low word.  A photon
// keeps three words, a step computes three for the whole warp (phi is equal
// in a group of photons), and each (photon, step) starts at round 3.
struct PhiloxPhoton {
  uint32_t a, b, c;
};
struct PhiloxStep {
  uint32_t lo1, hi, lo;
};
__device__ __forceinline__ PhiloxPhoton philox_photon(uint32_t plo, uint32_t s,
                                                      const uint32_t* __restrict__ rk) {
  const unsigned long long p0 = (unsigned long long)kPhiloxM0 * plo;
  const unsigned long long p1 =
      (unsigned long long)kPhiloxM1 * ((uint32_t)(p0 >> 32) ^ s ^ rk[1]);
  return {(uint32_t)(p1 >> 32) ^ rk[2], (uint32_t)p1, (uint32_t)p0 ^ rk[3]};
}
__device__ __forceinline__ PhiloxStep philox_step(uint32_t k, uint32_t phi,
                                                  const uint32_t* __restrict__ rk) {
  const unsigned long long p1 = (unsigned long long)kPhiloxM1 * k;
  const unsigned long long p0 =
      (unsigned long long)kPhiloxM0 * ((uint32_t)(p1 >> 32) ^ phi ^ rk[0]);
  return {(uint32_t)p1, (uint32_t)(p0 >> 32), (uint32_t)p0};
}
// philox(make_uint4(plo, phi, k, s), rk)
__device__ __forceinline__ uint4 philox_words(const PhiloxPhoton& p, const PhiloxStep& t,
                                              const uint32_t* __restrict__ rk) {
  uint4 c = make_uint4(p.a ^ t.lo1, p.b, t.hi ^ p.c, t.lo);
#pragma unroll
  for (int r = 2; r < 10; ++r) {
    const unsigned long long p0 = (unsigned long long)kPhiloxM0 * c.x;
    const unsigned long long p1 = (unsigned long long)kPhiloxM1 * c.z;
    c = make_uint4((uint32_t)(p1 >> 32) ^ c.y ^ rk[2 * r], (uint32_t)p1,
                   (uint32_t)(p0 >> 32) ^ c.w ^ rk[2 * r + 1], (uint32_t)p0);
  }
  return c;
}

// ---- two photons at a time ---------------------------------------------------
// A lane of the propagation kernel carries two photons, and their FP32 sums
// and products go through the packed f32x2 instructions: each half rounds as
// the scalar instruction does, at the same FP32 rate, in half the issue slots
// (measured on the GB300: 16 FFMA + 16 LOP3 take 37.4 issue cycles, 8 packed
// FFMA + 16 LOP3 28.8).
__device__ __forceinline__ unsigned long long pack2(float2 v) {
  unsigned long long d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(v.x), "f"(v.y));
  return d;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
  float2 d;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(v));
  return d;
}
__device__ __forceinline__ float2 dup2(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(pack2(a)), "l"(pack2(b)), "l"(pack2(c)));
  return unpack2(d);
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  unsigned long long d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(pack2(a)), "l"(pack2(b)));
  return unpack2(d);
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  unsigned long long d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(pack2(a)), "l"(pack2(b)));
  return unpack2(d);
}
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
  unsigned long long d;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(pack2(a)), "l"(pack2(b)));
  return unpack2(d);
}
struct Vec2 {  // the two photons' vectors
  float2 x, y, z;
};
__device__ __forceinline__ float3 first(const Vec2& v) { return make_float3(v.x.x, v.y.x, v.z.x); }
__device__ __forceinline__ float3 second(const Vec2& v) { return make_float3(v.x.y, v.y.y, v.z.y); }
__device__ __forceinline__ Vec2 both(float3 a, float3 b) {
  return {make_float2(a.x, b.x), make_float2(a.y, b.y), make_float2(a.z, b.z)};
}

// 24-bit uniform in (0, 1] (exact: integer <= 2^24 times 2^-24).
__device__ __forceinline__ float u01(uint32_t x) {
  return __uint2float_rn((x >> 8) + 1u) * 5.9604644775390625e-8f;
}

// ---- precision-selected primitives -----------------------------------------
__device__ __forceinline__ float approx_sqrt(float x) {
  float y;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float approx_rcp(float x) {
  float y;
  asm("rcp.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// The step loop's forms flush subnormals: without .ftz each call carries a
// compare and two scalings for subnormal operands, and here every operand is
// zero or normal (each use says why), so both forms give the same bits.
// (With the integer forms in scatter_cos_fast: 18.40 -> 17.13 ms per 1e8
// photons in the 400-module detector at the default tuning, same hits.)
__device__ __forceinline__ float ftz_sqrt(float x) {
  float y;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float ftz_rcp(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float ftz_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// (arguments: uniforms >= 2^-24 and products of such, never subnormal)
__device__ __forceinline__ float ftz_lg2(float x) {
  float y;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float approx_ex2(float x) {
  float y;
  asm("ex2.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

template <bool P>
__device__ __forceinline__ float f_log(float x) {
  if (P) return logf(x);
  return ftz_lg2(x) * 0.693147182f;  // ln(x) = log2(x) * ln(2)
}
template <bool P>
__device__ __forceinline__ float f_sqrt(float x) {
  return P ? __fsqrt_rn(x) : approx_sqrt(x);
}
template <bool P>
__device__ __forceinline__ float f_rcp(float x) {
  return P ? __frcp_rn(x) : approx_rcp(x);
}
template <bool P>
__device__ __forceinline__ float f_div(float a, float b) {
  return P ? __fdiv_rn(a, b) : a * approx_rcp(b);
}
// Cube root of a positive number: 2^(log2(x)/3).
template <bool P>
__device__ __forceinline__ float f_cbrt_pos(float x) {
  return P ? cbrtf(x) : approx_ex2(ftz_lg2(x) * 0.333333343f);
}
template <bool P>
__device__ __forceinline__ float f_exp(float x) {
  return P ? expf(x) : approx_ex2(x * 1.44269502f);
}
// sin / cos of 2*pi*u for u in (0, 1].  The fast form evaluates the SFU at
// 2*pi*u - pi, inside [-pi, pi] where its error is smallest, and flips signs.
template <bool P>
__device__ __forceinline__ void f_sincos_2pi(float u, float* s, float* c) {
  if (P) {
    sincosf(kTwoPi * u, s, c);
  } else {
    float ss, cc;
    __sincosf(fmaf(kTwoPi, u, -kPi), &ss, &cc);
    *s = -ss;
    *c = -cc;
  }
}
template <bool P>
__device__ __forceinline__ void f_sincos(float x, float* s, float* c) {
  if (P) sincosf(x, s, c); else __sincosf(x, s, c);
}

// a*b + c: fused in the fast variant, two roundings in the replay variant
// (which is compiled without contraction, like the oracle).
template <bool P>
__device__ __forceinline__ float madd(float a, float b, float c) {
  return P ? a * b + c : fmaf(a, b, c);
}

// uniform(minval, maxval) of src/photon_prop_cuda.jl:48-51 on a given uniform.
__device__ __forceinline__ float uniform_ab(float a, float b, float u) { return a + u * (b - a); }

// ---- geometry ----------------------------------------------------------------
// Rotation taking e_z onto the unit vector a, applied to b (rot_from_ez_fast,
// PhysicsTools; called at src/photon_prop_cuda.jl:92-95, :296).  Written in
// the Rodrigues form whose only division is well conditioned in each
// hemisphere of a; the expression order matches the oracle's.
template <bool P>
__device__ __forceinline__ float3 rot_from_ez(float3 a, float3 b) {
  const float s2 = P ? a.x * a.x + a.y * a.y : fmaf(a.y, a.y, a.x * a.x);
  // on the axis (the fast form counts a subnormal s2 as on it)
  if (P ? s2 == 0.0f : s2 < 1.17549435e-38f) {
    const float sg = a.z >= 0.0f ? 1.0f : -1.0f;
    return make_float3(sg * b.x, sg * b.y, sg * b.z);
  }
  // 1 / (1 + a.z), written as (1 - a.z) / s2 in the lower hemisphere where
  // 1 + a.z cancels; the fast form selects the operands of one reciprocal
  float f;
  if (P) {
    f = a.z >= 0.0f ? f_rcp<P>(1.0f + a.z) : f_div<P>(1.0f - a.z, s2);
  } else {
    const bool up = a.z >= 0.0f;
    f = (up ? 1.0f : 1.0f - a.z) * ftz_rcp(up ? 1.0f + a.z : s2);
  }
  if (P) {
    const float k = (a.x * b.y - a.y * b.x) * f;
    return make_float3(b.x * a.z + a.x * b.z - a.y * k, b.y * a.z + a.y * b.z + a.x * k,
                       b.z * a.z - (a.x * b.x + a.y * b.y));
  }
  // the same with every fused multiply-add written out (the fast variant is
  // compiled without automatic contraction, so its rounding is fixed here)
  const float k = fmaf(a.x, b.y, -(a.y * b.x)) * f;
  return make_float3(fmaf(a.x, b.z, fmaf(b.x, a.z, -(a.y * k))),
                     fmaf(a.y, b.z, fmaf(b.y, a.z, a.x * k)),
                     fmaf(b.z, a.z, -fmaf(a.x, b.x, a.y * b.y)));
}

// sph_to_cart(theta, phi) with phi = 2*pi*u_phi.
template <bool P>
__device__ __forceinline__ float3 sph_to_cart(float theta, float u_phi) {
  if (P) {
    const float phi = uniform_ab(0.0f, kTwoPi, u_phi);
    const float st = sinf(theta), ct = cosf(theta);
    return make_float3(st * cosf(phi), st * sinf(phi), ct);
  }
  float st, ct, sp, cp;
  __sincosf(theta, &st, &ct);
  f_sincos_2pi<false>(u_phi, &sp, &cp);
  return make_float3(st * cp, st * sp, ct);
}

// Direction with polar cosine ct and azimuth 2*pi*u_phi.  The replay variant
// goes through theta = acos(ct) as the reference does
// (initialize_direction_isotropic, src/photon_prop_cuda.jl:73-77); the fast
// one uses sin(theta) = sqrt(1 - ct^2).
template <bool P>
__device__ __forceinline__ float3 dir_from_cos(float ct, float u_phi) {
  if (P) return sph_to_cart<true>(acosf(ct), u_phi);
  const float st = approx_sqrt(fmaxf(1.0f - ct * ct, 0.0f));
  float sp, cp;
  f_sincos_2pi<false>(u_phi, &sp, &cp);
  return make_float3(st * cp, st * sp, ct);
}

// ---- tables ------------------------------------------------------------------
// Inverse-CDF spectrum sampled like a 1-D linear-filtered texture with
// normalised coordinates and clamp addressing (src/spectrum.jl:79-83,
// :137-138): texel i sits at (i + 0.5) / n.  FP32 weights instead of the
// texture unit's 8-bit fraction.
__device__ __forceinline__ float spectrum_sample(const float* __restrict__ k, int n, float u) {
  if (n <= 1) return __ldg(k);
  const float x = fminf(fmaxf(u * (float)n - 0.5f, 0.0f), (float)(n - 1));
  const int i = min((int)x, n - 2);
  const float f = x - (float)i;
  const float a = __ldg(k + i), b = __ldg(k + i + 1);
  return a + f * (b - a);
}

// Quantile table with knots at u = i / (n - 1).
__device__ __forceinline__ float quantile_sample(const float* __restrict__ q, int n, float u) {
  if (n <= 1) return __ldg(q);
  const float x = u * (float)(n - 1);
  const int i = min(max((int)x, 0), n - 2);
  const float f = x - (float)i;
  const float a = __ldg(q + i), b = __ldg(q + i + 1);
  return a + f * (b - a);
}

// Medium at wavelength wl: {sca_len, group velocity, abs_len, n}, linear in wl.
__device__ __forceinline__ float4 medium_at(const float4* __restrict__ t, int n, float wl_min,
                                            float inv_step, float wl) {
  const float x = fminf(fmaxf((wl - wl_min) * inv_step, 0.0f), (float)(n - 1));
  const int i = min((int)x, n - 2);
  const float f = x - (float)i;
  const float4 a = __ldg(t + i), b = __ldg(t + i + 1);
  return make_float4(a.x + f * (b.x - a.x), a.y + f * (b.y - a.y), a.z + f * (b.z - a.z),
                     a.w + f * (b.w - a.w));
}

// ---- scattering (update_direction, src/photon_prop_cuda.jl:280-298) ---------
// With probability hg_weight Henyey-Greenstein at g, else the second
// component: Einstein-Smoluchowski at b (MixedHGES, Cardano root of the cubic
// CDF) or simplified Liu at g (cos = 2 eta^((1-g)/(1+g)) - 1, the deep-ice
// mixture).  Both samples are computed and one is selected (a warp almost
// always needs both anyway); the second component's kind is uniform per
// launch.  Both forms take the step's random words: u_choice from wc, eta
// from we.

// The replay variant: the oracle's expression forms, IEEE division/sqrt/cbrt/pow.
__device__ __forceinline__ float scatter_cos_precise(const pp::PhaseDev& ph, uint32_t wc,
                                                     uint32_t we) {
  const float u_choice = u01(wc), eta = u01(we);
  float hg, other;
  const float g = ph.hg_g, b = ph.es_b;
  const float t = (1.0f - g * g) / (1.0f + g * (2.0f * eta - 1.0f));
  hg = 1.0f / (2.0f * g) * (1.0f + g * g - t * t);
  hg = hg < -1.0f ? -1.0f : (hg > 1.0f ? 1.0f : hg);
  if (ph.kind == PP_PHASE_HG_SL) {
    other = 2.0f * powf(eta, ph.sl_exp) - 1.0f;
  } else {
    const float q = (b + 3.0f) * (eta - 0.5f) / b;
    const float d = sqrtf(q * q + 1.0f / (b * b * b));
    other = cbrtf(q + d) + cbrtf(q - d);
  }
  return u_choice < ph.hg_weight ? hg : other;
}

// The fast variant takes two photons (words we.x and we.y are theirs) and
// works on the 24-bit integers of the uniforms where that is exact and cheaper
// than forming u = k 2^-24 first: the choice is one integer compare
// (PhaseDev::hg_words), 2 eta - 1 = k 2^-23 - 1, and the interval and fraction
// of the tabulated Einstein-Smoluchowski root (PhaseDev::es_table) are k's
// upper and lower bits (no float-to-integer conversions, which take the
// quarter-rate pipe).  Same values bit for bit.
__device__ __forceinline__ float es_root(const pp::PhaseDev& ph, uint32_t ke) {
  constexpr int kShift = 24 - pp::kEsTableBits;
  const float2 e = __ldg(reinterpret_cast<const float2*>(
      reinterpret_cast<const char*>(ph.es_table) + ((ke >> kShift) << 3)));
  // low bits as a fraction: 2^23 + l through the bit pattern, then l 2^-shift
  const float l = __uint_as_float(0x4B000000u | (ke & ((1u << kShift) - 1u)));
  constexpr float kFrac = 1.0f / (float)(1 << kShift);
  return fmaf(fmaf(l, kFrac, -8388608.0f * kFrac), e.y, e.x);
}
__device__ __forceinline__ float second_component(const pp::PhaseDev& ph, float kf) {
  const float eta = kf * 5.9604644775390625e-8f;
  // (a subnormal power and its logarithm round away against the 1)
  if (ph.kind == PP_PHASE_HG_SL) return fmaf(2.0f, ftz_ex2(ph.sl_exp * ftz_lg2(eta)), -1.0f);
  const float q = ph.es_k1 * (eta - 0.5f);
  const float d = approx_sqrt(fmaf(q, q, ph.es_k2));
  return f_cbrt_pos<false>(q + d) - f_cbrt_pos<false>(d - q);
}
__device__ __forceinline__ float2 scatter_cos_fast(const pp::PhaseDev& ph, uint2 wc, uint2 we) {
  const uint32_t k0 = (we.x >> 8) + 1u, k1 = (we.y >> 8) + 1u;  // eta = k 2^-24
  const float2 kf = make_float2(__uint2float_rn(k0), __uint2float_rn(k1));
  // (1 + g (2 eta - 1) lies in [1 - |g|, 1 + |g|]: normal)
  const float2 v = fma2(dup2(ph.hg_g), fma2(kf, dup2(1.1920928955078125e-7f), dup2(-1.0f)),
                        dup2(1.0f));
  const float2 t = mul2(dup2(ph.hg_1mg2), make_float2(ftz_rcp(v.x), ftz_rcp(v.y)));
  // (1 + g^2 - t^2) / 2g with both factors' signs turned
  const float2 h = mul2(fma2(t, t, dup2(ph.hg_n1pg2)), dup2(ph.hg_ninv2g));
  float2 other;
  if (ph.es_table)
    other = make_float2(es_root(ph, k0), es_root(ph, k1));
  else
    other = make_float2(second_component(ph, kf.x), second_component(ph, kf.y));
  return make_float2(wc.x < ph.hg_words ? fminf(fmaxf(h.x, -1.0f), 1.0f) : other.x,
                     wc.y < ph.hg_words ? fminf(fmaxf(h.y, -1.0f), 1.0f) : other.y);
}

// Back onto the unit sphere, for the fast variant: its SFU sine, cosine and
// square root leave |dir| off 1 by ~1e-6, and the reference's sphere test
// (b = a^2 - (|p - c|^2 - r^2), which assumes |dir| = 1) turns a norm error e
// into a shift 2 e a^2 of b -- at 100 m from a module comparable to r^2, and
// biased: photons then miss distant modules they should hit.  One Newton
// step of 1/sqrt(n2) from 1 (error ~ (n2 - 1)^2) on the FMA pipe.
__device__ __forceinline__ float3 renormalise(float3 d) {
  const float n2 = fmaf(d.z, d.z, fmaf(d.y, d.y, d.x * d.x));
  const float s = fmaf(-0.5f, n2, 1.5f);
  return make_float3(d.x * s, d.y * s, d.z * s);
}

// The new direction from the step's three random words (choice, eta, azimuth).
// Replay variant.
__device__ __forceinline__ float3 update_direction_precise(const pp::PhaseDev& ph, float3 dir,
                                                           uint32_t wc, uint32_t we, uint32_t wp) {
  const float c = scatter_cos_precise(ph, wc, we);
  const float s2 = 1.0f - c * c;
  const float st = f_sqrt<true>(s2 > 0.0f ? s2 : 0.0f);
  const float phi = uniform_ab(0.0f, kTwoPi, u01(wp));
  return rot_from_ez<true>(dir, make_float3(cosf(phi) * st, sinf(phi) * st, c));
}

// Fast variant, two photons: each half rounds as renormalise(rot_from_ez<false>(
// dir, (cos(2 pi u) st, sin(2 pi u) st, c))) of that photon; where a packed
// operand is needed negated, an exact sign change takes the place of the scalar
// instruction's operand modifier.
__device__ __forceinline__ Vec2 update_direction_fast(const pp::PhaseDev& ph, const Vec2& a,
                                                      uint2 wc, uint2 we, uint2 wp) {
  const float2 c = scatter_cos_fast(ph, wc, we);
  // 1 - c^2 (with its sign turned; it is 0 or at least 2^-24)
  const float2 n2 = fma2(c, c, dup2(-1.0f));
  const float2 st = make_float2(ftz_sqrt(fmaxf(-n2.x, 0.0f)), ftz_sqrt(fmaxf(-n2.y, 0.0f)));
  // 2 pi u - pi with u = k 2^-24, the scale folded into the constant (f_sincos_2pi)
  const float2 ang = fma2(dup2(kTwoPi * 5.9604644775390625e-8f),
                          make_float2(__uint2float_rn((wp.x >> 8) + 1u),
                                      __uint2float_rn((wp.y >> 8) + 1u)),
                          dup2(-kPi));
  float2 ss, cc;
  __sincosf(ang.x, &ss.x, &cc.x);
  __sincosf(ang.y, &ss.y, &cc.y);
  // the azimuth's sine and cosine are -ss and -cc
  const float2 nst = make_float2(-st.x, -st.y);
  const float2 bx = mul2(cc, nst), by = mul2(ss, nst), nbx = mul2(cc, st);
  // 1 / (1 + a.z), or (1 - a.z) / (a.x^2 + a.y^2) in the lower hemisphere, kept
  // finite on the lower axis, where it meets zeros (emission directions are
  // exact there, on_axis).  (2^-126 added to a.x^2 instead of the maximum would
  // turn the rounding of exact ties: 5 of 166,000 hits moved.)
  const float2 s2 = fma2(a.y, a.y, mul2(a.x, a.x));
  const float2 up = add2(a.z, dup2(1.0f)), down = sub2(dup2(1.0f), a.z);
  float2 f;
  {
    const bool u0 = a.z.x >= 0.0f, u1 = a.z.y >= 0.0f;
    const float d0 = u0 ? up.x : fmaxf(s2.x, 1.17549435e-38f);
    const float d1 = u1 ? up.y : fmaxf(s2.y, 1.17549435e-38f);
    f = mul2(make_float2(u0 ? 1.0f : down.x, u1 ? 1.0f : down.y),
             make_float2(ftz_rcp(d0), ftz_rcp(d1)));
  }
  const float2 k = mul2(fma2(a.x, by, mul2(a.y, nbx)), f);
  const float2 nk = make_float2(-k.x, -k.y);
  const float2 ox = fma2(a.x, c, fma2(bx, a.z, mul2(a.y, nk)));
  const float2 oy = fma2(a.y, c, fma2(by, a.z, mul2(a.x, k)));
  const float2 w = fma2(a.x, bx, mul2(a.y, by));
  const float2 oz = fma2(c, a.z, make_float2(-w.x, -w.y));
  const float2 s = fma2(dup2(-0.5f), fma2(oz, oz, fma2(oy, oy, mul2(ox, ox))), dup2(1.5f));
  return {mul2(ox, s), mul2(oy, s), mul2(oz, s)};
}

// ---- ray-sphere test (_intersect_nsphere, src/photon_prop_cuda.jl:309-343) --
// Hit iff the near intersection lies strictly inside (0, step).  Both
// variants evaluate it exactly as the reference's FP32 expression rounds --
// no fused multiply-adds, IEEE square root: b = a^2 - (|p - c|^2 - r^2)
// cancels heavily for distant spheres, so a different rounding order would
// shift which grazing photons hit (and is not the same everywhere the
// compiler inlines this); the test runs only in the grid walk, so exactness
// costs nothing measurable.
template <bool P>
__device__ __forceinline__ bool sphere_hit(float4 s, float3 pos, float3 dir, float step,
                                           float* d_out) {
  const float dx = __fsub_rn(pos.x, s.x), dy = __fsub_rn(pos.y, s.y), dz = __fsub_rn(pos.z, s.z);
  const float a = __fadd_rn(__fadd_rn(__fmul_rn(dir.x, dx), __fmul_rn(dir.y, dy)),
                            __fmul_rn(dir.z, dz));
  const float pp =
      __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
  const float b = __fsub_rn(__fmul_rn(a, a), __fsub_rn(pp, s.w));
  if (b >= 0.0f) {
    const float d = __fsub_rn(-a, __fsqrt_rn(b));
    if (d > 0.0f && d < step) {
      *d_out = d;
      return true;
    }
  }
  return false;
}

// Intersection with target j of a shaped-target list (check_intersection,
// src/photon_prop_cuda.jl:345-404): spheres by the sphere formula above;
// rectangles and discs lie in the plane z = z_j, met at d = (z_j - z) / dir_z
// when 0 <= d <= step and the point is strictly inside the shape.
template <bool P>
__device__ __forceinline__ bool shape_hit(const float4* __restrict__ shapes, int j, float3 pos,
                                          float3 dir, float step, float* d_out) {
  const float4 g = __ldg(shapes + 2 * j);
  const float4 h = __ldg(shapes + 2 * j + 1);
  const int kind = __float_as_int(h.y);
  if (kind == PP_TARGET_SPHERE) return sphere_hit<P>(g, pos, dir, step, d_out);
  if (dir.z == 0.0f) return false;
  const float d = f_div<P>(g.z - pos.z, dir.z);
  if (d < 0.0f || d > step) return false;
  const float x = madd<P>(dir.x, d, pos.x) - g.x;
  const float y = madd<P>(dir.y, d, pos.y) - g.y;
  const bool in = kind == PP_TARGET_RECTANGLE ? (fabsf(x) < g.w && fabsf(y) < h.x)
                                              : (x * x + y * y < g.w);
  if (in) *d_out = d;
  return in;
}

// First target in index order intersected within (0, step): the candidates
// come from a 3-D DDA walk over the uniform grid cells the segment crosses
// between t_lo and t_hi (0 <= t_lo < t_hi <= step: the part of the segment
// that may come near a target, inside the grid's box up to rounding; the sphere
// test itself always uses the whole segment) (Amanatides & Woo); among all intersected candidates the smallest index
// wins, which is exactly the reference's "first target in index order"
// (src/photon_prop_cuda.jl:497-506).  Returns the 0-based index or -1.
template <bool P>
__device__ __forceinline__ int first_hit(const pp::GridDev& g, const uint32_t* __restrict__ cells,
                                         const uint16_t* __restrict__ items,
                                         const float4* __restrict__ sph, float3 pos, float3 dir,
                                         float step, float t_lo, float t_hi) {
  // Reciprocal direction; zero components become a huge value of the same
  // sign as the step direction chosen below (+ for +0 and -0 alike).
  const float ix = ftz_rcp(fabsf(dir.x) > 1e-20f ? dir.x : 1e-20f);
  const float iy = ftz_rcp(fabsf(dir.y) > 1e-20f ? dir.y : 1e-20f);
  const float iz = ftz_rcp(fabsf(dir.z) > 1e-20f ? dir.z : 1e-20f);
  const int nx = g.dims[0], ny = g.dims[1], nz = g.dims[2];
  int cx = (int)floorf((fmaf(dir.x, t_lo, pos.x) - g.lo[0]) * g.inv_cell[0]);
  int cy = (int)floorf((fmaf(dir.y, t_lo, pos.y) - g.lo[1]) * g.inv_cell[1]);
  int cz = (int)floorf((fmaf(dir.z, t_lo, pos.z) - g.lo[2]) * g.inv_cell[2]);
  cx = min(max(cx, 0), nx - 1);
  cy = min(max(cy, 0), ny - 1);
  cz = min(max(cz, 0), nz - 1);
  const int sx = ix >= 0.0f ? 1 : -1;
  const int sy = iy >= 0.0f ? 1 : -1;
  const int sz = iz >= 0.0f ? 1 : -1;
  float tnx = (fmaf((float)(cx + (sx > 0)), g.cell[0], g.lo[0]) - pos.x) * ix;
  float tny = (fmaf((float)(cy + (sy > 0)), g.cell[1], g.lo[1]) - pos.y) * iy;
  float tnz = (fmaf((float)(cz + (sz > 0)), g.cell[2], g.lo[2]) - pos.z) * iz;
  const float tdx = g.cell[0] * fabsf(ix);
  const float tdy = g.cell[1] * fabsf(iy);
  const float tdz = g.cell[2] * fabsf(iz);
  const int strx = sx, stry = sy * nx, strz = sz * nx * ny;
  int cidx = (cz * ny + cy) * nx + cx;

  int best = 0x7fffffff;
  const int max_iter = nx + ny + nz + 3;
  for (int it = 0; it < max_iter; ++it) {
    const uint32_t w = cells[cidx];
    const uint32_t cnt = w >> pp::kCellStartBits;
    if (cnt) {
      const uint32_t first = w & pp::kCellStartMask;
      for (uint32_t k = 0; k < cnt; ++k) {
        const int j = items[first + k];
        float d;
        if (j < best && sphere_hit<P>(sph[j], pos, dir, step, &d)) {
          best = j;
        }
      }
    }
    // the axis whose boundary comes first (x, then y, on ties), stepped by
    // selects: lanes of a warp step different axes without diverging
    const bool ax = tnx <= tny && tnx <= tnz;
    const bool ay = !ax && tny <= tnz;
    const bool az = !ax && !ay;
    const float tn = ax ? tnx : (ay ? tny : tnz);
    if (tn > t_hi) break;
    cx += ax ? sx : 0;
    cy += ay ? sy : 0;
    cz += az ? sz : 0;
    if ((unsigned)cx >= (unsigned)nx || (unsigned)cy >= (unsigned)ny ||
        (unsigned)cz >= (unsigned)nz)
      break;
    tnx += ax ? tdx : 0.0f;
    tny += ay ? tdy : 0.0f;
    tnz += az ? tdz : 0.0f;
    cidx += ax ? strx : (ay ? stry : strz);
  }
  return best == 0x7fffffff ? -1 : best;
}

// ---- emitters (initialize_photon_state, src/photon_prop_cuda.jl:158-276) ----

// Gamma(shape, scale) by Marsaglia & Tsang (2000) from the photon's emitter
// stream (rand_gamma, PhysicsTools; called at :214).
template <bool P>
__device__ __forceinline__ float gamma_sample(float shape, float scale, uint32_t plo, uint32_t phi,
                                              uint32_t src, uint32_t k0, uint32_t k1) {
  float a = shape;
  const bool boost = a < 1.0f;
  if (boost) a += 1.0f;
  const float d = a - 1.0f / 3.0f;
  const float c = P ? 1.0f / sqrtf(9.0f * d) : rsqrtf(9.0f * d);
  for (int j = 0; j < kGammaMaxTries; ++j) {
    const uint4 r = philox(make_uint4(plo, phi, kExtraCall + (uint32_t)j, src), k0, k1);
    const float u0 = u01(r.x), u1 = u01(r.y), u2 = u01(r.z);
    float cs;
    if (P) {
      cs = cosf(kTwoPi * u1);
    } else {
      float sn;
      f_sincos_2pi<false>(u1, &sn, &cs);
    }
    const float x = f_sqrt<P>(-2.0f * f_log<P>(u0)) * cs;
    float v = 1.0f + c * x;
    if (v <= 0.0f) continue;
    v = v * v * v;
    const float x2 = x * x;
    if (u2 < 1.0f - 0.0331f * x2 * x2 || f_log<P>(u2) < 0.5f * x2 + d * (1.0f - v + f_log<P>(v))) {
      float gs = d * v;
      if (boost) gs *= (P ? powf(u01(r.w), 1.0f / shape) : f_exp<false>(f_log<false>(u01(r.w)) / shape));
      return gs * scale;
    }
  }
  return d * scale;
}

// Cherenkov cone about the emitter axis: theta_c = acos(1/n), phi ~ U(0, 2pi),
// optionally rotated onto a sampled track direction first
// (sample_cherenkov_direction, :80-111).
template <bool P>
__device__ __forceinline__ float3 cherenkov_dir(float3 axis, float ref_ix, float u_phi,
                                                float u_track, float u_track_phi, bool smear,
                                                const float* __restrict__ track, int n_track) {
  float3 ph = P ? sph_to_cart<true>(acosf(1.0f / ref_ix), u_phi)
                : dir_from_cos<false>(approx_rcp(ref_ix), u_phi);
  if (smear) {
    float ct = quantile_sample(track, n_track, u_track);
    ct = ct > 1.0f ? 1.0f : (ct < -1.0f ? -1.0f : ct);
    ph = rot_from_ez<P>(dir_from_cos<P>(ct, u_track_phi), ph);
  }
  return rot_from_ez<P>(axis, ph);
}

}  // namespace ppdev
