// pp_pmt.cu -- photon hits -> PMT hits on the device: the detection step that
// follows propagation in the reference (make_hits_from_photons and
// calc_pe_weight!, src/processing.jl:88-205), one thread per hit record.
//
// For a POM (src/pom.jl:246-305, POMAcceptance): with rel = (hit - centre) / r,
// for each of the 16 PMTs (unit vector p_i, group g_i)
//   pt_i  = acos(clamp(rel . p_i, -1, 1))
//   w_i   = Rayleigh_{sigma_g}(pt_i) / (sin(pt_i) / 2)   (0 where sin(pt_i) = 0)
//   prob_i = w_i * acc_g(wavelength) / 8
// the photon is detected when u1 < sum_i prob_i, by PMT i chosen with
// probability prob_i / sum (the first i whose running sum reaches u2 * sum).
// acc_g and the relative quantum efficiency are linear interpolations that
// are 0 outside their tables (Interpolations.jl, extrapolation_bc = 0).
// For a homogeneous module (src/detection.jl:57-84) the photon is detected
// when u1 < active_area / (4 pi r^2), as PMT 1.
// For a DOM (src/dom.jl:96-134) it is detected, as PMT 1, when
// u1 * polymax < poly(cos zenith of its direction) and u2 < wl_acc(wavelength)
// (the second test only when the model asks for the wavelength acceptance).
// For a multi-PMT module (src/detection.jl:90-131) it is detected when
// u1 <= sum_i max(dir . q_i, 0) * pmt_area / (pi r^2) (q_i the PMT axes in the
// module frame), by the PMT that StatsBase's weighted sample picks for u2 over
// the weights w_i = -(rel . p_i) (p_i the oriented axes): the first i whose
// running sum reaches u2 * sum_i w_i, else the last.
// u1, u2 are Philox4x32-10 uniforms of counter (hit index, 0x504d5400, 0),
// key = seed, so a CPU restatement can replay every decision (up to the
// rounding of the arithmetic: sin(pt) is evaluated as sqrt(1 - cos^2 pt),
// the Gaussian factor by exp2f).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <string>

#include "pp_device.cuh"
#include "pp_internal.h"

namespace {

constexpr int kPomPmts = 16;
constexpr uint32_t kPmtStream = 0x504d5400u;  // Philox counter word that tags this stream

struct PmtArgs {
  const pp_hit_record* rec;
  long long n;
  const pp_pmt_target* targets;
  int n_targets;
  const pp_pom_model* pom;  // device copies, each may be null
  const pp_dom_model* dom;
  const pp_multipmt_model* mpmt;
  uint32_t key0, key1;
  int32_t* pmt_id;
  float* qe_weight;         // may be null
};

// Linear interpolation on ascending knots, 0 outside [x[0], x[n-1]].
__device__ __forceinline__ float interp0(const float* x, const float* y, int n, float v) {
  if (n < 2 || !(v >= x[0]) || !(v <= x[n - 1])) return 0.0f;
  int lo = 0, hi = n - 1;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (x[mid] <= v) lo = mid;
    else hi = mid;
  }
  const float t = (v - x[lo]) / (x[hi] - x[lo]);
  return fmaf(t, y[hi] - y[lo], y[lo]);
}

template <class T>
__device__ __forceinline__ void stage(T* dst, const T* src) {
  static_assert(sizeof(T) % 4 == 0, "word copy");
  if (!src) return;
  const int* s = reinterpret_cast<const int*>(src);
  int* d = reinterpret_cast<int*>(dst);
  for (int w = threadIdx.x; w < (int)(sizeof(T) / 4); w += blockDim.x) d[w] = s[w];
}

// The models in shared memory (staged once per block; the grids stride).
struct Models {
  pp_pom_model pom;
  pp_dom_model dom;
  pp_multipmt_model mpmt;
};
// Rayleigh(pt; sigma) = pt / sigma^2 * 2^(pt^2 * (-log2(e) / (2 sigma^2))), per group
struct Rayleigh {
  float inv_s2_1, inv_s2_2, e2_1, e2_2;
};
__device__ __forceinline__ Rayleigh rayleigh(const pp_pom_model& m) {
  Rayleigh y;
  y.inv_s2_1 = 1.0f / (m.sigma_group1 * m.sigma_group1);
  y.inv_s2_2 = 1.0f / (m.sigma_group2 * m.sigma_group2);
  y.e2_1 = -0.72134752044448170368f * y.inv_s2_1;  // -log2(e) / 2
  y.e2_2 = -0.72134752044448170368f * y.inv_s2_2;
  return y;
}

// x a[0] + y a[1] + z a[2] with its roundings written out.
__device__ __forceinline__ float dot3(float x, float y, float z, const float* a) {
  return fmaf(z, a[2], fmaf(x, a[0], __fmul_rn(y, a[1])));
}

// The PMT (0: none) and QE weight of hit record i.  Every sum of products is an explicit
// FMA, so that the kernels that inline this, and any compiler, round alike.
__device__ __forceinline__ void detect(const PmtArgs& a, const Models& s, const Rayleigh& y,
                                       long long i, int& id, float& qe) {
  const pp_pom_model& sm = s.pom;
  const pp_dom_model& sdom = s.dom;
  const pp_multipmt_model& smp = s.mpmt;
  const float inv_s2_1 = y.inv_s2_1, inv_s2_2 = y.inv_s2_2, e2_1 = y.e2_1, e2_2 = y.e2_2;
  id = 0;
  qe = 0.0f;
  const float4* r = reinterpret_cast<const float4*>(a.rec + i);
  // the record's first 32 bytes: position, wavelength; direction, module
  const float4 pw = __ldg(r);
  const float4 dw = __ldg(r + 1);
  const int module = __float_as_int(dw.w);  // 1-based
  if (module >= 1 && module <= a.n_targets) {
    const pp_pmt_target t = a.targets[module - 1];
    const uint4 u = ppdev::philox(make_uint4((uint32_t)i, (uint32_t)((unsigned long long)i >> 32),
                                          kPmtStream, 0u),
                               a.key0, a.key1);
    const float u1 = ppdev::u01(u.x), u2 = ppdev::u01(u.y);
    if (t.kind == PP_PMT_HOMOGENEOUS) {
      const float frac = t.active_area / (4.0f * 3.14159265358979f * t.radius * t.radius);
      id = u1 < frac ? 1 : 0;
      qe = 1.0f;
    } else if (t.kind == PP_PMT_POM && a.pom) {
      const pp_pom_model& m = sm;
      const float inv_r = 1.0f / t.radius;
      const float rx = (pw.x - t.position[0]) * inv_r;
      const float ry = (pw.y - t.position[1]) * inv_r;
      const float rz = (pw.z - t.position[2]) * inv_r;
      const float acc1 = interp0(m.acc_wavelength, m.acc_group1, m.n_acc, pw.w);
      const float acc2 = interp0(m.acc_wavelength, m.acc_group2, m.n_acc, pw.w);
      float prob[kPomPmts];
      float total = 0.0f;
#pragma unroll
      for (int k = 0; k < kPomPmts; ++k) {
        const float c = fminf(fmaxf(dot3(rx, ry, rz, m.pmt_dir[k]), -1.0f), 1.0f);
        const float pt = acosf(c);
        const bool g1 = m.pmt_group[k] == 1;
        const float s = sqrtf(fmaxf(fmaf(-c, c, 1.0f), 0.0f));  // sin(acos(c)) for pt in [0, pi]
        const float pdf = pt * (g1 ? inv_s2_1 : inv_s2_2) * exp2f(pt * pt * (g1 ? e2_1 : e2_2));
        // w / 8 = pdf / (s / 2) / 8 = pdf / (4 s)
        prob[k] = s != 0.0f ? __fdividef(pdf, 4.0f * s) * (g1 ? acc1 : acc2) : 0.0f;
        total += prob[k];
      }
      if (u1 < total) {
        const float target = u2 * total;
        float cum = 0.0f;
        id = kPomPmts;
#pragma unroll
        for (int k = 0; k < kPomPmts; ++k) {
          cum += prob[k];
          if (cum >= target) {
            id = k + 1;
            break;
          }
        }
      }
      qe = interp0(m.qe_wavelength, m.qe, m.n_qe, pw.w);
    } else if (t.kind == PP_PMT_DOM && a.dom) {
      const pp_dom_model& m = sdom;
      const float cz = dot3(dw.x, dw.y, dw.z, m.zenith_axis);
      float poly = 0.0f;
      for (int k = m.n_poly - 1; k >= 0; --k) poly = fmaf(poly, cz, m.poly[k]);
      const bool ang = u1 * m.polymax < poly;
      const bool wl = !m.apply_wl_acceptance || u2 < interp0(m.wl, m.wl_acc, m.n_wl, pw.w);
      id = ang && wl ? 1 : 0;
      qe = 1.0f;
    } else if (t.kind == PP_PMT_MULTIPMT && a.mpmt) {
      const pp_multipmt_model& m = smp;
      float proj = 0.0f;
      for (int k = 0; k < m.n_pmt; ++k) {
        const float c = dot3(dw.x, dw.y, dw.z, m.pmt_dir_module[k]);
        if (c > 0.0f) proj += c;
      }
      const float prob = proj * m.pmt_area / (3.14159265358979f * t.radius * t.radius);
      if (u1 <= prob) {
        const float inv_r = 1.0f / t.radius;
        const float rx = (pw.x - t.position[0]) * inv_r;
        const float ry = (pw.y - t.position[1]) * inv_r;
        const float rz = (pw.z - t.position[2]) * inv_r;
        float wsum = 0.0f;
        for (int k = 0; k < m.n_pmt; ++k)
          wsum -= dot3(rx, ry, rz, m.pmt_dir[k]);
        const float target = u2 * wsum;
        int j = 0;
        float cw = -dot3(rx, ry, rz, m.pmt_dir[0]);
        while (cw < target && j < m.n_pmt - 1) {
          ++j;
          cw -= dot3(rx, ry, rz, m.pmt_dir[j]);
        }
        id = j + 1;
      }
      qe = interp0(m.qe_wavelength, m.qe, m.n_qe, pw.w);
    }
  }
}

__global__ void __launch_bounds__(256) pmt_kernel(const PmtArgs a) {
  __shared__ Models s;
  stage(&s.pom, a.pom);
  stage(&s.dom, a.dom);
  stage(&s.mpmt, a.mpmt);
  __syncthreads();
  const Rayleigh y = rayleigh(s.pom);
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < a.n;
       i += (long long)gridDim.x * blockDim.x) {
    int id;
    float qe;
    detect(a, s, y, i, id, qe);
    a.pmt_id[i] = id;
    if (a.qe_weight) a.qe_weight[i] = qe;
  }
}

// ---- many POM hits -----------------------------------------------------------
// Six or seven hits in a hundred are detected, and the others need no more than
// an upper bound of their detection probability: total = acc_1 S_1 + acc_2 S_2,
// S_g the group's summed angular weights, functions of the hit's direction from
// the module centre alone.  Their maxima over the cells of an octahedral map
// are tabulated (bound_kernel), a hit whose u1 is not below acc_1 S_1max + acc_2
// S_2max is undetected, and only the rest -- collected by each warp into full
// passes -- take the 16 PMTs' acos, sqrt and exp2.  The decisions are those of
// `detect`, bit for bit.  Issue bound before (1,800 instructions per 32 hits, 2.76
// ms for 5e7); now 0.76 ms, in which the 80-byte records and the results (4.4 GB) pass
// at 87% of the measured copy bandwidth.
constexpr int kMapSize = 64;             // cells per side
constexpr float kNormSlack = 1e-3f;      // |rel| within 1 +- this, else no bound is used
constexpr int kBuckets = 256;            // of a wavelength table's search

// The direction of map coordinates (u, v) in [-1, 1]^2.
__device__ __forceinline__ float3 oct_dir(float u, float v) {
  float3 d = make_float3(u, v, 1.0f - fabsf(u) - fabsf(v));
  if (d.z < 0.0f) {
    d.x = copysignf(1.0f - fabsf(v), u);
    d.y = copysignf(1.0f - fabsf(u), v);
  }
  const float n = rsqrtf(d.x * d.x + d.y * d.y + d.z * d.z);
  return make_float3(d.x * n, d.y * n, d.z * n);
}
// The map cell of a direction (of any length).
__device__ __forceinline__ int oct_cell(float x, float y, float z) {
  const float n = __fdividef(1.0f, fabsf(x) + fabsf(y) + fabsf(z));
  float u = x * n, v = y * n;
  if (z < 0.0f) {
    const float w = u;
    u = copysignf(1.0f - fabsf(v), u);
    v = copysignf(1.0f - fabsf(w), v);
  }
  const float h = 0.5f * kMapSize;
  const int iu = (int)fminf(fmaxf(fmaf(u, h, h), 0.0f), (float)(kMapSize - 1));
  const int iv = (int)fminf(fmaxf(fmaf(v, h, h), 0.0f), (float)(kMapSize - 1));
  return iv * kMapSize + iu;
}

// One thread per cell and PMT: bounds of the groups' summed weights prob / acc
// over the cell's directions.  A PMT's weight falls, then (towards the antipode)
// rises with the angle, so its maximum over the cell's range of angles is at an
// end; the range is widened by the map's rounding and by what kNormSlack does
// to the cosine.  The 16 PMTs' threads are neighbours and add up by shuffles.
constexpr int kBoundThreads = 256;
__global__ void __launch_bounds__(kBoundThreads)
    bound_kernel(const pp_pom_model* __restrict__ m, float2* __restrict__ out) {
  const int t = blockIdx.x * kBoundThreads + threadIdx.x;
  const int c = t / kPomPmts, k = t % kPomPmts;
  const float w = 2.0f / kMapSize;
  const float u0 = -1.0f + w * (c % kMapSize), v0 = -1.0f + w * (c / kMapSize);
  const float3 d = oct_dir(u0 + 0.5f * w, v0 + 0.5f * w);
  // the farthest point of a cell is a corner (the map's folds run along diagonals)
  const float3 e = oct_dir(fminf(u0 + w * (k & 1), 1.0f), fminf(v0 + w * (k >> 1 & 1), 1.0f));
  float cmin = fminf(d.x * e.x + d.y * e.y + d.z * e.z, 1.0f);
  cmin = fminf(cmin, __shfl_xor_sync(0xffffffffu, cmin, 1));
  cmin = fminf(cmin, __shfl_xor_sync(0xffffffffu, cmin, 2));
  const float rho = acosf(cmin) + 2e-3f;
  const bool g1 = m->pmt_group[k] == 1;
  const float sg = g1 ? m->sigma_group1 : m->sigma_group2;
  const float inv_s2 = 1.0f / (sg * sg);
  const float at = acosf(fminf(fmaxf(d.x * m->pmt_dir[k][0] + d.y * m->pmt_dir[k][1] +
                                     d.z * m->pmt_dir[k][2], -1.0f), 1.0f));
  float best = 0.0f;
  for (int side = 0; side < 2; ++side) {
    const float end = side ? fminf(at + rho, 3.14159265f) : fmaxf(at - rho, 0.0f);
    const float cc = fminf(fmaxf(cosf(end) + (side ? -2e-3f : 2e-3f), -1.0f), 1.0f);
    const float pt = acosf(cc);
    // the smallest non-zero sine of an FP32 cosine is 3.4e-4
    const float sn = fmaxf(sqrtf(fmaxf(1.0f - cc * cc, 0.0f)), 3e-4f);
    const float ratio = pt < 1e-2f ? 1.0001f : pt / sn;
    best = fmaxf(best, 0.25f * inv_s2 * ratio * expf(-0.5f * pt * pt * inv_s2));
  }
  float s1 = g1 ? best : 0.0f, s2 = g1 ? 0.0f : best;
  for (int o = 1; o < kPomPmts; o <<= 1) {
    s1 += __shfl_xor_sync(0xffffffffu, s1, o);
    s2 += __shfl_xor_sync(0xffffffffu, s2, o);
  }
  // (5% for the rounding of the weights near a PMT's axis)
  if (k == 0) out[c] = make_float2(1.05f * s1, 1.05f * s2);
}

// Last knot k <= n - 2 with x[k] <= v (the interval interp0's bisection ends at,
// for v in [x[0], x[n - 1]]), from a start at or before it.
__device__ __forceinline__ int knot_from(const float* x, int n, int k, float v) {
  while (k < n - 2 && x[k + 1] <= v) ++k;
  return k;
}

// One CTA of 1024 per SM, so that the map and the models are there once and the
// rest is L1 (5e7 hits, some of them off the modules' surfaces: 0.94 ms; 2 x 512
// threads 1.02, 4 x 256 1.08).
constexpr int kManyThreads = 1024;
__global__ void __launch_bounds__(kManyThreads, 1)
    pmt_many_kernel(const PmtArgs a, const float4* __restrict__ place,
                    const float2* __restrict__ bound) {
  __shared__ Models s;
  __shared__ float2 map[kMapSize * kMapSize];
  __shared__ float2 acc_max[kBuckets];          // of both groups, over a bucket's wavelengths
  __shared__ unsigned char qe_start[kBuckets];  // where a bucket's knot search starts
  __shared__ float4 qe_line[PP_POM_MAX_KNOTS];  // knot, interval, QE, its difference
  __shared__ long long waiting[kManyThreads / 32][64];
  stage(&s.pom, a.pom);
  stage(&s.dom, a.dom);
  stage(&s.mpmt, a.mpmt);
  for (int c = threadIdx.x; c < kMapSize * kMapSize; c += blockDim.x) map[c] = __ldg(bound + c);
  __syncthreads();
  const pp_pom_model& m = s.pom;
  const float acc_lo = m.acc_wavelength[0], acc_hi = m.acc_wavelength[m.n_acc - 1];
  const float qe_lo = m.qe_wavelength[0], qe_hi = m.qe_wavelength[m.n_qe - 1];
  const float acc_scale = kBuckets / (acc_hi - acc_lo), qe_scale = kBuckets / (qe_hi - qe_lo);
  for (int b = threadIdx.x; b < kBuckets; b += blockDim.x) {
    // the lines' maxima are at the ends or at knots (a bucket widened to each
    // side covers the rounding of its number)
    const float v0 = fmaxf(acc_lo + ((float)b - 0.25f) / acc_scale, acc_lo);
    const float v1 = fminf(acc_lo + ((float)b + 1.25f) / acc_scale, acc_hi);
    float2 top = make_float2(fmaxf(interp0(m.acc_wavelength, m.acc_group1, m.n_acc, v0),
                                   interp0(m.acc_wavelength, m.acc_group1, m.n_acc, v1)),
                             fmaxf(interp0(m.acc_wavelength, m.acc_group2, m.n_acc, v0),
                                   interp0(m.acc_wavelength, m.acc_group2, m.n_acc, v1)));
    for (int k = 0; k < m.n_acc; ++k)
      if (m.acc_wavelength[k] >= v0 && m.acc_wavelength[k] <= v1)
        top = make_float2(fmaxf(top.x, m.acc_group1[k]), fmaxf(top.y, m.acc_group2[k]));
    acc_max[b] = top;
    qe_start[b] = (unsigned char)knot_from(m.qe_wavelength, m.n_qe, 0,
                                           qe_lo + (float)(b - 1) / qe_scale);
  }
  for (int k = threadIdx.x; k + 1 < m.n_qe; k += blockDim.x)
    qe_line[k] = make_float4(m.qe_wavelength[k], m.qe_wavelength[k + 1] - m.qe_wavelength[k],
                             m.qe[k], m.qe[k + 1] - m.qe[k]);
  __syncthreads();
  const Rayleigh y = rayleigh(m);
  const int lane = threadIdx.x & 31;
  long long* mine = waiting[threadIdx.x >> 5];
  int n_wait = 0;  // rows in `mine` (warp-uniform)
  const long long stride = (long long)gridDim.x * blockDim.x;
  long long base = (long long)blockIdx.x * blockDim.x + (threadIdx.x & ~31);
  // the next record is requested before this one is worked on
  float4 pw_next = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  int module_next = 0;
  auto request = [&](long long i) {
    if (i < a.n) {
      const float4* r = reinterpret_cast<const float4*>(a.rec + i);
      pw_next = __ldg(r);
      module_next = __float_as_int(__ldg(reinterpret_cast<const float*>(r) + 7));
    }
  };
  request(base + lane);
  for (;; base += stride) {
    const bool more = base < a.n;
    if (more) {
      const long long i = base + lane;
      const float4 pw = pw_next;
      const int module = module_next;  // 1-based
      request(i + stride);
      bool wait = false;
      if (i < a.n) {
        float4 at = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (module >= 1 && module <= a.n_targets) at = __ldg(place + module - 1);
        if (at.w > 0.0f) {  // a POM
          const uint4 u = ppdev::philox(
              make_uint4((uint32_t)i, (uint32_t)((unsigned long long)i >> 32), kPmtStream, 0u),
              a.key0, a.key1);
          const float rx = (pw.x - at.x) * at.w, ry = (pw.y - at.y) * at.w,
                      rz = (pw.z - at.z) * at.w;
          const float n2 = rx * rx + ry * ry + rz * rz;
          float limit = 0.0f;  // outside the acceptance tables nothing is detected
          if (pw.w >= acc_lo && pw.w <= acc_hi) {
            const float2 w = map[oct_cell(rx, ry, rz)];
            const float2 acc = acc_max[min((int)((pw.w - acc_lo) * acc_scale), kBuckets - 1)];
            limit = acc.x * w.x + acc.y * w.y;
          }
          wait = !(fabsf(n2 - 1.0f) < 2.0f * kNormSlack - 1e-5f && ppdev::u01(u.x) >= limit);
          if (!wait) a.pmt_id[i] = 0;
          if (a.qe_weight) {
            float qe = 0.0f;
            if (pw.w >= qe_lo && pw.w <= qe_hi) {
              const float4 l = qe_line[knot_from(
                  m.qe_wavelength, m.n_qe,
                  qe_start[min((int)((pw.w - qe_lo) * qe_scale), kBuckets - 1)], pw.w)];
              qe = fmaf((pw.w - l.x) / l.y, l.w, l.z);
            }
            a.qe_weight[i] = qe;
          }
        } else {  // another kind, or no module of this call
          int id;
          float qe;
          detect(a, s, y, i, id, qe);
          a.pmt_id[i] = id;
          if (a.qe_weight) a.qe_weight[i] = qe;
        }
      }
      const unsigned w = __ballot_sync(0xffffffffu, wait);
      if (wait) mine[n_wait + __popc(w & ((1u << lane) - 1u))] = i;
      n_wait += __popc(w);
      __syncwarp();
    }
    if (n_wait >= 32 || (!more && n_wait > 0)) {
      const int take = min(n_wait, 32);
      n_wait -= take;
      if (lane < take) {
        const long long i = mine[n_wait + lane];
        int id;
        float qe;
        detect(a, s, y, i, id, qe);
        a.pmt_id[i] = id;
      }
      __syncwarp();
    }
    if (!more && n_wait == 0) break;
  }
}

// What pmt_many_kernel's bound needs of a POM model: unit PMT axes, positive
// widths, acceptances that are not negative, ascending tables.
bool bound_applies(const pp_pom_model& m) {
  if (!(m.sigma_group1 > 1e-3f && m.sigma_group1 < 1e3f && m.sigma_group2 > 1e-3f &&
        m.sigma_group2 < 1e3f))
    return false;
  for (int k = 0; k < kPomPmts; ++k) {
    const float* d = m.pmt_dir[k];
    if (!(std::fabs(d[0] * d[0] + d[1] * d[1] + d[2] * d[2] - 1.0f) < 1e-4f)) return false;
  }
  for (int k = 0; k < m.n_acc; ++k)
    if (!(m.acc_group1[k] >= 0.0f && m.acc_group1[k] < 1e6f && m.acc_group2[k] >= 0.0f &&
          m.acc_group2[k] < 1e6f) ||
        (k > 0 && !(m.acc_wavelength[k] > m.acc_wavelength[k - 1])))
      return false;
  for (int k = 1; k < m.n_qe; ++k)
    if (!(m.qe_wavelength[k] > m.qe_wavelength[k - 1])) return false;
  return std::isfinite(m.acc_wavelength[0]) && std::isfinite(m.acc_wavelength[m.n_acc - 1]) &&
         std::isfinite(m.qe_wavelength[0]) && std::isfinite(m.qe_wavelength[m.n_qe - 1]);
}
// Hits from which on the map's extra launch pays (3e5 hits: 54 us with it, 39
// without; 1e6: 72 and 83), whatever share of them POMs have: 400 modules of which one is
// a POM and the others DOMs 155 us (152 without) for 2^20 hits, 415 (445) for 2^24,
// multi-PMT modules 166 (162) and 562 (679), homogeneous ones 141 (142) and 361 (403); 20 POMs
// among DOMs 153 (187) and 445 (1,072).
constexpr long long kManyHits = 1 << 20;

// A call's targets and models reach the device as kernel parameters, which a launch
// takes when it is made: the caller's structures, and the image they are gathered
// in, are free when the call returns, also under stream capture and where a copy
// from pageable memory is asynchronous.
constexpr int kImageWords[] = {250, 1020, 2040};  // 16-byte words that a launch carries
template <int kWords>
struct ImagePart {
  uint4 w[kWords];
};
template <int kWords>
__global__ void __launch_bounds__(256)
    write_kernel(uint4* __restrict__ dst, const __grid_constant__ ImagePart<kWords> part, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[i] = part.w[i];
}
// Room for `bytes` (zeros) and, after them, for what a launch reads past the last part.
using HostImage = std::unique_ptr<unsigned char[]>;
HostImage host_image(size_t bytes) {
  HostImage image(new unsigned char[bytes + sizeof(ImagePart<kImageWords[2]>)]);
  memset(image.get(), 0, bytes);
  return image;
}
// The first `bytes` (a multiple of 16) of a host_image to device memory, in launches of
// the smallest size that holds what is left.  (400 mixed modules, 15 KB: one of 16 KB.)
cudaError_t write_image(void* dst, const HostImage& image, size_t bytes, cudaStream_t s) {
  const void* kernels[] = {(const void*)write_kernel<kImageWords[0]>,
                           (const void*)write_kernel<kImageWords[1]>,
                           (const void*)write_kernel<kImageWords[2]>};
  cudaError_t e = cudaSuccess;
  for (size_t words = bytes / 16, at = 0; e == cudaSuccess && at < words;) {
    int size = 0;
    while (size < 2 && words - at > (size_t)kImageWords[size]) ++size;
    int n = (int)std::min<size_t>(words - at, kImageWords[size]);
    uint4* to = static_cast<uint4*>(dst) + at;
    void* params[] = {&to, image.get() + 16 * at, &n};
    e = cudaLaunchKernel(kernels[size], dim3((unsigned)((n + 255) / 256)), dim3(256), params, 0, s);
    at += n;
  }
  return e;
}

__global__ void tres_kernel(const pp_hit_record* __restrict__ rec, long long n,
                            const double* __restrict__ tgeo, int n_targets, double t0,
                            double* __restrict__ tres) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const int module = rec[i].module_index;  // 1-based
    tres[i] = module >= 1 && module <= n_targets ? rec[i].time - tgeo[module - 1] - t0
                                                 : __longlong_as_double(0x7ff8000000000000ll);
  }
}

}  // namespace

extern "C" {

PP_API int pp_time_residuals(const pp_hit_record* d_records, int64_t n, const double* tgeo,
                             int32_t n_targets, double t0, double* d_tres, void* stream) {
  if (n < 0 || (n > 0 && (!d_records || !d_tres)) || n_targets < 0 || (n_targets > 0 && !tgeo))
    return pp::report_error(PP_ERR_INVALID, "pp_time_residuals: bad arguments");
  if (n == 0) return PP_OK;
  cudaStream_t s = (cudaStream_t)stream;
  double* d_tg = nullptr;
  const size_t tb = sizeof(double) * (size_t)(n_targets > 0 ? n_targets : 1);
  cudaError_t e = cudaMallocAsync((void**)&d_tg, tb, s);
  if (e == cudaSuccess && n_targets > 0)
    e = cudaMemcpyAsync(d_tg, tgeo, sizeof(double) * n_targets, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const long long blocks = std::min<long long>((n + 255) / 256, (long long)sms * 8);
    tres_kernel<<<(unsigned)blocks, 256, 0, s>>>(d_records, n, d_tg, n_targets, t0, d_tres);
    e = cudaGetLastError();
  }
  if (d_tg) cudaFreeAsync(d_tg, s);
  if (e != cudaSuccess)
    return pp::report_error(PP_ERR_CUDA, std::string("pp_time_residuals: ") + cudaGetErrorString(e));
  return PP_OK;
}

PP_API int pp_make_hits_from_photons_models(const pp_hit_record* d_records, int64_t n,
                                            const pp_pmt_target* targets, int32_t n_targets,
                                            const pp_detection_models* models, int64_t seed,
                                            int32_t* d_pmt_id, float* d_qe_weight, void* stream) {
  static const char* kWho = "pp_make_hits_from_photons: ";
  if (n < 0 || (n > 0 && (!d_records || !d_pmt_id)) || n_targets < 0 ||
      (n_targets > 0 && !targets))
    return pp::report_error(PP_ERR_INVALID, std::string(kWho) + "bad arguments");
  const pp_pom_model* pom = models ? models->pom : nullptr;
  const pp_dom_model* dom = models ? models->dom : nullptr;
  const pp_multipmt_model* mp = models ? models->multipmt : nullptr;
  if (pom && (pom->n_acc < 2 || pom->n_acc > PP_POM_MAX_KNOTS || pom->n_qe < 2 ||
              pom->n_qe > PP_POM_MAX_KNOTS))
    return pp::report_error(PP_ERR_INVALID, std::string(kWho) + "bad POM tables");
  if (dom && (dom->n_poly < 1 || dom->n_poly > PP_DOM_MAX_POLY || dom->n_wl < 2 ||
              dom->n_wl > PP_POM_MAX_KNOTS))
    return pp::report_error(PP_ERR_INVALID, std::string(kWho) + "bad DOM tables");
  if (mp && (mp->n_pmt < 1 || mp->n_pmt > PP_MULTIPMT_MAX_PMTS || mp->n_qe < 2 ||
             mp->n_qe > PP_POM_MAX_KNOTS))
    return pp::report_error(PP_ERR_INVALID, std::string(kWho) + "bad multi-PMT tables");
  for (int i = 0; i < n_targets; ++i) {
    const int k = targets[i].kind;
    if (k != PP_PMT_HOMOGENEOUS && k != PP_PMT_POM && k != PP_PMT_DOM && k != PP_PMT_MULTIPMT)
      return pp::report_error(PP_ERR_INVALID, std::string(kWho) + "unknown module kind");
    if ((k == PP_PMT_POM && !pom) || (k == PP_PMT_DOM && !dom) || (k == PP_PMT_MULTIPMT && !mp))
      return pp::report_error(PP_ERR_INVALID, std::string(kWho) + "module without its model");
    if (!(targets[i].radius > 0.0f))
      return pp::report_error(PP_ERR_INVALID, std::string(kWho) + "target radius <= 0");
  }
  if (n == 0) return PP_OK;
  cudaStream_t s = (cudaStream_t)stream;
  // one staging allocation: targets, then each model at a 16-byte boundary
  auto up16 = [](size_t b) { return (b + 15) & ~size_t(15); };
  const size_t tb = up16(sizeof(pp_pmt_target) * (size_t)(n_targets > 0 ? n_targets : 1));
  const size_t ob_pom = tb, ob_dom = ob_pom + (pom ? up16(sizeof(pp_pom_model)) : 0);
  const size_t ob_mp = ob_dom + (dom ? up16(sizeof(pp_dom_model)) : 0);
  const size_t ob_place = ob_mp + (mp ? up16(sizeof(pp_multipmt_model)) : 0);
  const bool many = pom && n >= kManyHits && bound_applies(*pom);
  const size_t total = ob_place + (many ? sizeof(float4) * (size_t)n_targets : 0);
  const size_t alloc = total + (many ? sizeof(float2) * kMapSize * kMapSize : 0);
  const HostImage image = host_image(total);
  if (n_targets > 0) memcpy(image.get(), targets, sizeof(pp_pmt_target) * n_targets);
  if (pom) memcpy(image.get() + ob_pom, pom, sizeof(pp_pom_model));
  if (dom) memcpy(image.get() + ob_dom, dom, sizeof(pp_dom_model));
  if (mp) memcpy(image.get() + ob_mp, mp, sizeof(pp_multipmt_model));
  if (many) {  // centre and 1 / radius of the POMs, 0 for the others
    float4* place = reinterpret_cast<float4*>(image.get() + ob_place);
    for (int i = 0; i < n_targets; ++i)
      place[i] = make_float4(targets[i].position[0], targets[i].position[1],
                             targets[i].position[2],
                             targets[i].kind == PP_PMT_POM ? 1.0f / targets[i].radius : 0.0f);
  }
  unsigned char* buf = nullptr;
  cudaError_t e = cudaMallocAsync((void**)&buf, alloc, s);
  if (e == cudaSuccess) e = write_image(buf, image, total, s);
  if (e != cudaSuccess) {
    if (buf) cudaFreeAsync(buf, s);
    return pp::report_error(PP_ERR_CUDA, std::string(kWho) + cudaGetErrorString(e));
  }
  PmtArgs a{};
  a.rec = d_records;
  a.n = n;
  a.targets = reinterpret_cast<const pp_pmt_target*>(buf);
  a.n_targets = n_targets;
  a.pom = pom ? reinterpret_cast<const pp_pom_model*>(buf + ob_pom) : nullptr;
  a.dom = dom ? reinterpret_cast<const pp_dom_model*>(buf + ob_dom) : nullptr;
  a.mpmt = mp ? reinterpret_cast<const pp_multipmt_model*>(buf + ob_mp) : nullptr;
  a.key0 = (uint32_t)(uint64_t)seed;
  a.key1 = (uint32_t)((uint64_t)seed >> 32);
  a.pmt_id = d_pmt_id;
  a.qe_weight = d_qe_weight;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const long long blocks = std::min<long long>((n + 255) / 256, (long long)sms * 8);
  if (many) {
    float2* bound = reinterpret_cast<float2*>(buf + total);
    bound_kernel<<<kMapSize * kMapSize * kPomPmts / kBoundThreads, kBoundThreads, 0, s>>>(a.pom,
                                                                                          bound);
    pmt_many_kernel<<<(unsigned)std::min<long long>((n + kManyThreads - 1) / kManyThreads, sms),
                      kManyThreads, 0, s>>>(a, reinterpret_cast<const float4*>(buf + ob_place), bound);
  } else {
    pmt_kernel<<<(unsigned)blocks, 256, 0, s>>>(a);
  }
  e = cudaGetLastError();
  cudaFreeAsync(buf, s);
  if (e != cudaSuccess)
    return pp::report_error(PP_ERR_CUDA, std::string(kWho) + cudaGetErrorString(e));
  return PP_OK;
}

PP_API int pp_make_hits_from_photons(const pp_hit_record* d_records, int64_t n,
                                     const pp_pmt_target* targets, int32_t n_targets,
                                     const pp_pom_model* pom, int64_t seed, int32_t* d_pmt_id,
                                     float* d_qe_weight, void* stream) {
  const pp_detection_models models{pom, nullptr, nullptr};
  return pp_make_hits_from_photons_models(d_records, n, targets, n_targets, &models, seed,
                                          d_pmt_id, d_qe_weight, stream);
}

}  // extern "C"
