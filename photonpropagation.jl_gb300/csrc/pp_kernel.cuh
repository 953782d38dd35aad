// pp_kernel.cuh -- the persistent photon-propagation kernel template.
//
// Included by two translation units: pp_propagate.cu instantiates the fast
// variant (SFU approximations, packed pairs), pp_propagate_precise.cu the
// replay variant (IEEE math library, compiled with -fmad=false so that every
// FP32 expression rounds exactly as the CPU oracle's does).
//
// Replaces cuda_propagate_photons! (PhotonPropagation.jl v0.9.3,
// src/photon_prop_cuda.jl:429-549) and its one-launch-per-source host loop
// (:927-943).  Design:
//   * persistent CTAs; every warp pulls chunks of photons of one source from a
//     device work queue, so one launch covers any number of sources with
//     uneven photon counts, and sources of few photons share groups (kMixed);
//   * photon i of source s draws its random numbers from Philox4x32-10 at
//     counter (i, call, s) and key = seed: results do not depend on the launch
//     shape and any photon range can be replayed;
//   * two photons per lane.  The kernel is bound by instruction issue, and the
//     packed f32x2 instructions do the two photons' sums and products in one
//     issue slot; the 64 photons of a warp also fill its clip and walk passes
//     twice as well.  16 warps of 128 registers replace 32 of 64: per photon step
//     8.7 warp instructions instead of 11.4 (1e8 photons, 400 modules: 16.66 ->
//     15.75 ms; 256 emitters 5.51 -> 4.97; histogram tables 6.22 -> 5.37).  Tables too
//     large for shared memory take 32 warps all the same (Tables);
//   * speculative stepping with deferred hit tests.  Each lane runs all
//     n_steps of its photons without waiting for the target test.  A step
//     segment is cleared cheaply when the safety field proves that no target
//     lies within the ball around its midpoint; the rare uncleared segments
//     go to a per-warp stack in shared memory.  When 32 of them wait, the warp
//     clips them, one per lane, by sphere tracing the safety field from both
//     ends (most vanish); the survivors wait on a second stack with the part
//     of the segment that may come near a target, and whenever 32 wait the
//     warp walks them, one per lane, through the uniform-grid DDA over that
//     part only.  A photon's hit is the earliest step with an intersection
//     and, within it, the lowest target index -- the reference's "first
//     target in index order" (:497-506).  Steps after the hit were computed
//     speculatively and are discarded, and not tested once the hit is known;
//   * the target grid (cells, candidate lists, spheres) is staged once per CTA
//     into shared memory with a TMA bulk copy completing on an mbarrier, waited
//     on with a time bound;
//   * hits are appended with one atomic per warp into 80-byte records written
//     as five 16-byte vector stores.
#pragma once

#include <cuda_runtime.h>

#include "pp_device.cuh"
#include "pp_internal.h"

namespace pp {
namespace {

using namespace ppdev;

__device__ __forceinline__ unsigned long long global_timer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ unsigned long long* u64(uint64_t* p) {
  return reinterpret_cast<unsigned long long*>(p);
}

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// Issue TMA bulk copies of `bytes` (multiple of 16, both ends 16-byte
// aligned) completing on the mbarrier at bar_a.
__device__ __forceinline__ void bulk_copy(unsigned char* dst, const unsigned char* src,
                                          uint32_t bytes, uint32_t bar_a) {
  constexpr uint32_t kChunk = 32768;
  for (uint32_t off = 0; off < bytes; off += kChunk) {
    const uint32_t n = bytes - off < kChunk ? bytes - off : kChunk;
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_addr(dst + off)),
        "l"(src + off), "r"(n), "r"(bar_a)
        : "memory");
  }
}

// Stage two global tables into shared memory with TMA bulk copies completing
// on one mbarrier.  Every thread then waits on the barrier's phase 0 for at
// most limit_ns.  Returns false on timeout.  skip_copies (a diagnostic, see
// pp_debug_staging_timeout) arms the barrier but issues no copy, so that the
// bounded wait runs out with nothing in flight.
__device__ bool stage_tables(unsigned char* dst0, const unsigned char* src0, uint32_t bytes0,
                             unsigned char* dst1, const unsigned char* src1, uint32_t bytes1,
                             unsigned long long* bar, unsigned long long limit_ns,
                             bool skip_copies) {
  const uint32_t bar_a = smem_addr(bar);
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar_a), "r"(1) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar_a),
                 "r"(bytes0 + bytes1)
                 : "memory");
    if (!skip_copies) {
      bulk_copy(dst0, src0, bytes0, bar_a);
      bulk_copy(dst1, src1, bytes1, bar_a);
    }
  }
  const unsigned long long t0 = global_timer_ns();
  while (true) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar_a), "r"(0)
        : "memory");
    if (done) return true;
    if (global_timer_ns() - t0 > limit_ns) return false;
  }
}

// Two points against the safety field, in units of the node spacing: q, the
// squared distance of m from the field's box, and w, the lower bound
// max(D(c) - |m' - c|, 0) at m's projection m' onto the box, c the nearest node.
// Adding and subtracting 2^23 rounds to the nearest node and leaves the node's
// index in the mantissa, so nothing is converted between float and integer:
// 45 instructions against 55-60 for floor, clamp and a Chebyshev box test,
// and sqrt(q + w^2) clears more than the larger of two bounds did.
constexpr float kRoundMagic = 8388608.0f;
struct FieldPoint2 {
  float2 q, w;
};
template <bool kShared>
__device__ __forceinline__ FieldPoint2 field_point2(const SafetyDev& s,
                                                    const unsigned char* __restrict__ f,
                                                    const Vec2& m) {
  const float2 inv = dup2(s.inv_cell), magic = dup2(kRoundMagic), nmagic = dup2(-kRoundMagic);
  const float2 ux = fma2(m.x, inv, dup2(-s.lo_sc[0]));
  const float2 uy = fma2(m.y, inv, dup2(-s.lo_sc[1]));
  const float2 uz = fma2(m.z, inv, dup2(-s.lo_sc[2]));
  auto clamp = [](float2 u, float hi) {
    return make_float2(fminf(fmaxf(u.x, 0.0f), hi), fminf(fmaxf(u.y, 0.0f), hi));
  };
  const float2 cx = clamp(ux, s.fmaxc[0]), cy = clamp(uy, s.fmaxc[1]), cz = clamp(uz, s.fmaxc[2]);
  const float2 ex = sub2(ux, cx), ey = sub2(uy, cy), ez = sub2(uz, cz);
  const float2 gx = add2(cx, magic);
  const float2 fx = add2(gx, nmagic);
  const float2 fy = add2(add2(cy, magic), nmagic), fz = add2(add2(cz, magic), nmagic);
  const float2 rx = sub2(cx, fx), ry = sub2(cy, fy), rz = sub2(cz, fz);
  const float2 id = fma2(fma2(fz, dup2(s.fdims[1]), fy), dup2(s.fdims[0]), gx);
  const uint32_t i0 = __float_as_uint(id.x) - 0x4B000000u, i1 = __float_as_uint(id.y) - 0x4B000000u;
  const uint32_t b0 = kShared ? f[i0] : __ldg(f + i0), b1 = kShared ? f[i1] : __ldg(f + i1);
  const float2 D = fma2(make_float2(__uint_as_float(0x4B000000u | b0),
                                    __uint_as_float(0x4B000000u | b1)),
                        dup2(s.quantum), dup2(-kRoundMagic * s.quantum));
  const float2 rr = fma2(rz, rz, fma2(ry, ry, mul2(rx, rx)));
  const float2 w = sub2(D, make_float2(ftz_sqrt(rr.x), ftz_sqrt(rr.y)));
  FieldPoint2 p;
  p.q = fma2(ez, ez, fma2(ey, ey, mul2(ex, ex)));
  p.w = make_float2(fmaxf(w.x, 0.0f), fmaxf(w.y, 0.0f));
  return p;
}

// Do the segments pos + t*dir, t in [0, L], of the two photons provably miss
// every target?  A segment lies inside the ball of radius L/2 about its
// midpoint, and no (inflated) sphere comes that near.
template <bool kShared>
__device__ __forceinline__ void segments_clear(const SafetyDev& s, const unsigned char* f,
                                               const Vec2& pos, const Vec2& dir, float2 L,
                                               bool* clear0, bool* clear1) {
  const float2 h = mul2(L, dup2(0.5f));
  const FieldPoint2 p = field_point2<kShared>(
      s, f, {fma2(dir.x, h, pos.x), fma2(dir.y, h, pos.y), fma2(dir.z, h, pos.z)});
  const float2 r = fma2(h, dup2(s.r_scale), dup2(s.r_slack));
  const float2 bound = fma2(p.w, p.w, p.q), r2 = mul2(r, r);
  *clear0 = bound.x > r2.x;
  *clear1 = bound.y > r2.y;
}

// Slack (m) taken off each clipped end: covers the rounding of the traced
// points and of the square root, well inside the 1 cm by which the field's
// spheres are inflated.
constexpr float kClipSlack = 5e-3f;

// Clip the raw entries [base, base + c) (c <= 32, one per lane): first to the
// grid's box (no target lies outside it), then by sphere tracing the safety
// field twice from each end of what is left, both ends in one packed test --
// no target lies within w of a point p -- and last by the step loop's ball test
// on each half of the rest, so the walk can skip [0, t0) and (t1, L].  Entries
// left with t0 < t1 go on top of the clipped stack with their interval; the
// others cannot hit anything and are dropped.  Returns the new height of the
// clipped stack.  (Two traces and one halving: 1e8 photons, 400 modules, 9%
// faster than two traces alone; one trace and one halving, two and two, or
// halvings alone are slower, as is a third pass of either kind.)
template <bool kShared>
__device__ __forceinline__ int clip_entries(WarpQueue& q, int base, int c, int n2,
                                            const GridDev& g, const SafetyDev& s,
                                            const unsigned char* __restrict__ f, int lane) {
  const int src = base + lane;
  bool keep = false;
  float4 ea, eb;
  float t0 = 0.0f, t1 = 0.0f;
  if (lane < c) {
    ea = q.raw_a[src];
    eb = q.raw_b[src];
    const float3 p = make_float3(ea.x, ea.y, ea.z), d = make_float3(eb.x, eb.y, eb.z);
    const float L = ea.w;
    // slab test against the grid box (the same one the walk clips to)
    const float ix = ftz_rcp(fabsf(d.x) > 1e-20f ? d.x : 1e-20f);
    const float iy = ftz_rcp(fabsf(d.y) > 1e-20f ? d.y : 1e-20f);
    const float iz = ftz_rcp(fabsf(d.z) > 1e-20f ? d.z : 1e-20f);
    const float tx0 = (g.lo[0] - p.x) * ix, tx1 = (g.hi[0] - p.x) * ix;
    const float ty0 = (g.lo[1] - p.y) * iy, ty1 = (g.hi[1] - p.y) * iy;
    const float tz0 = (g.lo[2] - p.z) * iz, tz1 = (g.hi[2] - p.z) * iz;
    t0 = fmaxf(fmaxf(fminf(tx0, tx1), fminf(ty0, ty1)), fmaxf(fminf(tz0, tz1), 0.0f));
    t1 = fminf(fminf(fmaxf(tx0, tx1), fmaxf(ty0, ty1)), fminf(fmaxf(tz0, tz1), L));
    auto at = [&](float2 t) {
      return field_point2<kShared>(s, f, {fma2(dup2(d.x), t, dup2(p.x)),
                                          fma2(dup2(d.y), t, dup2(p.y)),
                                          fma2(dup2(d.z), t, dup2(p.z))});
    };
#pragma unroll
    for (int it = 0; it < 2; ++it) {
      const float2 w = at(make_float2(t0, t1)).w;
      t0 = fmaf(w.x, s.cell, t0);
      t1 = fmaf(-w.y, s.cell, t1);
    }
    // the ball test on each half of what is left
    const float h = 0.25f * fmaxf(t1 - t0, 0.0f), mid = fmaf(2.0f, h, t0);
    const FieldPoint2 m = at(make_float2(t0 + h, t1 - h));
    const float r = fmaf(h, s.r_scale, s.r_slack);
    const bool clear0 = fmaf(m.w.x, m.w.x, m.q.x) > r * r;
    const bool clear1 = fmaf(m.w.y, m.w.y, m.q.y) > r * r;
    t0 = clear0 ? mid : t0;
    t1 = clear1 ? (clear0 ? -1.0f : mid) : t1;
    t0 = fmaxf(t0 - kClipSlack, 0.0f);
    t1 = fminf(t1 + kClipSlack, L);
    keep = t0 < t1;
  }
  const unsigned m = __ballot_sync(0xffffffffu, keep);
  if (keep) {
    const int dst = n2 + __popc(m & ((1u << lane) - 1u));
    q.clip_a[dst] = ea;
    q.clip_b[dst] = eb;
    q.clip_t[dst] = make_float2(t0, t1);
  }
  __syncwarp();
  return n2 + __popc(m);
}

// Test the clipped entries [base, base + c) (c <= 32) by the grid DDA over their
// intervals.  The pass lasts as long as its longest walk, so the 32 - c spare
// lanes go to the long intervals (the longest of 25 walks crossed 19 cells, the
// mean one 3): an entry of length l is cut into
// 1 + floor(l / (total / (32 - c))) equal pieces, overlapping by the clip slack,
// one lane each.  The earliest (step, target) per photon wins via a shared
// atomicMin on the key (step << 16 | target).  Returns whether there was a hit.
template <bool P>
__device__ __forceinline__ bool test_queue(WarpQueue& q, int base, int c,
                                           const GridDev& g, const uint32_t* cells,
                                           const uint16_t* items, const float4* sph, int lane) {
  // pieces of this lane's entry, in units of 1/64 m so that the sums are exact
  float2 iv = make_float2(0.0f, 0.0f);
  if (lane < c) iv = q.clip_t[base + lane];
  const unsigned units = (unsigned)(fminf(iv.y - iv.x, 1e6f) * 64.0f);
  const unsigned total = __reduce_add_sync(0xffffffffu, units);
  // (0.9999: the floors' sum stays at most 32 - c under rounding)
  const float per = 0.9999f * (float)(32 - c) * ftz_rcp((float)max(total, 1u));
  const int n = lane < c ? 1 + (int)((float)units * per) : 0;
  int end = n;  // inclusive scan
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, end, o);
    if (lane >= o) end += v;
  }
  // this lane's entry: the last whose first piece is at or before the lane
  const unsigned starts =
      __reduce_or_sync(0xffffffffu, lane < c ? 1u << (end - n) : 0u) & (0xffffffffu >> (31 - lane));
  const int el = __popc(starts) - 1;
  const int m = __shfl_sync(0xffffffffu, n, el);
  const int piece = lane - (31 - __clz(starts));
  const int e = base + el;
  int j = -1;
  if (piece < m) {
    const float4 ea = q.clip_a[e], eb = q.clip_b[e];
    const float2 t = q.clip_t[e];
    const float w = (t.y - t.x) * ftz_rcp((float)m);
    const float ta = piece == 0 ? t.x : fmaxf(fmaf((float)piece, w, t.x) - kClipSlack, t.x);
    const float tb =
        piece == m - 1 ? t.y : fminf(fmaf((float)(piece + 1), w, t.x) + kClipSlack, t.y);
    j = first_hit<P>(g, cells, items, sph, make_float3(ea.x, ea.y, ea.z),
                     make_float3(eb.x, eb.y, eb.z), ea.w, ta, tb);
    if (j >= 0) {
      const uint32_t meta = __float_as_uint(eb.w);
      atomicMin(&q.key[meta & (kGroup - 1u)], ((meta >> 8) << 16) | (uint32_t)j);
    }
  }
  __syncwarp();
  return __any_sync(0xffffffffu, j >= 0);
}

// Append one hit: one atomic per warp for all lanes that record in this pass;
// the record is written as five 16-byte stores in pp_hit_record's order.
__device__ __forceinline__ void record_hit(const LaunchArgs& a, float3 pos, float wl, float3 dir,
                                           float dist, float3 idir, float abs_w, double time,
                                           long long photon, int module_index, int n_steps,
                                           int source_index, bool* overflowed) {
  const unsigned act = __activemask();
  const int lane = threadIdx.x & 31;
  const int leader = __ffs(act) - 1;
  const unsigned rank = __popc(act & ((1u << lane) - 1u));
  unsigned long long base = 0;
  if (lane == leader) base = atomicAdd(u64(&a.counters->n_hits), (unsigned long long)__popc(act));
  base = __shfl_sync(act, base, leader);
  const unsigned long long slot = base + rank;
  if (slot < a.capacity) {
    float4* r = reinterpret_cast<float4*>(a.hits + slot);
    r[0] = make_float4(pos.x, pos.y, pos.z, wl);
    r[1] = make_float4(dir.x, dir.y, dir.z, __int_as_float(module_index));
    r[2] = make_float4(dist, idir.x, idir.y, idir.z);
    r[3] = make_float4(abs_w, __int_as_float(n_steps), __int_as_float(source_index), 0.0f);
    reinterpret_cast<double2*>(r)[4] = make_double2(time, __longlong_as_double(photon));
  } else {
    atomicOr(&a.counters->err_flags, (unsigned)PP_FLAG_OVERFLOW);
    *overflowed = true;
  }
}

// Initial state of photon p of source s (initialize_photon_state,
// src/photon_prop_cuda.jl:158-276): position, direction, emission time,
// wavelength and the medium at that wavelength {sca_len, v_group, abs_len,
// n}.  Deterministic in (p, s), so the step loop keeps only what it needs and
// the few photons that hit recompute the rest when their hit is recorded.
struct PhotonInit {
  float3 pos, dir;
  float t0, wl;
  float4 med;
};

template <bool kPrecise>
__device__ __forceinline__ PhotonInit init_photon(const LaunchArgs& a, int s, uint32_t plo,
                                                  uint32_t phi) {
  const pp_source* sp = a.sources + s;
  const int kind = __ldg(&sp->kind);
  const float3 spos = make_float3(__ldg(&sp->position[0]), __ldg(&sp->position[1]),
                                  __ldg(&sp->position[2]));
  const float3 saxis = make_float3(__ldg(&sp->direction[0]), __ldg(&sp->direction[1]),
                                   __ldg(&sp->direction[2]));
  const float stime = __ldg(&sp->time);
  const uint4 r0 = philox(make_uint4(plo, phi, 0u, (uint32_t)s), a.round_keys);
  const float u0 = u01(r0.x), u1 = u01(r0.y), u2 = u01(r0.z), u3 = u01(r0.w);
  const float wl = a.spectrum ? spectrum_sample(a.spectrum, a.n_spectrum, u0)
                              : a.mono_wavelength;
  const float4 med = medium_at(a.medium, a.n_medium, a.med_wl_min, a.med_inv_step, wl);

  // ---- initial state (initialize_photon_state) ----
  float3 pos = spos, dir;
  float t0 = stime;
  switch (kind) {
    case PP_SRC_POINTLIKE_ISOTROPIC:
    case PP_SRC_POINTLIKE_TIME_RANGE:
      dir = dir_from_cos<kPrecise>(uniform_ab(-1.0f, 1.0f, u1), u2);
      if (kind == PP_SRC_POINTLIKE_TIME_RANGE)
        t0 = uniform_ab(stime, __ldg(&sp->time_end), u3);
      break;
    case PP_SRC_COLLIMATED_ISOTROPIC:
      dir = dir_from_cos<kPrecise>(uniform_ab(__ldg(&sp->cut_angle_cos), 1.0f, u2), u1);
      break;
    case PP_SRC_PENCIL: {
      const float div = __ldg(&sp->beam_divergence);
      dir = div > 0.0f ? rot_from_ez<kPrecise>(
                             saxis, sph_to_cart<kPrecise>(
                                        f_sqrt<kPrecise>(uniform_ab(0.0f, div * div, u1)), u2))
                       : saxis;
      break;
    }
    case PP_SRC_AXICONE: {
      float th = __ldg(&sp->angle);
      const float div = __ldg(&sp->beam_divergence);
      if (div > 0.0f) {
        float cs;
        if (kPrecise) {
          cs = cosf(kTwoPi * u3);
        } else {
          float sn;
          f_sincos_2pi<false>(u3, &sn, &cs);
        }
        th += f_sqrt<kPrecise>(-2.0f * f_log<kPrecise>(u2)) * cs * div;
      }
      dir = rot_from_ez<kPrecise>(saxis, sph_to_cart<kPrecise>(th, u1));
      break;
    }
    case PP_SRC_EXTENDED_CHERENKOV:
    case PP_SRC_EXTENDED_CHERENKOV_NOSMEAR:
    case PP_SRC_POINTLIKE_CHERENKOV:
    case PP_SRC_CHERENKOV_TRACK: {
      float along = 0.0f;
      if (kind == PP_SRC_EXTENDED_CHERENKOV || kind == PP_SRC_EXTENDED_CHERENKOV_NOSMEAR) {
        along = gamma_sample<kPrecise>(__ldg(&sp->long_a), 1.0f / __ldg(&sp->long_b), plo, phi,
                                       (uint32_t)s, a.key0, a.key1) *
                __ldg(&sp->long_lrad);
      } else if (kind == PP_SRC_CHERENKOV_TRACK) {
        const uint4 re = philox(make_uint4(plo, phi, kExtraCall, (uint32_t)s), a.round_keys);
        along = uniform_ab(0.0f, __ldg(&sp->length), u01(re.x));
      }
      if (kind != PP_SRC_POINTLIKE_CHERENKOV) {
        pos = make_float3(spos.x + along * saxis.x, spos.y + along * saxis.y,
                          spos.z + along * saxis.z);
        t0 = stime + along / kCVac;
      }
      dir = cherenkov_dir<kPrecise>(
          saxis, med.w, u1, u2, u3, kind != PP_SRC_EXTENDED_CHERENKOV_NOSMEAR,
          a.track + (size_t)__ldg(&sp->smear_table) * (size_t)a.n_track, a.n_track);
      break;
    }
    default:
      dir = make_float3(0.0f, 0.0f, 1.0f);
      break;
  }

  PhotonInit in;
  in.pos = pos;
  in.dir = kPrecise ? dir : renormalise(dir);
  in.t0 = t0;
  in.wl = wl;
  in.med = med;
  return in;
}

// Where photons that have hit go on (m): outside every safety field by more than any
// step is long, and with a square that FP32 holds in units of any node spacing.
constexpr float kFarAway = 1e12f;

// The step lengths of the two photons from their first random words.
template <bool kPrecise>
__device__ __forceinline__ float2 step_lengths(uint32_t w0, uint32_t w1, float2 sca_len) {
  if constexpr (kPrecise)
    return make_float2(-f_log<true>(u01(w0)) * sca_len.x, -f_log<true>(u01(w1)) * sca_len.y);
  else
    return mul2(mul2(make_float2(ftz_lg2(u01(w0)), ftz_lg2(u01(w1))), dup2(-0.693147182f)),
                sca_len);
}

// An emission direction nearer to the z axis than FP32 can square counts as on
// it, exactly, so that the step's rotation divides nothing by zero.
__device__ __forceinline__ float3 on_axis(float3 d) {
  return fmaf(d.y, d.y, d.x * d.x) < 1.17549435e-38f ? make_float3(0.0f, 0.0f, d.z) : d;
}

// The two photons' state, moved over one step.
struct Walk2 {
  Vec2 pos, dir;
  float2 dist, comp;  // Kahan-compensated path lengths
};
template <bool kPrecise>
__device__ __forceinline__ void advance(const PhaseDev& ph, Walk2& w, float2 step, const uint4& r0,
                                        const uint4& r1) {
  if constexpr (kPrecise) {
    const float3 q0 = first(w.pos), q1 = second(w.pos), e0 = first(w.dir), e1 = second(w.dir);
    w.pos = both(make_float3(madd<true>(e0.x, step.x, q0.x), madd<true>(e0.y, step.x, q0.y),
                             madd<true>(e0.z, step.x, q0.z)),
                 make_float3(madd<true>(e1.x, step.y, q1.x), madd<true>(e1.y, step.y, q1.y),
                             madd<true>(e1.z, step.y, q1.z)));
  } else {
    w.pos = {fma2(w.dir.x, step, w.pos.x), fma2(w.dir.y, step, w.pos.y),
             fma2(w.dir.z, step, w.pos.z)};
  }
  const float2 y = sub2(step, w.comp), t = add2(w.dist, y);
  w.comp = sub2(sub2(t, w.dist), y);
  w.dist = t;
  if constexpr (kPrecise)
    w.dir = both(update_direction_precise(ph, first(w.dir), r0.y, r0.z, r0.w),
                 update_direction_precise(ph, second(w.dir), r1.y, r1.z, r1.w));
  else
    w.dir = update_direction_fast(ph, w.dir, make_uint2(r0.y, r1.y), make_uint2(r0.z, r1.z),
                                  make_uint2(r0.w, r1.w));
}

// Shaped targets: test the step segments of a lane's two photons (those that are
// open) against every target in index order and keep a photon's first hit, which
// closes it; a list of detector lines is searched line by line
// (src/photon_prop_cuda.jl:611-634): the 2-D test of the line, then its modules;
// the first crossed line ends the search.  Both photons take one pass over the
// list.  Horizontal shapes: shape_hit in packed operations, each half rounding as it
// does (1e6 photons, 20 discs of 50 m: 284 us with one photon per lane, 397 with a
// wider packed test before shape_hit, 283 now; 50 discs of 2 m: 1,270, 1,342 and
// 828).  Spheres and lines: packed operations decide first whether sphere_hit can
// succeed, the discriminant being below zero by no more than the rounding of either
// form (at most 1.5e-6 of the squared distance q).  1e7 photons, 400 spheres: 68 ms
// with one photon per lane, 97 with sphere_hit for one photon after the other, 54 now.
template <bool kPrecise>
__device__ __forceinline__ void search_shapes(const LaunchArgs& a, const Vec2& p, const Vec2& v,
                                              float2 steps, float2 dist0, uint32_t k,
                                              uint32_t* key, WarpBest& best, int lane,
                                              bool (&open)[2]) {
  const float3 pos[2] = {first(p), second(p)}, dir[2] = {first(v), second(v)};
  const float step[2] = {steps.x, steps.y};
  bool search[2] = {open[0], open[1]};
  int hit[2] = {-1, -1};  // 0-based module index to report
  float d[2] = {0.0f, 0.0f};
  int line_no = 0;
  // 1 / v.z as shape_hit's division takes it; in the replay variant, which divides, a
  // value that makes the way to a shape's height no longer than it is
  float2 rz;
  if constexpr (kPrecise)
    rz = make_float2(1.0f / copysignf(fmaxf(fabsf(v.z.x), 1e-30f), v.z.x),
                     1.0f / copysignf(fmaxf(fabsf(v.z.y), 1e-30f), v.z.y));
  else
    rz = make_float2(f_rcp<false>(v.z.x), f_rcp<false>(v.z.y));
  for (int j = 0; j < a.n_shapes && (search[0] || search[1]); ++j) {
    const float4 s = __ldg(a.shapes + 2 * j), h = __ldg(a.shapes + 2 * j + 1);
    const int kind = __float_as_int(h.y);
    const float2 dz = sub2(p.z, dup2(s.z));
    bool near0, near1;
    if (kind == PP_TARGET_SPHERE || kind == PP_TARGET_LINE) {
      const float2 dx = sub2(p.x, dup2(s.x)), dy = sub2(p.y, dup2(s.y));
      float2 c = fma2(v.x, dx, mul2(v.y, dy)), q = fma2(dx, dx, mul2(dy, dy));
      if (kind == PP_TARGET_SPHERE) {
        c = fma2(v.z, dz, c);
        q = fma2(dz, dz, q);
      }
      const float2 b = fma2(q, dup2(4e-6f), fma2(c, c, sub2(dup2(s.w), q)));
      near0 = b.x >= 0.0f;
      near1 = b.y >= 0.0f;
    } else {  // a horizontal shape: the way to its height is in the segment
      const float2 t = mul2(sub2(dup2(s.z), p.z), rz);
      if constexpr (kPrecise) {
        near0 = !(t.x < 0.0f || t.x > step[0] * 1.00001f);
        near1 = !(t.y < 0.0f || t.y > step[1] * 1.00001f);
      } else {  // and, rounding as in shape_hit, ends in the shape
        const float2 x = sub2(fma2(v.x, t, p.x), dup2(s.x));
        const float2 y = sub2(fma2(v.y, t, p.y), dup2(s.y));
        if (kind == PP_TARGET_RECTANGLE) {
          near0 = fabsf(x.x) < s.w && fabsf(y.x) < h.x;
          near1 = fabsf(x.y) < s.w && fabsf(y.y) < h.x;
        } else {
          const float2 r2 = add2(mul2(x, x), mul2(y, y));
          near0 = r2.x < s.w;
          near1 = r2.y < s.w;
        }
        near0 = near0 && !(t.x < 0.0f || t.x > step[0]);
        near1 = near1 && !(t.y < 0.0f || t.y > step[1]);
      }
    }
    if (near0 || near1) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        if (!(search[i] && (i ? near1 : near0))) continue;
        if (kind == PP_TARGET_LINE) {
          float dl;
          if (!sphere_hit<kPrecise>(s, make_float3(pos[i].x, pos[i].y, 0.0f),
                                    make_float3(dir[i].x, dir[i].y, 0.0f), step[i], &dl))
            continue;
          search[i] = false;
          const int nm = __float_as_int(h.x);
          for (int m = 1; m <= nm; ++m) {
            if (shape_hit<kPrecise>(a.shapes, j + m, pos[i], dir[i], step[i], &d[i])) {
              hit[i] = m + nm * (line_no + 1) - 1;
              break;
            }
          }
        } else if (shape_hit<kPrecise>(a.shapes, j, pos[i], dir[i], step[i], &d[i])) {
          hit[i] = j;
          search[i] = false;
        }
      }
    }
    if (kind == PP_TARGET_LINE) {
      ++line_no;
      j += __float_as_int(h.x);
    }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    if (hit[i] < 0) continue;
    open[i] = false;
    const int own = lane + 32 * i;
    key[own] = (k << 16) | (uint32_t)hit[i];
    best.hx[own] = madd<kPrecise>(dir[i].x, d[i], pos[i].x);
    best.hy[own] = madd<kPrecise>(dir[i].y, d[i], pos[i].y);
    best.hz[own] = madd<kPrecise>(dir[i].z, d[i], pos[i].z);
    best.ox[own] = dir[i].x;
    best.oy[own] = dir[i].y;
    best.oz[own] = dir[i].z;
    best.dist[own] = (i ? dist0.y : dist0.x) + d[i];
  }
}

// What a hit's record needs: the emission again, and the hit itself.
struct Hit {
  PhotonInit in;
  float3 pos, dir;
  float dist;
};

// The hit of photon (plo, phi) of source s in step k on the sphere `target`,
// from the photon's random numbers: its steps are taken again up to that one
// (as both photons of a pair, through the functions of the step loop, so the
// same values bit for bit).  A call for the few photons that hit -- 1e-4 of them
// in the 400-module detector -- keeps the emission data out of the step loop's
// registers and the path length and hit points out of the queue: 5.8 instead of
// 8.2 KB of shared memory a warp, the rest is L1.  With entries of whole float4s:
// 14.19 -> 13.56 ms per 1e8 photons.
template <bool kPrecise>
__device__ __noinline__ void replay_hit(const LaunchArgs& a, int s, uint32_t plo, uint32_t phi,
                                        int k_hit, float4 target, Hit* out) {
  const PhotonInit in = init_photon<kPrecise>(a, s, plo, phi);
  const PhiloxPhoton ph = philox_photon(plo, (uint32_t)s, a.round_keys);
  const float3 d0 = on_axis(in.dir);
  Walk2 w = {both(in.pos, in.pos), both(d0, d0), dup2(0.0f), dup2(0.0f)};
  float2 step;
#pragma unroll 1
  for (int k = 1;; ++k) {
    const uint4 r = philox_words(ph, philox_step((uint32_t)k, phi, a.round_keys), a.round_keys);
    step = step_lengths<kPrecise>(r.x, r.x, dup2(in.med.x));
    if (k >= k_hit) break;
    advance<kPrecise>(a.phase, w, step, r, r);
  }
  const float3 pos = first(w.pos), dir = first(w.dir);
  float d = 0.0f;
  sphere_hit<kPrecise>(target, pos, dir, step.x, &d);
  out->in = in;
  out->pos = make_float3(madd<kPrecise>(dir.x, d, pos.x), madd<kPrecise>(dir.y, d, pos.y),
                         madd<kPrecise>(dir.z, d, pos.z));
  out->dir = dir;
  out->dist = (w.dist.x - w.comp.x) + d;
}

// Photon i of source s: its number and the source.
struct PhotonId {
  int s;
  uint32_t lo, hi;
};
// Last s in [0, n) with prefix[s] <= i.
__device__ __forceinline__ int owner_of(const unsigned long long* __restrict__ prefix, int n,
                                        unsigned long long i) {
  int lo = 0, hi = n;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (__ldg(prefix + mid) <= i) lo = mid; else hi = mid;
  }
  return lo;
}
// Photon i of all sources' photons in order (mixed groups).
__device__ __forceinline__ PhotonId photon_of_all(const LaunchArgs& a, unsigned long long i) {
  const int s = owner_of(a.chunk_prefix, a.n_src, i);
  const unsigned long long p =
      (unsigned long long)__ldg(&a.sources[s].first_photon) + (i - __ldg(a.chunk_prefix + s));
  return {s, (uint32_t)p, (uint32_t)(p >> 32)};
}

// kShapes: shaped targets (a.shapes), every target tested at every step in
// index order (no grid, no deferred queue).
// kMixed: the photons of all sources are numbered one after the other
// (chunk_prefix holds photons), and a group takes 64 of them, of as many sources as they
// come from: for workloads of many sources of few photons, which would leave most of
// a group of one source's photons empty.
template <bool kPrecise, Tables kTables, bool kMixed>
__global__ void __launch_bounds__(small_ctas(kTables) ? kSmallThreads : kMaxBlockThreads,
                                  min_ctas(kTables))
    propagate_kernel(const __grid_constant__ LaunchArgs a) {
  constexpr bool kSmemGrid = kTables == Tables::kStaged, kShapes = kTables == Tables::kShapes;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(8) unsigned long long bar;

  const uint32_t* cells;
  const uint16_t* items;
  const float4* sph;
  const unsigned char* field;
  if (kSmemGrid) {
    if (!stage_tables(smem, a.blob, a.grid.blob_bytes, smem + a.safety_offset, a.safety,
                      a.sgrid.bytes, &bar, a.wait_limit_ns, a.skip_staging_copies != 0)) {
      atomicOr(&a.counters->err_flags, (unsigned)PP_FLAG_TIMEOUT);
      return;
    }
    cells = reinterpret_cast<const uint32_t*>(smem);
    items = reinterpret_cast<const uint16_t*>(smem + a.grid.off_items);
    sph = reinterpret_cast<const float4*>(smem + a.grid.off_spheres);
    field = smem + a.safety_offset;
  } else {
    cells = reinterpret_cast<const uint32_t*>(a.blob);
    items = reinterpret_cast<const uint16_t*>(a.blob + a.grid.off_items);
    sph = reinterpret_cast<const float4*>(a.blob + a.grid.off_spheres);
    field = a.safety;
  }
  const bool have_grid = a.grid.n_targets > 0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  WarpQueue& q = reinterpret_cast<WarpQueue*>(smem + a.state_offset)[warp];
  WarpBest& best = reinterpret_cast<WarpBest&>(q);  // shaped targets only
  const unsigned lanemask_lt = (1u << lane) - 1u;

  unsigned long long steps_acc = 0, sim_acc = 0;

  // The first chunk of every warp is its own, dealt out CTA by CTA so that a
  // small workload spreads over all SMs without a queue (1e5 photons: 45 -> 27
  // us); the others come from the queue.  (Asking for them one chunk ahead hides
  // nothing that the other warps do not: 13.19 against 13.15 ms per 1e8.)
  const unsigned long long n_warps = (unsigned long long)gridDim.x * a.warps_per_block;
  unsigned long long next = (unsigned long long)warp * gridDim.x + blockIdx.x;
  while (next < a.total_chunks) {
    const unsigned long long c = next;
    // The chunk's photons, of the source that owns it or of all.
    const int s = kMixed ? 0 : owner_of(a.chunk_prefix, a.n_src, c);
    const long long p0 =
        (long long)(kMixed ? c : c - __ldg(a.chunk_prefix + s)) * a.chunk_photons;
    const long long pend =
        min(p0 + (long long)a.chunk_photons,
            kMixed ? (long long)__ldg(a.chunk_prefix + a.n_src) : __ldg(a.src_photons + s));
    const long long first_photon = kMixed ? 0ll : __ldg(&a.sources[s].first_photon);

    int count;
    // A full hit buffer: a warp whose hits it did not take stops after this chunk, and so
    // does one that finds the flag now.  (Asking at the chunk's end, or at each group,
    // makes every warp wait for the counters' busy line: 13.08 -> 13.14 ms per 1e8.)
    bool full = false;
    unsigned stop = 0;
    if (lane == 0)
      stop = *reinterpret_cast<volatile unsigned*>(&a.counters->err_flags) & PP_FLAG_OVERFLOW;
    for (long long base = p0; base < pend; base += count) {
      // A group: up to 64 photons, lane l carrying the l-th and the (32 + l)-th; of one
      // source, all with the same high counter word.
      const long long pb = first_photon + base;
      count = (int)min(pend - base, (long long)kGroup);
      if (!kMixed) count = (int)min((long long)count, 0x100000000ll - (long long)(uint32_t)pb);
      auto photon = [&](int i) -> PhotonId {
        if (kMixed) return photon_of_all(a, (unsigned long long)(pb + i));
        return {s, (uint32_t)pb + (uint32_t)i, (uint32_t)((unsigned long long)pb >> 32)};
      };
      const bool active0 = lane < count, active1 = lane + 32 < count;
      // Lanes past the end replay the group's first photon (never recorded).
      const PhotonId id0 = photon(active0 ? lane : 0), id1 = photon(active1 ? lane + 32 : 0);
      Walk2 w;
      float2 sca_len;
#pragma unroll 1
      for (int j = 0; j < 2; ++j) {
        const PhotonInit in = init_photon<kPrecise>(a, kMixed && j ? id1.s : id0.s,
                                                    j ? id1.lo : id0.lo, kMixed && j ? id1.hi : id0.hi);
        if (j == 0) {
          w.pos.x.x = in.pos.x; w.pos.y.x = in.pos.y; w.pos.z.x = in.pos.z;
          const float3 d = on_axis(in.dir);
          w.dir.x.x = d.x; w.dir.y.x = d.y; w.dir.z.x = d.z;
          sca_len.x = in.med.x;
        } else {
          w.pos.x.y = in.pos.x; w.pos.y.y = in.pos.y; w.pos.z.y = in.pos.z;
          const float3 d = on_axis(in.dir);
          w.dir.x.y = d.x; w.dir.y.y = d.y; w.dir.z.y = d.z;
          sca_len.y = in.med.x;
        }
      }
      const PhiloxPhoton ph0 = philox_photon(id0.lo, (uint32_t)id0.s, a.round_keys);
      const PhiloxPhoton ph1 =
          philox_photon(id1.lo, (uint32_t)(kMixed ? id1.s : id0.s), a.round_keys);
      w.dist = dup2(0.0f);
      w.comp = dup2(0.0f);
      q.key[lane] = 0xffffffffu;
      q.key[lane + 32] = 0xffffffffu;
      __syncwarp();
      // heights of the raw and the clipped stack (warp-uniform)
      int n1 = 0, n2 = 0;
      bool open[2] = {active0, active1};  // shaped targets: the photon has not hit yet
      // The step loop holds neither the clip nor the walk: it stops when 32 raw
      // entries wait, they are clipped, 32 clipped ones are walked as soon as
      // they wait, and the loop resumes; after the last step the same code
      // takes what is left.
      int k = 1;
      while (true) {
        for (; k <= a.n_steps && n1 < 32; ++k) {
          const PhiloxStep pt0 = philox_step((uint32_t)k, id0.hi, a.round_keys);
          const PhiloxStep pt1 = kMixed ? philox_step((uint32_t)k, id1.hi, a.round_keys) : pt0;
          const uint4 r0 = philox_words(ph0, pt0, a.round_keys);
          const uint4 r1 = philox_words(ph1, pt1, a.round_keys);
          const float2 step = step_lengths<kPrecise>(r0.x, r1.x, sca_len);
          if constexpr (kShapes) {
            search_shapes<kPrecise>(a, w.pos, w.dir, step,
                                    make_float2(w.dist.x - w.comp.x, w.dist.y - w.comp.y),
                                    (uint32_t)k, q.key, best, lane, open);
            if (!__any_sync(0xffffffffu, open[0] || open[1])) break;
          } else {
            bool clear0, clear1;
            segments_clear<kSmemGrid>(a.sgrid, field, w.pos, w.dir, step, &clear0, &clear1);
            const bool need0 = have_grid && active0 && !clear0;
            const bool need1 = have_grid && active1 && !clear1;
            const unsigned m0 = __ballot_sync(0xffffffffu, need0);
            const unsigned m1 = __ballot_sync(0xffffffffu, need1);
            const uint32_t meta = (uint32_t)lane | ((uint32_t)k << 8);
            if (need0) {
              const int e = n1 + __popc(m0 & lanemask_lt);
              q.raw_a[e] = make_float4(w.pos.x.x, w.pos.y.x, w.pos.z.x, step.x);
              q.raw_b[e] = make_float4(w.dir.x.x, w.dir.y.x, w.dir.z.x, __uint_as_float(meta));
            }
            n1 += __popc(m0);
            if (need1) {
              const int e = n1 + __popc(m1 & lanemask_lt);
              q.raw_a[e] = make_float4(w.pos.x.y, w.pos.y.y, w.pos.z.y, step.y);
              q.raw_b[e] =
                  make_float4(w.dir.x.y, w.dir.y.y, w.dir.z.y, __uint_as_float(meta + 32u));
            }
            n1 += __popc(m1);
          }
          advance<kPrecise>(a.phase, w, step, r0, r1);
        }
        if (kShapes) break;
        __syncwarp();  // the raw entries are visible
        if (n1 > 0) {  // 32 wait, or the steps are done
          const int take = min(n1, 32);
          n1 -= take;
          n2 = clip_entries<kSmemGrid>(q, n1, take, n2, a.grid, a.sgrid, field, lane);
        }
        const bool last = k > a.n_steps && n1 == 0;
        if (n2 >= 32 || (last && n2 > 0)) {
          const int take = min(n2, 32);
          n2 -= take;
          const bool hits = test_queue<kPrecise>(q, n2, take, a.grid, cells, items, sph, lane);
          if (hits && !last) {
            // No later step of a photon with a hit: it goes on far from every target
            // (its hit is replayed), and the steps end when that is all of them.
            // Earlier steps may still wait.
            const bool hit0 = q.key[lane] != 0xffffffffu, hit1 = q.key[lane + 32] != 0xffffffffu;
            w.pos.x.x = hit0 ? kFarAway : w.pos.x.x;
            w.pos.x.y = hit1 ? kFarAway : w.pos.x.y;
            if (__all_sync(0xffffffffu, (hit0 || !active0) && (hit1 || !active1)))
              k = a.n_steps + 1;
          }
        }
        if (last && n2 == 0) break;
      }
      __syncwarp();

      constexpr uint32_t kNone = 0xffffffffu;
      const uint32_t key0 = active0 ? q.key[lane] : kNone;
      const uint32_t key1 = active1 ? q.key[lane + 32] : kNone;
      const bool hit0 = key0 != kNone, hit1 = key1 != kNone;
      if (active0) steps_acc += hit0 ? key0 >> 16 : (uint32_t)a.n_steps;
      if (active1) steps_acc += hit1 ? key1 >> 16 : (uint32_t)a.n_steps;
      sim_acc += (unsigned)active0 + (unsigned)active1;
      // The group's hits, gathered so that one lane takes each: a pass of replays lasts
      // as long as its latest hit, and 32 hits are one pass whichever photons have them.
      // (With this and the steps above: 5e6 photons beside a sphere that half of them
      // hit 1.09 -> 0.97 ms, 1e6 among 300 spheres of 3 m 0.52 -> 0.48, 1e8 in the
      // 400-module detector 13.15 -> 13.09.)
      const unsigned m0 = __ballot_sync(0xffffffffu, hit0), m1 = __ballot_sync(0xffffffffu, hit1);
      const int n_hit = __popc(m0) + __popc(m1);
      if (n_hit > 0) {
        int* list = reinterpret_cast<int*>(q.clip_t);  // (free, and past a WarpBest)
        if (hit0) list[__popc(m0 & lanemask_lt)] = lane;
        if (hit1) list[__popc(m0) + __popc(m1 & lanemask_lt)] = lane + 32;
        __syncwarp();
        for (int h = lane; h < n_hit; h += 32) {
          const int own = list[h];
          const uint32_t key = q.key[own];
          const PhotonId id = photon(own);
          const int steps_taken = (int)(key >> 16);
          Hit hit;
          if constexpr (kShapes) {
            hit.in = init_photon<kPrecise>(a, id.s, id.lo, id.hi);
            hit.pos = make_float3(best.hx[own], best.hy[own], best.hz[own]);
            hit.dir = make_float3(best.ox[own], best.oy[own], best.oz[own]);
            hit.dist = best.dist[own];
          } else {
            replay_hit<kPrecise>(a, id.s, id.lo, id.hi, steps_taken, sph[key & 0xffffu], &hit);
          }
          const float4 med = hit.in.med;
          const double time = (double)hit.in.t0 + (double)hit.dist / (double)med.y;
          const float abs_w = f_exp<kPrecise>(-f_div<kPrecise>(hit.dist, med.z));
          if (a.hist) {
            // arrival-time histogram of this source, weighted by absorption
            const float tres = (float)(time - (double)__ldg(a.hist_tgeo + id.s));
            const float u = log10f(fmaxf(tres + a.hist_t_offset, 1e-30f));
            const int bin = min(max((int)floorf((u - a.hist_log_lo) * a.hist_inv_log_width), 0),
                                a.hist_bins - 1);
            float* row = a.hist + (size_t)id.s * (size_t)(a.hist_bins + 1);
            atomicAdd(row, abs_w);
            atomicAdd(row + 1 + bin, abs_w);
            atomicAdd(u64(&a.counters->n_hits), 1ull);
          } else {
            bool overflowed = false;
            record_hit(a, hit.pos, hit.in.wl, hit.dir, hit.dist, hit.in.dir, abs_w, time,
                       (long long)(((unsigned long long)id.hi << 32) | id.lo),
                       (int)(key & 0xffffu) + 1, steps_taken, id.s, &overflowed);
            if (overflowed) {
              sim_acc -= 1;
              full = true;
            }
          }
        }
      }
      __syncwarp();  // the hits are read before the next group clears them
    }
    if (lane == 0) {
      next = n_warps < a.total_chunks ? n_warps + atomicAdd(u64(&a.counters->work_next), 1ull)
                                      : a.total_chunks;
      if (stop) next = a.total_chunks;
    }
    next = __shfl_sync(0xffffffffu, next, 0);
    if (__any_sync(0xffffffffu, full)) break;
  }

  // One atomic per CTA for each of the photon and step counters.
  __shared__ unsigned long long total_steps, total_sim;
  if (threadIdx.x == 0) total_steps = total_sim = 0ull;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    steps_acc += __shfl_xor_sync(0xffffffffu, steps_acc, o);
    sim_acc += __shfl_xor_sync(0xffffffffu, sim_acc, o);
  }
  __syncthreads();
  if (lane == 0) {
    atomicAdd(&total_steps, steps_acc);
    atomicAdd(&total_sim, sim_acc);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    atomicAdd(u64(&a.counters->photon_steps), total_steps);
    atomicAdd(u64(&a.counters->n_ph_sim), total_sim);
  }
}

template <bool P, bool kMixed>
const void* kernel_for(Tables t) {
  switch (t) {
    case Tables::kStaged:
      return reinterpret_cast<const void*>(&propagate_kernel<P, Tables::kStaged, kMixed>);
    case Tables::kGlobal:
      return reinterpret_cast<const void*>(&propagate_kernel<P, Tables::kGlobal, kMixed>);
    case Tables::kGlobalMany:
      return reinterpret_cast<const void*>(&propagate_kernel<P, Tables::kGlobalMany, kMixed>);
    default:
      return reinterpret_cast<const void*>(&propagate_kernel<P, Tables::kShapes, kMixed>);
  }
}
template <bool P>
const void* kernel_ptr(Tables t, bool mixed) {
  return mixed ? kernel_for<P, true>(t) : kernel_for<P, false>(t);
}

}  // namespace
}  // namespace pp
