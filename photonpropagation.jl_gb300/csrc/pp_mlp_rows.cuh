// pp_mlp_rows.cuh -- the training step of the surrogate in three kernels.
//
// A step used to be a chain of some 25 kernels (a GEMM per layer and direction,
// column sums, loss, gather, zeroing, Adam, ...), 7.6 us each on average, every
// one bound by its own latency: 190 us for 10.9 GFLOP at batch 8192.  The forward
// pass, the loss and the backward pass through the activations need nothing
// from other rows, so one kernel takes a CTA's 64 rows through all of them
// (rows_kernel), a second one reduces all layers' weight and bias gradients
// over the rows (dw_kernel), and a third is Adam.
//
// Layouts.  Every operand is written once in the core-matrix order in which the
// tensor core reads it (pp_tc.cuh), so that each is fetched as it stands:
//   * weights, twice (pack_offset): wf, K-major over the layer's input, for the
//     forward pass, and wb, the transposed product's operand, for the backward
//     pass; each as blocks of all of N x 64 of K;
//   * inputs, activations and pre-activations' gradients in blocks of 64 rows as
//     rows_kernel multiplies them from shared memory, K-major (pptc::core_offset):
//     one bulk store each; the weight gradients, whose K is the rows, read the
//     same core matrices MN-major.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "pp_device.cuh"
#include "pp_tc.cuh"

namespace pprows {

using bf16 = __nv_bfloat16;
constexpr int kMaxLayers = 17;
constexpr int kRows = 64;                        // rows per CTA (tcgen05 M)
constexpr int kChunk = 64;                       // K columns per weight chunk
constexpr uint32_t kSlotBytes = 256u * kChunk * 2u;
constexpr int kEpiThreads = 512;                 // 16 warps, 4 per TMEM lane quarter
constexpr int kRowsThreads = kEpiThreads + 64;   // + MMA issuer + weight producer
constexpr uint32_t kTileBytes = 64u * 128u * 2u;
constexpr int kColStride = 136;  // 8 rows of float2 in different banks
constexpr uint32_t kBatchTag = 0x42415443u;      // Philox counter word of the batch stream

// ---- layouts --------------------------------------------------------------------
// Element (n, k) of an N x K operand in blocks of 64 columns (the last may be
// narrower): its byte offset.
__host__ __device__ inline uint32_t pack_offset(int n, int k, int N, int K) {
  const int j = k / kChunk, kk = k % kChunk;
  const int kw = K - j * kChunk < kChunk ? K - j * kChunk : kChunk;
  return (uint32_t)(j * N * kChunk * 2 +
                    (((n >> 3) * (kw >> 3) + (kk >> 3)) * 128 + (kk & 7) * 2 + (n & 7) * 16));
}
// The backward operand of a weight matrix W[o][i]: n = i, k = o, with eight
// neighbouring i in a core matrix's row.
__host__ __device__ inline uint32_t pack_offset_t(int n, int k, int N, int K) {
  const int j = k / kChunk, kk = k % kChunk;
  const int kw = K - j * kChunk < kChunk ? K - j * kChunk : kChunk;
  return (uint32_t)(j * N * kChunk * 2 +
                    (((n >> 3) * (kw >> 3) + (kk >> 3)) * 128 + (kk & 7) * 16 + (n & 7) * 2));
}
// What a replayed step reads from device memory, so that one captured graph
// serves every run: Adam steps taken, the schedule, the batch stream's key.
struct TrainCtl {
  long long step, step0, total;
  float lr0, lr1;
  uint32_t key0, key1;
};

struct RowsParams {
  // the batch: rows 0 .. B - 1 of x, count, hist, or (n_table > 0) B rows drawn
  // from n_table by Philox (i, Adam step, tag) under ctl's key
  const float *x, *count, *hist;
  long long n_table;
  const TrainCtl* ctl;
  int B, n_in, in_pad, hidden, n_layers, out_pad, n_bins;
  float inv_b, time_weight;
  const unsigned char *wf, *wb;
  uint32_t wf_off[kMaxLayers], wb_off[kMaxLayers];
  const float* bias[kMaxLayers];
  // 64-row blocks; layer l of y and z at l * layer_bytes.  z: pre-activations in
  // rows_kernel's own order, and over them, once a CTA has read them, their gradients
  unsigned char *x0, *y, *z, *dout;
  size_t layer_bytes;
  float *gbias, *loss;                    // the head's bias gradient, the batch loss
  uint32_t act_bytes;                     // one activation buffer
  unsigned* err;
  unsigned long long wait_ns;
};

// Job n of a CTA: the matrix product that all roles work on next.
//   0 .. L - 1   forward through hidden layer n
//   L            head
//   L + 1        gradient of the last hidden layer's pre-activations
//   L + 2 .. 2 L gradient of layer (2 L - n)'s
struct Job {
  int K, N;
  const unsigned char* w;
};
template <int kHidden>
__device__ __forceinline__ Job job_of(const RowsParams& p, int n) {
  const int L = p.n_layers;
  Job j;
  j.K = n == 0 ? p.in_pad : (n == L + 1 ? p.out_pad : p.hidden);
  j.N = n == L ? p.out_pad : kHidden;
  j.w = n <= L ? p.wf + p.wf_off[n] : p.wb + p.wb_off[2 * L + 1 - n];
  return j;
}
// where job n's A operand, K columns of a CTA's rows, is kept for dw_kernel
// (n == 2 L + 1: the last job's result)
__device__ __forceinline__ unsigned char* operand_home(const RowsParams& p, int n, int K) {
  const int L = p.n_layers;
  unsigned char* base = n == 0       ? p.x0
                        : n <= L     ? p.y + (size_t)(n - 1) * p.layer_bytes
                        : n == L + 1 ? p.dout
                                     : p.z + (size_t)(2 * L + 1 - n) * p.layer_bytes;
  return base + (size_t)blockIdx.x * (size_t)(kRows * K * 2);
}
__device__ __forceinline__ void bulk_store(void* dst, uint32_t src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(src),
               "r"(bytes)
               : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
// Until every store so far has read its shared memory, or is complete.
__device__ __forceinline__ void bulk_stores_read() {
  asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}
__device__ __forceinline__ void bulk_stores_done() {
  asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes,
                                          uint64_t* bar) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(
                   pptc::smem_u32(bar)),
               "r"(bytes)
               : "memory");
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          dst),
      "l"(src), "r"(bytes), "r"(pptc::smem_u32(bar))
      : "memory");
}
// Loads of many small pieces go through cp.async of 16 bytes per thread: bulk copies
// of 2 KB each bring 21 bytes per clock and SM, whatever the number of SMs.
__device__ __forceinline__ void fetch16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void fetch_commit() {
  asm volatile("cp.async.commit_group;" ::: "memory");
}
// Until all but this thread's last N groups have landed, for the tensor core.
template <int N>
__device__ __forceinline__ void fetch_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
  pptc::fence_async_smem();
}

// The accumulator of an M = 64 product: row 16 i + j is TMEM lane 32 i + j.  A
// warp's 16x256b load of 8 columns gives each thread four values: columns
// 2 (lane % 4), + 1 of row lane / 4, then of row lane / 4 + 8.
__device__ __forceinline__ void tmem_ld_8(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x1.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_ld_16(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
                 "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
// A read-only load that stays where it is written: before a wait.
__device__ __forceinline__ float ld_early_if(const float* p, bool in) {  // or 0
  float v;
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\tmov.f32 %0, 0f00000000;\n\t"
      "@p ld.global.nc.f32 %0, [%1];\n\t}"
      : "=f"(v)
      : "l"(p), "r"((uint32_t)in));
  return v;
}
__device__ __forceinline__ float2 ld_early2(const float* p) {
  float2 v;
  asm volatile("ld.global.nc.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
  return v;
}

__device__ __forceinline__ void epi_sync() {
  asm volatile("bar.sync 1, %0;" ::"n"(kEpiThreads) : "memory");
}
__device__ __forceinline__ uint32_t bf16x2(float lo, float hi) { return pptc::bf16x2_from(lo, hi); }
__device__ __forceinline__ float bf16_lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }

// One CTA takes 64 rows of the batch through the forward pass, the loss and the
// backward pass through the activations.  One warp streams the weights into
// slots of 32 KB, one issues the MMAs and stores the operands that dw_kernel needs,
// 16 do the epilogues; two accumulators and two activation buffers alternate, and
// each 64-column chunk of a layer's input starts its MMAs when its epilogue is done,
// so that all but a layer's last chunk run under the epilogue before them.  Bound: the
// serial chain of 2 L + 1 products, epilogue and MMA latency: 25 us for 4 x 256, at
// batch 1024 (16 CTAs) as at 8192 (128).  With 128 rows per CTA, halves of a layer
// and one thread's waits between the MMAs it took 40 us, on 64 SMs.
template <int kHidden>
__global__ void __launch_bounds__(kRowsThreads, 1)
    rows_kernel(const __grid_constant__ RowsParams p) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  extern __shared__ __align__(128) unsigned char smem[];
  constexpr int kParts = kHidden / kChunk;
  // chunk k of a job's input and of its weights
  __shared__ __align__(8) uint64_t go[kParts], w_full[kParts], w_empty[kParts], acc_full, epi_done, mma_done;
  __shared__ float4 red[4][kRows];  // the loss: partial results per column group,
  __shared__ __align__(16) float col_sum[32 * kColStride];  // the head's gradient of row pairs,
  __shared__ float row_loss[32];                            // and their loss
  __shared__ uint32_t tmem_slot;
  __shared__ volatile int abort_flag;
  __shared__ long long s_row[kRows];
  unsigned char* ring = smem + 2 * p.act_bytes;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int L = p.n_layers, n_jobs = 2 * L + 1;
  const int row0 = (int)blockIdx.x * kRows;
  constexpr uint32_t kAccCols = kHidden < 128 ? 128 : kHidden;  // also the head's columns
  if (warp == 0) pptc::tmem_alloc(&tmem_slot, 2 * kAccCols);
  if (threadIdx.x == 32) {
    for (int i = 0; i < kParts; ++i) {
      pptc::mbar_init(&go[i], kEpiThreads / 32);
      pptc::mbar_init(&w_full[i], 1);
      pptc::mbar_init(&w_empty[i], 1);
    }
    pptc::mbar_init(&acc_full, 1);
    pptc::mbar_init(&epi_done, kEpiThreads / 32);
    pptc::mbar_init(&mma_done, 1);
    abort_flag = 0;
  }
  // the table row of each batch row (-1 past the batch)
  if (threadIdx.x >= 64 && threadIdx.x < 64 + kRows) {
    const int i = row0 + (int)threadIdx.x - 64;
    long long src = i < p.B ? i : -1;
    if (p.n_table > 0 && src >= 0) {
      const unsigned long long t = (unsigned long long)(p.ctl->step + 1);
      const uint4 r = ppdev::philox(
          make_uint4((uint32_t)i, (uint32_t)t, (uint32_t)(t >> 32), kBatchTag),
          p.ctl->key0, p.ctl->key1);
      src = (long long)__umul64hi(((unsigned long long)r.x << 32) | r.y,
                                  (unsigned long long)p.n_table);
    }
    s_row[threadIdx.x - 64] = src;
  }
  pptc::fence_before_sync();
  __syncthreads();
  pptc::fence_after_sync();
  const uint32_t tmem = tmem_slot;
  bool ok = true;

  if (warp > kEpiThreads / 32) {
    // ---------------- weights: chunk k of a job goes to slot k
    if (lane == 0) {
      uint32_t uses[kParts];
#pragma unroll
      for (int k = 0; k < kParts; ++k) uses[k] = 0;
      for (int n = 0; n < n_jobs && ok; ++n) {
        const Job j = job_of<kHidden>(p, n);
#pragma unroll
        for (int k = 0; k < kParts; ++k) {
          if (k * kChunk >= j.K) break;
          ok = !abort_flag && pptc::mbar_wait(&w_empty[k], (uses[k] & 1) ^ 1, p.wait_ns);
          if (!ok) break;
          ++uses[k];
          bulk_load(pptc::smem_u32(ring + k * kSlotBytes),
                    j.w + (size_t)k * j.N * kChunk * 2,
                    (uint32_t)(j.N * min(kChunk, j.K - k * kChunk) * 2), &w_full[k]);
        }
      }
      if (!ok) abort_flag = 1;
      // every copy has landed before shared memory goes
#pragma unroll
      for (int k = 0; k < kParts; ++k)
        if (uses[k] > 0) pptc::mbar_wait(&w_full[k], (uses[k] - 1) & 1, p.wait_ns);
    }
    __syncwarp();
  } else if (warp == kEpiThreads / 32) {
    // ---------------- MMA issuer
    // The four MMAs of a chunk (64 x 256 x 16: 128 cycles each) run while this warp
    // works out the next chunk and tests its two barriers, if that takes less than
    // their 512 cycles; the warp stays converged, as descriptors in uniform
    // registers need no move each.
    const bool leader = lane == 0;
    uint32_t turns = 0;  // parity of chunk k's barriers, bit k
    const uint32_t act0 = pptc::smem_u32(smem);
    const uint32_t full0 = pptc::smem_u32(&w_full[0]), go0 = pptc::smem_u32(&go[0]);
    const uint64_t b0 = pptc::smem_desc(pptc::smem_u32(ring), 128, (kChunk / 8) * 128u);
    for (int n = 0; n < n_jobs && ok; ++n) {
      const Job j = job_of<kHidden>(p, n);
      const uint32_t act = act0 + (uint32_t)(n & 1) * p.act_bytes;
      const uint32_t idesc =
          pptc::idesc_bf16(kRows, j.N) | (n > L ? 1u << 16 : 0u);  // B transposed backward
      const uint32_t d = tmem + (uint32_t)(n & 1) * kAccCols;
      const int last = (j.K + kChunk - 1) / kChunk - 1, tail = j.K - last * kChunk;
      uint64_t a = pptc::smem_desc(act, 128, (uint32_t)(j.K / 8) * 128u), b = b0;
      uint32_t turn = turns;
      turns ^= (2u << last) - 1;
      for (int k = 0; k <= last; ++k) {
        const bool there = pptc::mbar_test2(full0 + k * 8, turn & 1, go0 + k * 8, turn & 1);
        if (!__all_sync(0xffffffffu, there)) {
          ok = __all_sync(0xffffffffu, !abort_flag &&
                                           pptc::mbar_wait(&w_full[k], turn & 1, p.wait_ns) &&
                                           pptc::mbar_wait(&go[k], turn & 1, p.wait_ns));
          if (!ok) break;
        }
        pptc::fence_after_sync();
        if (k < last || tail == kChunk) {
#pragma unroll
          for (int s = 0; s < kChunk / 16; ++s)
            pptc::mma_f16_by(leader, d, a + (uint64_t)(s * 16), b + (uint64_t)(s * 16), idesc,
                             k > 0 || s > 0);
        } else {
          const uint64_t bn = pptc::smem_desc(pptc::smem_u32(ring + k * kSlotBytes), 128,
                                              (uint32_t)(tail / 8) * 128u);
          for (int s = 0; s < tail / 16; ++s)
            pptc::mma_f16_by(leader, d, a + (uint64_t)(s * 16), bn + (uint64_t)(s * 16), idesc,
                             k > 0 || s > 0);
        }
        if (k == last) {
          // The epilogue of this job overwrites the previous job's operand, which
          // has been read; this job's own goes to memory meanwhile.
          if (leader) {
            bulk_stores_read();
            pptc::mma_commit(&acc_full);
            pptc::mma_commit(&w_empty[k]);
            bulk_store(operand_home(p, n, j.K), act, (uint32_t)(kRows * j.K * 2));
          }
          __syncwarp();
        } else {
          pptc::mma_commit_by(leader, &w_empty[k]);
        }
        a += kChunk;
        b += kSlotBytes / 16;
        turn >>= 1;
      }
    }
    if (ok) ok = __all_sync(0xffffffffu, pptc::mbar_wait(&epi_done, 0, p.wait_ns));
    if (lane == 0) {
      if (ok)
        bulk_store(operand_home(p, n_jobs, kHidden),
                   pptc::smem_u32(smem + (size_t)(n_jobs & 1) * p.act_bytes),
                   (uint32_t)(kRows * kHidden * 2));
      bulk_stores_done();
      pptc::mma_commit(&mma_done);
      if (!pptc::mbar_wait(&mma_done, 0, p.wait_ns)) ok = false;
      if (!ok) abort_flag = 1;
    }
    __syncwarp();
  } else {
    // ---------------- epilogues
    const int t = threadIdx.x;
    const int quad = warp & 3, cgrp = warp >> 2;
    const int ra = quad * 16 + (lane >> 2), cl = 2 * (lane & 3);  // rows ra, ra + 8
    auto arrive = [&](uint64_t* bar) {
      pptc::fence_async_smem();
      pptc::fence_before_sync();
      __syncwarp();
      if (lane == 0) pptc::mbar_arrive(bar);
    };
    // (after a wait that ran out the work goes on, on whatever is there: every
    // barrier below counts all warps)
    auto wait_acc = [&](int n) {
      if (!abort_flag && !pptc::mbar_wait(&acc_full, n & 1, p.wait_ns)) abort_flag = 1;
      __syncwarp();
      pptc::fence_after_sync();
    };
    // the inputs: BF16, zero past n_in and past the batch
    for (int u = t; u < kRows * (p.in_pad >> 3); u += kEpiThreads) {
      const int rr = u & (kRows - 1), g = u / kRows;
      const long long src = s_row[rr];
      float v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int c = g * 8 + i;
        v[i] = src >= 0 && c < p.n_in ? __ldg(p.x + src * p.n_in + c) : 0.0f;
      }
      const uint4 q = make_uint4(bf16x2(v[0], v[1]), bf16x2(v[2], v[3]), bf16x2(v[4], v[5]),
                                 bf16x2(v[6], v[7]));
      *reinterpret_cast<uint4*>(smem + pptc::core_offset(rr, g, p.in_pad)) = q;
    }
    arrive(&go[0]);
    for (int n = 0; n < n_jobs; ++n) {
      unsigned char* out = smem + (size_t)((n + 1) & 1) * p.act_bytes;
      const uint32_t acc = tmem + (uint32_t)(n & 1) * kAccCols + ((uint32_t)(quad * 32) << 16);
      if (n != L) {
        const bool fwd = n < L;
        const int l = fwd ? n : 2 * L - n;  // whose pre-activations, or their gradients
        // pre-activations, kept for this thread's own use later in the order in
        // which it holds them
        uint4* zt = reinterpret_cast<uint4*>(p.z + (size_t)l * p.layer_bytes +
                                             (size_t)blockIdx.x * (kRows * kHidden * 2)) + t;
        float2 bias[kParts][2];
        uint4 zq[kParts];
#pragma unroll
        for (int k = 0; k < kParts; ++k) {  // requested before the wait
          if (fwd) {
#pragma unroll
            for (int q = 0; q < 2; ++q)
              bias[k][q] = ld_early2(p.bias[l] + k * kChunk + cgrp * 16 + 8 * q + cl);
          } else {
            zq[k] = zt[k * kEpiThreads];
          }
        }
        wait_acc(n);
        uint32_t v[2][8];
        tmem_ld_16(acc + (uint32_t)(cgrp * 16), v[0]);
#pragma unroll
        for (int k = 0; k < kParts; ++k) {
          pptc::tmem_wait();
          if (k + 1 < kParts)
            tmem_ld_16(acc + (uint32_t)((k + 1) * kChunk + cgrp * 16), v[(k + 1) & 1]);
          uint32_t z[4] = {zq[k].x, zq[k].y, zq[k].z, zq[k].w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {  // 8-column block e / 2, row ra + 8 (e % 2)
            float2 x = make_float2(__uint_as_float(v[k & 1][2 * e]),
                                   __uint_as_float(v[k & 1][2 * e + 1]));
            const float2 half = make_float2(0.5f, 0.5f), one = make_float2(1.0f, 1.0f);
            if (fwd) {  // pptc::silu
              x = ppdev::add2(x, bias[k][e >> 1]);
              z[e] = bf16x2(x.x, x.y);
              x = ppdev::mul2(x, half);
              x = ppdev::fma2(x, make_float2(pptc::tanh_approx(x.x), pptc::tanh_approx(x.y)), x);
            } else {  // pptc::silu_grad
              const float2 zz = make_float2(bf16_lo(z[e]), bf16_hi(z[e]));
              float2 s = ppdev::mul2(zz, half);
              s = ppdev::fma2(half, make_float2(pptc::tanh_approx(s.x), pptc::tanh_approx(s.y)),
                              half);
              x = ppdev::mul2(x, ppdev::mul2(s, ppdev::fma2(zz, ppdev::sub2(one, s), one)));
            }
            *reinterpret_cast<uint32_t*>(
                out + pptc::core_offset(ra + 8 * (e & 1), k * 8 + cgrp * 2 + (e >> 1), kHidden) +
                2 * cl) = bf16x2(x.x, x.y);
          }
          // (the pre-activations are written and read: their place is the bulk store's)
          if (!fwd && k + 1 == kParts) asm volatile("fence.proxy.async.global;" ::: "memory");
          if (n + 1 < n_jobs) arrive(&go[k]);
          if (fwd) zt[k * kEpiThreads] = make_uint4(z[0], z[1], z[2], z[3]);
        }
      } else {
        // the loss: Poisson + multinomial negative log-likelihood of each row and
        // its gradient with respect to the head's outputs.  A thread has up to
        // four 8-column blocks, from column cb on, of its two rows.
        const int nb = p.n_bins, per = (p.out_pad / 8 + 3) / 4, cb = cgrp * per * 8;
        const int blocks = max(0, min(per, p.out_pad / 8 - cgrp * per));
        const long long src[2] = {s_row[ra], s_row[ra + 8]};
        // (Columns that are no bin get a logit of -1e38 and a count of 0, by which they
        // take no part: nothing below branches on them.)
        float hist[4][4], e[4][4];
        float2 bias[4];
        const float* row_hist[2] = {p.hist + max(src[0], 0ll) * nb - 1,
                                    p.hist + max(src[1], 0ll) * nb - 1};
#pragma unroll
        for (int q = 0; q < 4; ++q) {  // requested before the wait
          if (q < blocks) {
            const int c = cb + 8 * q + cl;
            const bool bin0 = c >= 1 && c <= nb, bin1 = c + 1 <= nb;
            bias[q] = ld_early2(p.bias[L] + c);
            hist[q][0] = ld_early_if(row_hist[0] + c, bin0 && src[0] >= 0);
            hist[q][1] = ld_early_if(row_hist[0] + c + 1, bin1 && src[0] >= 0);
            hist[q][2] = ld_early_if(row_hist[1] + c, bin0 && src[1] >= 0);
            hist[q][3] = ld_early_if(row_hist[1] + c + 1, bin1 && src[1] >= 0);
          }
        }
        const bool first = cgrp == 0 && cl == 0;  // has column 0, the expected count
        float k[2], o0[2], mx[2] = {-1e38f, -1e38f};
#pragma unroll
        for (int i = 0; i < 2; ++i) k[i] = ld_early_if(p.count + max(src[i], 0ll), first);
        wait_acc(n);
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (q < blocks)
            tmem_ld_8(acc + (uint32_t)(cb + 8 * q), reinterpret_cast<uint32_t*>(e[q]));
        pptc::tmem_wait();
        o0[0] = fminf(e[0][0] + bias[0].x, 30.0f);
        o0[1] = fminf(e[0][2] + bias[0].x, 30.0f);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          if (q < blocks) {
            const int c = cb + 8 * q + cl;
            const bool bin0 = c >= 1 && c <= nb, bin1 = c + 1 <= nb;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              e[q][i] = (i & 1 ? bin1 : bin0) ? e[q][i] + (i & 1 ? bias[q].y : bias[q].x) : -1e38f;
              mx[i >> 1] = fmaxf(mx[i >> 1], e[q][i]);
            }
          }
        }
        // Sums of a row's column group relative to the group's maximum (over four
        // threads), then of the row relative to its maximum.
        auto over_four = [&](float a) {
          a += __shfl_xor_sync(0xffffffffu, a, 1);
          return a + __shfl_xor_sync(0xffffffffu, a, 2);
        };
        float se[2] = {0.0f, 0.0f}, hs[2] = {0.0f, 0.0f}, hx[2] = {0.0f, 0.0f};
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 1));
          mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 2));
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          if (q < blocks) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float x = e[q][i] - mx[i >> 1];
              hs[i >> 1] += hist[q][i];
              hx[i >> 1] += hist[q][i] * x;
              e[q][i] = __expf(x);
              se[i >> 1] += e[q][i];
            }
          }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          se[i] = over_four(se[i]);
          hs[i] = over_four(hs[i]);
          hx[i] = over_four(hx[i]);
          if (cl == 0) red[cgrp][ra + 8 * i] = make_float4(mx[i], se[i], hs[i], hx[i]);
        }
        epi_sync();
        float gw[2], scale[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          float4 g[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) g[j] = red[j][ra + 8 * i];
          const float top = fmaxf(fmaxf(g[0].x, g[1].x), fmaxf(g[2].x, g[3].x));
          scale[i] = __expf(mx[i] - top);
          se[i] = hs[i] = hx[i] = 0.0f;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float d = g[j].x - top;
            se[i] += g[j].y * __expf(d);
            hs[i] += g[j].z;
            hx[i] += fmaf(g[j].z, d, g[j].w);
          }
          gw[i] = src[i] >= 0 ? p.inv_b * p.time_weight : 0.0f;
          scale[i] /= se[i];
        }
        float lrow = 0.0f;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          if (q < blocks) {
            float g[4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
              g[i] = (hs[i >> 1] * (e[q][i] * scale[i >> 1]) - hist[q][i]) * gw[i >> 1];
            if (q == 0 && first) {
#pragma unroll
              for (int w = 0; w < 2; ++w) {
                const float lam = __expf(o0[w]);
                const float lt = -(hx[w] - hs[w] * __logf(se[w]));
                const bool in = src[w] >= 0;
                g[2 * w] = in ? (lam - k[w]) * p.inv_b : 0.0f;
                lrow += in ? (lam - k[w] * o0[w] + p.time_weight * lt) * p.inv_b : 0.0f;
              }
            }
#pragma unroll
            for (int w = 0; w < 2; ++w)
              *reinterpret_cast<uint32_t*>(
                  out + pptc::core_offset(ra + 8 * w, (cb >> 3) + q, p.out_pad) + 2 * cl) =
                  bf16x2(g[2 * w], g[2 * w + 1]);
            // the head's bias gradient: column sums of the FP32 gradients
            *reinterpret_cast<float2*>(
                &col_sum[(quad * 8 + (lane >> 2)) * kColStride + cb + 8 * q + cl]) =
                make_float2(g[0] + g[2], g[1] + g[3]);
          }
        }
        if (first) row_loss[quad * 8 + (lane >> 2)] = lrow;
        arrive(&go[0]);
        if (p.out_pad > kChunk) arrive(&go[1]);
      }
    }
    arrive(&epi_done);
    epi_sync();
    if (t <= p.n_bins) {
      float sum = 0.0f;
#pragma unroll 8
      for (int i = 0; i < 32; ++i) sum += col_sum[i * kColStride + t];
      atomicAdd(p.gbias + t, sum);
    }
    if (warp == kEpiThreads / 32 - 1) {
      float sum = row_loss[lane];
      for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      if (lane == 0) atomicAdd(p.loss, sum);
    }
  }
  pptc::fence_before_sync();
  __syncthreads();
  if (warp == 0) pptc::tmem_dealloc(tmem, 2 * kAccCols);
  if (threadIdx.x == 0 && (abort_flag || !ok)) atomicOr(p.err, 1u);
}

// ---- weight and bias gradients -----------------------------------------------------
// 13 us at batch 8192 (69 MB of operands out of L2, 9.4 MB of atomics; 17 us with
// bulk copies of an 8-row group each), 7 us at 1024.  Two CTAs per SM double the
// atomics: 13.7 and 10 us.
// Every 128 x 128 tile of every layer's dW = dZ^T X, its rows (K) split over
// blocks_per_split 64-row tiles per CTA so that all CTAs run at once, summed by
// float4 atomics; the first column tile's CTAs also sum dZ's columns (the bias
// gradients) from the operand in shared memory.
struct DwTile {
  const unsigned char *a, *b;   // its first column in the first block of each operand
  int a_cols, b_cols;           // columns of the operands' blocks
  int rows, cols;               // of the result tile (multiples of 16)
  float* out;
  int ldc;
  float* bias;                  // column sums of a, or null
};
constexpr int kMaxDwTiles = 4 * kMaxLayers;
struct DwParams {
  DwTile tile[kMaxDwTiles];
  int n_tiles, n_blocks, blocks_per_split;
  unsigned* err;
  unsigned long long wait_ns;
  // the captured step's schedule (sched != null): Adam's step size and bias
  // corrections for step ctl->step + 1
  float* sched;
  const TrainCtl* ctl;
  float b1, b2;
};
constexpr int kDwStages = 6;
constexpr uint32_t kDwStageBytes = 2 * kTileBytes;
constexpr int kDwFetch = 128;                       // 4 warps bring the operands
constexpr int kDwThreads = 256 + 32 + kDwFetch;     // 8 warps of sums and results, MMA issuer

// In double and rounded once, as pp_mlp_train_step computes them.
__device__ __noinline__ void schedule(const DwParams& p) {
  const TrainCtl c = *p.ctl;
  const long long done = c.step;
  const double frac = c.total > 1 ? (double)(done - c.step0) / (double)(c.total - 1) : 0.0;
  p.sched[0] = (float)((double)c.lr1 + 0.5 * ((double)c.lr0 - (double)c.lr1) *
                                           (1.0 + cos(3.14159265358979323846 * frac)));
  p.sched[1] = (float)(1.0 - pow((double)p.b1, (double)(done + 1)));
  p.sched[2] = (float)(1.0 - pow((double)p.b2, (double)(done + 1)));
}

__global__ void __launch_bounds__(kDwThreads, 1) dw_kernel(const __grid_constant__ DwParams p) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(8) uint64_t full[kDwStages], empty[kDwStages], done;
  __shared__ uint32_t tmem_slot;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const DwTile& w = p.tile[blockIdx.x % p.n_tiles];
  const int k0 = (int)(blockIdx.x / p.n_tiles) * p.blocks_per_split;
  const int k1 = min(p.n_blocks, k0 + p.blocks_per_split);
  const bool sums = w.bias != nullptr;
  if (warp == 0) pptc::tmem_alloc(&tmem_slot, 128);
  if (threadIdx.x == 32) {
    for (int i = 0; i < kDwStages; ++i) {
      pptc::mbar_init(&full[i], kDwFetch / 32);
      pptc::mbar_init(&empty[i], sums ? 9 : 1);  // the MMAs' commit, the summing warps
    }
    pptc::mbar_init(&done, 1);
  }
  pptc::fence_before_sync();
  __syncthreads();
  pptc::fence_after_sync();
  const uint32_t tmem = tmem_slot;
  bool ok = true;
  if (warp > 8) {
    // eight 8-row groups of each operand; a stage is announced when the one after
    // it has been requested
    const int t = (int)threadIdx.x - 256 - 32;
    auto announce = [&](int k) {
      __syncwarp();
      if (lane == 0) pptc::mbar_arrive(&full[(k - k0) % kDwStages]);
    };
    int k = k0;
    for (; k < k1; ++k) {
      const uint32_t c = (uint32_t)(k - k0), slot = c % kDwStages;
      ok = __all_sync(0xffffffffu,
                      pptc::mbar_wait(&empty[slot], ((c / kDwStages) & 1) ^ 1, p.wait_ns));
      if (!ok) break;
      const uint32_t dst = pptc::smem_u32(smem + slot * kDwStageBytes) + t * 16;
      const unsigned char* a = w.a + (size_t)k * 128 * w.a_cols + t * 16;
      const unsigned char* b = w.b + (size_t)k * 128 * w.b_cols + t * 16;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (t < w.rows) fetch16(dst + i * w.rows * 16, a + (size_t)i * 16 * w.a_cols);
        if (t < w.cols) fetch16(dst + kTileBytes + i * w.cols * 16, b + (size_t)i * 16 * w.b_cols);
      }
      fetch_commit();
      if (c >= 1) {
        fetch_wait<1>();
        announce(k - 1);
      }
    }
    fetch_wait<0>();
    if (ok)
      for (int q = max(k0, k - 1); q < k; ++q) announce(q);
  } else if (warp == 8) {
    // (the result tile's rows past w.rows take whatever follows in the stage)
    const uint32_t idesc = pptc::idesc_bf16(128, w.cols) | (1u << 15) | (1u << 16);
    const uint64_t a0 = pptc::smem_desc(pptc::smem_u32(smem), (uint32_t)w.rows * 16u, 128);
    const uint64_t b0 =
        pptc::smem_desc(pptc::smem_u32(smem) + kTileBytes, (uint32_t)w.cols * 16u, 128);
    bool there = false;  // the next stage has been seen complete
    uint32_t slot = 0, phase = 0;
    for (int k = k0; k < k1; ++k) {
      ok = __all_sync(0xffffffffu, there || pptc::mbar_wait(&full[slot], phase, p.wait_ns));
      if (!ok) break;
      pptc::fence_after_sync();
      const uint32_t at = slot;
      if (++slot == kDwStages) {
        slot = 0;
        phase ^= 1u;
      }
      there = k + 1 < k1 && pptc::mbar_test(pptc::smem_u32(&full[slot]), phase);
      const uint64_t a = a0 + (uint64_t)(at * (kDwStageBytes / 16));
      const uint64_t b = b0 + (uint64_t)(at * (kDwStageBytes / 16));
#pragma unroll
      for (int s = 0; s < 4; ++s)
        pptc::mma_f16_by(lane == 0, tmem, a + (uint64_t)(s * 2 * w.rows),
                         b + (uint64_t)(s * 2 * w.cols), idesc, k > k0 || s > 0);
      pptc::mma_commit_by(lane == 0, &empty[at]);
    }
    if (lane == 0) {
      pptc::mma_commit(&done);
      if (!pptc::mbar_wait(&done, 0, p.wait_ns)) ok = false;
    }
    __syncwarp();
  } else {
    // (by a CTA whose warps have no sums to do meanwhile)
    if (p.sched && (int)blockIdx.x == p.n_tiles - 1 && threadIdx.x == 0) schedule(p);
    __syncwarp();
    const int t = threadIdx.x;
    if (sums) {
      // columns 8 g .. 8 g + 7 of rows kp, kp + 16, kp + 32, kp + 48 of each block
      const int g = t >> 4, kp = t & 15;
      float s[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) s[i] = 0.0f;
      for (int k = k0; k < k1; ++k) {
        const uint32_t c = (uint32_t)(k - k0), slot = c % kDwStages;
        ok = __all_sync(0xffffffffu,
                        pptc::mbar_wait(&full[slot], (c / kDwStages) & 1, p.wait_ns));
        if (!ok) break;
        if (g * 8 < w.rows) {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const uint4 v = *reinterpret_cast<const uint4*>(
                smem + slot * kDwStageBytes + pptc::core_offset(kp + 16 * q, g, w.rows));
            const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              s[2 * i] += bf16_lo(u[i]);
              s[2 * i + 1] += bf16_hi(u[i]);
            }
          }
        }
        __syncwarp();
        if (lane == 0) pptc::mbar_arrive(&empty[slot]);
      }
#pragma unroll
      for (int i = 0; i < 8; ++i)
        for (int o = 1; o < 16; o <<= 1) s[i] += __shfl_xor_sync(0xffffffffu, s[i], o);
      if (ok && kp == 0 && g * 8 < w.rows) {
#pragma unroll
        for (int i = 0; i < 8; ++i) atomicAdd(w.bias + g * 8 + i, s[i]);
      }
    }
    ok = __all_sync(0xffffffffu, pptc::mbar_wait(&done, 0, p.wait_ns)) && ok;
    if (ok) {
      pptc::fence_after_sync();
      const int r = (warp & 3) * 32 + lane;
#pragma unroll 1
      for (int c0 = (warp >> 2) * 32; c0 < w.cols; c0 += 64) {
        uint32_t v[32];
        pptc::tmem_ld32_nowait(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c0, v);
        pptc::tmem_wait();
        if (r < w.rows) {
          float4* d = reinterpret_cast<float4*>(w.out + (size_t)r * w.ldc + c0);
#pragma unroll
          for (int q = 0; q < 8; ++q)
            if (c0 + 4 * q < w.cols)
              atomicAdd(d + q, make_float4(__uint_as_float(v[4 * q]), __uint_as_float(v[4 * q + 1]),
                                           __uint_as_float(v[4 * q + 2]),
                                           __uint_as_float(v[4 * q + 3])));
        }
      }
    }
  }
  pptc::fence_before_sync();
  ok = __syncthreads_and(ok);
  if (!ok && threadIdx.x == 0) atomicOr(p.err, 1u);
  if (warp == 0) pptc::tmem_dealloc(tmem, 128);
}

// ---- Adam ----------------------------------------------------------------------------
struct LayerMap {
  long long off_w, off_b;
  int rows, cols;
  uint32_t wf, wb;  // byte offsets of its two packs
};
struct AdamParams {
  float *w, *g, *m, *v;
  long long n;
  const float* sched;       // {lr, bc1, bc2} on the device, or null: the three below
  float lr, bc1, bc2, b1, b2, eps;
  bf16* w16;                // row-major BF16 copy (the layer-by-layer forward pass)
  unsigned char *wf, *wb;
  int n_layers;             // hidden layers
  LayerMap layer[kMaxLayers];
  float *loss_acc, *loss;   // the batch loss moves on, the accumulators are zeroed
  TrainCtl* ctl;            // its step count advances, or null
};
// The BF16 copies of parameters i .. i + 3 (i a multiple of 4; a layer's rows and
// columns are multiples of 16, so that the four are neighbours in all of them).
__device__ __forceinline__ void pack_weights(const AdamParams& p, long long i, float4 w) {
  const uint2 q = make_uint2(bf16x2(w.x, w.y), bf16x2(w.z, w.w));
  *reinterpret_cast<uint2*>(p.w16 + i) = q;
  int l = 0;
  while (l < p.n_layers && i >= p.layer[l + 1].off_w) ++l;
  const LayerMap& m = p.layer[l];
  const int at = (int)(i - m.off_w);
  if (at >= m.rows * m.cols) return;  // biases
  const int o = at / m.cols, c = at % m.cols;
  *reinterpret_cast<uint2*>(p.wf + m.wf + pack_offset(o, c, m.rows, m.cols)) = q;
  if (l > 0) *reinterpret_cast<uint2*>(p.wb + m.wb + pack_offset_t(c, o, m.cols, m.rows)) = q;
}
// Four parameters per thread: 869 blocks of one each took 5.2 us for 222 k
// parameters, launch included.
__global__ void adam_kernel(const __grid_constant__ AdamParams p) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const long long i = 4 * ((long long)blockIdx.x * blockDim.x + threadIdx.x);
  if (i >= p.n) return;
  const float lr = p.sched ? p.sched[0] : p.lr;
  const float bc1 = p.sched ? p.sched[1] : p.bc1, bc2 = p.sched ? p.sched[2] : p.bc2;
  const float4 g4 = *reinterpret_cast<const float4*>(p.g + i);
  const float4 m4 = *reinterpret_cast<const float4*>(p.m + i);
  const float4 v4 = *reinterpret_cast<const float4*>(p.v + i);
  const float4 w4 = *reinterpret_cast<const float4*>(p.w + i);
  const float g[4] = {g4.x, g4.y, g4.z, g4.w};
  float m[4] = {m4.x, m4.y, m4.z, m4.w}, v[4] = {v4.x, v4.y, v4.z, v4.w};
  float w[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    m[j] = p.b1 * m[j] + (1.0f - p.b1) * g[j];
    v[j] = p.b2 * v[j] + (1.0f - p.b2) * g[j] * g[j];
    w[j] -= lr * (m[j] / bc1) / (sqrtf(v[j] / bc2) + p.eps);
  }
  *reinterpret_cast<float4*>(p.g + i) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  *reinterpret_cast<float4*>(p.m + i) = make_float4(m[0], m[1], m[2], m[3]);
  *reinterpret_cast<float4*>(p.v + i) = make_float4(v[0], v[1], v[2], v[3]);
  *reinterpret_cast<float4*>(p.w + i) = make_float4(w[0], w[1], w[2], w[3]);
  pack_weights(p, i, make_float4(w[0], w[1], w[2], w[3]));
  if (i == 0) {
    *p.loss = *p.loss_acc;
    *p.loss_acc = 0.0f;
    if (p.ctl) p.ctl->step += 1;
  }
}
// The packs of the current parameters.
__global__ void pack_kernel(const __grid_constant__ AdamParams p) {
  const long long i = 4 * ((long long)blockIdx.x * blockDim.x + threadIdx.x);
  if (i < p.n) pack_weights(p, i, *reinterpret_cast<const float4*>(p.w + i));
}
// Without an update: the loss moves on and the accumulators are zeroed.
__global__ void clear_kernel(float* __restrict__ g, long long n, float* loss_acc, float* loss) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) g[i] = 0.0f;
  if (i == 0) {
    *loss = *loss_acc;
    *loss_acc = 0.0f;
  }
}
__global__ void set_ctl_kernel(TrainCtl* ctl, const TrainCtl v) { *ctl = v; }

}  // namespace pprows
