// pp_internal.h -- structures shared by the host runtime and the device
// kernels of the photon-transport library (not part of the public ABI).
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstdint>
#include <string>
#include <vector>

#include "pp_gb300.h"

namespace pp {

// Uniform culling grid over the targets.  The grid, its per-cell candidate
// lists and the sphere table live in one contiguous 16-byte aligned "blob"
// that each CTA stages into shared memory with one TMA bulk copy:
//   [cells  : uint32 x n_cells, (count << 20) | first_item]  padded to 16 B
//   [items  : uint16 x n_items, target indices]             padded to 16 B
//   [spheres: float4 x n_targets, (x, y, z, r^2)]
struct GridDev {
  float lo[3];        // origin of cell (0,0,0)
  float hi[3];        // lo + dims * cell
  float cell[3];      // cell edge per axis (m)
  float inv_cell[3];  // 1 / cell
  int dims[3];
  int n_cells;
  int n_targets;
  uint32_t off_items;    // byte offset of the item list in the blob
  uint32_t off_spheres;  // byte offset of the sphere table in the blob
  uint32_t blob_bytes;   // multiple of 16
};

// Safety field: a uniform grid of nodes lo + i * cell over a box that contains
// every (inflated) sphere; a node holds a lower bound of its distance to the
// nearest sphere surface, quantised down in kSafetyQuantum steps (uint8).  For
// a point m with projection m' onto the box and the node c nearest to m',
// every sphere is at least sqrt(|m - m'|^2 + w^2) away, w = max(D(c) - |m' - c|, 0):
// the distance to the spheres is 1-Lipschitz, and a convex box seen from
// outside lies behind its nearest point.
struct SafetyDev {
  float lo[3];
  float hi[3];
  float cell;      // node spacing (m), the same on every axis
  float inv_cell;
  int dims[3];     // nodes per axis, >= 2
  int n_cells;     // nodes, < 2^23
  uint32_t bytes;  // allocation, n_cells rounded up to 16 (padding bytes are 0)
  // Derived on the host (set_derived) so that the kernel's tests read them
  // as constant operands; the tests work in units of the spacing.
  float fdims[3];  // dims as float
  float fmaxc[3];  // dims - 1 as float (largest node coordinate)
  float lo_sc[3];  // lo * inv_cell
  float quantum;   // kSafetyQuantum * inv_cell
  float r_scale;   // ball radius in spacings = r_scale * (half the segment) + r_slack:
  float r_slack;   // 1e-4 relative and 0.1 mm above it
  void set_derived();
  // Nodes of spacing h (m, made coarser if they would be too many) over the
  // box [blo, bhi].
  void set_shape(const float* blo, const float* bhi, double h);
  // The automatic spacing for n spheres.
  static double auto_cell(const float* blo, const float* bhi, int n, bool staged = true);
};
constexpr float kSafetyQuantum = 0.5f;  // m per uint8 step (saturates at 127.5 m)

inline void SafetyDev::set_derived() {
  for (int a = 0; a < 3; ++a) {
    fdims[a] = (float)dims[a];
    fmaxc[a] = (float)(dims[a] - 1);
    lo_sc[a] = lo[a] * inv_cell;
  }
  quantum = kSafetyQuantum * inv_cell;
  r_scale = 1.0001f * inv_cell;
  r_slack = 1e-4f * inv_cell;
}

inline double safety_nodes(const float* blo, const float* bhi, double h) {
  double n = 1.0;
  for (int a = 0; a < 3; ++a)
    n *= std::ceil(std::max(1e-6, (double)bhi[a] - (double)blo[a]) / h) + 1.0;
  return n;
}

inline void SafetyDev::set_shape(const float* blo, const float* bhi, double h) {
  for (int guard = 0; guard < 512 && safety_nodes(blo, bhi, h) > 8.0e6; ++guard) h *= 1.25;
  n_cells = 1;
  for (int a = 0; a < 3; ++a) {
    dims[a] = (int)std::ceil(std::max(1e-6, (double)bhi[a] - (double)blo[a]) / h) + 1;
    lo[a] = blo[a];
    hi[a] = (float)((double)blo[a] + (dims[a] - 1) * h);
    n_cells *= dims[a];
  }
  cell = (float)h;
  inv_cell = (float)(1.0 / h);
  bytes = (uint32_t)(((size_t)n_cells + 15) & ~(size_t)15);
  set_derived();
}

// 120 nodes per sphere, 2k to 48k: the staged tables of a large detector leave 92
// KB of the SM to L1.  400 modules, ms per 1e8 photons (per 4e7 of 256 emitters):
// 34k nodes 13.54 (4.48), 48k 13.13 (4.46), 60k 13.16 (4.56), 72k 13.02 (4.54).
// Tables that stay in global memory (staged false: some 1,700 spheres and more) have
// no L1 to share: 60 nodes per sphere.  2e6 photons in a 600 m cube, ms with 48k nodes
// and with these, 16 warps an SM: 4,000 spheres 1.35 and 1.04, 20,000 3.94 and 2.34,
// 60,000 6.4 and 4.0 (120 nodes 3.8).
inline double SafetyDev::auto_cell(const float* blo, const float* bhi, int n, bool staged) {
  double vol = 1.0;
  for (int a = 0; a < 3; ++a) vol *= std::max(1e-6, (double)bhi[a] - (double)blo[a]);
  double nodes = std::min(std::max(120.0 * n, 2048.0), 48000.0);
  if (!staged) nodes = std::max(nodes, 60.0 * n);
  double h = std::max(1e-3, std::cbrt(vol / nodes));
  for (int guard = 0; guard < 512 && safety_nodes(blo, bhi, h) > nodes; ++guard) h *= 1.02;
  return h;
}

// A lane of the propagation kernel carries two photons.  pp_tuning's
// block_threads counts 1024 for all the warps an SM holds: that many, or the
// same share of them, make a CTA.
constexpr int kGroup = 64;     // photons a warp carries at a time
// (16 warps of 128 registers: 24 of 80 issue 73% of the time against 68%, but
// spill, and both take 13.6 ms per 1e8 photons; the FMA and ALU pipes bound both.)
constexpr int kSmWarps = 16;
constexpr int kMaxBlockThreads = 32 * kSmWarps;
inline int propagate_warps(int block_threads) {
  return (block_threads * kSmWarps + 1023) / 1024;
}
// Where a kernel's tables are.  The last two run small CTAs, so that registers and not
// a CTA's size set the warps of an SM.
enum class Tables {
  kStaged,      // in shared memory
  kGlobal,      // kept in global memory, or too large and a workload of one round of warps
  kGlobalMany,  // too large for shared memory, more chunks than kManyChunks an SM
  kShapes       // no tables: a list of shapes
};
// Tables that are too large: 32 warps of 64 registers, whose spills cost less than the
// latency of L2 with 16 warps to hide it, as soon as 16 do not take the whole
// workload at once.  60,000 spheres in a cube of 600 m, 2e6 photons: 4.02 ms with 16
// warps, 3.29 with 24, 2.64 with 32 (200,000 photons 0.55 and 0.39, 155,000 0.338 and
// 0.385); of 120 m: 5.12, 4.22, 3.28; 4,000 of 600 m: 1.05, 0.93, 0.83.  Shapes: 20 of
// 96 (1e6 photons, 50 discs of 2 m: 1,059 us with 16 warps, 828 with 20; 400 spheres in
// the unculled loop, 2e6 photons: 13.8 and 10.9 ms).
constexpr int kManyChunks = 16;
constexpr bool small_ctas(Tables t) { return t == Tables::kGlobalMany || t == Tables::kShapes; }
constexpr int min_ctas(Tables t) {  // of an SM
  return t == Tables::kGlobalMany ? 8 : t == Tables::kShapes ? 5 : 1;
}
constexpr int kSmallBlock = 256;  // in units of block_threads
constexpr int kSmallThreads = 32 * (kSmallBlock * kSmWarps / 1024);

constexpr double kMixedFrom = 1.1;  // photons that groups have room for, over photons

// Per-warp shared-memory state of the propagation kernel: the step segments
// whose hit test is deferred (two stacks: those not yet clipped by the safety
// field, and those clipped, which wait for the grid walk over [t0, t1]) and,
// per photon, the earliest hit found so far.
constexpr int kRawCap = 32 - 1 + kGroup;  // clipped as soon as 32 wait
constexpr int kClippedCap = 32 - 1 + 32;  // walked as soon as 32 wait
struct alignas(16) WarpQueue {
  float4 raw_a[kRawCap];       // segment start, length
  float4 raw_b[kRawCap];       // direction, owner (lane + 32 * photon) | step << 8
  float4 clip_a[kClippedCap];
  float4 clip_b[kClippedCap];
  float2 clip_t[kClippedCap];  // part of the segment the grid walk must cover
  uint32_t key[kGroup];        // step << 16 | target index; ~0 = none
};
// Shaped targets (no queue): per photon, the hit itself.
struct WarpBest {
  float hx[kGroup], hy[kGroup], hz[kGroup];
  float ox[kGroup], oy[kGroup], oz[kGroup];
  float dist[kGroup];
};

constexpr uint32_t kCellStartBits = 20;                    // first item index
constexpr uint32_t kCellStartMask = (1u << kCellStartBits) - 1u;
constexpr uint32_t kCellMaxCount = (1u << (32 - kCellStartBits)) - 1u;
// Automatic cells: 8 per target, 16 for lists that are too dense for that.  (400
// modules: 8 15.0 ms per 1e8 photons, 16 15.7, 4 15.2: fewer cells to cross against
// more spheres per cell.)
constexpr double kAutoCellsPerTarget[] = {8.0, 16.0};
constexpr int kAutoCells = 2;
constexpr int kGridTooDense = 1;                           // of build_grid, build_grid_into
constexpr float kGridMargin = 0.01f;                       // m, AABB inflation

// Phase-function constants derived once per medium.
struct PhaseDev {
  float hg_weight;  // P(Henyey-Greenstein)
  float hg_g;
  float hg_1mg2;    // 1 - g^2
  float hg_n1pg2;   // -(1 + g^2)
  float hg_ninv2g;  // -1 / (2 g)
  float es_k1;      // (b + 3) / b
  float es_k2;      // 1 / b^3
  float es_b;       // Einstein-Smoluchowski b
  int kind;         // PP_PHASE_*
  float sl_exp;     // simplified Liu: (1 - g) / (1 + g)
  // u = ((w >> 8) + 1) 2^-24 < hg_weight as a compare of the random word: w < hg_words
  uint32_t hg_words;
  // Einstein-Smoluchowski inverse CDF for the fast kernel: kEsTable intervals
  // of eta on [0, 1], entry i = {q(i / N), q((i + 1) / N) - q(i / N)}, then one
  // entry {q(1), 0} (set by pp_set_medium; null: the Cardano formula)
  const float2* es_table;
};

// Intervals of the tabulated Einstein-Smoluchowski inverse CDF.  q(eta) is
// smooth on [0, 1] (its derivative is 1 / pdf, and pdf ~ 1 + b cos^2 is
// bounded away from 0), so linear interpolation on 1024 intervals is exact to
// ~1e-7, below the SFU cube roots of the formula it replaces.
constexpr int kEsTableBits = 10;
constexpr int kEsTable = 1 << kEsTableBits;

// The table of PhaseDev::es_table for parameter b (kEsTable + 1 entries), in
// double and rounded once:
// q = cbrt(Q + D) + cbrt(Q - D), Q = (b + 3)(eta - 1/2) / b, D = sqrt(Q^2 + 1/b^3)
// (the Cardano root of the ES CDF's cubic, as the replay kernel evaluates it).
inline void make_es_table(float b, float2* out) {
  const double bb = b, k1 = (bb + 3.0) / bb, k2 = 1.0 / (bb * bb * bb);
  double prev = 0.0;
  for (int i = 0; i <= kEsTable; ++i) {
    const double q = k1 * ((double)i / kEsTable - 0.5);
    const double d = std::sqrt(q * q + k2);
    const double v = std::cbrt(q + d) + std::cbrt(q - d);
    if (i > 0) out[i - 1] = make_float2((float)prev, (float)(v - prev));
    prev = v;
  }
  // eta = 1: the last interval's end, as its interpolation rounds
  const float2 e = out[kEsTable - 1];
  out[kEsTable] = make_float2((float)((double)e.x + (double)e.y), 0.0f);
}

// The phase function of a medium, validated: nullptr on success, else the
// reason.  Shared by pp_set_medium and pp_propagate_static.
inline const char* make_phase(const pp_medium* m, PhaseDev* p) {
  if (m->phase_kind != PP_PHASE_HG_ES && m->phase_kind != PP_PHASE_HG_SL)
    return "phase_kind must be PP_PHASE_HG_ES or PP_PHASE_HG_SL";
  if (!(m->hg_weight >= 0.0f && m->hg_weight <= 1.0f)) return "hg_weight must be in [0, 1]";
  const float g = m->hg_g;
  if (m->hg_weight > 0.0f && !(std::fabs(g) >= 1e-3f && std::fabs(g) < 1.0f))
    return "hg_g must satisfy 1e-3 <= |g| < 1";
  if (m->phase_kind == PP_PHASE_HG_ES && m->hg_weight < 1.0f && !(m->es_b > 0.0f))
    return "es_b must be > 0 when the ES component is used";
  if (m->phase_kind == PP_PHASE_HG_SL && m->hg_weight < 1.0f && !(g > -1.0f && g < 1.0f))
    return "the simplified-Liu component needs -1 < g < 1";
  const float b = m->es_b > 0.0f ? m->es_b : 1.0f;
  p->hg_weight = m->hg_weight;
  p->hg_g = g;
  p->hg_1mg2 = 1.0f - g * g;
  p->hg_n1pg2 = -(1.0f + g * g);
  p->hg_ninv2g = m->hg_weight > 0.0f ? -1.0f / (2.0f * g) : 0.0f;
  p->es_k1 = (b + 3.0f) / b;
  p->es_k2 = 1.0f / (b * b * b);
  p->es_b = b;
  p->kind = m->phase_kind;
  p->sl_exp = (1.0f - g) / (1.0f + g);
  // k 2^-24 < hg_weight, k = (w >> 8) + 1 in 1 .. 2^24
  const double c = std::ceil((double)m->hg_weight * 16777216.0);
  p->hg_words = c >= 1.0 ? ((uint32_t)c - 1u) << 8 : 0u;
  return nullptr;
}

// The work queue of sources with nph[i] photons in chunks of `chunk`: cumulative chunks
// of each source, or, for many sources of few photons, the cumulative photons, whose
// chunks are of all sources.  Returns the number of chunks.
// Mixed when groups of one source's photons would be more than 10% empty and more than
// the GPU's warps (as many as these run side by side whatever they hold).  us with
// groups of 32 photons of one source, of 64, mixed: 100,000 sources of 1 photon 480,
// 690, 45; of 20 602, 777, 367; 10,000 of 32 100, 107, 78; of 54 161, 115, 109; of 64
// 170, 118, 134.
inline unsigned long long make_queue(const long long* nph, int n, long long chunk, int num_sms,
                                     unsigned long long* prefix, bool* mixed) {
  unsigned long long groups = 0, photons = 0;
  for (int i = 0; i < n; ++i) {
    photons += (unsigned long long)nph[i];
    groups += (unsigned long long)((nph[i] + kGroup - 1) / kGroup);
  }
  *mixed = groups > (unsigned long long)(kSmWarps * num_sms) &&
           (double)groups * kGroup > kMixedFrom * (double)photons;
  prefix[0] = 0;
  for (int i = 0; i < n; ++i)
    prefix[i + 1] =
        prefix[i] + (unsigned long long)(*mixed ? nph[i] : (nph[i] + chunk - 1) / chunk);
  return *mixed ? (photons + (unsigned long long)chunk - 1) / (unsigned long long)chunk : prefix[n];
}

// Everything one launch of the propagation kernel needs (kernel parameter,
// passed as __grid_constant__).
struct LaunchArgs {
  const pp_source* sources;
  const unsigned long long* chunk_prefix;  // [n_src + 1] cumulative chunks, or photons (mixed)
  bool mixed;                              // groups of several sources' photons
  const long long* src_photons;            // [n_src] photons after scaling
  unsigned long long total_chunks;
  int n_src;
  int chunk_photons;                       // photons per queued chunk

  const unsigned char* blob;               // grid blob (global memory)
  GridDev grid;
  const unsigned char* safety;             // safety field (global memory)
  SafetyDev sgrid;
  // Shaped targets (no grid): 2 float4 per target, {x, y, z, p0} {p1, kind}:
  // sphere p0 = r^2; rectangle p0, p1 = half lengths; disc p0 = r^2.
  const float4* shapes;
  int n_shapes;

  const float4* medium;                    // {sca_len, v_group, abs_len, n}
  int n_medium;
  float med_wl_min;
  float med_inv_step;
  PhaseDev phase;

  const float* spectrum;                   // inverse CDF knots or nullptr
  int n_spectrum;
  float mono_wavelength;
  const float* track;                      // cos(theta) quantiles or nullptr
  int n_track;

  uint32_t key0, key1;                     // Philox key = seed
  uint32_t round_keys[20];                 // Philox round keys (set_seed)
  int n_steps;

  // key = seed; round r of Philox4x32-10 uses (key0 + r W0, key1 + r W1),
  // precomputed once per launch so that the per-step generator takes them as
  // kernel-parameter operands instead of recomputing them
  void set_seed(uint64_t seed) {
    key0 = (uint32_t)(seed & 0xffffffffu);
    key1 = (uint32_t)(seed >> 32);
    for (int r = 0; r < 10; ++r) {
      round_keys[2 * r] = key0 + (uint32_t)r * 0x9E3779B9u;
      round_keys[2 * r + 1] = key1 + (uint32_t)r * 0xBB67AE85u;
    }
  }

  pp_hit_record* hits;
  unsigned long long capacity;
  pp_counters* counters;
  unsigned long long wait_limit_ns;        // bound on the TMA staging wait
  int skip_staging_copies;                 // diagnostic: arm the barrier, copy nothing

  // Histogram mode (hist != nullptr): instead of hit records, every hit adds
  // its absorption weight to hist[s * (bins + 1)] (count) and to bin
  // 1 + b of log10(t - tgeo[s] + hist_t_offset) on [hist_log_lo, hist_log_hi).
  float* hist;
  const float* hist_tgeo;
  int hist_bins;
  float hist_t_offset;
  float hist_log_lo;
  float hist_inv_log_width;

  uint32_t safety_offset;                  // shared-memory offset of the staged field
  uint32_t state_offset;                   // shared-memory offset of the warp state
  int warps_per_block;
};

// Dynamic shared memory of one CTA: [grid blob | safety field] when staged,
// then the per-warp state (the queues, whose room the shaped targets' hits use).
static_assert(sizeof(WarpBest) <= offsetof(WarpQueue, clip_t), "shares the stacks' room");
static_assert(sizeof(int) * kGroup <= sizeof(float2) * kClippedCap, "the list of a group's hits");
inline size_t propagate_smem_bytes(uint32_t blob_bytes, uint32_t safety_bytes, bool smem_tables,
                                   int block_threads, uint32_t* safety_offset,
                                   uint32_t* state_offset) {
  const size_t blob = ((size_t)blob_bytes + 15) & ~(size_t)15;
  const size_t field = ((size_t)safety_bytes + 15) & ~(size_t)15;
  const size_t off = smem_tables ? blob + field : 0;
  if (safety_offset) *safety_offset = (uint32_t)blob;
  if (state_offset) *state_offset = (uint32_t)off;
  return off + (size_t)propagate_warps(block_threads) * sizeof(WarpQueue);
}
// Largest dynamic shared memory per CTA for which CTAs of block_threads
// still fill an SM: the
// SM's 228 KB less 1 KB reserved per CTA and the static barrier, at most the
// 227 KB one CTA may opt into.
inline size_t smem_budget(int block_threads) {
  const int ctas = block_threads >= 1024 ? 1 : 1024 / (block_threads > 0 ? block_threads : 1);
  const size_t b = (size_t)228 * 1024 / (size_t)ctas - 1024 - 64;
  return b < (size_t)227 * 1024 - 64 ? b : (size_t)227 * 1024 - 64;
}

// Host-side launch of the propagation kernel (pp_propagate.cu).
cudaError_t launch_propagate(const LaunchArgs& args, int block_threads, int ctas_per_sm,
                             bool precise, bool smem_grid, int num_sms, cudaStream_t stream,
                             int* grid_out);
// Grid build on the device (pp_grid.cu).  targets_dev: n spheres in device
// memory.  Returns 0 on success, kGridTooDense or -1; *blob_out is allocated with
// cudaMalloc.
int build_grid(const pp_sphere* targets_dev, int n, float cell_size, cudaStream_t stream,
               GridDev* grid_out, unsigned char** blob_out, long long* n_items_out,
               std::string* err);

// Set the calling thread's last error (pp_abi.cu); returns code.
int report_error(int code, const std::string& message);

// Grid build into caller-provided device memory (pp_grid.cu): `shape` holds
// the box, cell sizes and dims; d_counts/d_start/d_cursor have n_cells entries,
// d_totals two.  Used by the entry point that allocates nothing.
int build_grid_into(const pp_sphere* targets_dev, int n, const GridDev& shape, unsigned* d_counts,
                    unsigned* d_start, unsigned* d_cursor, unsigned* d_totals,
                    unsigned char* d_blob, size_t blob_capacity, cudaStream_t stream,
                    GridDev* grid_out, long long* n_items_out, std::string* err);
// Safety field into caller-provided device memory of shape.bytes bytes.
int build_safety_into(const pp_sphere* targets_dev, int n, const SafetyDev& shape,
                      unsigned char* d_field, cudaStream_t stream, std::string* err);

// Safety field over the grid box (pp_grid.cu); *field_out is cudaMalloc'd.
int build_safety(const pp_sphere* targets_dev, int n, const GridDev& grid, float cell,
                 cudaStream_t stream, SafetyDev* out, unsigned char** field_out, std::string* err);

// Scatter hit records into columns on the device (pp_grid.cu).
cudaError_t launch_hits_to_columns(const pp_hit_record* rec, long long n, const pp_hits& out,
                                   cudaStream_t stream);

// Philox on the device for the ABI diagnostic (pp_grid.cu).
cudaError_t launch_debug_philox(const uint32_t* ctr, int n, uint32_t k0, uint32_t k1,
                                uint32_t* out, cudaStream_t stream);

// FFMA throughput kernel (pp_grid.cu); returns flops per launch.
cudaError_t launch_fp32_peak(float* sink, int blocks, int threads, int iters, cudaStream_t stream);

}  // namespace pp
