// pp_propagate.cu -- fast variant of the propagation kernel and the host-side
// launch (grid sizing from the occupancy calculator, dynamic shared memory for
// the staged target grid).
#include <cuda_runtime.h>

#include <algorithm>

#include "pp_kernel.cuh"

namespace pp {

// Replay variant, instantiated in pp_propagate_precise.cu.
const void* precise_kernel_ptr(Tables t, bool mixed);

namespace {

const void* select_kernel(bool precise, Tables t, bool mixed) {
  return precise ? precise_kernel_ptr(t, mixed) : kernel_ptr<false>(t, mixed);
}

}  // namespace

cudaError_t launch_propagate(const LaunchArgs& args, int block_threads, int ctas_per_sm,
                             bool precise, bool smem_grid, int num_sms, cudaStream_t stream,
                             int* grid_out) {
  if (block_threads > 1024 || block_threads % 32) return cudaErrorInvalidValue;
  if (args.shapes) smem_grid = false;
  const bool fit = propagate_smem_bytes(args.grid.blob_bytes, args.sgrid.bytes, true, block_threads,
                                        nullptr, nullptr) <= smem_budget(block_threads);
  const Tables t =
      args.shapes ? Tables::kShapes
      : smem_grid ? Tables::kStaged
      : !fit && args.total_chunks > (unsigned long long)(kManyChunks * num_sms) ? Tables::kGlobalMany
                                                                                : Tables::kGlobal;
  const void* k = select_kernel(precise, t, args.mixed);
  if (small_ctas(t)) {  // the same share of an SM
    ctas_per_sm = (std::min(ctas_per_sm, 32) * block_threads * min_ctas(t) + 1023) / 1024;
    block_threads = kSmallBlock;
  }
  const int threads = propagate_warps(block_threads) * 32;
  LaunchArgs a = args;
  const size_t smem = propagate_smem_bytes(args.grid.blob_bytes, args.sgrid.bytes, smem_grid,
                                           block_threads, &a.safety_offset, &a.state_offset);
  a.warps_per_block = threads / 32;
  cudaError_t e;
  if (smem > 48 * 1024) {
    e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  int occ = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k, threads, smem);
  if (e != cudaSuccess) return e;
  if (occ < 1) return cudaErrorInvalidConfiguration;
  const int per_sm = ctas_per_sm > 0 ? (ctas_per_sm < occ ? ctas_per_sm : occ) : occ;
  int grid = per_sm * num_sms;
  // Never launch more CTAs than there are chunks of work.
  if (args.total_chunks < (unsigned long long)grid)
    grid = (int)(args.total_chunks > 0 ? args.total_chunks : 1);
  if (grid_out) *grid_out = grid;
  void* params[] = {&a};
  return cudaLaunchKernel(k, dim3(grid), dim3(threads), params, smem, stream);
}

}  // namespace pp
