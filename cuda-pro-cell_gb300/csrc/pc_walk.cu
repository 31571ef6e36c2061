// Instantiations and launchers of the tree walk (pc_walk.cuh), plain and batched.
#include "pc_walk.cuh"

namespace pc {

static size_t walk_smem_bytes(bool batched) { return batched ? sizeof(WalkSmem<true>) : sizeof(WalkSmem<false>); }

int walk_occupancy(bool batched, int* blocks_per_sm) {
  auto* k = batched ? k_walk<true> : k_walk<false>;
  const size_t smem = walk_smem_bytes(batched);
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, k, kWalkThreads, smem);
  return (int)e;
}

uint32_t walk_warps_per_block() { return kWalkWarps; }

// A stack holds at most about 32 cells per generation; a region that overflows all the same (parked
// cells may come back to a deep stack) sets an error bit and the run goes to the level sweeps, which
// a build with a small region makes happen for a test.
uint32_t walk_region_cells(uint32_t gmax) {
#ifdef PC_WALK_REGION_CELLS
  (void)gmax;
  return PC_WALK_REGION_CELLS;
#else
  return 32u * (gmax + 2u) + 512u;
#endif
}

int launch_walk(const WalkArgs& w, int blocks, void* stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)blocks);
  cfg.blockDim = dim3((unsigned)kWalkThreads);
  cfg.dynamicSmemBytes = walk_smem_bytes(w.a.btypes != nullptr);
  cfg.stream = (cudaStream_t)stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return (int)cudaLaunchKernelEx(&cfg, w.a.btypes ? k_walk<true> : k_walk<false>, w);
}

}  // namespace pc
