// launch.cuh — launches with programmatic stream serialization (programmatic dependent launch).
//
// A kernel launched through launch_pdl may start while the kernel before it in the stream still runs: it must execute pdl_wait()
// before it touches anything an earlier kernel writes, and before it writes anything an earlier kernel reads.  pdl_wait()
// returns when every kernel the launch depends on has completed and its writes are visible; without a programmatic edge
// (first kernel of a stream, after a copy) it returns at once.  pdl_launch_dependents() lets the next such kernel start: called
// early only by short kernels that leave room on the SMs.  With it at the start of the large ones too (tensor-core tiles, attention,
// row sweeps, layout passes) the waiting CTAs took registers and shared memory from the running ones and cost more than the launch
// latency they hid (UNet 5.27 -> 5.46 ms, decoder with one prompt 1.66 -> 1.73 ms).
// A kernel that allocates tensor memory calls it behind the allocation and a barrier: some kernels allocate ahead of their pdl_wait(),
// and one that held an SM's columns while a CTA of the kernel it waits for still asked for them would wait for good.
#pragma once

#include <cuda_runtime.h>

#include <utility>

#include "common.h"

namespace mb {
namespace {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// The same for kernels of either size: a launch whose CTAs are on the SMs all at once loses nothing to the waiting ones.  Attention and the
// one-pass RMSNorm, which a GEMM that fetches its weights ahead follows: one prompt of 1000 tokens 1100 -> 1033 us, encoder at batch 40
// 269.7 -> 264.5 us.  (Not the convolutions' chain of layout passes, sweeps and tiles: with it and dependency waits throughout the
// UNet of 3 samples took 613 -> 686 us, the conv stack 7.17 -> 7.38 ms.  Nor with a kernel's set-up moved ahead of its wait: attention
// of 8 samples x 128 tokens lost 2 us a launch.)
// `early` is pdl_small_grid() of the launch: at most two CTAs per SM, which both kernels have room for (their launch bounds and shared memory).
inline bool pdl_small_grid(unsigned ctas) { return ctas <= 2u * static_cast<unsigned>(ctx().sm_count); }
__device__ __forceinline__ void pdl_early_if(int early) {
  if (early) pdl_launch_dependents();
}

template <class... P, class... A>
int launch_pdl(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, int cluster, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cluster > 1) {
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = static_cast<unsigned>(cluster);
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.numAttrs = 2;
  }
  MB_CUDA(cudaLaunchKernelEx(&cfg, kern, std::forward<A>(args)...));
  return MIMIR_B200_OK;
}

}  // namespace
}  // namespace mb
