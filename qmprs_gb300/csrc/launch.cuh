// Programmatic launches: a kernel's blocks take their places while the
// kernel before it in the stream still runs.
//
// grid_wait returns when that kernel is complete and its writes are visible,
// and lets the next one start.  Every block of every kernel launched here
// calls it, also one without work, before it writes global memory or reads
// what its predecessor wrote; a kernel has therefore waited for everything
// before its predecessor when it starts, and may read that at once (the tile
// passes build their offset tables, the polar kernel loads its gates).  After
// a copy, a fill or another library's kernel the launch is an ordinary one.
// Measured: about 2.8 us a launch (2400 launches of the blocked
// eigensolver's rounds, 43.7 -> 37.2 ms).
#pragma once

#include <cuda_runtime.h>

__device__ __forceinline__ void grid_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// ... in clusters of `ranks` blocks
template <class... P, class... A>
static void launch_ranks_after(void (*k)(P...), int ranks, dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                               A... args) {
  cudaLaunchAttribute at[2] = {};
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = ranks;
  at[1].val.clusterDim.y = 1;
  at[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = at;
  cfg.numAttrs = ranks > 1 ? 2 : 1;
  cudaLaunchKernelEx(&cfg, k, args...);   // an error stays for cudaGetLastError, as after <<<>>>
}

template <class... P, class... A>
static void launch_after(void (*k)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A... args) {
  launch_ranks_after(k, 1, grid, block, smem, s, args...);
}
