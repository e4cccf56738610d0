// Programmatic dependent launch: a kernel of a dependent chain starts while its
// predecessor still runs, loads what no kernel of the chain writes (index
// arrays, matrix values, diagonals), and waits for the predecessor before it
// touches a vector.  Every kernel launched through launch_chain calls
// pdl_trigger() first and pdl_wait() in every thread, before its first access
// to chained data: then each kernel completes after its predecessor, and
// waiting for the direct predecessor is waiting for the whole chain.
//
// Why: a chain of small SpMM kernels in a CUDA graph takes 1.39 / 1.69 / 2.44
// us per kernel at 200 / 2000 / 30000 rows; launched this way 0.96 / 1.07 /
// 1.60 us (B200).
#pragma once

#include <cuda_runtime.h>

#include <utility>

#include "emg_internal.h"

namespace emg {

__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// chained: the kernel may start before its predecessor in the stream is done
// (its unwaited loads must then be older than the predecessor)
template <typename... P, typename... A>
inline void launch_chain(void (*kern)(P...), unsigned grid, unsigned block, cudaStream_t s, bool chained, A &&...args) {
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.stream = s;
  cfg.attrs = at;
  cfg.numAttrs = chained ? 1 : 0;
  EMG_CUDA(cudaLaunchKernelEx(&cfg, kern, static_cast<P>(std::forward<A>(args))...));
}

}  // namespace emg
