// Kernel launches with programmatic dependent launch (sm_90 and later).
//
// A launch made with launch() may be processed by the device while the
// kernel before it in the stream is still finishing, instead of after a full
// stream serialisation: on GB300 a chain of dependent kernels of about 10 us
// each took 10.8 us per kernel this way against 12.3 us with plain launches
// (the gap between them shrinks from about 2.3 us to under 1 us).  In
// exchange every kernel of this library calls pdl_wait(), which returns once the
// preceding grid in the stream has completed and its memory writes are visible,
// before it touches any buffer that another kernel or a copy writes; so each
// kernel sees exactly what it would after a plain launch.  Most begin with it.
// Before it a kernel may only fill its own shared and tensor memory, and read
// its arguments and the tables that init_device_tables writes once per device
// (the hash kernels on lanes, the path checks and the tree's subtrees load such
// tables, the tensor-core ones copy theirs and allocate tensor memory).  That
// early allocation waits for nothing of the grid before: no kernel here triggers
// its dependents, so a CTA starts after all CTAs of that grid have left and
// freed theirs; a CTA of another stream's tensor kernel does not share an SM
// with it (their registers do not fit) and would free its columns by itself.
// (griddepcontrol.wait returns at once in a kernel that was launched without
// the attribute.)
#pragma once
#include <cuda_runtime.h>

#include <utility>

#include "gpu_shape.h"

namespace whir {
namespace gpu {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// kernel<<<grid, block, smem, stream>>>(args...) with the attribute set; the
// arguments are converted to the kernel's parameter types as <<<>>> does.
// Errors are also left for cudaGetLastError().
template <class... P, class... A>
inline cudaError_t launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem,
                          cudaStream_t st, A &&...args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

}  // namespace gpu
}  // namespace whir
