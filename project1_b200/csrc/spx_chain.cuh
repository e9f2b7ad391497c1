// Chains of dependent kernels by programmatic launches: each kernel lets the next one's CTAs
// start as soon as its own have all started (release_next) and waits, before it reads what
// the one before wrote or overwrites what it read, until that has finished (await_previous,
// by every CTA). The first kernel of a chain is an ordinary launch, so what came before is
// complete by then. Launched otherwise, both do nothing.
//
// What a kernel of the chain writes is not constant while the next one runs, so that one reads it
// after the wait with ordinary loads through pointers that are neither __restrict__ nor given to
// __ldg: read-only loads may be moved over the wait. Data complete before the chain starts
// (the products M, tables from the host) may be read in any way and before the wait.
//
// One-slab split calls: 96 columns, 160 pairs, 4 frequencies 24.6 us unchained, 20.5 chained;
// 403 columns, 12201 pairs, 12 frequencies 447 and 430. GEMMs and panels of the dielectric
// inverse: 24 matrices of 1200 8.41 and 8.35 ms, 4 of 168 277 and 260 us.
#pragma once
#include <cuda_runtime.h>

namespace spx {

__device__ __forceinline__ void release_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void await_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
template <typename... P, typename... A>
static cudaError_t launch_chained(void (*kernel)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t s,
                                  bool chained, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = chained ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace spx
