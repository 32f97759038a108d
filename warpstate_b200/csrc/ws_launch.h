// Launches of a scan's kernel chain with programmatic dependent launch: a
// kernel may be set up while the one before it in the stream still runs, and
// waits on the device (pdl_wait) until that one has completed.  A scan is eight
// to fourteen kernels, most of a few microseconds.  Measured, us a scan without
// and with it: 100 literals over 16 MiB 24.5 -> 19.5, 500 regexes over 64 MiB
// 63 -> 51, 40 anchored ones over 32 MiB 56 -> 42, 60 unbounded ones over 200
// MiB 113 -> 93; a 4 KiB host record 75 -> 62.
//
// Rules: every kernel of the chain starts with pdl_begin() or, where it has
// work that touches only tables no kernel writes, ends that work with
// pdl_wait(); nothing else is read or written before.  All threads of a kernel
// call it, so a kernel completes only after its predecessor has, and the order
// carries over along the chain.  The first kernel of a scan is launched the
// ordinary way, after everything the caller enqueued.
#pragma once
#include <cuda_runtime.h>

#include <utility>

#include "ws_internal.h"

namespace ws {

__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_begin() {
  pdl_trigger();
  pdl_wait();
}

// `first`: the first kernel of a scan, launched the ordinary way.
template <class... P, class... A>
void launch_scan(bool first, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = smem;
  c.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  c.attrs = at;
  c.numAttrs = first ? 0 : 1;
  check_cuda(cudaLaunchKernelEx(&c, kernel, static_cast<P>(std::forward<A>(args))...), "kernel launch");
}

template <class... P, class... A>
void launch_pdl(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
  launch_scan(false, kernel, grid, block, smem, st, std::forward<A>(args)...);
}

}  // namespace ws
