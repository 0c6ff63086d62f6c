// Kernels that follow one another on a stream, each started while the one before it drains.
//
// A launch made with launch_chained may begin before the kernel in front of it has ended (programmatic
// stream serialisation): its blocks are set up, and a tensor-core pass initialises its barriers and
// takes its tensor memory, while that kernel's last blocks run.  Every such kernel calls chain_wait
// in all its threads before it touches global memory: the wait ends when the kernel in front has
// ended and its writes are visible.  The next kernel may start from chain_next on, which follows the
// wait, so that at most two of a chain are resident together; a pass, whose run time is long, calls
// it when it has loaded its last operand.  Behind anything but such a kernel (a copy, an event, a plain
// launch) the order is the usual one, and so it is in a captured graph.
//
// Small products are bound by launches: FP64 K x at n=2000, M=10k (six kernels) takes 30.5 us instead of
// 39.1, a CG solve at 5,003 x 20,011 1.00 ms instead of 1.20, an AI-REML at 2,000 x 10,000 48.8 ms
// instead of 55.2.  Passes that let the next kernel in at their start ran 1 to 2 % longer.
#pragma once

#include <cuda_runtime.h>

#include "cs_internal.h"

namespace cs {

__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// The next kernel of the chain may start when every block has called this (one thread does) or ended.
__device__ __forceinline__ void chain_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_enter() {
    chain_wait();
    chain_next();
}

// `attrs`: room for one more attribute behind the cfg.numAttrs that are set.
inline void chain(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attrs) {
    attrs[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[cfg.numAttrs].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attrs;
    ++cfg.numAttrs;
}

template <class... P, class... A>
void launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A&&... args) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    chain(cfg, attr);
    CS_CUDA(cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...));
}

}  // namespace cs
