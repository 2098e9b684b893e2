// launch.cuh -- kernel launches that may begin before their predecessor in the
// stream has ended (programmatic dependent launch).
//
// Between two kernels of a chain the chip drains, the next grid is set up and its
// blocks start cold.  With the launch attribute the next grid is set up while its
// predecessor still runs: every kernel of a chain calls chain_begin() before it
// touches global memory, which lets its own successor be set up and then waits
// until all of its predecessor's work is complete and visible.  A kernel must
// not return before that call, so that completion of a kernel implies completion
// of everything before it in the chain.
//
// What another kernel of the chain writes is read with ordinary loads through
// parameters without __restrict__, never with __ldg: a waiting kernel is resident
// while its predecessors write, so the memory is not constant over its lifetime as
// the read-only path requires, and a load that the compiler may take for invariant
// could also be moved above the wait.  __restrict__ stays on what is constant over
// the chain (work items, channel records, the caller's data) and on what a kernel
// only writes.
//
// Used where one stream runs kernel after kernel with nothing beside it: the
// steps of a context without markers (400 x 80: 6.2 -> 4.0 us a step) and the
// step's bookkeeping kernels (512 x 160 with 40 capsules: 31.7 -> 27.6 us).  Not on
// the forcing sweeps: there the waiting blocks take the places of the side
// streams' kernels (256 learned channels 538 -> 556 us a step, 96 x 40 with two
// capsules 114.6 -> 116.8 us).
#pragma once
#include <cuda_runtime.h>

namespace sfg {

__device__ __forceinline__ void chain_begin() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// `chained`: the stream's previous operation is a kernel of the chain and no
// event wait lies between.
template <typename... P, typename... A>
inline void launch_chain(bool chained, void (*kernel)(P...), int grid, int block, size_t smem,
                         cudaStream_t st, A... args) {
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = chained ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace sfg
