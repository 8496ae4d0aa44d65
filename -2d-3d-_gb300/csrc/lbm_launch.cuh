// lbm_launch.cuh - launches of the step kernels that overlap with the end of the kernel before.
//
// Consecutive kernels of a step depend on each other, so on small lattices most of a step was
// the way from one kernel's end to the next one's first load.  A kernel launched by launch_after
// may start while the one before it drains: it computes its indices and then waits
// (wait_for_previous) until that kernel has finished and its writes are visible, before its first
// access to memory.  start_next, after a block's stores, lets the next kernel be brought up while
// this one's last writes are made visible.  Earlier it costs more than it gives: the next kernel's
// blocks then fill what the first SMs to finish have free, and a small grid ends up on a few SMs
// (GB300, us per step without / early / late: plain FP64 2D 256x128 19.4 / 55 / 18.2, FP64
// accuracy 256x128 5.3 / 6.5 / 4.0 and 128x64 4.4 / 4.2 / 3.6).
// Every kernel launched this way waits, so each one also finds everything before its predecessor
// finished.
// What such a kernel reads was written during its own lifetime, so it takes no read-only loads
// (__ldg, or what the compiler makes of a const __restrict__ kernel parameter): those may be moved
// above the wait or served from a cache that does not see the writes.
#pragma once

#include <cuda_runtime.h>

namespace lbm {

__device__ __forceinline__ void start_next() { asm volatile("griddepcontrol.launch_dependents;"); }
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class... P, class... A>
static void launch_after(void (*kernel)(P...), unsigned grid, unsigned block, cudaStream_t s, A&&... args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.stream = s;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace lbm
