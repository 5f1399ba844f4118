// Kernel launches that overlap their predecessor's end.
//
// A step is a chain of short kernels (5 to 20 of 3 to 90 us), each reading
// what the one before wrote, so between two of them the GPU drains, launches
// and fills again.  launch_chained allows the launch while the kernel before
// it in the stream is still running (programmatic stream serialization);
// inside, chain_release lets the next kernel's CTAs take the places that
// this grid's last wave leaves free, and chain_wait stops until every kernel
// before has finished and its writes are visible.  Before chain_wait a kernel
// touches only what no kernel writes: its launch parameters and the model's
// tables.  A kernel launched the ordinary way passes chain_wait at once.
// For the same reason a chained kernel qualifies only tables __restrict__: of
// a buffer that the kernel before still writes or reads the qualifier would
// say that nothing else touches it, and the compiler could load from it before
// chain_wait or through the non-coherent path.
//
// chain_release stands before a kernel's last phase, not at its start: with
// an early release several small grids wait on the SMs at once and new CTAs
// no longer spread over all of them (a 792-element step 25.0 against 20.7 us,
// a 64-element FP64 tendency 11 to 21 against 10 us, larger meshes the same
// or up to 2% slower).  One-wave kernels whose balance over the SMs decides
// (the column substitution) are launched the ordinary way for that reason:
// chained, a HEVI step took 1.218 against 1.075 ms.
//
// Measured per step, ordinary launches against chained ones: 792 elements
// 30.7 / 20.7 us, the 1 M-node bubble 179 / 167 us, the cubed-shell GCM
// 164 / 149 us, with hyperdiffusion 412 / 347 us, the Smagorinsky LES
// 762 / 720 us, 720,000 nodes as grid arrays 225 / 210 us, a 24-member
// ensemble 1430 / 1393 us.
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace cmdg {
namespace {

__device__ __forceinline__ void chain_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... Formal, typename... Actual>
cudaError_t launch_chained(cudaStream_t s, void (*kernel)(Formal...), unsigned grid, unsigned block, size_t smem,
                           Actual&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid, 1, 1);
    cfg.blockDim = dim3(block, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, std::forward<Actual>(args)...);
    const cudaError_t last = cudaGetLastError();
    return e != cudaSuccess ? e : last;
}

}  // namespace
}  // namespace cmdg
