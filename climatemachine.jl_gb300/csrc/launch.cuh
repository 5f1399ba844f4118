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
// chain_release stands before a kernel's last phase, not at its start, and
// only in a grid of more CTAs than the next kernel can keep resident on the
// whole GPU (chain_ctas).  The CTAs of a smaller next kernel all start at
// once, on whichever SMs still hold the fewest of this one's, and no longer
// spread evenly; where one SM's pipe is the bound that costs up to what its
// share grows by.  The release of a small grid against none, us per step: 252
// FP64 elements (N = 4) 123 / 75, an FP64 LES of 120 (N = 5) 391 / 245,
// horizontal FP64 hyperdiffusion of 288 shell elements (N = 4) 525 / 302, 729
// mixed elements (N = 3) 18.8 / 16.0; of a large one: 1,560 FP64 elements (N =
// 3) 202 / 214, an FP64 LES of 729 (N = 4) 725 / 810, the 425,250-node GCM with
// hyperdiffusion 276 / 291.  Without the release the next grid starts when
// every CTA has ended, still ahead of an ordinary launch (16.0 / 17.9 us for
// the 729 elements).  A grid of at most half the SMs releases too: both grids'
// CTAs find SMs of their own (64 FP64 elements with hyperdiffusion, N = 4,
// 133 / 139).  Of FP32 CTAs of two warps (N = 2) an SM issues two at once, and
// grids of up to twice the SMs release (252 elements with hyperdiffusion 45.3 /
// 48.8).  The element-wise kernels release first: a successor's
// CTAs find their SMs evenly loaded.  One-wave kernels whose balance over the
// SMs decides (the column substitution) are launched the ordinary way: chained
// behind an early release, a HEVI step took 1.218 against 1.075 ms.
//
// Measured per step, ordinary launches against chained ones: 792 elements
// 30.7 / 20.7 us, the 1 M-node bubble 179 / 167 us, the cubed-shell GCM
// 164 / 149 us, with hyperdiffusion 412 / 347 us, the Smagorinsky LES
// 762 / 720 us, 720,000 nodes as grid arrays 225 / 210 us, a 24-member
// ensemble 1430 / 1393 us.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>
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

// whether a grid of this many CTAs releases the next kernel, which the device
// keeps next_ctas CTAs of resident; light: FP32 CTAs of two warps
inline int chain_releases(int64_t grid, int next_ctas, bool light = false) {
    constexpr int64_t SMS = 152;
    return grid > next_ctas || 2 * grid <= (light ? 4 * SMS : SMS);
}

// CTAs of kernel K that the current device keeps resident, 0 if it cannot be
// asked
template <auto K>
int chain_ctas(unsigned block, size_t smem, int dev = -1) {
    static std::atomic<uint64_t> known[64];  // per device: block size and CTAs
    int per_sm = 0, sms = 0;
    if (dev < 0 && cudaGetDevice(&dev) != cudaSuccess) return 0;
    std::atomic<uint64_t>& slot = known[dev & 63];
    const uint64_t v = slot.load(std::memory_order_relaxed);
    if ((unsigned)(v >> 32) == block) return (int)(uint32_t)v;
    if (cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, K, (int)block, smem) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    slot.store((uint64_t)block << 32 | (uint32_t)(per_sm * sms), std::memory_order_relaxed);
    return per_sm * sms;
}

}  // namespace
}  // namespace cmdg
