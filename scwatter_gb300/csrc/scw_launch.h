// Kernel launches whose start overlaps the end of the kernel before.
#pragma once

#include <cuda_runtime.h>
#include <utility>

namespace scw {

// A kernel that may be set up while the one before it in the stream still runs; launched plainly, a dependent pair
// is 2.2 us apart.  Every kernel launched so calls chain_wait in all its threads (also those without work) before
// it touches what another kernel writes, or writes what another reads: the wait ends when the one before has ended
// and its writes are visible.  chain_trigger, after the wait, lets the next one's blocks come once all of this
// one's are there; without it they come as this one's end.  The output kernels do not call it: with the next evaluation's
// blocks already there a small volume took 30.4 us in place of 18.0.  Neither does the contraction (1816 us
// with, 1809 without on a large volume).
// A launch under capture is a plain one.
// In the solver the products, their splits, the one-column products and the triangular blocks go out so, each
// waiting at its top: solves of 4 slices of 25 harmonics, 10 of 108 and 20 of 324 took 3.64 / 12.99 / 90.3 ms
// launched plainly, 3.25 / 12.17 / 88.3 ms so.
template <class... P, class... A>
inline cudaError_t launch_chained(bool chained, cudaStream_t stream, dim3 grid, unsigned block, size_t smem,
                                  void (*kernel)(P...), A&&... args) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (chained && (cudaStreamIsCapturing(stream, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone)) chained = false;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = &at;
    cfg.numAttrs = chained ? 1 : 0;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
    return e != cudaSuccess ? cudaGetLastError() : e;         // a refused launch leaves nothing for later checks
}
#ifdef __CUDACC__
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
#endif

}  // namespace scw
