// Programmatic dependent launch: the kernels of one call sequence follow each other on one stream, and at small batches the gap
// between two of them costs as much as the work.  A kernel launched with launch_pdl may start while its predecessor drains; it
// reads constants (tables, plans, keys) right away and waits for the predecessor's results only then.
//
// Rules that keep this safe: pdl_wait() stands before the first access to any buffer that another kernel of the stream writes or
// reads (the buffer pool hands buffers on in stream order), every block executes it, and pointers to such buffers are not
// __restrict__ const (the compiler may hoist a read-only load over the wait).  A kernel without the wait is launched the
// ordinary way and so starts only when everything before it has finished.
#pragma once
#include <cuda_runtime.h>
#include <utility>

namespace hb {

// the predecessor has finished and its writes are visible; from here on the successor may be scheduled
__device__ __forceinline__ void pdl_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// the error is returned and not left for the next cudaGetLastError, which would blame another call
template <class... P, class... A>
inline cudaError_t launch_pdl(cudaStream_t st, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, A &&...args) {
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = st;
    cfg.attrs = at; cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, P(std::forward<A>(args))...);
    if (e != cudaSuccess) cudaGetLastError();
    return e;
}

} // namespace hb
