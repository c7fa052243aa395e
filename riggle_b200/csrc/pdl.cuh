// Programmatic dependent launch.  The short kernels of the pipeline's chains have a PDL variant
// (template flag PDL) that starts with pdl_wait(): it returns once the grid launched before it on
// the stream has completed and its memory is visible, so nothing is read or written before it.
// pdl_release() lets the next grid of the stream be scheduled before this one finishes; that grid
// still waits in pdl_wait() for this one to complete.  Large runs launch the variants without
// either instruction.
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace rgl {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Launches a short kernel of a pipeline chain: with `pdl` its PDL variant (which begins with
// pdl_wait()) with programmatic stream serialization, so that it may be scheduled while the previous
// grid of the stream is finishing; else its plain variant.  PDL is used for small runs, where the
// launch latency between the short kernels of a chain is a visible share of the run.
template <typename... K, typename... A>
cudaError_t launch_chain(bool pdl, void (*with_pdl)(K...), void (*plain)(K...), dim3 grid, dim3 block, size_t smem,
                         cudaStream_t st, A&&... args) {
    if (!pdl) {
        plain<<<grid, block, smem, st>>>(std::forward<A>(args)...);  // errors surface at the next check
        return cudaSuccess;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, with_pdl, std::forward<A>(args)...);
}

}  // namespace rgl
