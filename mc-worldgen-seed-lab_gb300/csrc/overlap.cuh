/* overlap.cuh -- kernels of one stream that run at the same time (programmatic dependent launch).
 *
 * A kernel of a batch calls overlap_next() at its start; the next one, launched with launch_on(true, ...), may then begin as soon as
 * its predecessor's blocks are all running and leave room, instead of after the last one's tail.  It does not read what the
 * predecessor writes; overlap_wait() before its end makes its completion imply the predecessor's, so that whatever follows in the
 * stream (launched without the flag) sees both complete.  Without the flag both calls do nothing. */
#ifndef MG_OVERLAP_CUH
#define MG_OVERLAP_CUH
#include <cuda_runtime.h>

namespace mg {

__device__ __forceinline__ void overlap_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void overlap_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... P, typename... A>
cudaError_t launch_on(bool overlap, void (*kernel)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t st, A... args) {
    cudaLaunchConfig_t c = {};
    cudaLaunchAttribute a = {};
    a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    a.val.programmaticStreamSerializationAllowed = 1;
    c.gridDim = dim3(grid);
    c.blockDim = dim3(block);
    c.dynamicSmemBytes = smem;
    c.stream = st;
    c.attrs = &a;
    c.numAttrs = overlap ? 1 : 0;
    return cudaLaunchKernelEx(&c, kernel, P(args)...);
}

}  // namespace mg
#endif
