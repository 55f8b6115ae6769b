// Programmatic dependent launch of short kernels that follow one another on a stream: the next
// kernel's blocks take their places while the last blocks of the one before still run, and
// wait there for its end.  Every kernel that is launched so calls follow_wait() before its
// first access to memory, in every block: a kernel behind it may then rely on everything
// before.  follow_next() lets the next kernel's blocks in once all of this one's have started.
// Both do nothing in an ordinary launch.
#pragma once

#include <cuda_runtime.h>

namespace gain {

__device__ __forceinline__ void follow_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void follow_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <class... P, class... A>
cudaError_t launch_following(void (*kernel)(P...), unsigned blocks, unsigned threads, cudaStream_t st, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(threads);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

}  // namespace gain
