// Dependent launches: a kernel launched with launch_after may have its blocks brought onto the device while
// the kernel before it on the stream still runs; its first statement is after_previous(), which waits until
// that kernel has finished and its writes are visible, so the order of the work does not change.  What is
// saved is the launch itself (about a microsecond a kernel) between short kernels.  The kernel before
// lets it in by let_next_in() (every block, or its exit).
//
// What such a kernel may read, and how.  Its lifetime begins while the kernel before it still writes, so what
// that kernel may write (any buffer a launch of the library or of its caller writes) is read after
// after_previous() and by plain loads: not by __ldg, and not through a `const ... __restrict__` parameter of the
// kernel, both of which promise that the words do not change from the kernel's start to its end and leave the
// compiler free to move a load above the wait.  The read-only path is for what no launch writes: the tables of
// a batch, a batch's bind poses, skin weights, rest data and indices, the training samples.  (A frame's graph starts
// when the launches before it have ended, so inside it only its own kernels count.)
#pragma once
#include <cuda_runtime.h>

namespace tfx {

__device__ __forceinline__ void after_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_next_in() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <class... P, class... A>
cudaError_t launch_after(void (*kernel)(P...), unsigned blocks, unsigned threads, size_t smem, cudaStream_t s, A... args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace tfx
