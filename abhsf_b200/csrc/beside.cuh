// beside.cuh -- kernels of one product that run side by side on one stream.
//
// A product is up to three kernels over disjoint rows of y (chains, sliced rows,
// the ring or streaming kernel).  The first is an ordinary launch, so it starts
// after everything queued before it.  Each of the others is launched with the
// programmatic-serialization attribute: it may start once every CTA of the one
// before it runs (they let it at their start), and one of its threads waits for
// the one before to complete before it ends.  So the last kernel of the product
// ends after all of them, and whatever comes next on the stream after that.  A
// second stream with two events and two waits did the same for about 6 us a
// product more.
#pragma once

#include "common.cuh"

namespace abhsf {

// The kernels of one product queued so far.
struct beside {
    bool any = false;
};

template <typename... P, typename... A>
void launch_beside(beside& b, void (*kern)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t st, A... args)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = b.any ? 1 : 0;
    ABHSF_CUDA(cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...));
    b.any = true;
}

// At a kernel's start, by every thread: the next kernel of the product may start.
__device__ __forceinline__ void beside_begin() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// At the end, by every thread that gets there (thread 0 of CTA 0 must): the
// kernel before is complete.
__device__ __forceinline__ void beside_end()
{
    if (threadIdx.x == 0 && blockIdx.x == 0 && blockIdx.y == 0)
        asm volatile("griddepcontrol.wait;" ::: "memory");
}

}  // namespace abhsf
