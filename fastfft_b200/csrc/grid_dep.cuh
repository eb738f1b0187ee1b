// Programmatic dependent launch: a pass may be scheduled while the pass before it drains.
//
// A transform is a chain of two to five kernels on one stream, each a few microseconds long at
// ordinary sizes, and the gap between two of them (the last blocks' tail, the launch and the first
// blocks' start) is comparable with the kernel itself.  Every pass kernel therefore starts with
// grid_dependency() and is launched with launch_dependent(): it is set up early, its blocks are
// placed once the last block of the earlier grid has left, and they wait in the hardware until
// that grid has completed and its writes are visible.  Nothing is read or written before that
// wait, so the order of all memory accesses is that of ordinary launches.
//
// No pass releases its successor early (griddepcontrol.launch_dependents).  Measured on B200 with
// the release as the first instruction: blocks of the next pass then crowd the multiprocessors
// that the running one leaves empty and keep the side stream's kernels out (us per call, plain
// launches / early release / this form: 1536 x 1280 round trip 35.5 / 43.2 / 27.2, 64-template
// search 538 / 591 / 533, 64^3 -> 256^3 -> 128^3 82 / 74 / 71, complex 512^2 28.2 / 24.5 / 18.7);
// released before the last stores it is as without a release.
#pragma once

#include <cuda_runtime.h>

namespace ffb {

__device__ __forceinline__ void grid_dependency() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class Args, class... More>
inline cudaError_t launch_dependent(void (*fn)(Args, More...), dim3 grid, int threads, size_t smem, cudaStream_t st,
                                    const Args& a, const More&... more) {
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, fn, a, more...);
}

}  // namespace ffb
