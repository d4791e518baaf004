// Programmatic dependent launch: the kernels of a frame are launched before their predecessor has ended and wait for its
// completion before they touch memory that a kernel writes, so that the launch latency overlaps the predecessor's end.
// No kernel triggers its successor explicitly: with a trigger at the start, the successor's CTAs filled the first SMs that
// fell free and left the others idle (1000 x 937 fixed frame 82 us without, 97 with the early trigger, 70 with the
// implicit one at the end; 256 x 240 54, 49, 44).
//
// A kernel that starts before its predecessor has ended may not read what that one writes through the read-only path: that path
// (and a load that the compiler makes of a const __restrict__ parameter) is for memory that stays unchanged while the kernel runs,
// and such loads may be moved above the wait.  So the signal, the image and the buffers between the passes are read by ordinary
// loads; __ldg is for the job's vectors and the plan's tables, which are uploaded by copies, not by kernels.
//
// Every CTA of a kernel launched through `launch` calls pdl_wait, early exits included: a grid that completed without
// waiting would let its own successor start while its predecessor still runs.
#pragma once

#include <cuda_runtime.h>

namespace pfa {
namespace {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class... P, class... A>
cudaError_t launch(void (*fn)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A &&...args) {
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, fn, static_cast<P>(args)...);
}

}  // namespace
}  // namespace pfa
