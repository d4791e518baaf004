// The barriers of the persistent kernels that stage tiles ahead by bulk copies (k_fl_pass1_runs, k_fl_resample2,
// k_fx_pass1_runs, k_fx_resample2): per buffer one for its copies (full) and one for the warps that are done with it (empty).
//
// Every wait is bounded and taken by a whole warp.  Once one has run out nobody may trust a buffer: the warp leaves the
// pipeline (it reads no window, hands no buffer back and stages nothing, so that no other warp overwrites one that is still
// read or re-arms a barrier whose copies are still on their way), and the waits of the other warps end too.  The
// kernel writes zeros for what it could not form, sets its error flag, and waits for the copies that are still in flight.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "tc_sm100.cuh"

namespace pfa {
namespace {

// Polls of a wait (each try_wait may suspend for a while): a bulk copy lands in microseconds.
constexpr uint32_t kStageWaitPolls = 1u << 22;
// both barriers of each buffer, the test hook's barrier, the two words of the ring's state
constexpr size_t stage_ring_bytes(int bufs) { return (size_t)16 * bufs + 16; }

// Opts a kernel in to `limit` bytes of dynamic shared memory: always the most that any job of it may take, so that plans of
// other jobs on other host threads cannot lower it between this thread's call and its launch.
template <class K>
cudaError_t allow_smem(K fn, size_t limit) {
    return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)limit);
}
constexpr size_t kMaxSmem = 227 * 1024;

template <int BUFS>
struct StageRing {
    uint64_t *full, *empty, *unarmed;   // unarmed: nothing arrives on it (test hook)
    volatile int *lost;                 // a wait has run out
    volatile int *staged;               // units staged so far (they are staged in order)

    __device__ explicit StageRing(unsigned char *at)
        : full(reinterpret_cast<uint64_t *>(at)), empty(full + BUFS), unarmed(empty + BUFS),
          lost(reinterpret_cast<volatile int *>(unarmed + 1)), staged(lost + 1) {}

    // by one thread, before a block barrier
    __device__ void init(int warps) {
        for (int b = 0; b < BUFS; ++b) {
            tc::mbar_init(full + b, 1);
            tc::mbar_init(empty + b, warps);
        }
        tc::mbar_init(unarmed, 1);
        *lost = 0;
        *staged = 0;
        tc::mbar_fence_init();
    }
    // by a whole warp
    __device__ __forceinline__ bool wait(uint64_t *bar, uint32_t parity, uint32_t polls = kStageWaitPolls) {
        bool got = tc::mbar_wait(bar, parity, 1);
        for (uint32_t i = 1; !got && i < polls && !*lost; ++i) got = tc::mbar_wait(bar, parity, 1);
        got = __all_sync(0xffffffffu, got);
        if (!got) *lost = 1;
        return got;
    }
    // the copies of unit `it` (counted from the CTA's first) have landed
    __device__ __forceinline__ bool landed(int it) { return wait(full + it % BUFS, (it / BUFS) & 1); }
    // every warp is done with unit `it`
    __device__ __forceinline__ bool released(int it) { return wait(empty + it % BUFS, (it / BUFS) & 1); }
    // this warp is done with unit `it`
    __device__ __forceinline__ void release(int it) {
        __syncwarp();
        if ((threadIdx.x & 31) == 0) tc::mbar_arrive(empty + it % BUFS);
    }
    // by the whole block, at the end of the kernel
    __device__ __forceinline__ void finish(int *err) {
        __syncthreads();
        if (threadIdx.x == 0 && *lost) {
            atomicExch(err, 1);                              // the frame is not valid
            // leave no copy in flight behind, as far as a bounded wait can tell: the last unit of each buffer
            for (int it = *staged - 1; it >= 0 && it >= *staged - BUFS; --it)
                (void)tc::mbar_wait(full + it % BUFS, (it / BUFS) & 1, kStageWaitPolls);
        }
    }
};

}  // namespace
}  // namespace pfa
