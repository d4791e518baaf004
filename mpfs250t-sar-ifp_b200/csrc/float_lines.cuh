// What the float kernels of pfa_pass2.cu, pfa_fft2.cu and pfa_autofocus.cu share: the line FFT and its CTA shapes, the cluster
// of the corner turn, the packed pass-2 brackets, and launch helpers.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "fft_f32.cuh"
#include "interp_f32.cuh"
#include "pfa_internal.h"

namespace pfa {
namespace {

// FFT: register Stockham radix-16 (fft_f32.cuh).
template <int L, int E>
using F32Fft = StockhamFft<L, E>;

// resident CTAs per SM the line kernels are compiled for: 64 registers a thread for tiles of up to 16
// values, 128 for the 32-value tile (its radix-32 passes hold 64 floats of data)
constexpr int fl_min_ctas(int L, int E) {
    return E >= 32 ? (((1 << L) / E >= 512) ? 1 : 2) : (((1 << L) / E >= 1024) ? 1 : (((1 << L) / E >= 512) ? 2 : 4));
}

// Corner turn #2 fused into the cross FFT: a cluster of kCT CTAs holds kCT adjacent range bins; after
// their FFTs each CTA writes a 1/kCT slice of cross bins for all kCT rows (kCT * 8-byte runs) into the
// transposed buffer, reading the other rows from the cluster's distributed shared memory.  Four CTAs:
// a run fills one 32-byte sector, and 4-CTA clusters pack a GPC's SMs more fully than 8-CTA ones
// (pass 2 at 8192^2: 0.87 ms with 4, 0.95 with 2, 0.99 with 8).
constexpr int kCT = 4;
static_assert(8 % kCT == 0, "npad (a multiple of 8) must hold whole clusters");

// packed pass-2 bracket (written by the forward pass 2 of an autofocus gradient for the adjoint), on the
// ascending view of the pass-2 sources: bit 31 = outside the span, bits 17..30 = lower index ja, bits 0..16 =
// the lerp weight toward ja + 1 (x 131071) or, for an interior bracket of the float sinc (15 <= ja <= m-17,
// where no lerp weight is needed), the sinc phase
__device__ __forceinline__ uint32_t pack_br(int dead, int lowi, float f) {
    const uint32_t q = (uint32_t)fminf(fmaxf(rintf(f * 131071.f), 0.f), 131071.f);
    return ((uint32_t)dead << 31) | ((uint32_t)lowi << 17) | q;
}
__device__ __forceinline__ uint32_t pack_br_phase(int lowi, int ph) { return ((uint32_t)lowi << 17) | (uint32_t)ph; }
__device__ __forceinline__ int br_low(uint32_t p) { return (int)((p >> 17) & 0x3fffu); }

// Blocks of `fn` resident on the whole device at once (the L2 prefetch distance of the line kernels).
template <class K>
int resident_blocks(K fn, int threads, size_t smem) {
    int dev = 0, sms = 0, per = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, threads, smem) != cudaSuccess) {
        (void)cudaGetLastError();           // no prefetch; leave no error behind for the launch check
        return 0;
    }
    return sms * per;
}

template <int L>
struct Cfg {
    static constexpr int N = 1 << L;
    static constexpr int E = (N >= 512) ? 16 : (N / 32);
    static constexpr int T = N / E;
};

}  // namespace
}  // namespace pfa
