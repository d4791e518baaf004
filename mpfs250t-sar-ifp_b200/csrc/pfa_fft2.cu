// Range FFT and detection of the float PFA datapath (src/form_image_pfa.py:225-240, mpfs/host/accel.py:43).
//
//   k_fl_fft2  per cross bin: FP32 FFT along range (length n2, rows j >= n are the zero pad),
//              fused detection store (|z|, |z|^2 or complex with the (-1)^(u+v) centring sign)
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>

#include "float_lines.cuh"
#include "pdl.cuh"

namespace pfa {
namespace {

// ------------------------------------------------------------------------------------------ K3f
struct FFft2Args {
    const float2 *y1t;
    const float2 *tw;
    void *out;
    int n, npad, centred, detect, inverse;
    float scale;
    int pf;               // L2 prefetch distance in lines (the resident blocks of the grid), 0 = none
    int nlines;
};

template <int L, int E>
__global__ void __launch_bounds__((1 << L) / E, fl_min_ctas(L, E)) k_fl_fft2(FFft2Args a) {
    pdl_wait();
    using F = F32Fft<L, E>;
    constexpr int N = F::N, T = F::T;
    extern __shared__ __align__(16) unsigned char smem[];
    float2 *xbuf = reinterpret_cast<float2 *>(smem);
    const int tid = threadIdx.x;
    const int k = blockIdx.x;                  // cross bin (row of the output image)
    if (a.pf && k + a.pf < a.nlines) l2_prefetch(a.y1t + (size_t)(k + a.pf) * a.npad, (size_t)8 * a.npad, tid);
    float2 x[E];
    const float2 *rowk = a.y1t + (size_t)k * a.npad;
#pragma unroll
    for (int u = 0; u < E; ++u) {
        const int j = tid + T * u;
        x[u] = j < a.n ? __ldcs(rowk + j) : make_float2(0.f, 0.f);
    }
    F::run(x, xbuf, a.tw, tid);
    const size_t base = (size_t)k * N;
    const float cs = a.inverse ? -a.scale : a.scale;     // inverse: conj(FFT(conj(x))) / (m2 n2)
#pragma unroll
    for (int v = 0; v < E; ++v) {
        const int col = tid + T * v;
        float2 z = make_float2(x[v].x * a.scale, x[v].y * cs);
        if (a.detect == PFA_DETECT_MAG) {
            static_cast<float *>(a.out)[base + col] = sqrtf(fmaf(z.x, z.x, z.y * z.y));
        } else if (a.detect == PFA_DETECT_POWER) {
            static_cast<float *>(a.out)[base + col] = fmaf(z.x, z.x, z.y * z.y);
        } else {
            if (a.centred && ((k + col) & 1)) { z.x = -z.x; z.y = -z.y; }
            static_cast<float2 *>(a.out)[base + col] = z;
        }
    }
}

template <int L, int E>
cudaError_t launch_fft2(const FloatDev &d, void *out, int detect, float scale, cudaStream_t st) {
    using F = F32Fft<L, E>;
    FFft2Args p{d.y1, d.twn, out, d.n, d.npad, d.layout == PFA_LAYOUT_CENTRED, detect, d.sgn > 0, scale, 0, d.m2};
    size_t sm = (size_t)8 * F::xbuf_elems();
    auto fn = k_fl_fft2<L, E>;
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    p.pf = resident_blocks(fn, (1 << L) / E, sm);
    (void)launch(fn, d.m2, (1 << L) / E, sm, st, p);
    return cudaGetLastError();
}

template <int L>
cudaError_t fft2_tile(const FloatDev &d, void *out, int detect, float scale, cudaStream_t st) {
    if constexpr (L >= 8 && L <= 13) {
        if (d.ept_range == 8) return launch_fft2<L, 8>(d, out, detect, scale, st);
    }
    if constexpr (L >= 13) {               // the automatic choice (0) for these lines: 32 (measured faster)
        if (d.ept_range == 32 || d.ept_range == 0) return launch_fft2<L, 32>(d, out, detect, scale, st);
    }
    return launch_fft2<L, Cfg<L>::E>(d, out, detect, scale, st);
}

}  // namespace

cudaError_t float_fft2(const FloatDev &d, void *out, int detect, float scale, cudaStream_t st) {
    switch (d.Ln) {
        case 6: return fft2_tile<6>(d, out, detect, scale, st);
        case 7: return fft2_tile<7>(d, out, detect, scale, st);
        case 8: return fft2_tile<8>(d, out, detect, scale, st);
        case 9: return fft2_tile<9>(d, out, detect, scale, st);
        case 10: return fft2_tile<10>(d, out, detect, scale, st);
        case 11: return fft2_tile<11>(d, out, detect, scale, st);
        case 12: return fft2_tile<12>(d, out, detect, scale, st);
        case 13: return fft2_tile<13>(d, out, detect, scale, st);
        case 14: return fft2_tile<14>(d, out, detect, scale, st);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace pfa
