// Pass 2 of the float PFA datapath: the cross resample of form_image_pfa.resample_kspace (src/form_image_pfa.py:199-222),
// the Hamming window, the FFT along cross and corner turn #2.
//
//   k_fl_pass2_fft  per range bin j: source KR[j] * tan_s (FP64), bracket, gather, float32 Hamming
//                   product window, (-1)^(j+k) centring modulation, FP32 FFT along cross (length m2)
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>

#include "float_lines.cuh"
#include "pdl.cuh"
#include "tc_sm100.cuh"
#include "tma_sm100.cuh"

namespace pfa {
namespace {

// ------------------------------------------------------------------------------------------ K2f
struct FPass2Args {
    CUtensorMap p1_map;   // TMA map of the pass-1 output rows (boxes of 256 samples)
    const double *tan_s, *kr_grid, *kc_grid, *ham_m, *ham_n;
    const int16_t *tabq;
    const float2 *tw;
    float2 *y1t;          // [m2][npad] cross-FFT output, transposed: row = cross bin, col = range bin
    uint32_t *pk_out;     // packed brackets [j][k] for the autofocus adjoint, or nullptr
    float2 *rp_out;       // float sinc, autofocus forward: R2 p1 [j][k] before the window (the adjoint's
                          // W^2 R2 p1 term), or nullptr
    int *err;             // set when the row load's bounded wait runs out
    int m, n, mpad, npad, centred, window, inverse;
    int probe;            // test hook: > 0 = first wait this many polls on a barrier nothing arrives on
    double *ysum;         // PK (autofocus forward): += sum |y1|^2 over the frame (S / n2, by Parseval)
};

// Polls of the pass-2 row-load wait (each try_wait may suspend for a while): a TMA row load lands in
// microseconds, so running out means the copy is lost; the frame is then flagged, not waited for.
constexpr uint32_t kRowWaitPolls = 1u << 22;

// Shared-memory bytes of pass 2's region A: the row as whole 256-sample boxes, or the FFT exchange buffer.
__host__ __device__ constexpr size_t pass2_region_a(int m, size_t xbuf_elems) {
    return ((size_t)2048 * ((m + 255) / 256) > (size_t)8 * xbuf_elems ? (size_t)2048 * ((m + 255) / 256)
                                                                       : (size_t)8 * xbuf_elems);
}

// PK: also store the packed brackets for the autofocus adjoint (lerp only; a separate instantiation so
// that the frame's pass 2 carries no extra register pressure)
template <int L, int E, bool SINC, bool PK = false>
__global__ void __cluster_dims__(kCT, 1, 1) __launch_bounds__((1 << L) / E, fl_min_ctas(L, E))
k_fl_pass2_fft(const __grid_constant__ FPass2Args a) {
    pdl_wait();
    using F = F32Fft<L, E>;
    constexpr int N = F::N, T = F::T;
    extern __shared__ __align__(1024) unsigned char smem[];
    // layout: [region A: the row (whole TMA boxes) | exchange buffer] [sinc table] [row mbarrier, probe]
    // [PK: T / 32 doubles of the |y1|^2 reduction].  No static shared memory: region A starts the window.
    const int m = a.m;
    const size_t regA = pass2_region_a(m, F::xbuf_elems());
    float2 *row = reinterpret_cast<float2 *>(smem);
    float2 *xbuf = reinterpret_cast<float2 *>(smem);
    int16_t *tab = reinterpret_cast<int16_t *>(smem + regA);
    uint64_t *row_bar = reinterpret_cast<uint64_t *>(smem + regA + (SINC ? 2 * kTabShorts : 0));
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const int tid = threadIdx.x;
    // clusters in reverse range-bin order (a cluster's CTAs stay adjacent, rank order kept): pass 1 wrote
    // the high range-bin rows of p1 last, so the first clusters find their rows in L2
    const int j = (int)(gridDim.x - kCT - (blockIdx.x & ~(kCT - 1)) + (blockIdx.x & (kCT - 1)));
    const bool live = j < a.n;                 // grid is padded to a multiple of the cluster size
    float2 x[E];
    bool landed = true, issued = false;
    if (live) {
    // The row (256-sample boxes of the p1 tensor map) and the sinc table stream into shared memory by TMA
    // while the brackets are computed; warp 0 issues the copies.
    issued = (tma::saddr(row) & 127) == 0;          // CTA-uniform; a misaligned box is never issued
    if (tid == 0) {
        tc::mbar_init(row_bar, 1);
        tc::mbar_init(row_bar + 1, 1);     // the test hook's barrier: never arrived on
        tc::mbar_fence_init();
        tc::fence_smem_to_async();
    }
    __syncthreads();
    if (tid < 32 && issued) {
        const int nbox = (m + 255) >> 8;
        if (tid == 0) tma::arrive_expect_tx(row_bar, 2048u * nbox + (SINC ? 2u * kTabShorts : 0u));
        __syncwarp();
        for (int b = tid; b < nbox; b += 32) tma::load_2d(row + 256 * b, &a.p1_map, 256 * b, j, row_bar);
        if (SINC && tid == 0) tma::bulk_load(tab, a.tabq, 2u * kTabShorts, row_bar);
    }
    const double krj = a.kr_grid[j];
    const double s0 = krj * a.tan_s[0], s1 = krj * a.tan_s[m - 1];
    const bool asc = s1 >= s0;
    auto xa = [&](int t) { return krj * __ldg(a.tan_s + (asc ? t : m - 1 - t)); };
    const double lo_v = asc ? s0 : s1, hi_v = asc ? s1 : s0;
    const double inv_span = (double)(m - 1) / (hi_v - lo_v);
    const double hn = a.window ? a.ham_n[j] : 1.0;
    int bl[E];      // packed bracket: lower natural index | phase << 16 | reversed << 24; -1 = outside
    float bf[E];    // lerp weight toward the upper sample
    constexpr int CH = 2;
#pragma unroll
    for (int u0 = 0; u0 < E; u0 += CH) {
        double q[CH];
        bool ok[CH];
#pragma unroll
        for (int c = 0; c < CH; ++c) {
            const int k = tid + T * (u0 + c);
            ok[c] = k < m;
            q[c] = ok[c] ? __ldg(a.kc_grid + k) : 0.0;
        }
        int ja[CH];
        Frac fr[CH];
        interp_brackets<SINC, CH>(xa, m, lo_v, hi_v, inv_span, q, ok, ja, fr);
#pragma unroll
        for (int c = 0; c < CH; ++c) {
            const int u = u0 + c;
            if constexpr (PK) {
                // the adjoint's brackets on the ascending view (fraction and phase before any mirroring)
                if (ok[c]) {
                    uint32_t pkv;
                    if (ja[c] < 0) pkv = pack_br(1, q[c] < lo_v ? 0 : m - 2, 0.f);
                    else if (SINC && ja[c] >= 15 && ja[c] <= m - 17) pkv = pack_br_phase(ja[c], fr[c].ph);
                    else pkv = pack_br(0, ja[c], fr[c].f);
                    a.pk_out[(size_t)j * a.mpad + tid + T * u] = pkv;
                }
            }
            bl[u] = -1;
            bf[u] = 0.f;
            if (ja[c] >= 0) {
                int lowi = ja[c];
                if (!asc) { lowi = m - 2 - ja[c]; mirror_frac(fr[c]); }
                bl[u] = lowi | (fr[c].ph << 16) | (fr[c].rev << 24);
                bf[u] = fr[c].f;
            }
        }
    }
    // sinc: warp 0 waits for the row and the block barrier passes its view of the landed bytes to the other
    // warps; lerp: every thread waits (each measured the faster of the two for its kernel, by ~1 %)
    const bool probe_ok = a.probe <= 0 || tc::mbar_wait(row_bar + 1, 0, (uint32_t)a.probe);
    if constexpr (SINC) {
        bool got = true;
        if (tid < 32) got = issued && probe_ok && tc::mbar_wait(row_bar, 0, kRowWaitPolls);
        landed = __syncthreads_and(got) != 0;
    } else {
        landed = issued && probe_ok && tc::mbar_wait(row_bar, 0, kRowWaitPolls);
        __syncthreads();
    }
    if (!landed) atomicExch(a.err, 1);      // any thread whose wait ran out: the frame is not valid
#pragma unroll
    for (int u = 0; u < E; ++u) {
        const int k = tid + T * u;
        float2 val = make_float2(0.f, 0.f);
        if (k < m && landed) {
            if (bl[u] >= 0) {
                const int lowi = bl[u] & 0xffff;
                const Frac fr{bf[u], (bl[u] >> 16) & 0xff, (bl[u] >> 24) & 1};
                val = gather_f32<SINC>(row, 0, m, lowi, fr, tab);
                if constexpr (PK && SINC) a.rp_out[(size_t)j * a.mpad + k] = val;   // R2 p1 for the adjoint
                // np.outer(hamming(m), hamming(n)).astype(float32)[k, j]
                const float wgt = a.window ? (float)(a.ham_m[k] * hn) : 1.0f;
                const float sg = (a.centred && ((j + k) & 1)) ? -wgt : wgt;
                val.x *= sg;
                val.y *= sg;
            } else if constexpr (PK && SINC) {
                a.rp_out[(size_t)j * a.mpad + k] = make_float2(0.f, 0.f);
            }
        }
        x[u] = a.inverse ? make_float2(val.x, -val.y) : val;
    }
    F::run(x, xbuf, a.tw, tid);
    if constexpr (PK) {
        // the autofocus needs S = sum |z|^2 before its range adjoint: z = F_range y1 along zero-padded lines
        // of n2, so S = n2 sum |y1|^2 (Parseval), summed here where y1 is formed
        double *ysum_red = reinterpret_cast<double *>(row_bar + 2);   // dynamic: static shared memory
        double sq = 0.0;                                              // would move region A off 128 bytes
#pragma unroll
        for (int v = 0; v < E; ++v) sq += (double)fmaf(x[v].x, x[v].x, x[v].y * x[v].y);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
        if ((tid & 31) == 0) ysum_red[tid >> 5] = sq;
        __syncthreads();
        if (tid == 0) {
            double t = 0.0;
            for (int w = 0; w < T / 32; ++w) t += ysum_red[w];
            atomicAdd(a.ysum, t);
        }
    }
    } else {
#pragma unroll
        for (int v = 0; v < E; ++v) x[v] = make_float2(0.f, 0.f);
    }
    // exchange buffer: this CTA's FFT row in natural frequency order (stays conjugated for the inverse)
    __syncthreads();
#pragma unroll
    for (int v = 0; v < E; ++v) xbuf[tid + T * v] = x[v];
    cluster.sync();
    const int rank = (int)cluster.block_rank();
    const int j0 = j - rank;
    constexpr int SLICE = N / kCT;
#pragma unroll
    for (int s2 = 0; s2 < E; ++s2) {
        const int item = tid + T * s2;         // item = kk * kCT + r
        const int r = item % kCT;
        const int k = rank * SLICE + item / kCT;
        const float2 *remote = cluster.map_shared_rank(xbuf, r);
        a.y1t[(size_t)k * a.npad + j0 + r] = remote[k];
    }
    cluster.sync();                            // keep this CTA's shared memory alive for the readers
    if (issued && !landed) (void)tc::mbar_wait(row_bar, 0, kRowWaitPolls);   // no copy left in flight at exit
}

template <int L, int E, bool SINC>
cudaError_t launch_pass2(const FloatDev &d, cudaStream_t st) {
    using F = F32Fft<L, E>;
    FPass2Args p{d.p1_map, d.tan_s, d.kr, d.kc, d.ham_m64, d.ham_n64, d.tabq, d.twm, d.y1, d.pk_out, d.rp_out, d.wait_err,
                 d.m, d.n, d.mpad, d.npad, d.layout == PFA_LAYOUT_CENTRED, d.window, d.sgn > 0,
                 d.mixed ? 0 : d.mx_probe, d.pk_out ? d.af_acc : nullptr};
    // + 2 mbarriers + the autofocus forward's reduction scratch
    const size_t sm = pass2_region_a(d.m, F::xbuf_elems()) + (SINC ? kTabShorts * 2 : 0) + 16 +
                      (d.pk_out ? (size_t)8 * std::max(1, F::T / 32) : 0);
    auto fn = k_fl_pass2_fft<L, E, SINC>;
    if (d.pk_out) fn = k_fl_pass2_fft<L, E, SINC, true>;
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    (void)launch(fn, d.npad, (1 << L) / E, sm, st, p);
    return cudaGetLastError();
}

// FFT register tile: 16 complex values per thread; 8 on request (twice the CTA size) for lines of 256
// points and more; 32 (half the CTA size, radix-32 passes: one shared-memory exchange fewer) for lines
// of 8192 and 16384 points, on request and by default for the range FFT (0 = automatic).  The cross
// FFT of pass 2 stays at 16 by default: that kernel is latency bound and loses more to the halved
// CTA than it gains from the saved exchange.
template <int L, bool SINC>
cudaError_t pass2_tile(const FloatDev &d, cudaStream_t st) {
    if constexpr (L >= 8 && L <= 13) {      // 2^L / 8 threads must stay within a CTA's 1024
        if (d.ept_cross == 8) return launch_pass2<L, 8, SINC>(d, st);
    }
    if constexpr (L >= 13) {
        if (d.ept_cross == 32) return launch_pass2<L, 32, SINC>(d, st);
    }
    return launch_pass2<L, Cfg<L>::E, SINC>(d, st);
}

template <bool SINC>
cudaError_t dispatch_pass2(const FloatDev &d, cudaStream_t st) {
    switch (d.Lm) {
        case 6: return pass2_tile<6, SINC>(d, st);
        case 7: return pass2_tile<7, SINC>(d, st);
        case 8: return pass2_tile<8, SINC>(d, st);
        case 9: return pass2_tile<9, SINC>(d, st);
        case 10: return pass2_tile<10, SINC>(d, st);
        case 11: return pass2_tile<11, SINC>(d, st);
        case 12: return pass2_tile<12, SINC>(d, st);
        case 13: return pass2_tile<13, SINC>(d, st);
        case 14: return pass2_tile<14, SINC>(d, st);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace

cudaError_t float_pass2(const FloatDev &d, cudaStream_t st) {
    if (d.p2_runs && d.az_sinc) {
        const cudaError_t e = float_resample2(d, st);
        return e != cudaSuccess ? e : float_row_fft(d, st);
    }
    return d.az_sinc ? dispatch_pass2<true>(d, st) : dispatch_pass2<false>(d, st);
}

}  // namespace pfa
