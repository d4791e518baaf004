// Image-entropy autofocus of the float PFA: the gradient of the image entropy with respect to the per-pulse phase and the
// descent step on the device.  The reference has no autofocus; the image it differentiates is form_image_pfa.pfa
// (src/form_image_pfa.py:243-246).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>

#include <string>

#include "float_lines.cuh"
#include "pdl.cuh"

namespace pfa {
namespace {

// ------------------------------------------------------------------------------------------ autofocus
// Image-entropy autofocus gradient.  With x = s exp(-j theta) (applied in pass 1), p1 = R1 x,
// z = F_range F_cross (W . R2 p1), I = |z|^2 and E = -sum p log p (p = I / S):
//   g_z  = dE/dconj(z) = -(1/S)(log(I/S) + E) z                     (0 where I = 0)
//   g_p1 = R2^H (W . F_cross^H F_range^H g_z)
//   dE/dtheta_i = 2 Im sum_j conj(g_p1[j, slot_i]) p1[j, slot_i]     (pass 1 is linear and per pulse,
//                 so its adjoint never has to be formed)
// The range FFT is recomputed from the cross-FFT buffer in the adjoint pass instead of storing z.  One
// pass over z suffices: S = n2 sum |y1|^2 comes from the forward pass 2 (Parseval), the range adjoint
// takes the part -(1/S) log(I/S) z of g_z and sums I log I on the way, and the part -(E/S) z, whose
// adjoint is -(E/S) n2 m2 R2^H (W^2 . R2 p1) (F^H F = N on the zero-padded lines), is added in the cross
// adjoint, when E is known.
struct AfRangeArgs {
    const float2 *y1t;      // [m2][npad] forward cross-FFT output, transposed
    const float2 *tw;       // range twiddles (n2)
    double *acc;            // [0] sum |y1|^2 (from the forward pass 2), [1] += sum I log I
    float2 *zadj_t;         // [n][m2] F_range^H (-(1/S) log(I/S) z), range-bin rows
    int n, npad, m2;
};

template <int L, int E>
__device__ __forceinline__ void af_load_range_row(float2 (&x)[E], const AfRangeArgs &a, int k) {
    constexpr int T = (1 << L) / E;
    const float2 *row = a.y1t + (size_t)k * a.npad;
#pragma unroll
    for (int u = 0; u < E; ++u) {
        const int j = threadIdx.x + T * u;
        x[u] = j < a.n ? __ldcs(row + j) : make_float2(0.f, 0.f);
    }
}

template <int L, int E>
__global__ void __cluster_dims__(kCT, 1, 1) __launch_bounds__((1 << L) / E, fl_min_ctas(L, E))
k_af_range_adjoint(AfRangeArgs a) {
    pdl_wait();
    namespace cg = cooperative_groups;
    using F = F32Fft<L, E>;
    constexpr int N = F::N, T = F::T;
    extern __shared__ __align__(16) unsigned char smem[];
    float2 *xbuf = reinterpret_cast<float2 *>(smem);
    cg::cluster_group cluster = cg::this_cluster();
    const int tid = threadIdx.x;
    const int k = blockIdx.x;                         // cross bin
    const double S = a.acc[0] * (double)N;
    const float invS = (float)(1.0 / S), off = (float)(-log(S));
    __shared__ double hred[T / 32];
    float2 x[E];
    af_load_range_row<L, E>(x, a, k);
    F::run(x, xbuf, a.tw, tid);                       // recompute z along range
    float hf = 0.f;                                   // this thread's sum I log I (E values; double beyond)
#pragma unroll
    for (int v = 0; v < E; ++v) {
        const float in = fmaf(x[v].x, x[v].x, x[v].y * x[v].y);
        const float lg = in > 0.f ? logf(in) : 0.f;
        hf = fmaf(in, lg, hf);
        const float c = in > 0.f ? -invS * (lg + off) : 0.f;            // -(1/S) log(I/S)
        x[v] = make_float2(c * x[v].x, -c * x[v].y);                    // conj of that part of g_z
    }
    double h = (double)hf;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) h += __shfl_xor_sync(0xffffffffu, h, o);
    if ((tid & 31) == 0) hred[tid >> 5] = h;
    F::run(x, xbuf, a.tw, tid);                       // F^H g = conj(F conj(g))
    __syncthreads();                                  // hred complete
    if (tid == 0) {
        double t = 0.0;
        for (int w = 0; w < T / 32; ++w) t += hred[w];
        atomicAdd(a.acc + 1, t);
    }
    __syncthreads();
#pragma unroll
    for (int v = 0; v < E; ++v) xbuf[tid + T * v] = make_float2(x[v].x, -x[v].y);   // range index j
    cluster.sync();
    const int rank = (int)cluster.block_rank();
    const int k0 = k - rank;
    constexpr int SLICE = N / kCT;
#pragma unroll
    for (int s2 = 0; s2 < E; ++s2) {
        const int item = tid + T * s2;
        const int r = item % kCT;
        const int j = rank * SLICE + item / kCT;
        if (j < a.n) {
            const float2 *remote = cluster.map_shared_rank(xbuf, r);
            a.zadj_t[(size_t)j * a.m2 + k0 + r] = remote[j];
        }
    }
    cluster.sync();
}

struct AfCrossArgs {
    const float2 *zadj_t;   // [n][m2]
    const float2 *p1;       // [n][mpad] forward pass-1 output (phase corrected)
    const uint32_t *pk;     // [n][mpad] packed brackets of the forward pass 2 (ascending view)
    const float2 *rp;       // sinc: [n][mpad] R2 p1 of the forward pass 2 (before the window)
    const double *ham_m, *ham_n;
    const double *kr_grid, *tan_s;   // the direction of range bin j's pass-2 source axis
    const int16_t *tabq;    // float sinc table (Q15 taps, [phase][kTabRow])
    const float2 *tw;       // cross twiddles (m2)
    float *dacc;            // [mpad] per-slot Im sum conj(g_p1) p1
    const double *acc;      // [0] sum |y1|^2, [1] sum I log I (complete once the range adjoint has run)
    int m, n, mpad, window, n2;
};

// Shared-memory positions of bracket k and of W . F^H g at cross index k in the cross adjoint.  Its
// segmented reduction has lane t walk indices near 16 t; XOR-ing the low four index bits with bits of
// the group index (a permutation inside each aligned group of 16) spreads those lanes over the banks
// (4-byte brackets: bits 5..8; 8-byte values: bits 4..7), and consecutive writers stay conflict free.
__device__ __forceinline__ int pk_at(int k) { return k ^ ((k >> 5) & 15); }
__device__ __forceinline__ int y_at(int k) { return k ^ ((k >> 4) & 15); }
__device__ __forceinline__ float br_w(uint32_t p) { return (float)(p & 0x1ffffu) * (1.0f / 131071.f); }

// R2^H as an atomics-free segmented reduction.  On the ascending view of the sources, bracket k (lower index
// l_k, monotone in k) touches slots l_k and l_k + 1 (lerp: weights 1 - f and f) or, for an interior float
// sinc bracket, slots l_k - 15 .. l_k + 16 (weight tab[phase][u - l_k + 15] / 2^15).  So slot u collects
// the contiguous run of k with l_k in [u - 16, u + 15] (sinc) or [u - 1, u] (lerp).  Each thread owns E
// consecutive slots: the lerp walks one run per slot; the sinc reads each bracket of the union of its
// slots' runs once and adds it to every slot it reaches.  A descending source axis maps ascending slot u to
// natural slot m - 1 - u (the forward mirrors the bracket and reverses the taps, which is the same map).
template <int L, int E, bool SINC>
__global__ void __launch_bounds__((1 << L) / E, fl_min_ctas(L, E)) k_af_cross_adjoint(AfCrossArgs a) {
    pdl_wait();
    using F = F32Fft<L, E>;
    constexpr int N = F::N, T = F::T;
    constexpr int REACH_LO = SINC ? 16 : 1, REACH_HI = SINC ? 15 : 0;
    extern __shared__ __align__(16) unsigned char smem[];
    float2 *xbuf = reinterpret_cast<float2 *>(smem);
    uint32_t *pk = reinterpret_cast<uint32_t *>(smem + (size_t)8 * F::xbuf_elems());
    const int tid = threadIdx.x;
    const int j = blockIdx.x;                         // range bin (< n)
    const int m = a.m;
    int16_t *tab = reinterpret_cast<int16_t *>(smem + (size_t)8 * F::xbuf_elems() + (size_t)4 * ((m + 15) & ~15));
    // the forward pass-2 brackets of this range bin (stored by the forward pass 2 of this gradient)
    {
        const uint32_t *src = a.pk + (size_t)j * a.mpad;
        for (int k = tid; k < m; k += T) pk[pk_at(k)] = __ldcs(src + k);
        if (SINC) {
            const uint4 *t4 = reinterpret_cast<const uint4 *>(a.tabq);
            for (int c = tid; c < kTabShorts / 8; c += T) reinterpret_cast<uint4 *>(tab)[c] = __ldg(t4 + c);
        }
    }
    const double krj = a.kr_grid[j];
    const bool asc = krj * a.tan_s[m - 1] >= krj * a.tan_s[0];    // as the forward pass 2 decides
    // adjoint of the cross FFT
    const float2 *row = a.zadj_t + (size_t)j * N;
    float2 x[E];
#pragma unroll
    for (int u = 0; u < E; ++u) {
        const float2 v = __ldcs(row + tid + T * u);
        x[u] = make_float2(v.x, -v.y);
    }
    F::run(x, xbuf, a.tw, tid);
    const double hn = a.window ? a.ham_n[j] : 1.0;
    // the -(E/S) z part of g_z: -(E/S) n2 m2 W^2 . R2 p1 at cross index k, R2 p1 from the forward brackets
    const double S = a.acc[0] * (double)a.n2;
    const double Ent = log(S) - a.acc[1] / S;
    const float beta = (float)(-(Ent / S) * (double)a.n2 * (double)N);
    const float2 *p1row = a.p1 + (size_t)j * a.mpad;
    auto nat = [&](int t) { return asc ? t : m - 1 - t; };   // ascending-view source -> natural slot
    __syncthreads();
    // four cross indices at a time: their two lerp samples are loaded (clamped indices, so unconditionally)
    // before any is used, so the loads of the four overlap
    constexpr int QB = E >= 4 ? 4 : E;
    static_assert(E % QB == 0, "tile of whole load batches");
#pragma unroll
    for (int v0 = 0; v0 < E; v0 += QB) {
        uint32_t bb[QB];
        float2 s0[QB], s1[QB];
#pragma unroll
        for (int c = 0; c < QB; ++c) {
            const int k = tid + T * (v0 + c);
            bb[c] = k < m ? pk[pk_at(k)] : 0x80000000u;
            if constexpr (SINC) {
                // the forward pass 2 stored R2 p1 (its 32-tap gathers): one coalesced load per cross index
                s0[c] = k < m ? __ldcs(a.rp + (size_t)j * a.mpad + k) : make_float2(0.f, 0.f);
            } else {
                const int l = min(br_low(bb[c]), m - 2);
                s0[c] = p1row[nat(l)];
                s1[c] = p1row[nat(l + 1)];
            }
        }
#pragma unroll
        for (int c = 0; c < QB; ++c) {
            const int v = v0 + c;
            const int k = tid + T * v;
            const float w = k < m ? (a.window ? (float)(a.ham_m[k] * hn) : 1.0f) : 0.f;
            float2 fw = make_float2(0.f, 0.f);          // (R2 p1)[k]
            if constexpr (SINC) {
                fw = s0[c];
            } else if (!(bb[c] >> 31)) {
                const float f = br_w(bb[c]);
                fw = make_float2(fmaf(f, s1[c].x - s0[c].x, s0[c].x), fmaf(f, s1[c].y - s0[c].y, s0[c].y));
            }
            const float bw = beta * w * w;
            // W . F_cross^H g, cross index k
            xbuf[y_at(k)] = make_float2(fmaf(bw, fw.x, w * x[v].x), fmaf(bw, fw.y, -w * x[v].y));
        }
    }
    __syncthreads();
    const int r_lo = tid * E;
    float2 gs[E];
#pragma unroll
    for (int s2 = 0; s2 < E; ++s2) gs[s2] = make_float2(0.f, 0.f);
    if (r_lo < m) {
        // The brackets of queries outside the row's source span carry no weight.  They are a prefix of k
        // (packed with lower index 0) and a suffix (lower index m - 2), so they sit inside the runs of
        // the first and the last slots; walking them would cost those threads (and their CTA) one step per
        // dead bracket and slot.  The walks cover only the live range [k0, k1).
        int k0, k1;
        {
            int lo = 0, hi = m;                         // first k past the dead prefix
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                const uint32_t b = pk[pk_at(mid)];
                if ((b >> 31) && br_low(b) == 0) lo = mid + 1; else hi = mid;
            }
            k0 = lo;
            hi = m;                                     // first dead k at or after k0: the dead suffix
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (!(pk[pk_at(mid)] >> 31)) lo = mid + 1; else hi = mid;
            }
            k1 = lo;
        }
        int lo = k0, hi = k1;                           // first live k with lower index >= r_lo - REACH_LO
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (br_low(pk[pk_at(mid)]) < r_lo - REACH_LO) lo = mid + 1; else hi = mid;
        }
        int kp = lo;
        if constexpr (SINC) {
            // Bracket-outer: every live bracket whose taps reach one of this thread's E slots (lower index
            // l in [r_lo - 16, r_lo + E + 14]) is read once and added to each slot it reaches, in the same
            // increasing-k order per slot as a slot-by-slot walk.  Interior brackets add tap r - l + 15 of
            // their phase row as the integer Q15 value, edge brackets their lerp weights times 2^15; the
            // sums are scaled by 2^-15 at the end (a power of two commutes with every rounding, so each sum
            // is the one the float taps give).
            for (int kk = kp; kk < k1; ++kk) {
                const uint32_t b = pk[pk_at(kk)];
                const int l = br_low(b);
                if (l > r_lo + E - 1 + REACH_HI) break;
                const float2 y = xbuf[y_at(kk)];
                if (l >= 15 && l <= m - 17) {
                    const int16_t *row = tab + (b & 0xffu) * kTabRow;
                    const int t0 = r_lo - l + 15;          // tap of slot r_lo
#pragma unroll
                    for (int s2 = 0; s2 < E; ++s2) {
                        if ((unsigned)(t0 + s2) < 32u) {
                            const float w = s16f(row[t0 + s2]);
                            gs[s2].x = fmaf(w, y.x, gs[s2].x);
                            gs[s2].y = fmaf(w, y.y, gs[s2].y);
                        }
                    }
                } else if (!(b >> 31)) {
                    const float f = br_w(b);
                    const float w0 = (1.0f - f) * 32768.f, w1 = f * 32768.f;
#pragma unroll
                    for (int s2 = 0; s2 < E; ++s2) {
                        const int r = r_lo + s2;
                        if (r == l) {
                            gs[s2].x = fmaf(w0, y.x, gs[s2].x);
                            gs[s2].y = fmaf(w0, y.y, gs[s2].y);
                        } else if (r == l + 1) {
                            gs[s2].x = fmaf(w1, y.x, gs[s2].x);
                            gs[s2].y = fmaf(w1, y.y, gs[s2].y);
                        }
                    }
                }
            }
#pragma unroll
            for (int s2 = 0; s2 < E; ++s2) {
                gs[s2].x *= 1.0f / 32768.f;
                gs[s2].y *= 1.0f / 32768.f;
                if (r_lo + s2 >= m) gs[s2] = make_float2(0.f, 0.f);
            }
        } else {
#pragma unroll
            for (int s2 = 0; s2 < E; ++s2) {
                const int r = r_lo + s2;
                if (r < m) {
                    float2 gsum = make_float2(0.f, 0.f);
                    for (int kk = kp; kk < k1; ++kk) {
                        const uint32_t b = pk[pk_at(kk)];
                        const int l = br_low(b);
                        if (l > r + REACH_HI) break;
                        if (b >> 31) continue;
                        const float f = br_w(b);
                        const float wgt = (l == r) ? 1.0f - f : (l == r - 1 ? f : 0.f);
                        const float2 y = xbuf[y_at(kk)];
                        gsum.x = fmaf(wgt, y.x, gsum.x);
                        gsum.y = fmaf(wgt, y.y, gsum.y);
                    }
                    while (kp < k1 && br_low(pk[pk_at(kp)]) < r + 1 - REACH_LO) ++kp;
                    gs[s2] = gsum;
                }
            }
        }
    }
    // the slot sums go through shared memory (padded: a thread's E consecutive slots hit distinct banks)
    // so that the p1 loads and the accumulation run slot-coalesced, all of a thread's loads in flight
    __syncthreads();
#pragma unroll
    for (int s2 = 0; s2 < E; ++s2) xbuf[F::pad(r_lo + s2)] = gs[s2];
    __syncthreads();
    float2 pv[E];
#pragma unroll
    for (int v = 0; v < E; ++v) {
        const int r = tid + T * v;
        pv[v] = r < m ? __ldcs(p1row + r) : make_float2(0.f, 0.f);
    }
#pragma unroll
    for (int v = 0; v < E; ++v) {
        const int r = tid + T * v;                    // natural slot
        if (r < m) {
            const float2 g = xbuf[F::pad(asc ? r : m - 1 - r)];
            atomicAdd(a.dacc + r, g.x * pv[v].y - g.y * pv[v].x);   // Im(conj(g) p1)
        }
    }
}

__global__ void k_af_finish(const float *dacc, const int32_t *order, const double *acc, float *dtheta, double *ent, int m,
                            int n2) {
    pdl_wait();
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r < m && dtheta) dtheta[order[r]] = 2.0f * dacc[r];
    if (r == 0 && ent) {
        const double S = acc[0] * (double)n2;
        ent[0] = log(S) - acc[1] / S;
    }
}

// One step of the autofocus descent on the device: g = dE/dtheta (2 dacc in slot order), theta <- theta -
// step (g - mean g) / max |g - mean g| (a constant phase does not change the image).  One block.
__global__ void __launch_bounds__(1024) k_af_update(const float *dacc, const int32_t *order, float *theta, int m,
                                                    float step) {
    pdl_wait();
    __shared__ double red[32];
    __shared__ float bc[2];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    double s = 0.0;
    for (int r = tid; r < m; r += blockDim.x) s += 2.0 * (double)dacc[r];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) red[warp] = s;
    __syncthreads();
    if (tid == 0) {
        double t = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w];
        bc[0] = (float)(t / m);
    }
    __syncthreads();
    const float mean = bc[0];
    float mx = 0.f;
    for (int r = tid; r < m; r += blockDim.x) mx = fmaxf(mx, fabsf(2.0f * dacc[r] - mean));
    mx = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(mx)));   // non-negative floats
    if (lane == 0) red[warp] = mx;
    __syncthreads();
    if (tid == 0) {
        float t = 0.f;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t = fmaxf(t, (float)red[w]);
        bc[1] = fmaxf(t, 1e-30f);
    }
    __syncthreads();
    const float scale = step / bc[1];
    for (int r = tid; r < m; r += blockDim.x) theta[order[r]] -= scale * (2.0f * dacc[r] - mean);
}

template <int L>
cudaError_t launch_af_range(const FloatDev &d, cudaStream_t st) {
    using F = F32Fft<L, Cfg<L>::E>;
    AfRangeArgs p{d.y1, d.twn, d.af_acc, d.af_zadj, d.n, d.npad, d.m2};
    const size_t sm = (size_t)8 * F::xbuf_elems();
    auto f2 = k_af_range_adjoint<L, Cfg<L>::E>;
    const cudaError_t e = cudaFuncSetAttribute(f2, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    (void)launch(f2, d.m2, Cfg<L>::T, sm, st, p);
    return cudaGetLastError();
}

template <int L>
cudaError_t launch_af_cross(const FloatDev &d, cudaStream_t st) {
    using F = F32Fft<L, Cfg<L>::E>;
    AfCrossArgs p{d.af_zadj, d.p1, d.af_pk, d.af_rp, d.ham_m64, d.ham_n64, d.kr, d.tan_s, d.tabq, d.twm, d.af_dacc, d.af_acc,
                  d.m, d.n, d.mpad, d.window, d.n2};
    // exchange buffer, packed brackets (whole groups of 16), sinc table
    const size_t sm = (size_t)8 * F::xbuf_elems() + (size_t)4 * ((d.m + 15) & ~15) + (d.az_sinc ? kTabShorts * 2 : 0);
    auto fn = d.az_sinc ? k_af_cross_adjoint<L, Cfg<L>::E, true> : k_af_cross_adjoint<L, Cfg<L>::E, false>;
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    (void)launch(fn, d.n, Cfg<L>::T, sm, st, p);
    return cudaGetLastError();
}

cudaError_t af_range(const FloatDev &d, cudaStream_t st) {
#define CALL(Lx) launch_af_range<Lx>(d, st)
    switch (d.Ln) {
        case 6: return CALL(6); case 7: return CALL(7); case 8: return CALL(8); case 9: return CALL(9);
        case 10: return CALL(10); case 11: return CALL(11); case 12: return CALL(12); case 13: return CALL(13);
        case 14: return CALL(14);
        default: return cudaErrorInvalidValue;
    }
#undef CALL
}

cudaError_t af_cross(const FloatDev &d, cudaStream_t st) {
#define CALL(Lx) launch_af_cross<Lx>(d, st)
    switch (d.Lm) {
        case 6: return CALL(6); case 7: return CALL(7); case 8: return CALL(8); case 9: return CALL(9);
        case 10: return CALL(10); case 11: return CALL(11); case 12: return CALL(12); case 13: return CALL(13);
        case 14: return CALL(14);
        default: return cudaErrorInvalidValue;
    }
#undef CALL
}

// Entropy and its gradient w.r.t. the per-pulse phase correction theta (float32; lerp or float sinc passes).
cudaError_t autofocus_grad(const FloatDev &d0, const float2 *sig, const float *theta, float *dtheta, double *ent,
                           cudaStream_t st, StageProf *prof) {
    StageProf none;
    StageProf &pf = prof ? *prof : none;
    pf.count = 0;
    cudaError_t e = pf.mark(st, "start");
    if (e != cudaSuccess) return e;
    FloatDev d = d0;
    d.layout = PFA_LAYOUT_NATURAL;      // |z| (so E) does not depend on the centring
    d.sgn = -1;
    d.pk_out = d.af_pk;                 // the forward pass 2 keeps its brackets for the cross adjoint
    d.rp_out = d.az_sinc && !d.p2_runs ? d.af_rp : nullptr;   // and, float sinc, its resampled rows (p2_runs: in g2 anyway)
    if ((e = cudaMemsetAsync(d.af_acc, 0, 256 + sizeof(float) * d.mpad, st)) != cudaSuccess) return e;     // and af_dacc behind it
    if ((e = float_pass1(d, sig, theta, st)) != cudaSuccess) return e;
    if ((e = pf.mark(st, "pass1_phase")) != cudaSuccess) return e;
    if ((e = float_pass2(d, st)) != cudaSuccess) return e;
    if ((e = pf.mark(st, "pass2_win_fft1")) != cudaSuccess) return e;
    if ((e = af_range(d, st)) != cudaSuccess) return e;
    if ((e = pf.mark(st, "range_entropy_adjoint")) != cudaSuccess) return e;
    if ((e = af_cross(d, st)) != cudaSuccess) return e;
    if ((e = pf.mark(st, "cross_adjoint_pass2T")) != cudaSuccess) return e;
    (void)launch(k_af_finish, (d.m + 255) / 256, 256, 0, st, d.af_dacc, d.order, d.af_acc, dtheta, ent, d.m, d.n2);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    return pf.mark(st, "finish");
}

}  // namespace
}  // namespace pfa

// ------------------------------------------------------------------------------------------ C ABI
namespace {
pfa_status ffail(pfa_plan *p, pfa_status st, const char *msg) {
    if (p) p->err = msg;
    return st;
}
struct DevGuard {
    int prev = -1;
    explicit DevGuard(int dev) { if (cudaGetDevice(&prev) != cudaSuccess) prev = -1; if (prev != dev) cudaSetDevice(dev); }
    ~DevGuard() { int cur = -1; if (prev >= 0 && cudaGetDevice(&cur) == cudaSuccess && cur != prev) cudaSetDevice(prev); }
};
pfa_status fcuda(pfa_plan *p, cudaError_t e, const char *where) {
    if (p) p->err = std::string(where) + ": " + cudaGetErrorString(e);
    return e == cudaErrorMemoryAllocation ? PFA_ERR_ALLOC : PFA_ERR_CUDA;
}
}  // namespace

extern "C" {

static pfa_status autofocus_common(pfa_plan *p, const float *sig_dev, const float *theta_dev, float *dtheta_dev,
                                   double *entropy_dev, void *stream);

pfa_status pfa_autofocus_step(pfa_plan *p, const float *sig_dev, float *theta_dev, float step, double *entropy_dev,
                              void *stream) {
    if (!p || !sig_dev || !theta_dev) return PFA_ERR_BAD_ARG;
    pfa_status st = autofocus_common(p, sig_dev, theta_dev, nullptr, entropy_dev, stream);
    if (st != PFA_OK) return st;
    DevGuard dg(p->device);
    (void)pfa::launch(pfa::k_af_update, 1, 1024, 0, reinterpret_cast<cudaStream_t>(stream), p->fl.af_dacc, p->fl.order, theta_dev,
                      p->fl.m, step);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? PFA_OK : fcuda(p, e, "autofocus update");
}

pfa_status pfa_autofocus_grad(pfa_plan *p, const float *sig_dev, const float *theta_dev, float *dtheta_dev,
                              double *entropy_dev, void *stream) {
    if (!p || !sig_dev || !theta_dev || !dtheta_dev) return PFA_ERR_BAD_ARG;
    return autofocus_common(p, sig_dev, theta_dev, dtheta_dev, entropy_dev, stream);
}

static pfa_status autofocus_common(pfa_plan *p, const float *sig_dev, const float *theta_dev, float *dtheta_dev,
                                   double *entropy_dev, void *stream) {
    if (p->cfg.mode != PFA_MODE_FLOAT32 && p->cfg.mode != PFA_MODE_MIXED) return ffail(p, PFA_ERR_BAD_CONFIG, "plan is not float mode");
    if (!p->job_ready) return ffail(p, PFA_ERR_NOT_READY, "pfa_set_float_job not called");
    pfa::FloatDev &d = p->fl;
    if (reinterpret_cast<uintptr_t>(sig_dev) & 7) return ffail(p, PFA_ERR_BAD_ARG, "signal must be 8-byte aligned");
    DevGuard dg(p->device);
    cudaError_t e;
    if (!d.af_blocks && (e = pfa::Arena::allocate(d.af_blocks, [&](pfa::Arena &a) {
            a.take(d.af_acc, 2); a.take(d.af_dacc, d.mpad);          // cleared together
            (void)a.together();
            a.take(d.af_zadj, (size_t)d.n * d.m2); a.take(d.af_pk, (size_t)d.n * d.mpad);
            // whichever pass 2 the job takes, now or later
            if (d.az_sinc && d.g2) d.af_rp = d.g2;
            else if (d.az_sinc) a.take(d.af_rp, (size_t)d.n * d.mpad);
        })) != cudaSuccess)
        return fcuda(p, e, "autofocus workspace");
    e = pfa::autofocus_grad(d, reinterpret_cast<const float2 *>(sig_dev), theta_dev, dtheta_dev, entropy_dev,
                            reinterpret_cast<cudaStream_t>(stream), &p->prof);
    if (e != cudaSuccess) return fcuda(p, e, "autofocus");
    return PFA_OK;
}

}  // extern "C"
