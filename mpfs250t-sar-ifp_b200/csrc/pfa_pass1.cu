// Pass 1 of the float PFA datapath: the per-pulse range resample of form_image_pfa.resample_kspace
// (src/form_image_pfa.py:177-198) and corner turn #1.
//
//   k_fl_pass1<SINC>   per pulse: FP64 source wavenumbers kr = (2 freq / c) pr, np.interp bracket (xp[j] <= x < xp[j+1],
//                      zero outside [xp0, xp_last]), FP32 lerp or the 32-tap float sinc
//   k_fl_pass1_runs    the float sinc where the output grid is about as fine as the samples
//
// All evaluate the source wavenumbers kr = (2 freq / c) pr and the brackets in FP64, apply the optional per-pulse
// phase and write range-bin rows of tan(phi)-sorted pulses.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>

#include "fft_f32.cuh"
#include "interp_f32.cuh"
#include "pfa_internal.h"
#include "pdl.cuh"
#include "stage_ring.cuh"
#include "tc_sm100.cuh"
#include "tma_sm100.cuh"

namespace pfa {
namespace {

constexpr double kC = 299792458.0;

// ------------------------------------------------------------------------------------------ K1f
// Each warp owns a double-buffered window of its pulse's samples: the window of the next pulse streams
// in (cp.async) while the current one is gathered.  The KR grid lies inside every pulse's own span, so
// F1_BINS consecutive bins cover at most F1_BINS + 1 source intervals; a wider window (not produced by
// prepare_tables) falls back to gathering from global memory.
constexpr int F1_SLOTS = 32, F1_WARPS = 8, F1_WMAX = 144;
// range bins per CTA: the sinc variant takes a narrower tile so three CTAs (with the 20 KB table) fit an SM
constexpr int f1_bins(bool sinc) { return sinc ? 64 : 128; }

struct FPass1Args {
    const float2 *sig;
    const double *f0, *df, *flast, *pr, *kr_grid;
    const int32_t *order;
    const int16_t *tabq;
    const uint16_t *tabr;
    const float *theta;     // per-pulse phase correction exp(-j theta_i) (autofocus), or nullptr
    float2 *p1;
    int m, n, mpad;
    int *err;               // set when a bounded wait runs out
    const int32_t *each;    // the runs: nonzero where the plan's present job is not one for them
    int probe;              // test hook of the runs: > 0 = first wait this many polls on a barrier nothing arrives on
};

// per-slot pulse constants, computed once per CTA
struct F1Pulse {
    double f0, df, sc, kfirst, klast, inv_dk;
    float2 rot;
    int i;          // source pulse, -1 for a slot past the last pulse
    int asc;
};

__device__ __forceinline__ F1Pulse pulse_of(const FPass1Args &a, int r) {
    F1Pulse p{};
    p.i = -1;
    p.rot = make_float2(1.f, 0.f);
    if (r < a.m) {
        const int i = a.order[r];
        const double f0 = a.f0[i], df = a.df[i], pri = a.pr[i];
        p.i = i;
        p.f0 = f0;
        p.df = df;
        p.sc = 2.0 * pri / kC;
        // kr[i, k] = (2 freq[i, k] / c) pr[i] (form_image_pfa.py:176-187).  The end points are evaluated
        // with the reference's exact IEEE operations (KR's first and last samples coincide with some
        // pulse's end points, where np.interp returns the end sample); interior samples use the affine
        // model freq = f0 + k df.
        p.kfirst = __dmul_rn(__ddiv_rn(__dmul_rn(2.0, f0), kC), pri);
        p.klast = __dmul_rn(__ddiv_rn(__dmul_rn(2.0, a.flast[i]), kC), pri);
        p.inv_dk = 1.0 / fabs(p.sc * df);               // the source axis is affine in the sample index
        // the phase correction commutes with the (linear, per-pulse) interpolation: rotate the output
        if (a.theta) {
            float sn, cs;
            sincosf(a.theta[i], &sn, &cs);
            p.rot = make_float2(cs, -sn);
        }
    }
    return p;
}

constexpr size_t f1_smem(bool sinc) {
    return (size_t)f1_bins(sinc) * (F1_SLOTS + 1) * 8 + (size_t)F1_WARPS * 2 * F1_WMAX * 8 + (sinc ? kTabShorts * 2 : 0);
}

template <bool SINC>
__global__ void __launch_bounds__(256, SINC ? 3 : 4) k_fl_pass1(FPass1Args a) {
    pdl_wait();
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int F1_BINS = f1_bins(SINC), TB = F1_BINS / 32, SPW = F1_SLOTS / F1_WARPS;
    constexpr size_t TILE_BYTES = (size_t)F1_BINS * (F1_SLOTS + 1) * 8;
    float2(*tile)[F1_SLOTS + 1] = reinterpret_cast<float2(*)[F1_SLOTS + 1]>(smem);
    float2(*win)[2][F1_WMAX] = reinterpret_cast<float2(*)[2][F1_WMAX]>(smem + TILE_BYTES);
    int16_t *tab = reinterpret_cast<int16_t *>(smem + TILE_BYTES + (size_t)F1_WARPS * 2 * F1_WMAX * 8);
    __shared__ F1Pulse prm[F1_SLOTS];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int r0 = blockIdx.x * F1_SLOTS, j0 = blockIdx.y * F1_BINS;
    const int n = a.n;
    if (SINC) {
        const uint4 *src = reinterpret_cast<const uint4 *>(a.tabq);
        uint4 *dst = reinterpret_cast<uint4 *>(tab);
#pragma unroll
        for (int i = 0; i < kTabShorts / 8 / 256; ++i) dst[tid + 256 * i] = __ldg(src + tid + 256 * i);
    }
    if (tid < F1_SLOTS) {
        prm[tid] = pulse_of(a, r0 + tid);
    }
    // the query wavenumbers of this CTA's bins are the same for every pulse
    double q[TB];
#pragma unroll
    for (int t = 0; t < TB; ++t) {
        const int j = j0 + lane + 32 * t;
        q[t] = j < n ? a.kr_grid[j] : 0.0;
    }
    __syncthreads();

    // start the copy of a window (every lane commits one group per slot, possibly empty)
    auto fetch = [&](const F1Pulse &p, int wlo, int whi, float2 *w) {
        if (p.i >= 0 && whi - wlo <= F1_WMAX) {
            const float2 *row = a.sig + (size_t)p.i * n;
            for (int k = wlo + lane; k < whi; k += 32) cp_async8(w + (k - wlo), row + k);
        }
        cp_async_commit();
    };

    // iteration s brackets slot s and starts its window, then gathers slot s - 1 while that copy flies
    int jj[TB], jn[TB];
    Frac fr[TB], fn[TB];
    int wlo = 0, whi = 0, wlo_n = 0, whi_n = 0;
#pragma unroll
    for (int s = 0; s <= SPW; ++s) {
        if (s < SPW) {
            // np.interp bracket of this warp's bins on pulse pn, and the sample window [wlo, whi) they read
            const F1Pulse &pn = prm[warp + F1_WARPS * s];
            wlo_n = whi_n = 0;
            if (pn.i >= 0) {
                auto kr = [&](int k) {
                    return k == 0 ? pn.kfirst : (k == n - 1 ? pn.klast : pn.sc * (pn.f0 + (double)k * pn.df));
                };
                const bool asc = kr(n - 1) >= kr(0);
                auto xa = [&](int t) { return asc ? kr(t) : kr(n - 1 - t); };
                const double xa0 = xa(0), xa1 = xa(n - 1);
                const bool fin = isfinite(pn.inv_dk);
                // xa(ja) for ja in [0, n-2]: xa0 at ja = 0 (the exact end point), the affine model inside
                auto xa_lo = [&](int ja) {
                    return ja == 0 ? xa0 : pn.sc * (pn.f0 + (double)(asc ? ja : n - 1 - ja) * pn.df);
                };
                int lo_i = 1 << 30, hi_i = -1;
#pragma unroll
                for (int t = 0; t < TB; ++t) {
                    jn[t] = -1;
                    fn[t] = Frac{0.f, 0, 0};
                    if (j0 + lane + 32 * t < n && q[t] >= xa0 && q[t] <= xa1) {
                        // closed-form bracket on the affine axis; the end points are exact
                        const double pos = (q[t] - xa0) * pn.inv_dk;
                        const int ja = fin ? min(max((int)floor(pos), 0), n - 2) : 0;
                        const double fd = (q[t] - xa_lo(ja)) * pn.inv_dk;
                        fn[t].f = (float)fd;
                        fn[t].ph = sinc_phase(fd);
                        // natural-order index of the lower sample and the weight toward the upper one
                        int lowi;
                        if (asc) { lowi = ja; } else { lowi = n - 2 - ja; mirror_frac(fn[t]); }
                        jn[t] = lowi;
                        lo_i = min(lo_i, lowi);
                        hi_i = max(hi_i, lowi);
                    }
                }
                lo_i = __reduce_min_sync(0xffffffffu, lo_i);
                hi_i = __reduce_max_sync(0xffffffffu, hi_i);
                if (hi_i >= 0) {
                    wlo_n = max(0, lo_i - (SINC ? 15 : 0));
                    whi_n = min(n, hi_i + (SINC ? 17 : 2));
                }
            } else {
#pragma unroll
                for (int t = 0; t < TB; ++t) jn[t] = -1;
            }
            fetch(pn, wlo_n, whi_n, win[warp][s & 1]);
        }
        if (s > 0) {
            if (s < SPW) cp_async_wait_group<1>(); else cp_async_wait_group<0>();
            __syncwarp();
            const int slot = warp + F1_WARPS * (s - 1);
            const F1Pulse &p = prm[slot];
            if (p.i < 0) {
#pragma unroll
                for (int t = 0; t < TB; ++t) tile[lane + 32 * t][slot] = make_float2(0.f, 0.f);
            } else {
                const bool fits = whi - wlo <= F1_WMAX;
                const float2 *w = win[warp][(s - 1) & 1];
                const float2 *row = a.sig + (size_t)p.i * n;
#pragma unroll
                for (int t = 0; t < TB; ++t) {
                    const int jb = lane + 32 * t;
                    float2 out = make_float2(0.f, 0.f);
                    if (jj[t] >= 0)
                        out = fits ? gather_f32<SINC>(w, wlo, n, jj[t], fr[t], tab)
                                   : gather_f32<SINC>(row, 0, n, jj[t], fr[t], tab);
                    tile[jb][slot] = a.theta ? cmul(out, p.rot) : out;
                }
            }
            __syncwarp();
        }
#pragma unroll
        for (int t = 0; t < TB; ++t) {
            jj[t] = jn[t];
            fr[t] = fn[t];
        }
        wlo = wlo_n;
        whi = whi_n;
    }
    __syncthreads();
    // two slots per lane, two bins per warp store (mpad is a multiple of 32: every slot of the CTA exists)
    const int half = lane >> 4, l2 = 2 * (lane & 15);
    for (int jb = 2 * warp + half; jb < F1_BINS; jb += 2 * F1_WARPS) {
        const int j = j0 + jb;
        if (j >= n) break;
        const float2 u0 = tile[jb][l2], u1 = tile[jb][l2 + 1];
        *reinterpret_cast<float4 *>(a.p1 + (size_t)j * a.mpad + r0 + l2) = make_float4(u0.x, u0.y, u1.x, u1.y);
    }
}

// ------------------------------------------------------------------------------------------ K1f, sinc runs
// A lane owns one of 32 sorted pulses and a thread forms eight consecutive range bins of it (sinc_run), so a warp
// writes one 256-byte row segment of p1 per bin straight from registers: no transposing tile.  One persistent CTA
// per SM walks its share of the (32 pulses x 128 bins) tiles, the same pulses as long as possible; the sample windows of
// the next two tiles arrive by one bulk copy per pulse while a tile is formed, and the 16 warps run ahead of one
// another by up to a tile (full and empty barriers per buffer; a block barrier per tile cost 12 %, and a grid of
// whole CTAs left 14 % of the SMs' time to the last wave).  The windows' pitch is an odd number of 16-byte units, so that
// lanes at equal offsets read distinct bank groups.
// For jobs whose source axes ascend and whose output spacing is within 1/7 of every pulse's sample spacing (so that
// eight outputs stay within a run); the others keep k_fl_pass1<true>.
// What bounds it: ALU and issue slots (three permutes, a packed add and four FMAs per tap pair); the earlier
// lane-per-bin gather was bound by its 105 shared-memory wavefronts per warp and output.
// 8167 x 8192: 1.05 -> 0.56 ms; 2326 x 2054: 0.087 -> 0.061 ms.
constexpr int S1_WARPS = 16, S1_BINS = S1_WARPS * kRunT, S1_BUFS = 3;
constexpr int S1_SLACK = 64;            // samples past the last window that a run may touch (and discard)

// one buffer: the 32 windows, the tile's query wavenumbers, the windows' bounds
constexpr size_t s1_buf(int pitch) { return (size_t)8 * F1_SLOTS * pitch + 8 * S1_BINS + 8 * F1_SLOTS; }
constexpr size_t s1_smem(int pitch) { return (size_t)kRunTabBytes + S1_BUFS * s1_buf(pitch) + 8 * S1_SLACK + stage_ring_bytes(S1_BUFS); }
constexpr int kMaxPitch = 206;          // an odd number of 16-byte units that keeps one CTA within 227 KB
static_assert(s1_smem(kMaxPitch) <= 227 * 1024 && kMaxPitch % 4 == 2, "windows fit beside the table");

// A frame captured in a graph keeps its kernels when the plan gets another job.  Where that one is not for runs, every output
// by itself, as k_fl_pass1<true> forms it.
__device__ __noinline__ void pass1_each(const FPass1Args &a) {
    const int n = a.n;
    const long long total = (long long)n * a.mpad, stride = (long long)gridDim.x * blockDim.x;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total; e += stride) {
        const int j = (int)(e / a.mpad);
        const F1Pulse p = pulse_of(a, (int)(e - (long long)j * a.mpad));
        const double q = a.kr_grid[j];
        const bool asc = p.klast >= p.kfirst;
        const double xa0 = asc ? p.kfirst : p.klast, xa1 = asc ? p.klast : p.kfirst;
        float2 z = make_float2(0.f, 0.f);
        if (p.i >= 0 && q >= xa0 && q <= xa1) {
            const double pos = (q - xa0) * p.inv_dk;
            const int ja = isfinite(p.inv_dk) ? min(max((int)floor(pos), 0), n - 2) : 0;
            const double xl = ja == 0 ? xa0 : p.sc * (p.f0 + (double)(asc ? ja : n - 1 - ja) * p.df);
            const double fd = (q - xl) * p.inv_dk;
            Frac fr{(float)fd, sinc_phase(fd), 0};
            if (!asc) mirror_frac(fr);
            z = gather_f32<true>(a.sig + (long long)p.i * n, 0, n, asc ? ja : n - 2 - ja, fr, a.tabq);
        }
        a.p1[e] = a.theta ? cmul(z, p.rot) : z;
    }
}

__global__ void __launch_bounds__(32 * S1_WARPS, 1) k_fl_pass1_runs(const __grid_constant__ FPass1Args a, int pitch) {
    extern __shared__ __align__(16) unsigned char smem[];
    unsigned char *tab = smem;
    const size_t bufb = s1_buf(pitch);
    auto win_of = [&](int b) { return reinterpret_cast<float2 *>(smem + kRunTabBytes + b * bufb); };
    auto q_of = [&](int b) { return reinterpret_cast<double *>(smem + kRunTabBytes + b * bufb + (size_t)8 * F1_SLOTS * pitch); };
    auto bounds_of = [&](int b) { return reinterpret_cast<int2 *>(q_of(b) + S1_BINS); };
    StageRing<S1_BUFS> ring(smem + kRunTabBytes + S1_BUFS * bufb + 8 * S1_SLACK);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n = a.n, ntiles = (n + S1_BINS - 1) / S1_BINS, groups = a.mpad / F1_SLOTS;
    const int units = ntiles * groups;                       // unit u: tile u % ntiles of pulse group u / ntiles
    const int u0 = (int)((long long)units * blockIdx.x / gridDim.x), u1 = (int)((long long)units * (blockIdx.x + 1) / gridDim.x);
    if (tid == 0) ring.init(S1_WARPS);
    const int each = *a.each;
    run_table_fill(tab, a.tabr, tid, 32 * S1_WARPS);
    pdl_wait();                                              // the tables above belong to the job
    __syncthreads();
    if (each) {
        pass1_each(a);
        return;
    }
    if (u0 >= u1) return;
    constexpr double kMagic = 6755399441055744.0;            // 1.5 * 2^52: an integer in the low word
    // The staging warp's view of the pulses (the warps take turns, so that none falls behind): the copies of unit u, one
    // per pulse, and the tile's query wavenumbers.
    int sg = -1, si = -1;
    double sxa0 = 0.0, sinv = 0.0;
    auto stage = [&](int u) {
        const int g = u / ntiles, b = (u - u0) % S1_BUFS;
        if (g != sg) {
            const F1Pulse q = pulse_of(a, g * F1_SLOTS + lane);
            si = q.i; sxa0 = q.kfirst; sinv = q.inv_dk;
            sg = g;
        }
        // sample window [lo, hi) of this lane's pulse, its ends moved to 16-byte boundaries inside the signal
        const int j0 = (u - g * ntiles) * S1_BINS, cnt = min(S1_BINS, n - j0);
        int lo = 0, hi = 0;
        if (si >= 0) {
            // np.interp's lower index on the affine axis, clamped to [0, n - 2] (floor by a directed rounding)
            auto lower = [&](double q) { return min(max(__double2loint(__dadd_rd((q - sxa0) * sinv, kMagic)), 0), n - 2); };
            const int la = lower(__ldg(a.kr_grid + j0)), lb = lower(__ldg(a.kr_grid + j0 + cnt - 1));
            lo = max(0, min(la, lb) - 15);
            hi = min(n, max(la, lb) + 18);
            const long long e0 = (long long)si * n;
            const int odd = (int)((reinterpret_cast<uintptr_t>(a.sig) >> 3) & 1);
            if ((odd + e0 + lo) & 1) lo += e0 + lo > 0 ? -1 : 1;
            if ((odd + e0 + hi) & 1) hi += e0 + hi < (long long)a.m * n ? 1 : -1;
            if (hi - lo > pitch || hi < lo) hi = lo;         // (not staged: gathered from global memory)
        }
        bounds_of(b)[lane] = make_int2(lo, hi);
        const uint32_t bytes = 8u * (uint32_t)(hi - lo), qbytes = 8u * ((cnt + 1) & ~1);   // kr_grid has a pad element
        const uint32_t total = __reduce_add_sync(0xffffffffu, bytes) + qbytes;
        __syncwarp();
        if (lane == 0) {
            tma::arrive_expect_tx(ring.full + b, total);
            tma::bulk_load(q_of(b), a.kr_grid + j0, qbytes, ring.full + b);
            *ring.staged = u - u0 + 1;
        }
        __syncwarp();
        if (bytes) tma::bulk_load(win_of(b) + lane * pitch, a.sig + (long long)si * n + lo, bytes, ring.full + b);
    };
    if (warp == S1_WARPS - 1) {
        stage(u0);
        if (u0 + 1 < u1) stage(u0 + 1);
    }
    const bool live = a.probe <= 0 || ring.wait(ring.unarmed, 0, (uint32_t)a.probe);
    int cur = -1;
    F1Pulse p{};
    int u = live ? u0 : u1;
    for (; u < u1; ++u) {
        const int it = u - u0, g = u / ntiles, k = u - g * ntiles, b = it % S1_BUFS;
        if (warp == it % S1_WARPS && u + 2 < u1) {
            // the buffer of unit u + 2 is free once every warp is done with unit u - 1
            if (it >= 1 && !ring.released(it - 1)) break;
            stage(u + 2);
        }
        if (g != cur) {
            p = pulse_of(a, g * F1_SLOTS + lane);
            cur = g;
        }
        if (!ring.landed(it)) break;
        const double xa0 = p.kfirst, xa1 = p.klast;
        const int2 bnd = bounds_of(b)[lane];
        const int wlo = bnd.x, whi = bnd.y;
        const double *qs = q_of(b) + warp * kRunT;
        const float2 *w = win_of(b) + lane * pitch;
        const int j0 = k * S1_BINS + warp * kRunT;
        float2 *dst = a.p1 + (size_t)j0 * a.mpad + g * F1_SLOTS + lane;
        // bracket of output t: the lower index and the phase
        int l[kRunT], ph[kRunT], lo = 1 << 30, hi = -(1 << 30);
#pragma unroll
        for (int t = 0; t < kRunT; ++t) {
            const double q = qs[t];
            const double tt = __dadd_rd((q - xa0) * p.inv_dk, kMagic);
            l[t] = __double2loint(tt);
            // interior of a run: 15 <= l, so xa(l) is the affine model (the clamped ends take the other path)
            const double fd = (q - p.sc * (p.f0 + (tt - kMagic) * p.df)) * p.inv_dk;
            ph[t] = min(max(__double2loint(fma(fd, 32768.0, kMagic)), 0), 32767) >> 7;
            lo = min(lo, l[t] - t);
            hi = max(hi, l[t] - t);
        }
        const bool inside = p.i >= 0 && hi - lo <= 1 && lo >= 15 && lo + kRunT <= n - 17 && lo - 15 >= wlo &&
                            lo + kRunT + 17 <= whi;
        // nothing to form (the queries ascend): zeros
        const bool dead = p.i < 0 || qs[kRunT - 1] < xa0 || qs[0] > xa1;
        if (j0 + kRunT <= n && __all_sync(0xffffffffu, inside || dead)) {
            const int at = dead ? 0 : lo - 15 - wlo;
            int o[kRunT];
            float2 out[kRunT];
#pragma unroll
            for (int t = 0; t < kRunT; ++t) {
                o[t] = dead ? 0 : l[t] - t - lo + (at & 1);
                ph[t] = dead ? 0 : ph[t];
            }
            sinc_run(w + (at & ~1), ph, o, tab, out);
            if (dead) {
#pragma unroll
                for (int t = 0; t < kRunT; ++t) out[t] = make_float2(0.f, 0.f);
            }
            if (a.theta) {
#pragma unroll
                for (int t = 0; t < kRunT; ++t) out[t] = cmul(out[t], p.rot);
            }
#pragma unroll
            for (int t = 0; t < kRunT; ++t, dst += a.mpad) *dst = out[t];
        } else {
            const bool fin = isfinite(p.inv_dk);
#pragma unroll 1
            for (int t = 0; t < kRunT && j0 + t < n; ++t) {
                const double q = qs[t];
                float2 z = make_float2(0.f, 0.f);
                if (p.i >= 0 && q >= xa0 && q <= xa1) {
                    const int ja = fin ? min(max(__double2loint(__dadd_rd((q - xa0) * p.inv_dk, kMagic)), 0), n - 2) : 0;
                    const double xl = ja == 0 ? xa0 : p.sc * (p.f0 + (double)ja * p.df);
                    const double fd = (q - xl) * p.inv_dk;
                    const Frac fr{(float)fd, sinc_phase(fd), 0};
                    const bool sinc = ja >= 15 && ja <= n - 17;
                    const bool in = sinc ? ja - 15 >= wlo && ja + 17 <= whi : ja >= wlo && ja + 2 <= whi;
                    const float2 *src = in ? w - wlo : a.sig + (long long)p.i * n;
                    if (sinc) {
#pragma unroll 8
                        for (int i = 0; i < 32; ++i) {
                            const float c = run_tap(tab, fr.ph, i);
                            const float2 x = src[ja - 15 + i];
                            z.x = fmaf(c, x.x, z.x);
                            z.y = fmaf(c, x.y, z.y);
                        }
                        z.x *= 1.0f / 32768.0f;
                        z.y *= 1.0f / 32768.0f;
                    } else {
                        z = gather_f32<false>(src, 0, n, ja, fr, nullptr);
                    }
                }
                dst[(size_t)t * a.mpad] = a.theta ? cmul(z, p.rot) : z;
            }
        }
        ring.release(it);                                    // this warp has read the windows of unit u
    }
    for (u = live ? u : u0; u < u1; ++u) {                   // a copy is lost: zeros
        const int g = u / ntiles, j0 = (u - g * ntiles) * S1_BINS + warp * kRunT;
        for (int j = j0; j < min(j0 + kRunT, n); ++j) a.p1[(size_t)j * a.mpad + g * F1_SLOTS + lane] = make_float2(0.f, 0.f);
    }
    ring.finish(a.err);
}

}  // namespace

cudaError_t float_pass1(const FloatDev &d, const float2 *sig, const float *theta, cudaStream_t st) {
    FPass1Args p{sig, d.f0, d.df, d.flast, d.pr, d.kr, d.order, d.tabq, d.tabr, theta, d.p1, d.m, d.n, d.mpad, d.wait_err, d.each, d.mx_probe};
    const int groups = (d.m + F1_SLOTS - 1) / F1_SLOTS;
    cudaError_t e;
    if (d.range_sinc && d.p1_runs) {
        // windows of a 128-bin tile at the job's widest spacing, an odd number of 16-byte units
        const int pitch = std::min(kMaxPitch, ((int)std::ceil((S1_BINS - 1) * d.p1_ratio) + 38) / 4 * 4 + 2);
        const size_t sm = s1_smem(pitch);
        const int units = (d.n + S1_BINS - 1) / S1_BINS * groups;
        if ((e = allow_smem(k_fl_pass1_runs, kMaxSmem)) != cudaSuccess) return e;
        (void)launch(k_fl_pass1_runs, std::min(units, d.sms), 32 * S1_WARPS, sm, st, p, pitch);
    } else {
        auto k1 = d.range_sinc ? k_fl_pass1<true> : k_fl_pass1<false>;
        const size_t sm = f1_smem(d.range_sinc);
        if ((e = cudaFuncSetAttribute(k1, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm)) != cudaSuccess) return e;
        (void)launch(k1, dim3(groups, (d.n + f1_bins(d.range_sinc) - 1) / f1_bins(d.range_sinc)), 256, sm, st, p);
    }
    return cudaGetLastError();
}

}  // namespace pfa
