// Pass 2's resample of the float PFA datapath on its own: the cross resample of form_image_pfa.resample_kspace
// (src/form_image_pfa.py:199-222) from the range-bin rows of pass 1 to the KC grid, with the Hamming window and the centring
// sign; the FFT along cross follows in another kernel (k_fl_row_fft or the tensor-core one).
//
// A lane owns one of 32 adjacent range bins and a thread forms eight consecutive cross samples of it.  Adjacent
// range bins have nearly the same brackets, so the query grid, tan(phi) and the tapers are read as broadcasts from
// shared memory, where the fused kernel (a lane per cross sample) read five different doubles a lane; the FP64 bracket
// of a run needs one search and then at most two steps per output.  The 32 rows' sample windows of a 128-sample tile
// arrive by one bulk copy each, ahead of the tile, as in pass 1.
//
// For jobs with ascending source axes whose pulses are nearly uniform in tan(phi) and whose output spacing is near the
// sources' (pass2_rule, host_rules.h); the others keep the fused k_fl_pass2_fft.  2326 x 2054: pass 2 178 -> 119 us;
// 8167 x 8192: 1.69 -> 1.15 ms (0.78 of it here).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>

#include "float_lines.cuh"
#include "pdl.cuh"
#include "stage_ring.cuh"
#include "tc_sm100.cuh"
#include "tma_sm100.cuh"

namespace pfa {
namespace {

constexpr int R2_ROWS = 32;
// Warps (eight cross samples each) and buffers of a CTA.  Sinc: one CTA per SM, 16 warps, three buffers beside the 64 KB
// table.  Lerp: two CTAs of 12 warps with three buffers each.
constexpr int r2_warps(bool sinc) { return sinc ? 16 : 12; }
constexpr int R2_BUFS = 3;
constexpr int r2_tile(bool sinc) { return r2_warps(sinc) * kRunT; }
// window pitch and tan segment for a job's widest output spacing (in source samples) and slack of the affine guess
constexpr int r2_reach(bool sinc, double ratio, int slack) {
    return (int)((r2_tile(sinc) - 1) * ratio) + 1 + 2 * slack + (sinc ? 42 : 12);
}
constexpr int R2_SLACK = 64;            // samples past the last window that a run may touch (and discard)

struct Resample2Args {
    const float2 *p1;                   // [n][mpad]
    const double *tan_s, *kr_grid, *kc_grid, *ham_m, *ham_n;
    const uint16_t *tabr;
    const int16_t *tabq;
    const int32_t *each;                // nonzero where the plan's present job is not one for this kernel
    float2 *g2;                         // [n][mpad]
    uint32_t *pk_out;                   // sinc: [n][mpad] packed brackets for the autofocus adjoint, or nullptr
    int *err;
    int m, n, mpad, centred, window;
    int pitch, tlen, slack;             // window pitch (samples), tan segment length, slack of the affine guess (samples)
    int probe;                          // test hook: > 0 = first wait this many polls on a barrier nothing arrives on
};

// one buffer: 32 windows, the tile's queries and tapers, the tan segment, the windows' starts and ends, the segment's start
__host__ __device__ constexpr size_t r2_buf(bool sinc, int pitch, int tlen) {
    return (size_t)8 * R2_ROWS * pitch + 16 * r2_tile(sinc) + 8 * tlen + 8 * R2_ROWS + 16;
}
constexpr size_t r2_smem(bool sinc, int pitch, int tlen) {
    return (sinc ? kRunTabBytes : 0) + R2_BUFS * r2_buf(sinc, pitch, tlen) + 8 * R2_SLACK + stage_ring_bytes(R2_BUFS);
}

// 1 / d for a normal positive d well inside the float range, to the last bit or two (Newton from the float reciprocal)
__device__ __forceinline__ double recip_newton(double d) {
    double r = (double)__frcp_rn((float)d);
    r = fma(fma(-d, r, 1.0), r, r);
    return fma(fma(-d, r, 1.0), r, r);
}

// A frame captured in a graph keeps its kernels when the plan gets another job.  Where that one is not for this kernel, every
// output by itself, as the fused kernels form it.
template <bool SINC>
__device__ __noinline__ void resample_each(const Resample2Args &a) {
    const int m = a.m;
    const long long total = (long long)a.n * a.mpad, stride = (long long)gridDim.x * blockDim.x;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total; e += stride) {
        const int j = (int)(e / a.mpad), k = (int)(e - (long long)j * a.mpad);
        if (k >= m) continue;
        const double krj = a.kr_grid[j], q = a.kc_grid[k], s0 = krj * a.tan_s[0], s1 = krj * a.tan_s[m - 1];
        const bool asc = s1 >= s0;
        auto xa = [&](int t) { return krj * __ldg(a.tan_s + (asc ? t : m - 1 - t)); };
        const double lo_v = asc ? s0 : s1, hi_v = asc ? s1 : s0, inv_span = (double)(m - 1) / (hi_v - lo_v);
        const int g = isfinite(inv_span) ? min(max((int)((q - lo_v) * inv_span), 0), m - 2) : 0;
        Frac f{0.f, 0, 0};
        const int ja = interp_bracket<SINC>(xa, m, lo_v, hi_v, q, g, f);
        if (SINC && a.pk_out)
            a.pk_out[e] = ja < 0 ? pack_br(1, q < lo_v ? 0 : m - 2, 0.f)
                                 : ja >= 15 && ja <= m - 17 ? pack_br_phase(ja, f.ph) : pack_br(0, ja, f.f);
        float2 z = make_float2(0.f, 0.f);
        if (ja >= 0) {
            if (!asc) mirror_frac(f);
            z = gather_f32<SINC>(a.p1 + (size_t)j * a.mpad, 0, m, asc ? ja : m - 2 - ja, f, a.tabq);
        }
        const float wgt = a.window ? (float)(a.ham_m[k] * a.ham_n[j]) : 1.0f;
        const float sg = (a.centred && ((j + k) & 1)) ? -wgt : wgt;
        a.g2[e] = make_float2(z.x * sg, z.y * sg);
    }
}

template <bool SINC>
__global__ void __launch_bounds__(32 * r2_warps(SINC), SINC ? 1 : 2) k_fl_resample2(const __grid_constant__ Resample2Args a) {
    constexpr int R2_WARPS = r2_warps(SINC), R2_TILE = r2_tile(SINC), BUFS = R2_BUFS;
    extern __shared__ __align__(16) unsigned char smem[];
    unsigned char *tab = smem, *bufs = smem + (SINC ? kRunTabBytes : 0);
    const int pitch = a.pitch, tlen = a.tlen;
    const size_t bufb = r2_buf(SINC, pitch, tlen);
    auto win_of = [&](int b) { return reinterpret_cast<float2 *>(bufs + b * bufb); };
    auto q_of = [&](int b) { return reinterpret_cast<double *>(bufs + b * bufb + (size_t)8 * R2_ROWS * pitch); };
    auto ham_of = [&](int b) { return q_of(b) + R2_TILE; };
    auto tan_of = [&](int b) { return q_of(b) + 2 * R2_TILE; };
    auto bounds_of = [&](int b) { return reinterpret_cast<int2 *>(tan_of(b) + tlen); };
    StageRing<BUFS> ring(bufs + BUFS * bufb + 8 * R2_SLACK);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int m = a.m, n = a.n, ntiles = (m + R2_TILE - 1) / R2_TILE, groups = (n + R2_ROWS - 1) / R2_ROWS;
    const int units = ntiles * groups;                       // unit u: tile u % ntiles of row group u / ntiles
    const int u0 = (int)((long long)units * blockIdx.x / gridDim.x), u1 = (int)((long long)units * (blockIdx.x + 1) / gridDim.x);
    if (tid == 0) ring.init(R2_WARPS);
    const int each = *a.each;
    if (SINC) run_table_fill(tab, a.tabr, tid, 32 * R2_WARPS);
    pdl_wait();                                              // the tables above belong to the job
    __syncthreads();
    if (each) {
        resample_each<SINC>(a);
        return;
    }
    if (u0 >= u1) return;
    const double tan0 = a.tan_s[0], tan1 = a.tan_s[m - 1];
    // This lane's row: scale of the sources, span, and samples per wavenumber of the affine guess.
    struct Row { double kr, lo, hi, inv; };
    auto row_of = [&](int j) {
        Row r;
        r.kr = a.kr_grid[min(j, n - 1)];
        r.lo = r.kr * tan0;
        r.hi = r.kr * tan1;
        r.inv = (double)(m - 1) / (r.hi - r.lo);
        return r;
    };
    auto guess = [&](const Row &r, double q) { return min(max((int)((q - r.lo) * r.inv), 0), m - 2); };
    // The warps take turns to stage a unit: one window per row, the tile's queries and tapers, the tan segment.
    int sg = -1;
    Row sr{};
    auto stage = [&](int u) {
        const int g = u / ntiles, b = (u - u0) % BUFS, j = g * R2_ROWS + lane;
        if (g != sg) {
            sr = row_of(j);
            sg = g;
        }
        const int k0 = (u - g * ntiles) * R2_TILE, cnt = min(R2_TILE, m - k0);
        int lo = 0, hi = 0, tl = m;
        if (j < n) {
            const int ga = guess(sr, __ldg(a.kc_grid + k0)), gb = guess(sr, __ldg(a.kc_grid + k0 + cnt - 1));
            lo = max(0, min(ga, gb) - a.slack - (SINC ? 15 : 1)) & ~1;
            hi = min(a.mpad, (max(ga, gb) + a.slack + (SINC ? 23 : 5)) & ~1);             // rows are whole 32-sample groups
            if (hi - lo > pitch) hi = lo;                    // (not staged: gathered from global memory)
            tl = max(0, min(ga, gb) - a.slack - 1);
        }
        tl = __reduce_min_sync(0xffffffffu, tl) & ~1;
        bounds_of(b)[lane] = make_int2(lo, hi);
        if (lane == 0) *reinterpret_cast<int *>(bounds_of(b) + R2_ROWS) = tl;
        const uint32_t bytes = 8u * (uint32_t)(hi - lo), qbytes = 8u * ((cnt + 1) & ~1);     // padded vectors
        const uint32_t tbytes = 8u * (uint32_t)tlen;                                         // tan_s is padded by tlen
        const uint32_t total = __reduce_add_sync(0xffffffffu, bytes) + (a.window ? 2 : 1) * qbytes + tbytes;
        __syncwarp();
        if (lane == 0) {
            tma::arrive_expect_tx(ring.full + b, total);
            tma::bulk_load(q_of(b), a.kc_grid + k0, qbytes, ring.full + b);
            if (a.window) tma::bulk_load(ham_of(b), a.ham_m + k0, qbytes, ring.full + b);
            tma::bulk_load(tan_of(b), a.tan_s + tl, tbytes, ring.full + b);
            *ring.staged = u - u0 + 1;
        }
        __syncwarp();
        if (bytes) tma::bulk_load(win_of(b) + lane * pitch, a.p1 + (size_t)j * a.mpad + lo, bytes, ring.full + b);
    };
    if (warp == R2_WARPS - 1) {
        stage(u0);
        if (BUFS > 2 && u0 + 1 < u1) stage(u0 + 1);
    }
    const bool live = a.probe <= 0 || ring.wait(ring.unarmed, 0, (uint32_t)a.probe);
    constexpr int AHEAD = BUFS - 1;
    int cur = -1;
    Row r{};
    double hn = 1.0;
    int u = live ? u0 : u1;
    for (; u < u1; ++u) {
        const int it = u - u0, g = u / ntiles, kt = u - g * ntiles, b = it % BUFS, j = g * R2_ROWS + lane;
        if (warp == it % R2_WARPS && u + AHEAD < u1) {
            // the buffer of unit u + AHEAD is free once every warp is done with unit u - 1
            if (it >= 1 && !ring.released(it - 1)) break;
            stage(u + AHEAD);
        }
        if (g != cur) {
            r = row_of(j);
            hn = a.window ? a.ham_n[min(j, n - 1)] : 1.0;
            cur = g;
        }
        if (!ring.landed(it)) break;
        const int2 bnd = bounds_of(b)[lane];
        const int wlo = bnd.x, whi = bnd.y, tl = *reinterpret_cast<const int *>(bounds_of(b) + R2_ROWS);
        const double *qs = q_of(b) + warp * kRunT, *hs = ham_of(b) + warp * kRunT, *tn = tan_of(b);
        const float2 *w = win_of(b) + lane * pitch;
        const int k0 = kt * R2_TILE + warp * kRunT;
        if (k0 >= a.mpad) {                                  // warp-uniform: past the row
            ring.release(it);
            continue;
        }
        // np.interp's bracket of the first output: l with x(l) <= q < x(l + 1), x(l) = kr tan[l], searched from the affine
        // guess among the staged sources
        bool inside = j < n && k0 + kRunT <= m;
        int lb;                                              // lower index of output t minus t, at least
        {
            const double q = qs[0];
            int l = guess(r, q);
            const int e0 = max(l - a.slack, 0), e1 = min(l + a.slack, m - 2);
            l = e0;
            if (e0 < tl || e1 + 1 - tl >= tlen) inside = false;
            else
                while (l < e1 && q >= r.kr * tn[l + 1 - tl]) ++l;
            lb = l - 1;
        }
        if (lb < tl || lb + kRunT + 2 - tl >= tlen || lb + kRunT + 2 > m - 1) inside = false;
        const double *tx = tn + (inside ? lb - tl : 0);
        int l[kRunT], ph[kRunT], lo = 1 << 30, hi = -(1 << 30);
        float fr[kRunT];
        uint32_t pk[kRunT];
        double x0 = r.kr * tx[0], x1 = r.kr * tx[1], x2 = r.kr * tx[2];
#pragma unroll
        for (int t = 0; t < kRunT; ++t) {
            const double q = qs[t], x3 = r.kr * tx[t + 3];
            // sources lb + t .. lb + t + 3: the bracket is one of the three intervals, or the run is given up
            const bool s1 = q >= x1, s2 = q >= x2;
            const double xa = s2 ? x2 : s1 ? x1 : x0, xb = s2 ? x3 : s1 ? x2 : x1;
            inside = inside && q >= x0 && q < x3;
            l[t] = lb + t + (s1 ? 1 : 0) + (s2 ? 1 : 0);
            if constexpr (SINC) {
                const double fd = (q - xa) * recip_newton(xb - xa);
                ph[t] = min(max(__double2loint(fma(fd, 32768.0, 6755399441055744.0)), 0), 32767) >> 7;
                pk[t] = pack_br_phase(l[t], ph[t]);
                lo = min(lo, l[t] - t);
                hi = max(hi, l[t] - t);
            } else {
                fr[t] = __fdiv_rn((float)(q - xa), (float)(xb - xa));
            }
            x0 = x1;
            x1 = x2;
            x2 = x3;
        }
        if constexpr (SINC) {
            inside = inside && lo >= 15 && lo + kRunT + 1 <= m - 17 && lo - 15 >= wlo && lo + kRunT + 19 <= whi &&
                     hi - lo + ((lo - 15 - wlo) & 1) <= 2;
        } else {
            inside = inside && qs[0] >= r.lo && qs[kRunT - 1] <= r.hi && l[0] >= wlo && l[kRunT - 1] + 2 <= whi;
#pragma unroll
            for (int t = 1; t < kRunT; ++t) inside = inside && l[t] >= wlo && l[t] + 2 <= whi;
        }
        // nothing to form (the queries ascend): zeros
        const bool dead = j >= n || k0 >= m || qs[min(kRunT, m - k0) - 1] < r.lo || qs[0] > r.hi;
        float2 out[kRunT];
        const bool runs = __all_sync(0xffffffffu, inside || (dead && !(SINC && a.pk_out)) || j >= n);
        if (runs) {
            if constexpr (SINC) {
                const int at = dead ? 0 : lo - 15 - wlo;
                int o[kRunT];
#pragma unroll
                for (int t = 0; t < kRunT; ++t) {
                    o[t] = dead ? 0 : l[t] - t - lo + (at & 1);
                    ph[t] = dead ? 0 : ph[t];
                }
                sinc_run(w + (at & ~1), ph, o, tab, out);
            } else {
#pragma unroll
                for (int t = 0; t < kRunT; ++t) {
                    const float2 *s = w + (dead ? 0 : l[t] - wlo);
                    const float2 v0 = s[0], v1 = s[1];
                    out[t] = make_float2(fmaf(fr[t], v1.x - v0.x, v0.x), fmaf(fr[t], v1.y - v0.y, v0.y));
                }
            }
            if (dead) {
#pragma unroll
                for (int t = 0; t < kRunT; ++t) out[t] = make_float2(0.f, 0.f);
            }
        } else {
            // edges of the span, irregular sources, windows that were not staged: one output at a time
            auto xa = [&](int i) { return r.kr * __ldg(a.tan_s + i); };
#pragma unroll
            for (int t = 0; t < kRunT; ++t) out[t] = make_float2(0.f, 0.f);
#pragma unroll 1
            for (int t = 0; t < kRunT; ++t) {
                const bool valid = j < n && k0 + t < m;
                const double q = valid ? qs[t] : 0.0;
                Frac f{0.f, 0, 0};
                const int lt = valid ? interp_bracket<SINC>(xa, m, r.lo, r.hi, q, guess(r, q), f) : -1;
                float2 z = make_float2(0.f, 0.f);
                const bool sinc = SINC && lt >= 15 && lt <= m - 17;
                if (lt >= 0) {
                    const bool in = sinc ? lt - 15 >= wlo && lt + 17 <= whi : lt >= wlo && lt + 2 <= whi;
                    const float2 *src = in ? w - wlo : a.p1 + (size_t)j * a.mpad;
                    if (sinc) {
#pragma unroll 8
                        for (int i = 0; i < 32; ++i) {
                            const float c = run_tap(tab, f.ph, i);
                            const float2 x = src[lt - 15 + i];
                            z.x = fmaf(c, x.x, z.x);
                            z.y = fmaf(c, x.y, z.y);
                        }
                        z.x *= 1.0f / 32768.0f;
                        z.y *= 1.0f / 32768.0f;
                    } else {
                        z = gather_f32<false>(src, 0, m, lt, f, nullptr);
                    }
                }
                const uint32_t p = !SINC || !a.pk_out ? 0u
                                   : lt < 0           ? pack_br(1, q < r.lo ? 0 : m - 2, 0.f)
                                   : sinc             ? pack_br_phase(lt, f.ph)
                                                      : pack_br(0, lt, f.f);
#pragma unroll
                for (int s = 0; s < kRunT; ++s)              // (registers: no indexed store)
                    if (s == t) { out[s] = z; pk[s] = p; }
            }
        }
        if (j < n) {
            // np.outer(hamming(m), hamming(n)).astype(float32)[k, j], and the centring sign
#pragma unroll
            for (int t = 0; t < kRunT; ++t) {
                const float wgt = a.window ? (float)(hs[t] * hn) : 1.0f;
                const float sg2 = (a.centred && ((j + t) & 1)) ? -wgt : wgt;         // k0 is a multiple of 8
                out[t].x *= sg2;
                out[t].y *= sg2;
            }
            float4 *dst = reinterpret_cast<float4 *>(a.g2 + (size_t)j * a.mpad + k0);
#pragma unroll
            for (int t = 0; t < kRunT / 2; ++t) dst[t] = make_float4(out[2 * t].x, out[2 * t].y, out[2 * t + 1].x, out[2 * t + 1].y);
            if (SINC && a.pk_out) {
                uint4 *pd = reinterpret_cast<uint4 *>(a.pk_out + (size_t)j * a.mpad + k0);
                pd[0] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
                pd[1] = make_uint4(pk[4], pk[5], pk[6], pk[7]);
            }
        }
        ring.release(it);                                    // this warp has read the buffer of unit u
    }
    for (u = live ? u : u0; u < u1; ++u) {                   // a copy is lost: zeros
        const int g = u / ntiles, j = g * R2_ROWS + lane, k0 = (u - g * ntiles) * R2_TILE + warp * kRunT;
        for (int k = k0; k < k0 + kRunT && j < n && k0 < a.mpad; ++k) {
            a.g2[(size_t)j * a.mpad + k] = make_float2(0.f, 0.f);
            if (SINC && a.pk_out) a.pk_out[(size_t)j * a.mpad + k] = pack_br(1, 0, 0.f);
        }
    }
    ring.finish(a.err);
}

// ------------------------------------------------------------------------------------------ cross FFT
struct RowFftArgs {
    const float2 *g2;                   // [n][mpad] resampled rows
    const double *ham_m, *ham_n;        // WIN: the window is still to be applied
    const float2 *tw;
    float2 *y1t;                        // [m2][npad] transposed: row = cross bin, col = range bin
    double *ysum;                       // WIN (autofocus forward): += sum |y1|^2 over the frame (S / n2, by Parseval)
    int m, n, mpad, npad, inverse, window;
    int pf;                             // L2 prefetch distance in rows, 0 = none
};

// FFT along cross of a resampled row and corner turn #2 (the clusters of k_fl_pass2_fft).  WIN: the autofocus forward,
// whose rows are kept without the window for the adjoint.
template <int L, int E, bool WIN>
__global__ void __cluster_dims__(kCT, 1, 1) __launch_bounds__((1 << L) / E, fl_min_ctas(L, E)) k_fl_row_fft(RowFftArgs a) {
    pdl_wait();
    using F = F32Fft<L, E>;
    constexpr int N = F::N, T = F::T;
    extern __shared__ __align__(1024) unsigned char smem[];
    float2 *xbuf = reinterpret_cast<float2 *>(smem);
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const int tid = threadIdx.x;
    // clusters in reverse range-bin order: the resample wrote the high rows last
    const int j = (int)(gridDim.x - kCT - (blockIdx.x & ~(kCT - 1)) + (blockIdx.x & (kCT - 1)));
    const bool live = j < a.n;
    float2 x[E];
    if (live) {
        if (a.pf && j >= a.pf) l2_prefetch(a.g2 + (size_t)(j - a.pf) * a.mpad, (size_t)8 * a.mpad, tid);
        const float2 *row = a.g2 + (size_t)j * a.mpad;
        const double hn = WIN && a.window ? a.ham_n[j] : 1.0;
#pragma unroll
        for (int u = 0; u < E; ++u) {
            const int k = tid + T * u;
            float2 v = k < a.m ? (WIN ? row[k] : __ldcs(row + k)) : make_float2(0.f, 0.f);
            if (WIN && a.window && k < a.m) {
                const float wgt = (float)(a.ham_m[k] * hn);
                v.x *= wgt;
                v.y *= wgt;
            }
            x[u] = a.inverse ? make_float2(v.x, -v.y) : v;
        }
        F::run(x, xbuf, a.tw, tid);
        if constexpr (WIN) {
            double *red = reinterpret_cast<double *>(smem + (size_t)8 * F::xbuf_elems());
            double sq = 0.0;
#pragma unroll
            for (int v = 0; v < E; ++v) sq += (double)fmaf(x[v].x, x[v].x, x[v].y * x[v].y);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
            if ((tid & 31) == 0) red[tid >> 5] = sq;
            __syncthreads();
            if (tid == 0) {
                double t = 0.0;
                for (int w = 0; w < T / 32; ++w) t += red[w];
                atomicAdd(a.ysum, t);
            }
        }
    } else {
#pragma unroll
        for (int v = 0; v < E; ++v) x[v] = make_float2(0.f, 0.f);
    }
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
}

template <int L, int E>
cudaError_t launch_row_fft(const FloatDev &d, cudaStream_t st) {
    using F = F32Fft<L, E>;
    const bool win = d.pk_out != nullptr;
    RowFftArgs p{d.g2, d.ham_m64, d.ham_n64, d.twm, d.y1, d.af_acc, d.m, d.n, d.mpad, d.npad, d.sgn > 0, d.window, 0};
    const size_t sm = (size_t)8 * F::xbuf_elems() + (win ? (size_t)8 * std::max(1, F::T / 32) : 0);
    auto fn = win ? k_fl_row_fft<L, E, true> : k_fl_row_fft<L, E, false>;
    const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    p.pf = resident_blocks(fn, F::T, sm);
    (void)launch(fn, d.npad, F::T, sm, st, p);
    return cudaGetLastError();
}

template <int L>
cudaError_t row_fft_tile(const FloatDev &d, cudaStream_t st) {
    if constexpr (L >= 8 && L <= 13) {
        if (d.ept_cross == 8) return launch_row_fft<L, 8>(d, st);
    }
    if constexpr (L >= 13) {
        if (d.ept_cross == 32) return launch_row_fft<L, 32>(d, st);
    }
    return launch_row_fft<L, Cfg<L>::E>(d, st);
}

}  // namespace

bool resample2_shape(bool sinc, double ratio, int slack, double spread, int *pitch, int *tlen) {
    const int reach = r2_reach(sinc, ratio, slack);
    *pitch = reach / 4 * 4 + 6;                              // an odd number of 16-byte units
    *tlen = (reach + (int)std::ceil(spread) + 16 + 1) & ~1;
    return *tlen <= 512 && r2_smem(sinc, *pitch, *tlen) <= (sinc ? 227 : 113) * 1024;
}

cudaError_t float_resample2(const FloatDev &d, cudaStream_t st) {
    Resample2Args p{d.p1, d.tan_s, d.kr, d.kc, d.ham_m64, d.ham_n64, d.tabr, d.tabq, d.each + 1, d.g2, d.pk_out, d.wait_err, d.m, d.n, d.mpad,
                    d.pk_out ? 0 : d.layout == PFA_LAYOUT_CENTRED, d.pk_out ? 0 : d.window, d.p2_pitch, d.p2_tlen, d.p2_slack,
                    d.mixed ? 0 : d.mx_probe};
    const bool sinc = d.az_sinc != 0;
    const int units = (d.m + r2_tile(sinc) - 1) / r2_tile(sinc) * ((d.n + R2_ROWS - 1) / R2_ROWS);
    auto fn = sinc ? k_fl_resample2<true> : k_fl_resample2<false>;
    const size_t sm = r2_smem(sinc, d.p2_pitch, d.p2_tlen);
    const cudaError_t e = allow_smem(fn, kMaxSmem);
    if (e != cudaSuccess) return e;
    (void)launch(fn, std::min(units, (sinc ? 1 : 2) * d.sms), 32 * r2_warps(sinc), sm, st, p);
    return cudaGetLastError();
}

cudaError_t float_row_fft(const FloatDev &d, cudaStream_t st) {
    switch (d.Lm) {
        case 6: return row_fft_tile<6>(d, st);
        case 7: return row_fft_tile<7>(d, st);
        case 8: return row_fft_tile<8>(d, st);
        case 9: return row_fft_tile<9>(d, st);
        case 10: return row_fft_tile<10>(d, st);
        case 11: return row_fft_tile<11>(d, st);
        case 12: return row_fft_tile<12>(d, st);
        case 13: return row_fft_tile<13>(d, st);
        case 14: return row_fft_tile<14>(d, st);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace pfa
