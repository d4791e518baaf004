// Pass 1 of the fixed-point datapath with the 32-tap sinc, in runs of eight outputs (silicon_emulator.py:60-122, 142-148):
// the same integers as k_fx_pass1<true>, arranged as the float mode's k_fl_pass1_runs.
//
//   k_fx_quant       Q0 quantise of the complex64 signal into packed int16 I/Q words (the layout of the int16 input)
//   k_fx_pass1_runs  bracket, 32-tap Q15 sinc, corner turn #1
//
// A lane owns one of 32 sorted pulses and a thread forms eight consecutive range bins of it from one sliding register window of
// samples; the Q15 taps are shifted into place by byte permutes (table in four copies in shared memory, see
// interp_f32.cuh).  A warp writes one 128-byte row segment of p1 per bin.  Persistent CTAs; the 32 pulses' sample windows of the
// next tiles arrive by bulk copies.  The bracket's weight needs floor/round of an exact FP64 quotient: it is formed from the
// affine spacing's reciprocal, whose error is bounded per pulse, and a quotient too near a rounding boundary is
// divided exactly.
// What bounds it: the multiply-add pipe (68 byte-pair dot products per output at half rate) and ALU; the earlier gather was
// bound by shared memory (32 sample and 4 tap loads per output).  5634 x 4319: 0.493 -> 0.224 ms and 0.042 for the quantiser; 2962 x 3755 int16: 0.201 -> 0.110 ms.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>

#include "fixed_math.cuh"
#include "interp_f32.cuh"
#include "pfa_internal.h"
#include "pdl.cuh"
#include "stage_ring.cuh"
#include "tc_sm100.cuh"
#include "tma_sm100.cuh"

namespace pfa {
namespace {

// floor(x / lsb) for the power of two lsb: a product with 1 / lsb is the correctly rounded value of the same number where
// both are normal floats (PROD)
template <bool PROD>
__device__ __forceinline__ uint32_t quant_pair(float re, float im, float s) {
    if constexpr (PROD)
        return pack16(sat16((int)fmaxf(fminf(floorf(__fmul_rn(re, s)), 32767.0f), -32768.0f)),
                      sat16((int)fmaxf(fminf(floorf(__fmul_rn(im, s)), 32767.0f), -32768.0f)));
    else
        return pack16(q0_quantise(re, s), q0_quantise(im, s));
}

template <bool PROD>
__device__ __forceinline__ void quant_sweep(const float4 *sig4, uint4 *__restrict__ out4, long long total, float s) {
    const long long n4 = total >> 2, stride = (long long)gridDim.x * blockDim.x;       // groups of four samples
    auto group = [&](long long i, float4 a, float4 b) {
        out4[i] = make_uint4(quant_pair<PROD>(a.x, a.y, s), quant_pair<PROD>(a.z, a.w, s), quant_pair<PROD>(b.x, b.y, s),
                             quant_pair<PROD>(b.z, b.w, s));
    };
    // back to front: the maximum's sweep left the end of the signal in L2; four loads in flight
    long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    for (; r + stride < n4; r += 2 * stride) {
        const long long i = n4 - 1 - r, k = i - stride;
        const float4 a = __ldcs(sig4 + 2 * i), b = __ldcs(sig4 + 2 * i + 1), c = __ldcs(sig4 + 2 * k), e = __ldcs(sig4 + 2 * k + 1);
        group(i, a, b);
        group(k, c, e);
    }
    if (r < n4) {
        const long long i = n4 - 1 - r;
        group(i, __ldcs(sig4 + 2 * i), __ldcs(sig4 + 2 * i + 1));
    }
    if (blockIdx.x == 0 && threadIdx.x < (total & 3)) {
        const long long i = 4 * n4 + threadIdx.x;
        const float2 z = reinterpret_cast<const float2 *>(sig4)[i];
        reinterpret_cast<uint32_t *>(out4)[i] = quant_pair<PROD>(z.x, z.y, s);
    }
}

__global__ void __launch_bounds__(256) k_fx_quant(const float4 *sig4, uint4 *__restrict__ out4, long long total,
                                                  const int32_t *ctrl) {
    pdl_wait();
    const int e = q0_exponent((uint32_t)ctrl[0]);
    if (e >= -126 && e <= 126) quant_sweep<true>(sig4, out4, total, (float)ldexp(1.0, -e));
    else quant_sweep<false>(sig4, out4, total, (float)ldexp(1.0, e));
}

struct RunArgs {
    const uint32_t *sig;                // [m][n] packed int16x2
    const float *f0, *df, *fac, *krp;
    const int32_t *order;
    const uint16_t *tab;                // [phase][32] taps
    uint32_t *p1;                       // [n][mpad]
    const int32_t *each;                // nonzero where the plan's present job is not one for runs
    int *err;                           // set when a bounded wait runs out
    int m, n, mpad, pitch;
    int probe;                          // test hook: > 0 = first wait this many polls on a barrier nothing arrives on
};

constexpr int X1_SLOTS = 32, X1_WARPS = 16, X1_BINS = X1_WARPS * kRunT, X1_BUFS = 4;
constexpr int X1_SLACK = 64;            // samples past the last window that a run may touch (and discard)
__host__ __device__ constexpr size_t x1_buf(int pitch) { return (size_t)4 * X1_SLOTS * pitch + 4 * X1_BINS + 8 * X1_SLOTS; }
constexpr size_t x1_smem(int pitch) { return (size_t)kRunTabBytes + X1_BUFS * x1_buf(pitch) + 4 * X1_SLACK + stage_ring_bytes(X1_BUFS); }
constexpr int kX1MaxPitch = 300;        // an odd number of 16-byte units that keeps one CTA within 227 KB
static_assert(x1_smem(kX1MaxPitch) <= 227 * 1024 && kX1MaxPitch % 8 == 4, "windows fit beside the table");

// (acc) += a0 b0 + a1 b1 for int16 pairs a and the low (signed) or high (unsigned) byte pair of b
__device__ __forceinline__ void dot_hi(int &acc, uint32_t a, uint32_t b) {
    asm("dp2a.lo.s32.s32 %0, %1, %2, %0;" : "+r"(acc) : "r"(a), "r"(b));
}
__device__ __forceinline__ void dot_lo(int &acc, uint32_t a, uint32_t b) {
    asm("dp2a.hi.s32.u32 %0, %1, %2, %0;" : "+r"(acc) : "r"(a), "r"(b));
}

// The table's word k holds taps 2k and 2k + 1 as bytes (high 2k, high 2k + 1, low 2k, low 2k + 1), tap = 256 high + low with a
// signed high and an unsigned low byte: two byte-pair products with a pair of samples of one component replace two
// multiply-adds each and need no sign extension.
__device__ __forceinline__ uint32_t tap_word(uint32_t two_taps) { return __byte_perm(two_taps, 0u, 0x2031); }

// sinc_run on packed int16 samples: x0 8-byte aligned, 42 of them readable.  The sums of the high and low bytes' products
// stay below 2^28 and 2^29 for any int16 taps; floor((256 H + L + 2^14) / 2^15) = floor((H + floor((L + 2^14) / 256)) / 128).
__device__ __forceinline__ void sinc_run_q15(const uint32_t *x0, const int (&ph)[kRunT], const int (&o)[kRunT],
                                             const unsigned char *tab, uint32_t (&out)[kRunT]) {
    constexpr int T = kRunT;
    const uint2 *xs = reinterpret_cast<const uint2 *>(x0);
    const unsigned char *tl = tab + 16 * (threadIdx.x % kRunCopies);
    // component pairs of the window's positions: er[i] = (2i, 2i + 1), qr[i] = (2i + 1, 2i + 2)
    uint32_t er[8], ei[8], qr[8], qi[8], last = 0u, prev[T], sel[T];
    int hr[T], hi[T], lr[T], li[T];
    auto re2 = [](uint32_t a, uint32_t b) { return __byte_perm(a, b, 0x5410); };
    auto im2 = [](uint32_t a, uint32_t b) { return __byte_perm(a, b, 0x7632); };
    // positions 2i, 2i + 1 (i >= 1 also closes the odd pair before them)
    auto put = [&](int i, uint2 v) {
        er[i] = re2(v.x, v.y);
        ei[i] = im2(v.x, v.y);
        if (i) {
            qr[i - 1] = re2(last, v.x);
            qi[i - 1] = im2(last, v.x);
        }
        last = v.y;
    };
#pragma unroll
    for (int t = 0; t < T; ++t) {
        hr[t] = hi[t] = lr[t] = li[t] = 0;
        prev[t] = 0u;
        sel[t] = o[t] == 0 ? 0x7654u : o[t] == 1 ? 0x6341u : 0x3210u;
    }
    auto dots = [&](int t, int i, uint32_t s) {              // i: even position offset of the word
        const int at = (t + i) >> 1;
        const uint32_t xr = (t & 1) ? qr[at] : er[at], xi = (t & 1) ? qi[at] : ei[at];
        dot_hi(hr[t], xr, s);
        dot_hi(hi[t], xi, s);
        dot_lo(lr[t], xr, s);
        dot_lo(li[t], xi, s);
    };
#pragma unroll
    for (int i = 0; i < 4; ++i) put(i, xs[i]);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
#pragma unroll
        for (int i = 0; i < 4; ++i) put(4 + i, xs[4 * (q + 1) + i]);
#pragma unroll
        for (int t = 0; t < T; ++t) {
            const uint4 u = *reinterpret_cast<const uint4 *>(tl + ph[t] * (64 * kRunCopies) + q * (16 * kRunCopies));
            const uint32_t w[5] = {prev[t], u.x, u.y, u.z, u.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) dots(t, 2 * e, __byte_perm(w[e], w[e + 1], sel[t]));
            prev[t] = u.w;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) { er[i] = er[4 + i]; ei[i] = ei[4 + i]; }
#pragma unroll
        for (int i = 0; i < 3; ++i) { qr[i] = qr[4 + i]; qi[i] = qi[4 + i]; }
    }
    const uint32_t x40 = x0[40];
    qr[3] = re2(last, x40);
    qi[3] = im2(last, x40);
#pragma unroll
    for (int t = 0; t < T; ++t) {
        dots(t, 0, __byte_perm(prev[t], 0u, sel[t]));
        out[t] = pack16(sat16((hr[t] + ((lr[t] + (1 << 14)) >> 8)) >> 7), sat16((hi[t] + ((li[t] + (1 << 14)) >> 8)) >> 7));
    }
}

// the run table's copies with the taps as byte-pair words
__device__ __forceinline__ void fill_tap_words(unsigned char *tab, const uint16_t *src, int tid, int threads) {
    for (int i = tid; i < 256 * 4; i += threads) {
        uint4 u = __ldg(reinterpret_cast<const uint4 *>(src) + i);
        u = make_uint4(tap_word(u.x), tap_word(u.y), tap_word(u.z), tap_word(u.w));
#pragma unroll
        for (int c = 0; c < kRunCopies; ++c) reinterpret_cast<uint4 *>(tab)[i * kRunCopies + c] = u;
    }
}

// one output at its bracket on an ascending axis of sn samples (apply_sinc, silicon_emulator.py:88-122): from the staged window
// [wlo, whi) or, past it, from the row in global memory
__device__ uint32_t gather_edge(Bracket br, int sn, int wlo, int whi, const uint32_t *win, const uint32_t *row, const unsigned char *tab) {
    if (br.idx < 0) return 0u;
    const bool sinc = br.idx >= 15 && br.idx <= sn - 17;
    const bool in = sinc ? br.idx - 15 >= wlo && br.idx + 17 <= whi : br.idx >= wlo && br.idx + 2 <= whi;
    const uint32_t *src = in ? win - wlo : row;
    if (!sinc) {
        const uint32_t va = src[br.idx], vb = src[br.idx + 1];
        const int r0 = lo16(va), i0 = hi16(va);
        return pack16(sat16(r0 + (((lo16(vb) - r0) * br.wq) >> 15)), sat16(i0 + (((hi16(vb) - i0) * br.wq) >> 15)));
    }
    const unsigned char *tr = tab + (br.wq >> 7) * (64 * kRunCopies) + 16 * (threadIdx.x % kRunCopies);
    int h[2][2] = {{0, 0}, {0, 0}};                          // int32 half sums, as sinc_gather keeps them
#pragma unroll
    for (int s = 0; s < 2; ++s)
#pragma unroll 8
        for (int e = 16 * s; e < 16 * s + 16; ++e) {
            const unsigned char *tw = tr + (e >> 3) * (16 * kRunCopies) + 4 * ((e & 7) >> 1) + (e & 1);
            const int c = (int)*reinterpret_cast<const signed char *>(tw) * 256 + (int)tw[2];
            const uint32_t x = src[br.idx - 15 + e];
            h[s][0] += c * lo16(x);
            h[s][1] += c * hi16(x);
        }
    const long long sr = (long long)h[0][0] + h[1][0], si = (long long)h[0][1] + h[1][1];
    return pack16((int)sat16ll((sr + (1 << 14)) >> 15), (int)sat16ll((si + (1 << 14)) >> 15));
}

// per-pulse constants: the exact source axis kr(k) = fac (f0 + k df) in float64 (silicon_emulator.py:144; k df is exact in
// float64, so a fused multiply-add rounds like the two operations) and the affine estimate
struct RunPulse {
    double fac, f0, df, inv, c0;
    double scale, thr;                  // 32768 inv; bound on the error of (q - kr(k)) scale against 32768 times the quotient
    double first, last;
    int i;
};

// A frame captured in a graph keeps its kernels when the plan gets another job.  Where that one is not for runs, every output
// by itself, as k_fx_pass1<true> forms it.
__device__ __noinline__ void pass1_each(const RunArgs &a, const unsigned char *tab) {
    const int n = a.n;
    const long long total = (long long)n * a.mpad, stride = (long long)gridDim.x * blockDim.x;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total; e += stride) {
        const int j = (int)(e / a.mpad), r = (int)(e - (long long)j * a.mpad);
        uint32_t z = 0u;
        if (r < a.m) {
            const int i = a.order[r];
            const double fac = (double)a.fac[i], f0 = (double)a.f0[i], df = (double)a.df[i], q = (double)a.krp[j];
            auto kr = [&](int k) { return __dmul_rn(fac, __dadd_rn(f0, __dmul_rn((double)k, df))); };
            const bool asc = kr(n - 1) >= kr(0);
            auto xa = [&](int t) { return asc ? kr(t) : kr(n - 1 - t); };
            const double inv_step = 1.0 / (fac * df), kest = q * inv_step - f0 / df;
            int g = 0;
            if (isfinite(kest) && isfinite(inv_step))
                g = (int)fmin(fmax(asc ? ceil(kest) : ceil((double)(n - 1) - kest), -1.0), (double)n + 1.0);
            z = gather_edge(bracket_from_count(xa, n, asc, q, lower_bound_from(xa, n, q, g)), n, 0, 0, nullptr,
                            a.sig + (long long)i * n, tab);
        }
        a.p1[e] = z;
    }
}

__global__ void __launch_bounds__(32 * X1_WARPS, 1) k_fx_pass1_runs(const __grid_constant__ RunArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    unsigned char *tab = smem, *bufs = smem + kRunTabBytes;
    const int pitch = a.pitch, n = a.n;
    const size_t bufb = x1_buf(pitch);
    auto win_of = [&](int b) { return reinterpret_cast<uint32_t *>(bufs + b * bufb); };
    auto q_of = [&](int b) { return reinterpret_cast<float *>(bufs + b * bufb + (size_t)4 * X1_SLOTS * pitch); };
    auto bounds_of = [&](int b) { return reinterpret_cast<int2 *>(q_of(b) + X1_BINS); };
    StageRing<X1_BUFS> ring(bufs + X1_BUFS * bufb + 4 * X1_SLACK);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ntiles = (n + X1_BINS - 1) / X1_BINS, groups = a.mpad / X1_SLOTS;
    const int units = ntiles * groups;                       // unit u: tile u % ntiles of pulse group u / ntiles
    const int u0 = (int)((long long)units * blockIdx.x / gridDim.x), u1 = (int)((long long)units * (blockIdx.x + 1) / gridDim.x);
    if (tid == 0) ring.init(X1_WARPS);
    const int each = *a.each;
    fill_tap_words(tab, a.tab, tid, 32 * X1_WARPS);
    pdl_wait();                                              // the tables above belong to the job
    __syncthreads();
    if (each) {
        pass1_each(a, tab);
        return;
    }
    if (u0 >= u1) return;
    constexpr double kMagic = 6755399441055744.0;            // 1.5 * 2^52: an integer in the low word
    auto pulse = [&](int r) {
        RunPulse p{};
        p.i = -1;
        if (r < a.m) {
            p.i = a.order[r];
            p.fac = (double)a.fac[p.i];
            p.f0 = (double)a.f0[p.i];
            p.df = (double)a.df[p.i];
            p.inv = 1.0 / (p.fac * p.df);
            p.c0 = p.f0 / p.df;
            p.first = __dmul_rn(p.fac, p.f0);
            p.last = __dmul_rn(p.fac, fma((double)(n - 1), p.df, p.f0));
            // kr(k) and kr(k + 1) are each within half an ulp of the affine axis, (f0 + k df) too: in units of the spacing
            // the quotient moves by less than 4 ulp(kr) / spacing; bounded here with a factor of four to spare
            p.scale = 32768.0 * p.inv;
            p.thr = 32768.0 * 0x1p-48 * (fmax(fabs(p.first), fabs(p.last)) * fabs(p.inv) + 1.0);
        }
        return p;
    };
    int sg = -1;
    RunPulse sp{};
    auto stage = [&](int u) {
        const int g = u / ntiles, b = (u - u0) % X1_BUFS;
        if (g != sg) {
            sp = pulse(g * X1_SLOTS + lane);
            sg = g;
        }
        const int j0 = (u - g * ntiles) * X1_BINS, cnt = min(X1_BINS, n - j0);
        int lo = 0, hi = 0;
        if (sp.i >= 0) {
            // lower index by the affine estimate, give or take one
            auto lower = [&](double q) { return min(max(__double2loint(__dadd_rd(fma(q, sp.inv, -sp.c0), kMagic)), 0), n - 2); };
            const int la = lower((double)__ldg(a.krp + j0)), lb = lower((double)__ldg(a.krp + j0 + cnt - 1));
            lo = max(0, min(la, lb) - 17);
            hi = min(n, max(la, lb) + 20);
            // window ends at 16-byte boundaries (four samples) inside the signal
            const long long e0 = (long long)sp.i * n, total = (long long)a.m * n;
            const int mis = (int)((reinterpret_cast<uintptr_t>(a.sig) >> 2) & 3);
            const int down = (int)((mis + e0 + lo) & 3), up = (int)(-(mis + e0 + hi) & 3);
            lo += e0 + lo - down >= 0 ? -down : 4 - down;
            hi += e0 + hi + up <= total ? up : up - 4;
            if (hi - lo > pitch || hi < lo) hi = lo;         // (not staged: gathered from global memory)
        }
        bounds_of(b)[lane] = make_int2(lo, hi);
        const uint32_t bytes = 4u * (uint32_t)(hi - lo), qbytes = 4u * ((cnt + 3) & ~3);    // the job block goes on past krp
        const uint32_t total = __reduce_add_sync(0xffffffffu, bytes) + qbytes;
        __syncwarp();
        if (lane == 0) {
            tma::arrive_expect_tx(ring.full + b, total);
            tma::bulk_load(q_of(b), a.krp + j0, qbytes, ring.full + b);
            *ring.staged = u - u0 + 1;
        }
        __syncwarp();
        if (bytes) tma::bulk_load(win_of(b) + lane * pitch, a.sig + (long long)sp.i * n + lo, bytes, ring.full + b);
    };
    constexpr int AHEAD = X1_BUFS - 1;
    if (warp == X1_WARPS - 1)
        for (int k = 0; k < AHEAD && u0 + k < u1; ++k) stage(u0 + k);
    const bool live = a.probe <= 0 || ring.wait(ring.unarmed, 0, (uint32_t)a.probe);
    int cur = -1;
    RunPulse p{};
    int u = live ? u0 : u1;
    for (; u < u1; ++u) {
        const int it = u - u0, g = u / ntiles, k = u - g * ntiles, b = it % X1_BUFS;
        if (warp == it % X1_WARPS && u + AHEAD < u1) {
            // the buffer of unit u + AHEAD is free once every warp is done with unit u - 1
            if (it >= 1 && !ring.released(it - 1)) break;
            stage(u + AHEAD);
        }
        if (g != cur) {
            p = pulse(g * X1_SLOTS + lane);
            cur = g;
        }
        if (!ring.landed(it)) break;
        const int2 bnd = bounds_of(b)[lane];
        const int wlo = bnd.x, whi = bnd.y;
        const float *qs = q_of(b) + warp * kRunT;
        const uint32_t *w = win_of(b) + lane * pitch;
        const int j0 = k * X1_BINS + warp * kRunT;
        uint32_t *dst = a.p1 + (size_t)j0 * a.mpad + g * X1_SLOTS + lane;
        auto kr = [&](double t) { return __dmul_rn(p.fac, fma(t, p.df, p.f0)); };
        // interp_coeffs: l with kr(l) < q <= kr(l + 1) and the weight's phase round(32768 quotient) >> 7
        int l[kRunT], ph[kRunT], lo = 1 << 30, hi = -(1 << 30);
        bool all = true;
#pragma unroll
        for (int t = 0; t < kRunT; ++t) {
            const double q = (double)qs[t];
            const double tt = __dadd_ru(fma(q, p.inv, -p.c0), kMagic - 1.0);        // ceil(estimate) - 1
            const double d = q - kr(tt - kMagic);
            l[t] = __double2loint(tt);
            // the quotient lies within thr of d scale: the estimate's bracket holds (0 < quotient < 1; the sign of d is
            // exact) and both ends of that interval round to the same phase
            const double v0 = fma(d, p.scale, -p.thr), v1 = fma(d, p.scale, p.thr);
            const int r0 = __double2loint(v0 + kMagic), r1 = __double2loint(v1 + kMagic);
            ph[t] = r1 >> 7;
            all = all && __double2hiint(d) > 0 && v1 < 32767.5 && (r0 >> 7) == ph[t];
            lo = min(lo, l[t] - t);
            hi = max(hi, l[t] - t);
        }
        const bool inside = p.i >= 0 && all && hi - lo <= 1 && lo >= 15 && lo + kRunT <= n - 17 && lo - 15 >= wlo &&
                            lo + kRunT + 17 <= whi;
        // nothing to form (the queries ascend): zeros
        const bool dead = p.i < 0 || (double)qs[kRunT - 1] <= p.first || (double)qs[0] > p.last;
        if (j0 + kRunT <= n && __all_sync(0xffffffffu, inside || dead)) {
            const int at = dead ? 0 : lo - 15 - wlo;
            int o[kRunT];
            uint32_t out[kRunT];
#pragma unroll
            for (int t = 0; t < kRunT; ++t) {
                o[t] = dead ? 0 : l[t] - t - lo + (at & 1);
                ph[t] = dead ? 0 : ph[t];
            }
            sinc_run_q15(w + (at & ~1), ph, o, tab, out);
#pragma unroll
            for (int t = 0; t < kRunT; ++t, dst += a.mpad) *dst = dead ? 0u : out[t];
        } else {
            auto xa = [&](int t) { return kr((double)t); };
#pragma unroll 1
            for (int t = 0; t < kRunT && j0 + t < n; ++t) {
                uint32_t z = 0u;
                if (p.i >= 0) {
                    const double q = (double)qs[t], est = fma(q, p.inv, -p.c0);
                    const int gs = isfinite(est) ? (int)fmin(fmax(ceil(est), -1.0), (double)n + 1.0) : 0;
                    const Bracket br = bracket_from_count(xa, n, true, q, lower_bound_from(xa, n, q, gs));
                    z = gather_edge(br, n, wlo, whi, w, a.sig + (long long)p.i * n, tab);
                }
                dst[(size_t)t * a.mpad] = z;
            }
        }
        ring.release(it);                                    // this warp has read the windows of unit u
    }
    for (u = live ? u : u0; u < u1; ++u) {                   // a copy is lost: zeros
        const int g = u / ntiles, j0 = (u - g * ntiles) * X1_BINS + warp * kRunT;
        for (int j = j0; j < min(j0 + kRunT, n); ++j) a.p1[(size_t)j * a.mpad + g * X1_SLOTS + lane] = 0u;
    }
    ring.finish(a.err);
}

// ------------------------------------------------------------------------------------------ pass 2
// The cross resample of pass 2 and the Q15 window (silicon_emulator.py:150-156, 165-195) in a kernel of its own, as the float
// mode's k_fl_resample2: a lane per range bin, eight consecutive cross samples per thread; the BFP FFT follows in
// k_fx_row_fft.  Sources are float32 products KRp[j] tan_s (exact in the comparisons), the weight's quotient of their
// float64 differences comes from one Newton step on a float reciprocal (relative error below 2^-45), and a phase within
// 2^-28 of a boundary is divided exactly.  5634 x 4319: 0.252 ms and 0.285 for the row FFT, 0.675 fused (a lane per cross
// sample, 32 + 32 shared-memory loads per output, the sinc and 13 FFT stages unrolled in one kernel).  For jobs with ascending, nearly affine sources (pfa_set_fixed_job).
struct Resample2Args {
    const uint32_t *p1;                 // [n][mpad]
    const float *tan_s, *krp, *kcp;
    const int32_t *hamr, *hamc;
    const uint16_t *tab;
    uint32_t *g2;                       // [n][mpad] windowed rows
    const int32_t *each;                // nonzero where the plan's present job is not one for this kernel
    int *err;
    int m, n, mpad, pitch, tlen, slack;
    int probe;                          // test hook, as in RunArgs
};

constexpr int X2_ROWS = 32, X2_WARPS = 16, X2_TILE = X2_WARPS * kRunT, X2_BUFS = 4;
constexpr int X2_SLACK = 64;
__host__ __device__ constexpr size_t x2_buf(int pitch, int tlen) {
    return (size_t)4 * X2_ROWS * pitch + 8 * X2_TILE + 4 * tlen + 8 * X2_ROWS + 16;
}
constexpr size_t x2_smem(int pitch, int tlen) {
    return (size_t)kRunTabBytes + X2_BUFS * x2_buf(pitch, tlen) + 4 * X2_SLACK + stage_ring_bytes(X2_BUFS);
}

// every output by itself, as k_fx_pass2_fft<.., true> forms it (see pass1_each)
__device__ __noinline__ void resample_each(const Resample2Args &a, const unsigned char *tab) {
    const int m = a.m;
    const long long total = (long long)a.n * a.mpad, stride = (long long)gridDim.x * blockDim.x;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total; e += stride) {
        const int j = (int)(e / a.mpad), k = (int)(e - (long long)j * a.mpad);
        if (k >= m) continue;
        const float krj = a.krp[j];
        const bool asc = __fmul_rn(krj, a.tan_s[m - 1]) >= __fmul_rn(krj, a.tan_s[0]);
        auto xa = [&](int t) { return (double)__fmul_rn(krj, __ldg(a.tan_s + (asc ? t : m - 1 - t))); };
        const double lo_v = xa(0), hi_v = xa(m - 1), inv_span = (double)(m - 1) / (hi_v - lo_v), q = (double)a.kcp[k];
        Bracket b{-1, 0};
        if (q > lo_v && q <= hi_v) b = bracket_from_count(xa, m, asc, q, lower_bound_from(xa, m, q, (int)((q - lo_v) * inv_span) + 1));
        const uint32_t v = gather_edge(b, m, 0, 0, nullptr, a.p1 + (size_t)j * a.mpad, tab);
        const int cw = wrap16((a.hamr[j] * a.hamc[k]) >> 15);
        a.g2[e] = pack16((lo16(v) * cw) >> 15, (hi16(v) * cw) >> 15);
    }
}

__global__ void __launch_bounds__(32 * X2_WARPS, 1) k_fx_resample2(const __grid_constant__ Resample2Args a) {
    extern __shared__ __align__(16) unsigned char smem[];
    unsigned char *tab = smem, *bufs = smem + kRunTabBytes;
    const int pitch = a.pitch, tlen = a.tlen;
    const size_t bufb = x2_buf(pitch, tlen);
    auto win_of = [&](int b) { return reinterpret_cast<uint32_t *>(bufs + b * bufb); };
    auto q_of = [&](int b) { return reinterpret_cast<float *>(bufs + b * bufb + (size_t)4 * X2_ROWS * pitch); };
    auto ham_of = [&](int b) { return reinterpret_cast<int32_t *>(q_of(b) + X2_TILE); };
    auto tan_of = [&](int b) { return q_of(b) + 2 * X2_TILE; };
    auto bounds_of = [&](int b) { return reinterpret_cast<int2 *>(tan_of(b) + tlen); };
    StageRing<X2_BUFS> ring(bufs + X2_BUFS * bufb + 4 * X2_SLACK);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int m = a.m, n = a.n, ntiles = (m + X2_TILE - 1) / X2_TILE, groups = (n + X2_ROWS - 1) / X2_ROWS;
    const int units = ntiles * groups;                       // unit u: tile u % ntiles of row group u / ntiles
    const int u0 = (int)((long long)units * blockIdx.x / gridDim.x), u1 = (int)((long long)units * (blockIdx.x + 1) / gridDim.x);
    if (tid == 0) ring.init(X2_WARPS);
    const int each = *a.each;
    fill_tap_words(tab, a.tab, tid, 32 * X2_WARPS);
    pdl_wait();                                              // the tables above belong to the job
    __syncthreads();
    if (each) {
        resample_each(a, tab);
        return;
    }
    if (u0 >= u1) return;
    const float tan0 = a.tan_s[0], tan1 = a.tan_s[m - 1];
    struct Row { float kr, lo, hi, inv; };
    auto row_of = [&](int j) {
        Row r;
        r.kr = a.krp[min(j, n - 1)];
        r.lo = __fmul_rn(r.kr, tan0);
        r.hi = __fmul_rn(r.kr, tan1);
        r.inv = (float)(m - 1) / (r.hi - r.lo);
        return r;
    };
    // affine estimate of the lower index (slack covers its error, the float32 arithmetic included)
    auto guess = [&](const Row &r, float q) { return min(max((int)((q - r.lo) * r.inv), 0), m - 2); };
    int sg = -1;
    Row sr{};
    auto stage = [&](int u) {
        const int g = u / ntiles, b = (u - u0) % X2_BUFS, j = g * X2_ROWS + lane;
        if (g != sg) {
            sr = row_of(j);
            sg = g;
        }
        const int k0 = (u - g * ntiles) * X2_TILE, cnt = min(X2_TILE, m - k0);
        int lo = 0, hi = 0, tl = m;
        if (j < n) {
            const int ga = guess(sr, __ldg(a.kcp + k0)), gb = guess(sr, __ldg(a.kcp + k0 + cnt - 1));
            lo = max(0, min(ga, gb) - a.slack - 15) & ~3;
            hi = min(a.mpad, (max(ga, gb) + a.slack + 26) & ~3);             // rows are whole 32-sample groups
            if (hi - lo > pitch) hi = lo;                    // (not staged: gathered from global memory)
            tl = max(0, min(ga, gb) - a.slack - 1);
        }
        tl = __reduce_min_sync(0xffffffffu, tl) & ~3;
        bounds_of(b)[lane] = make_int2(lo, hi);
        if (lane == 0) *reinterpret_cast<int *>(bounds_of(b) + X2_ROWS) = tl;
        const uint32_t bytes = 4u * (uint32_t)(hi - lo), qbytes = 4u * ((cnt + 3) & ~3), tbytes = 4u * (uint32_t)tlen;
        const uint32_t total = __reduce_add_sync(0xffffffffu, bytes) + 2 * qbytes + tbytes;      // the job block goes on past these
        __syncwarp();
        if (lane == 0) {
            tma::arrive_expect_tx(ring.full + b, total);
            tma::bulk_load(q_of(b), a.kcp + k0, qbytes, ring.full + b);
            tma::bulk_load(ham_of(b), a.hamc + k0, qbytes, ring.full + b);
            tma::bulk_load(tan_of(b), a.tan_s + tl, tbytes, ring.full + b);
            *ring.staged = u - u0 + 1;
        }
        __syncwarp();
        if (bytes) tma::bulk_load(win_of(b) + lane * pitch, a.p1 + (size_t)j * a.mpad + lo, bytes, ring.full + b);
    };
    constexpr int AHEAD = X2_BUFS - 1;
    if (warp == X2_WARPS - 1)
        for (int k = 0; k < AHEAD && u0 + k < u1; ++k) stage(u0 + k);
    const bool live = a.probe <= 0 || ring.wait(ring.unarmed, 0, (uint32_t)a.probe);
    int cur = -1, hr = 0;
    Row r{};
    int u = live ? u0 : u1;
    for (; u < u1; ++u) {
        const int it = u - u0, g = u / ntiles, kt = u - g * ntiles, b = it % X2_BUFS, j = g * X2_ROWS + lane;
        if (warp == it % X2_WARPS && u + AHEAD < u1) {
            // the buffer of unit u + AHEAD is free once every warp is done with unit u - 1
            if (it >= 1 && !ring.released(it - 1)) break;
            stage(u + AHEAD);
        }
        if (g != cur) {
            r = row_of(j);
            hr = a.hamr[min(j, n - 1)];
            cur = g;
        }
        if (!ring.landed(it)) break;
        const int2 bnd = bounds_of(b)[lane];
        const int wlo = bnd.x, whi = bnd.y, tl = *reinterpret_cast<const int *>(bounds_of(b) + X2_ROWS);
        const float *qs = q_of(b) + warp * kRunT, *tn = tan_of(b);
        const int32_t *hs = ham_of(b) + warp * kRunT;
        const uint32_t *w = win_of(b) + lane * pitch;
        const int k0 = kt * X2_TILE + warp * kRunT;
        if (k0 >= a.mpad) {                                  // warp-uniform: past the row
            ring.release(it);
            continue;
        }
        // bracket of the first output: l with x(l) < q <= x(l + 1), searched from the affine guess among the staged sources
        bool inside = j < n && k0 + kRunT <= m;
        int lb;                                              // lower index of output t minus t, at least
        {
            const float q = qs[0];
            const int gq = guess(r, q), e0 = max(gq - a.slack, 0), e1 = min(gq + a.slack, m - 2);
            int l = e0;
            if (e0 < tl || e1 + 1 - tl >= tlen) inside = false;
            else
                while (l < e1 && q > __fmul_rn(r.kr, tn[l + 1 - tl])) ++l;
            lb = l - 1;
        }
        if (lb < tl || lb + kRunT + 2 - tl >= tlen || lb + kRunT + 2 > m - 1) inside = false;
        const float *tx = tn + (inside ? lb - tl : 0);
        int l[kRunT], ph[kRunT], lo = 1 << 30, hi = -(1 << 30);
        float x0 = __fmul_rn(r.kr, tx[0]), x1 = __fmul_rn(r.kr, tx[1]), x2 = __fmul_rn(r.kr, tx[2]);
#pragma unroll
        for (int t = 0; t < kRunT; ++t) {
            const float q = qs[t], x3 = __fmul_rn(r.kr, tx[t + 3]);
            const bool s1 = q > x1, s2 = q > x2;
            const float xa = s2 ? x2 : s1 ? x1 : x0, xb = s2 ? x3 : s1 ? x2 : x1;
            inside = inside && q > x0 && q <= x3;
            l[t] = lb + t + (s1 ? 1 : 0) + (s2 ? 1 : 0);
            // 32768 (q - xa) / (xb - xa): exact float64 differences, reciprocal to 2^-45
            const double s = (double)xb - (double)xa, d = (double)q - (double)xa;
            double rc = (double)__frcp_rn(xb - xa);
            rc = fma(fma(-s, rc, 1.0), rc, rc);
            constexpr double kMagic = 6755399441055744.0, kThr = 0x1p-28;
            const double v = d * rc;
            const int r0 = __double2loint(fma(v, 32768.0, -kThr) + kMagic), r1 = __double2loint(fma(v, 32768.0, kThr) + kMagic);
            ph[t] = min(r1, 32767) >> 7;
            inside = inside && (min(max(r0, 0), 32767) >> 7) == ph[t];
            lo = min(lo, l[t] - t);
            hi = max(hi, l[t] - t);
            x0 = x1;
            x1 = x2;
            x2 = x3;
        }
        inside = inside && lo >= 15 && lo + kRunT + 1 <= m - 17 && lo - 15 >= wlo && lo + kRunT + 19 <= whi &&
                 hi - lo + ((lo - 15 - wlo) & 1) <= 2;
        // nothing to form (the queries ascend): zeros
        const bool dead = j >= n || k0 >= m || qs[min(kRunT, m - k0) - 1] <= r.lo || qs[0] > r.hi;
        uint32_t out[kRunT];
        if (__all_sync(0xffffffffu, inside || dead)) {
            const int at = dead ? 0 : lo - 15 - wlo;
            int o[kRunT];
#pragma unroll
            for (int t = 0; t < kRunT; ++t) {
                o[t] = dead ? 0 : l[t] - t - lo + (at & 1);
                ph[t] = dead ? 0 : ph[t];
            }
            sinc_run_q15(w + (at & ~1), ph, o, tab, out);
            if (dead) {
#pragma unroll
                for (int t = 0; t < kRunT; ++t) out[t] = 0u;
            }
        } else {
            auto xa = [&](int t) { return (double)__fmul_rn(r.kr, __ldg(a.tan_s + t)); };
#pragma unroll
            for (int t = 0; t < kRunT; ++t) out[t] = 0u;
#pragma unroll 1
            for (int t = 0; t < kRunT; ++t) {
                uint32_t z = 0u;
                if (j < n && k0 + t < m) {
                    const float qf = qs[t];
                    const double q = (double)qf;
                    Bracket br{-1, 0};
                    if (q > (double)r.lo && q <= (double)r.hi)
                        br = bracket_from_count(xa, m, true, q, lower_bound_from(xa, m, q, guess(r, qf) + 1));
                    z = gather_edge(br, m, wlo, whi, w, a.p1 + (size_t)j * a.mpad, tab);
                }
#pragma unroll
                for (int s = 0; s < kRunT; ++s)              // (registers: no indexed store)
                    if (s == t) out[s] = z;
            }
        }
        if (j < n) {
            // window_fixed: cw = (int16)((hr * hc) >> 15); out = (int16)((x * cw) >> 15)
#pragma unroll
            for (int t = 0; t < kRunT; ++t) {
                const int cw = wrap16((hr * hs[t]) >> 15);
                out[t] = pack16((lo16(out[t]) * cw) >> 15, (hi16(out[t]) * cw) >> 15);
            }
            uint4 *dst = reinterpret_cast<uint4 *>(a.g2 + (size_t)j * a.mpad + k0);
            dst[0] = make_uint4(out[0], out[1], out[2], out[3]);
            dst[1] = make_uint4(out[4], out[5], out[6], out[7]);
        }
        ring.release(it);                                    // this warp has read the buffer of unit u
    }
    for (u = live ? u : u0; u < u1; ++u) {                   // a copy is lost: zeros
        const int g = u / ntiles, j = g * X2_ROWS + lane, k0 = (u - g * ntiles) * X2_TILE + warp * kRunT;
        for (int k = k0; k < k0 + kRunT && j < n && k0 < a.mpad; ++k) a.g2[(size_t)j * a.mpad + k] = 0u;
    }
    ring.finish(a.err);
}

}  // namespace

cudaError_t fixed_pass1_runs(const FixedDev &d, const float *sig_c64, const uint32_t *sig_iq, cudaStream_t st) {
    if (sig_c64) {
        const long long groups = ((long long)d.m * d.n + 3) / 4;
        const int blocks = (int)std::min<long long>(8LL * d.sms, (groups + 511) / 512);       // two groups a thread
        (void)launch(k_fx_quant, blocks, 256, 0, st, reinterpret_cast<const float4 *>(sig_c64), reinterpret_cast<uint4 *>(d.sq),
                                              (long long)d.m * d.n, d.ctrl);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    // windows of a 128-bin tile at the job's widest spacing, an odd number of 16-byte units
    const int need = (int)std::ceil((X1_BINS - 1) * d.p1_ratio) + 46, pitch = std::min(kX1MaxPitch, need / 8 * 8 + 12);
    RunArgs a{sig_c64 ? d.sq : sig_iq, d.f0, d.df, d.fac, d.krp, d.order, d.sinc_pm, d.p1, d.each, d.ctrl + kFixedErrWord, d.m, d.n, d.mpad, pitch,
              d.probe};
    const int units = (d.n + X1_BINS - 1) / X1_BINS * (d.mpad / X1_SLOTS);
    const size_t sm = x1_smem(pitch);
    const cudaError_t e = allow_smem(k_fx_pass1_runs, kMaxSmem);
    if (e != cudaSuccess) return e;
    (void)launch(k_fx_pass1_runs, std::min(units, d.sms), 32 * X1_WARPS, sm, st, a);
    return cudaGetLastError();
}

bool fixed_resample2_shape(double ratio, int slack, double spread, int *pitch, int *tlen) {
    const int reach = (int)std::ceil((X2_TILE - 1) * ratio) + 2 * slack + 46;
    *pitch = reach / 8 * 8 + 12;                             // an odd number of 16-byte units
    *tlen = (reach + (int)std::ceil(spread) + 16 + 3) & ~3;
    return *tlen <= 512 && x2_smem(*pitch, *tlen) <= 227 * 1024;
}

cudaError_t fixed_resample2(const FixedDev &d, uint32_t *g2, cudaStream_t st) {
    Resample2Args a{d.p1, d.tan_s, d.krp, d.kcp, d.hamr, d.hamc, d.sinc_pm, g2, d.each + 1, d.ctrl + kFixedErrWord, d.m, d.n, d.mpad,
                    d.p2_pitch, d.p2_tlen, d.p2_slack, d.probe};
    const int units = (d.m + X2_TILE - 1) / X2_TILE * ((d.n + X2_ROWS - 1) / X2_ROWS);
    const size_t sm = x2_smem(d.p2_pitch, d.p2_tlen);
    const cudaError_t e = allow_smem(k_fx_resample2, kMaxSmem);
    if (e != cudaSuccess) return e;
    (void)launch(k_fx_resample2, std::min(units, d.sms), 32 * X2_WARPS, sm, st, a);
    return cudaGetLastError();
}

}  // namespace pfa
