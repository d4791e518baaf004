// Fixed-point helpers shared by the kernels of pfa_fixed.cu and pfa_fixed_runs.cu: saturation and packing, the Q0 exponent and
// quantiser, the FP64 bracket of serialize_inputs.interp_coeffs (mpfs/host/serialize_inputs.py:67-94).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace pfa {
namespace {

constexpr int kSincTaps = 32;
constexpr int kSincFirst = -15;

__device__ __forceinline__ int sat16(int v) { return min(max(v, -32768), 32767); }
__device__ __forceinline__ long long sat16ll(long long v) { return v < -32768 ? -32768 : (v > 32767 ? 32767 : v); }
__device__ __forceinline__ uint32_t pack16(int re, int im) {
    return (uint32_t)(uint16_t)re | ((uint32_t)(uint16_t)im << 16);
}
__device__ __forceinline__ int lo16(uint32_t p) { return (int)(int16_t)(p & 0xffffu); }
__device__ __forceinline__ int hi16(uint32_t p) { return (int)(int16_t)(p >> 16); }
__device__ __forceinline__ int wrap16(int v) { return (int)(int16_t)(v & 0xffff); }

// Source samples are packed int16 I/Q words (pass-2 rows) or unpacked int32 pairs (pass-1 windows,
// one 8-byte shared load per tap instead of a load and two sign extensions).
__device__ __forceinline__ int re_of(uint32_t v) { return lo16(v); }
__device__ __forceinline__ int im_of(uint32_t v) { return hi16(v); }
__device__ __forceinline__ int re_of(int2 v) { return v.x; }
__device__ __forceinline__ int im_of(int2 v) { return v.y; }

// Smallest e with M <= 32767 * 2^e, i.e. ceil(log2(M / 32767)) of fixedpoint.fit_scale for a float32
// maximum M (exact: M/32767 is either an exact power of two or at least 2^-24 away from one).
__device__ __forceinline__ int q0_exponent(uint32_t bits) {
    float M = __uint_as_float(bits);
    if (!(M > 0.0f)) return 0;
    double md = (double)M;
    int e = ilogb(md) - 15;
    while (md > ldexp(32767.0, e)) ++e;
    return e;
}

// floor(x / lsb) in float32 (the emulator divides float32 planes by a weak float scalar), sat16.
__device__ __forceinline__ int q0_quantise(float x, float lsb) {
    return sat16((int)fmaxf(fminf(floorf(__fdiv_rn(x, lsb)), 32767.0f), -32768.0f));
}

// lower_bound over a non-decreasing sequence xa(0..n-1): first t with xa(t) >= q (n if none).
// Starts from a guess and walks; falls back to bisection after a few steps.
template <class F>
__device__ __forceinline__ int lower_bound_from(const F &xa, int n, double q, int g) {
    int t = min(max(g, 0), n);
    int steps = 0;
    while (t < n && xa(t) < q) {
        ++t;
        if (++steps > 6) {
            int lo = t, hi = n;
            while (lo < hi) {
                int mid = (lo + hi) >> 1;
                if (xa(mid) < q) lo = mid + 1; else hi = mid;
            }
            return lo;
        }
    }
    while (t > 0 && xa(t - 1) >= q) {
        --t;
        if (++steps > 6) {
            int lo = 0, hi = t;
            while (lo < hi) {
                int mid = (lo + hi) >> 1;
                if (xa(mid) < q) lo = mid + 1; else hi = mid;
            }
            return lo;
        }
    }
    return t;
}

struct Bracket {
    int idx;   // natural-order lower index, -1 = out of span
    int wq;    // Q15 weight
};

// interp_coeffs (serialize_inputs.py:67-94) for one query, given the count of ascending-view
// source coordinates below q and an accessor of the ascending view.
template <class F>
__device__ __forceinline__ Bracket bracket_from_count(const F &xa, int n, bool asc, double q, int cnt) {
    Bracket b{-1, 0};
    int k = cnt - 1;
    if (k < 0 || k >= n - 1) return b;
    double x0 = xa(k), x1 = xa(k + 1);
    double fa = __ddiv_rn(__dsub_rn(q, x0), __dsub_rn(x1, x0));
    double w = asc ? fa : __dsub_rn(1.0, fa);
    double r = rint(__dmul_rn(w, 32768.0));
    r = fmin(fmax(r, 0.0), 32767.0);
    b.idx = asc ? k : (n - 2 - k);
    b.wq = (int)r;
    return b;
}

}  // namespace
}  // namespace pfa
