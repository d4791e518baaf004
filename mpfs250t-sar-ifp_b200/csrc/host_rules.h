// Host-side decisions without CUDA: how a plan's buffers share device allocations, and which jobs the passes in runs take.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstddef>
#include <vector>

namespace pfa {

// ------------------------------------------------------------------------------------------ allocations
// The driver maps device memory in steps of 2 MiB and serves small requests from what it has mapped (10 us or less); a new
// mapping takes 300 to 400 us, and as much again to give back.  So a plan of small buffers packs them into allocations of
// at most 1 MiB (a larger buffer by itself), which plans share the mapped memory with: 256 x 256 float plan 8 us, 360 in one
// allocation; 300 x 300 fixed 9 us, 360.  Every other plan takes a single allocation: 1000 x 1000 fixed 340 us, 1010 with one
// for each buffer.  The first `head` buffers stay together.
constexpr size_t kSmallAlloc = size_t(1) << 20, kSmallBuffer = size_t(5) << 18;
constexpr int kMaxBlocks = 12;

struct Packing {
    std::vector<size_t> block;       // bytes of each allocation
    std::vector<int> in;             // buffer -> allocation
    std::vector<size_t> offset;      // buffer -> offset in it
};

inline Packing pack_buffers(const std::vector<size_t> &bytes, size_t head) {
    auto pack = [&](size_t limit) {
        Packing p;
        size_t i = 0;
        while (i < bytes.size()) {
            const size_t end = i == 0 && head ? head : i + 1;        // the buffers that go in together
            size_t sum = 0;
            for (size_t k = i; k < end; ++k) sum += bytes[k];
            if (p.block.empty() || p.block.back() + sum > limit) p.block.push_back(0);
            for (; i < end; ++i) {
                p.in.push_back((int)p.block.size() - 1);
                p.offset.push_back(p.block.back());
                p.block.back() += bytes[i];
            }
        }
        return p;
    };
    const Packing small = pack(kSmallAlloc);
    const bool fits = std::all_of(small.block.begin(), small.block.end(), [](size_t b) { return b <= kSmallBuffer; });
    return fits && small.block.size() <= kMaxBlocks ? small : pack((size_t)-1);
}

// ------------------------------------------------------------------------------------------ routes
// Up to so many pulses the fused pass 2's one launch wins over the resample in a kernel of its own (float 256 x 240 frame: 28 us,
// 34 with the split, 400 x 380: 41, 37; fixed: 44, 50 and 69, 57).
constexpr int kFusedPulses = 256;

// Which jobs the passes in runs may take.  The kernels give up single runs by themselves, whatever the vectors hold, so most of
// a rule is an estimate of what pays; what they rely on is: ascending sources and queries (zeros for a run whose
// queries lie outside the sources' span), finite values, and sources whose far end is where the affine axis has it.
// Comparisons are written so that a NaN fails them.
struct RunsRule {
    bool runs = false;
    double ratio = 1.0;              // widest output spacing in source samples
};

// Pass 1 of the float sinc: every step of the output grid is 6/7 to 8/7 of the sample spacing of every pulse (eight brackets then
// advance by one sample each, give or take one in all).
inline RunsRule float_pass1_rule(int m, int n, const double *f0, const double *df, const double *f_last, const double *pr,
                                 const double *kr) {
    double smax = 0.0, smin = INFINITY, dmax = 0.0, dmin = INFINITY;
    bool ok = true;
    for (int j = 1; j < n; ++j) {
        ok = ok && kr[j] > kr[j - 1];
        smax = std::max(smax, kr[j] - kr[j - 1]);
        smin = std::min(smin, kr[j] - kr[j - 1]);
    }
    for (int i = 0; i < m; ++i) {
        const double dk = 2.0 / 299792458.0 * pr[i] * df[i];
        // the last eight samples before the end belong to no run: there the given end sample counts
        ok = ok && dk > 0.0 && std::fabs((f_last[i] - f0[i]) / df[i] - (n - 1)) <= 8.0;
        dmax = std::max(dmax, dk);
        dmin = std::min(dmin, dk);
    }
    RunsRule r;
    r.ratio = smax / dmin;
    r.runs = ok && std::isfinite(dmax) && smin / dmax >= 6.0 / 7.0 && r.ratio <= 8.0 / 7.0;
    return r;
}

// Pass 1 of the fixed-point sinc: eight steps of the output grid (float32 values) stay within a sample of eight of every pulse's.
inline RunsRule fixed_pass1_rule(int m, int n, const float *f0, const float *df, const float *fac, const float *kr) {
    double smin = INFINITY, smax = -INFINITY, wide = 0.0, tmin = INFINITY, tmax = -INFINITY;
    bool ok = n >= 64;
    for (int j = 0; j + 1 < n; ++j) {
        const double s1 = (double)kr[j + 1] - (double)kr[j];
        ok = ok && s1 > 0.0;
        wide = std::max(wide, s1);
        if (j + 8 < n) {
            smin = std::min(smin, (double)kr[j + 8] - (double)kr[j]);
            smax = std::max(smax, (double)kr[j + 8] - (double)kr[j]);
        }
    }
    for (int i = 0; i < m; ++i) {
        const double dk = (double)fac[i] * (double)df[i];
        ok = ok && dk > 0.0 && std::isfinite(f0[i]);
        tmin = std::min(tmin, dk);
        tmax = std::max(tmax, dk);
    }
    RunsRule r;
    r.ratio = smax / (8.0 * tmin);
    r.runs = ok && std::isfinite(tmax) && smin >= 7.0 * tmax && smax <= 9.0 * tmin && wide <= 2.0 * tmin;
    return r;
}

// Pass 2 in a kernel of its own: the sources ascend and lie near an affine axis, the output spacing is near theirs (in eight outputs
// the brackets gain or lose less than one and a half samples), and 32 adjacent range bins share their brackets closely enough
// for one staged segment of tan(phi).  `step`: outputs over which the spacing is taken (float32 queries: eight).
struct SplitRule : RunsRule {
    int slack = 0;                   // of the affine guess, in samples
    double spread = 0.0;             // samples by which the brackets of 32 adjacent range bins differ
};

template <class T>
SplitRule pass2_rule(int m, int n, const T *tn, const T *kc, const T *kr, int step) {
    SplitRule r;
    if (m <= kFusedPulses) return r;
    const double span = (double)tn[m - 1] - (double)tn[0], cell = span / (m - 1);
    double dev = 0.0, irr = 0.0, gap = INFINITY, krmin = INFINITY, krmax = -INFINITY, qmax = 0.0, qmin = INFINITY;
    bool ok = span > 0.0 && std::isfinite(span);
    for (int i = 0; i < m && ok; ++i) {
        dev = std::max(dev, std::fabs(((double)tn[i] - (double)tn[0]) / cell - i));
        if (i + 8 < m) irr = std::max(irr, std::fabs(((double)tn[i + 8] - (double)tn[i]) / cell - 8.0));
        if (i + step < m) {
            qmax = std::max(qmax, ((double)kc[i + step] - (double)kc[i]) / step);
            qmin = std::min(qmin, ((double)kc[i + step] - (double)kc[i]) / step);
        }
        if (i + 1 < m) {
            ok = tn[i + 1] >= tn[i] && kc[i + 1] >= kc[i];
            if (tn[i + 1] > tn[i]) gap = std::min(gap, (double)tn[i + 1] - (double)tn[i]);
        }
    }
    for (int j = 0; j < n && ok; ++j) {
        ok = kr[j] > T(0) && std::isfinite(kr[j]);
        krmin = std::min(krmin, (double)kr[j]);
        krmax = std::max(krmax, (double)kr[j]);
    }
    if (!ok) return r;
    for (int j = 0; j < n; j += 32) {
        const double a = kr[j], b = kr[std::min(j + 31, n - 1)];
        r.spread = std::max(r.spread, std::fabs(a / b - 1.0) * std::max(std::fabs((double)tn[0]), std::fabs((double)tn[m - 1])) / cell);
    }
    const double rmin = qmin / (krmax * cell);
    r.ratio = qmax / (krmin * cell);
    r.slack = (int)std::ceil(std::min(dev, 1e6)) + 1;
    const double drift = 8.0 * std::max(std::fabs(r.ratio - 1.0), std::fabs(rmin - 1.0));
    r.runs = dev <= 3.0 && r.spread <= 64.0 && irr + drift <= 1.5 && krmin * gap > 1e-30 && krmax * span < 1e30;
    return r;
}

}  // namespace pfa
