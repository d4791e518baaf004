// Float PFA datapath on sm_100a: the drop-in for form_image_pfa.pfa + detection
// (src/form_image_pfa.py:165-246, mpfs/host/accel.py:39-44).
//
//   pfa_pass1.cu   per pulse: range resample, corner turn #1
//   pfa_pass2.cu   per range bin: cross resample, window, FFT along cross, corner turn #2
//   pfa_resample2.cu  the cross resample in a kernel of its own, and the FFT of its rows
//   pfa_fft2.cu    per cross bin: FFT along range, detection
//   pfa_autofocus.cu  the entropy gradient over these
//
// This file: the plan's device state, the job upload, the frame and its entry points.
//
// Centring: fftshift(fft(ifftshift(x)))[v] = (-1)^v fft((-1)^a x[a])[v] for even N with N/2 even, so the
// shifts of form_image_pfa.transform2d (:144-147) cost one sign flip on load and one on store.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <string>
#include <vector>

#include "fft_f32.cuh"
#include "interp_f32.cuh"
#include "pfa_internal.h"
#include "tma_sm100.cuh"

namespace pfa {
const int16_t *builtin_sinc_table();

namespace {

int ilog2i(int v) { int l = 0; while ((1 << l) < v) ++l; return l; }

// W_N^k = exp(-2 pi i k / N), k < N (the inverse transform conjugates data, not twiddles)
void full_twiddles(int N, std::vector<float2> &out) {
    out.resize(N);
    for (int k = 0; k < N; ++k) {
        const double th = -2.0 * M_PI * (double)k / (double)N;
        out[k] = make_float2((float)std::cos(th), (float)std::sin(th));
    }
    // the factors of every tile's passes, in reading order (fft_f32.cuh)
    out.resize(tw_offset(N, 32, 99));
    for (int E = 2; E <= 32; E *= 2) {
        if (N / E < 32) continue;
        for (int p = 1; fft_pass(N, E, p).NS < N; ++p) {
            const FftPass ps = fft_pass(N, E, p);
            float2 *dst = out.data() + tw_offset(N, E, p);
            for (int a = 0; a < tw_arrays(ps.R); ++a) {
                const int r = ps.R <= 4 ? a + 1 : (a ? 4 * a : 1);
                for (int k = 0; k < ps.NS; ++k) dst[a * ps.NS + k] = out[r * k * (N / (ps.NS * ps.R))];
            }
        }
    }
}

}  // namespace

size_t float_workspace_bytes(int m, int n, bool rows) {
    const int m2 = 1 << ilog2i(m), mpad = (m + 31) / 32 * 32;
    const int npad = (n + 7) / 8 * 8;
    return (size_t)(rows ? 16 : 8) * n * mpad + (size_t)8 * npad * m2;
}

cudaError_t float_alloc(FloatDev &d, int m, int n, bool rows) {
    d.m = m; d.n = n;
    d.Lm = ilog2i(m); d.Ln = ilog2i(n);
    d.m2 = 1 << d.Lm; d.n2 = 1 << d.Ln;
    d.mpad = (m + 31) / 32 * 32;
    d.npad = (n + 7) / 8 * 8;             // whole clusters of the FP32 (kCT) and mixed pass-2 kernels
    if (d.m2 < 64 || d.n2 < 64 || d.m2 > 16384 || d.n2 > 16384) return cudaErrorInvalidValue;
    cudaError_t e;
#define TRY(x) do { e = (x); if (e != cudaSuccess) return e; } while (0)
    TRY(Arena::allocate(d.blocks, [&](Arena &a) {
        a.take(d.f0, m); a.take(d.df, m); a.take(d.flast, m); a.take(d.pr, m);
        a.take(d.tan_s, m + 512);             // the pass-2 resample stages whole segments
        a.take(d.order, m); a.take(d.each, 2);
        a.take(d.kr, n + 1); a.take(d.kc, m + 1); a.take(d.ham_m64, m + 1);       // staged in 16-byte units
        a.take(d.ham_n64, n);
        d.job_bytes = a.together();
        a.take(d.twm, tw_offset(d.m2, 32, 99)); a.take(d.twn, tw_offset(d.n2, 32, 99));
        a.take(d.tabq, kTabShorts); a.take(d.tabr, 256 * 32); a.take(d.wait_err, 1);
        a.take(d.p1, (size_t)n * d.mpad);
        if (rows) a.take(d.g2, (size_t)n * d.mpad);
        a.take(d.y1, (size_t)d.npad * d.m2);
    }));
    int dev = 0;
    TRY(cudaGetDevice(&dev));
    TRY(cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, dev));
    TRY(cudaMemset(d.wait_err, 0, sizeof(int)));
    // pass 2 reads its range-bin row of p1 as 256-sample boxes (2 KB; the last one zero-filled past mpad)
    TRY(tma::encode_2d(&d.p1_map, d.p1, 8, (uint64_t)d.mpad, (uint64_t)n, (uint64_t)8 * d.mpad, 256, 1));
#undef TRY
    return cudaSuccess;
}

void float_free(FloatDev &d) {
    d.blocks.free();
    d.af_blocks.free();
    d.af_zadj = nullptr;
    mixed_free(d);
}

cudaError_t float_form(const FloatDev &d, const float2 *sig, void *out, int detect, cudaStream_t st, StageProf *prof,
                       const float *theta) {
    StageProf none;
    StageProf &pf = prof ? *prof : none;
    pf.count = 0;
    cudaError_t e = pf.mark(st, "start");
    if (e != cudaSuccess) return e;
    if ((e = float_pass1(d, sig, theta, st)) != cudaSuccess) return e;
    if ((e = pf.mark(st, "pass1")) != cudaSuccess) return e;
    // mixed mode: tensor-core FFTs on the axes whose lines are 2048..8192 points, FP32 FFTs elsewhere
    if (d.mixed && mixed_axis(d.Lm)) e = mixed_pass2(d, st);
    else e = float_pass2(d, st);
    if (e != cudaSuccess) return e;
    if ((e = pf.mark(st, "pass2_win_fft1")) != cudaSuccess) return e;
    const float scale = d.sgn > 0 ? 1.0f / ((float)d.m2 * (float)d.n2) : 1.0f;
    if (d.mixed && mixed_axis(d.Ln)) e = mixed_fft2(d, out, detect, scale, st);
    else e = float_fft2(d, out, detect, scale, st);
    if (e != cudaSuccess) return e;
    return pf.mark(st, "fft2_detect");
}

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

pfa_status pfa_set_float_job(pfa_plan *p, const pfa_float_job *job) {
    if (!p || !job) return PFA_ERR_BAD_ARG;
    if (p->cfg.mode != PFA_MODE_FLOAT32 && p->cfg.mode != PFA_MODE_MIXED) return ffail(p, PFA_ERR_BAD_CONFIG, "plan is not float mode");
    if (!job->f0 || !job->df || !job->f_last || !job->pr || !job->tan_s || !job->order || !job->kr_grid || !job->kc_grid)
        return ffail(p, PFA_ERR_BAD_ARG, "missing job vector");
    if (job->layout != PFA_LAYOUT_CENTRED && job->layout != PFA_LAYOUT_NATURAL) return ffail(p, PFA_ERR_BAD_ARG, "bad layout");
    DevGuard dg(p->device);
    pfa::FloatDev &d = p->fl;
    const int m = d.m, n = d.n;
    std::vector<int> seen(m, 0);
    for (int i = 0; i < m; ++i) {
        const int r = job->order[i];
        if (r < 0 || r >= m || seen[r]++) return ffail(p, PFA_ERR_BAD_ARG, "order is not a permutation");
    }
    d.sgn = job->sgn < 0 ? -1 : 1;
    d.layout = job->layout;
    d.window = (job->ham_m && job->ham_n) ? 1 : 0;
    cudaError_t e;
#define CPY(dst, src, cnt) do { e = cudaMemcpy(dst, src, sizeof(*(dst)) * (cnt), cudaMemcpyHostToDevice); \
        if (e != cudaSuccess) return fcuda(p, e, "float job upload"); } while (0)
    if (!d.consts_ready) {      // twiddles and the sinc table depend on the plan's shape only
        std::vector<float2> twm, twn;
        pfa::full_twiddles(d.m2, twm);
        pfa::full_twiddles(d.n2, twn);
        std::vector<int16_t> tabq(pfa::kTabShorts, 0);
        const int16_t *tq = pfa::builtin_sinc_table();
        for (int i = 0; i < 256 * 32; ++i) tabq[(i >> 5) * pfa::kTabRow + (i & 31)] = tq[i];   // [phase][tap], padded rows
        CPY(d.twm, twm.data(), twm.size()); CPY(d.twn, twn.data(), twn.size());
        CPY(d.tabq, tabq.data(), pfa::kTabShorts);
        std::vector<uint16_t> tabr(256 * 32);
        for (int i = 0; i < 256 * 32; ++i) tabr[i] = (uint16_t)(tq[i] + 32768);
        CPY(d.tabr, tabr.data(), 256 * 32);
        d.consts_ready = true;
    }
#undef CPY
    const pfa::RunsRule r1 = pfa::float_pass1_rule(m, n, job->f0, job->df, job->f_last, job->pr, job->kr_grid);
    d.p1_runs = r1.runs;
    d.p1_ratio = r1.ratio;
    // Pass 2 in a kernel of its own, sinc (and mixed mode) only: 8167 x 8192 pass 2 1.69 -> 1.15 ms; with the FP32 lerp the extra
    // trip through memory cost about what the cheaper brackets save (0.79 against 0.81 ms there, 30 against 25 us at
    // 1024^2, measured with a resample 8 % slower than now).  The fused kernel takes the other jobs.
    const pfa::SplitRule r2 = pfa::pass2_rule(m, n, job->tan_s, job->kc_grid, job->kr_grid, 1);
    d.p2_slack = r2.slack;
    d.p2_runs = r2.runs && d.g2 && pfa::resample2_shape(d.az_sinc != 0, r2.ratio, r2.slack, r2.spread, &d.p2_pitch, &d.p2_tlen);
    // the job's vectors go up as one copy of their host image
    std::vector<unsigned char> &img = p->job_host;
    img.resize(d.job_bytes);
    auto put = [&](const void *dst, const void *src, size_t bytes) {
        std::memcpy(img.data() + (static_cast<const unsigned char *>(dst) - static_cast<const unsigned char *>(d.blocks.at[0])), src, bytes);
    };
    put(d.f0, job->f0, 8u * m); put(d.df, job->df, 8u * m); put(d.flast, job->f_last, 8u * m); put(d.pr, job->pr, 8u * m);
    put(d.tan_s, job->tan_s, 8u * m); put(d.order, job->order, 4u * m); put(d.kr, job->kr_grid, 8u * n);
    put(d.kc, job->kc_grid, 8u * m);
    if (d.window) { put(d.ham_m64, job->ham_m, 8u * m); put(d.ham_n64, job->ham_n, 8u * n); }
    // a frame captured in a graph under another job may replay the kernels of that job's route with these vectors
    const int32_t each[2] = {!d.p1_runs, !d.p2_runs};
    put(d.each, each, sizeof(each));
    if ((e = cudaMemcpy(d.blocks.at[0], img.data(), img.size(), cudaMemcpyHostToDevice)) != cudaSuccess) return fcuda(p, e, "float job upload");
    p->job_ready = true;
    return PFA_OK;
}

pfa_status pfa_form_float(pfa_plan *p, const float *sig_dev, void *out_dev, int32_t detect, void *stream) {
    if (!p || !sig_dev || !out_dev) return PFA_ERR_BAD_ARG;
    if (p->cfg.mode != PFA_MODE_FLOAT32 && p->cfg.mode != PFA_MODE_MIXED) return ffail(p, PFA_ERR_BAD_CONFIG, "plan is not float mode");
    if (!p->job_ready) return ffail(p, PFA_ERR_NOT_READY, "pfa_set_float_job not called");
    if (detect < PFA_DETECT_MAG || detect > PFA_DETECT_COMPLEX) return ffail(p, PFA_ERR_BAD_ARG, "bad detect mode");
    if (reinterpret_cast<uintptr_t>(sig_dev) & 7) return ffail(p, PFA_ERR_BAD_ARG, "signal must be 8-byte aligned");
    if (p->fl.mixed && (reinterpret_cast<uintptr_t>(out_dev) & 15))
        return ffail(p, PFA_ERR_BAD_ARG, "mixed mode: output must be 16-byte aligned");
    DevGuard dg(p->device);
    cudaError_t e = pfa::float_form(p->fl, reinterpret_cast<const float2 *>(sig_dev), out_dev, detect,
                                    reinterpret_cast<cudaStream_t>(stream), &p->prof);
    if (e != cudaSuccess) return fcuda(p, e, "float form");
    return PFA_OK;
}

static pfa_status wait_timeout_check(pfa_plan *p);

pfa_status pfa_form_float_host(pfa_plan *p, const float *sig_host, void *out_host, int32_t detect) {
    if (!p || !sig_host || !out_host) return PFA_ERR_BAD_ARG;
    if (p->cfg.mode != PFA_MODE_FLOAT32 && p->cfg.mode != PFA_MODE_MIXED) return ffail(p, PFA_ERR_BAD_CONFIG, "plan is not float mode");
    DevGuard dg(p->device);
    const size_t in_b = sizeof(float) * 2 * (size_t)p->fl.m * p->fl.n;
    const size_t out_b = (detect == PFA_DETECT_COMPLEX ? 8 : 4) * (size_t)p->fl.m2 * p->fl.n2;
    cudaError_t e;
    if (!p->host_stream && (e = cudaStreamCreateWithFlags(&p->host_stream, cudaStreamNonBlocking)) != cudaSuccess)
        return fcuda(p, e, "stream");
    if (p->staging_in_bytes < in_b) {
        if (p->staging_in) cudaFree(p->staging_in);
        p->staging_in = nullptr;
        if ((e = cudaMalloc(reinterpret_cast<void **>(&p->staging_in), in_b)) != cudaSuccess) { p->staging_in_bytes = 0; return fcuda(p, e, "staging"); }
        p->staging_in_bytes = in_b;
    }
    if (p->staging_out_bytes < out_b) {
        if (p->staging_out) cudaFree(p->staging_out);
        p->staging_out = nullptr;
        if ((e = cudaMalloc(&p->staging_out, out_b)) != cudaSuccess) { p->staging_out_bytes = 0; return fcuda(p, e, "staging"); }
        p->staging_out_bytes = out_b;
    }
    if ((e = cudaMemcpyAsync(p->staging_in, sig_host, in_b, cudaMemcpyHostToDevice, p->host_stream)) != cudaSuccess)
        return fcuda(p, e, "h2d");
    pfa_status st = pfa_form_float(p, p->staging_in, p->staging_out, detect, p->host_stream);
    if (st != PFA_OK) return st;
    if ((e = cudaMemcpyAsync(out_host, p->staging_out, out_b, cudaMemcpyDeviceToHost, p->host_stream)) != cudaSuccess)
        return fcuda(p, e, "d2h");
    if ((e = cudaStreamSynchronize(p->host_stream)) != cudaSuccess) return fcuda(p, e, "sync");
    return wait_timeout_check(p);
}

// A bounded wait that ran out (pass 2's TMA row load; in mixed mode also a tensor-core completion) sets a
// device flag; synchronous entry points read (and clear) it after their frames and report PFA_ERR_TIMEOUT.
static pfa_status wait_timeout_check(pfa_plan *p) {
    if (!p->fl.wait_err) return PFA_OK;
    int flag = 0;
    cudaError_t e = cudaMemcpy(&flag, p->fl.wait_err, sizeof(int), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return fcuda(p, e, "timeout flag");
    if (!flag) return PFA_OK;
    cudaMemset(p->fl.wait_err, 0, sizeof(int));
    return ffail(p, PFA_ERR_TIMEOUT, "a bounded wait on the device timed out (frame not valid)");
}

static pfa_status float_frame(pfa_plan *p, const void *in, void *out, cudaStream_t st, int32_t detect) {
    return pfa_form_float(p, static_cast<const float *>(in), out, detect, st);
}

pfa_status pfa_form_float_host_frames(pfa_plan *p, const float *const *sig_hosts, void *const *out_hosts,
                                      int32_t detect, int32_t nframes) {
    if (!p) return PFA_ERR_BAD_ARG;
    if (p->cfg.mode != PFA_MODE_FLOAT32 && p->cfg.mode != PFA_MODE_MIXED) return ffail(p, PFA_ERR_BAD_CONFIG, "plan is not float mode");
    if (detect < PFA_DETECT_MAG || detect > PFA_DETECT_COMPLEX) return ffail(p, PFA_ERR_BAD_ARG, "bad detect mode");
    DevGuard dg(p->device);
    const size_t in_b = sizeof(float) * 2 * (size_t)p->fl.m * p->fl.n;
    const size_t out_b = (detect == PFA_DETECT_COMPLEX ? 8 : 4) * (size_t)p->fl.m2 * p->fl.n2;
    const pfa_status st = pfa::run_host_frames(p, reinterpret_cast<const void *const *>(sig_hosts), out_hosts, nframes,
                                               in_b, out_b, float_frame, detect);
    return st != PFA_OK ? st : wait_timeout_check(p);
}

pfa_status pfa_form_float_phase(pfa_plan *p, const float *sig_dev, const float *theta_dev, void *out_dev, int32_t detect,
                                void *stream) {
    if (!p || !sig_dev || !theta_dev || !out_dev) return PFA_ERR_BAD_ARG;
    if (p->cfg.mode != PFA_MODE_FLOAT32 && p->cfg.mode != PFA_MODE_MIXED) return ffail(p, PFA_ERR_BAD_CONFIG, "plan is not float mode");
    if (!p->job_ready) return ffail(p, PFA_ERR_NOT_READY, "pfa_set_float_job not called");
    if (detect < PFA_DETECT_MAG || detect > PFA_DETECT_COMPLEX) return ffail(p, PFA_ERR_BAD_ARG, "bad detect mode");
    if (reinterpret_cast<uintptr_t>(sig_dev) & 7) return ffail(p, PFA_ERR_BAD_ARG, "signal must be 8-byte aligned");
    if (p->fl.mixed && (reinterpret_cast<uintptr_t>(out_dev) & 15))
        return ffail(p, PFA_ERR_BAD_ARG, "mixed mode: output must be 16-byte aligned");
    DevGuard dg(p->device);
    cudaError_t e = pfa::float_form(p->fl, reinterpret_cast<const float2 *>(sig_dev), out_dev, detect,
                                    reinterpret_cast<cudaStream_t>(stream), &p->prof, theta_dev);
    if (e != cudaSuccess) return fcuda(p, e, "float form");
    return PFA_OK;
}

}  // extern "C"
