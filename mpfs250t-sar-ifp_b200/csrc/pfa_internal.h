// Internal plan state shared by the C-ABI glue and the kernel launchers.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <new>
#include <string>
#include <vector>

#include "../../include/pfa_b200.h"
#include "host_rules.h"

namespace pfa {

// FixedDev::ctrl word that a bounded wait of the passes in runs sets when it runs out (cleared by the first frame of the
// entry points that report it)
constexpr int kFixedErrWord = 8;

// The device allocations of a plan's buffers (host_rules.h says how the buffers share them).
struct Blocks {
    void *at[kMaxBlocks] = {};
    explicit operator bool() const { return at[0] != nullptr; }
    void free() {
        for (void *&b : at) {
            if (b) cudaFree(b);
            b = nullptr;
        }
    }
};

// Hands out the buffers of a layout, 256-byte aligned: a first walk over the layout collects their sizes, a second one their
// places in `blocks`.
class Arena {
  public:
    template <class T>
    void take(T *&p, size_t count) {
        if (!blocks_) bytes_.push_back((std::max<size_t>(count, 1) * sizeof(T) + 255) / 256 * 256);
        else p = reinterpret_cast<T *>(static_cast<unsigned char *>(blocks_->at[pack_.in[next_]]) + pack_.offset[next_]), ++next_;
    }
    // the buffers so far lie in a row at the start of the first block; their bytes
    size_t together() {
        if (!blocks_) head_ = bytes_.size();
        size_t sum = 0;
        for (size_t i = 0; i < head_; ++i) sum += bytes_[i];
        return sum;
    }
    template <class F>
    static cudaError_t allocate(Blocks &blocks, F &&layout) {
        Arena a;
        try {
            layout(a);
            a.pack_ = pack_buffers(a.bytes_, a.head_);
        } catch (const std::bad_alloc &) {                   // (no exception leaves the C entry points)
            return cudaErrorMemoryAllocation;
        }
        for (size_t i = 0; i < a.pack_.block.size(); ++i) {
            const cudaError_t e = cudaMalloc(&blocks.at[i], a.pack_.block[i]);
            if (e != cudaSuccess) {
                blocks.at[i] = nullptr;
                blocks.free();
                return e;
            }
        }
        a.blocks_ = &blocks;
        layout(a);
        return cudaSuccess;
    }

  private:
    std::vector<size_t> bytes_;
    size_t head_ = 0, next_ = 0;
    Packing pack_;
    const Blocks *blocks_ = nullptr;
};

// Device-resident fixed-point job + workspace for one (m, n, G) frame.
struct FixedDev {
    int m = 0, n = 0, G = 0, L = 0, mpad = 0;
    int range_sinc = 0, az_sinc = 0;
    int range_cubic = 0, az_cubic = 0;      // 4-tap Lagrange variant (sinc flags off)
    int fused_detect = 0;                   // silicon detect order
    // job vectors (device)
    float *f0 = nullptr, *df = nullptr, *fac = nullptr, *tan_s = nullptr;
    float *krp = nullptr, *kcp = nullptr;
    int32_t *order = nullptr;          // sorted slot -> pulse index
    int32_t *hamr = nullptr, *hamc = nullptr;
    uint32_t *tw = nullptr;            // stage-contiguous twiddles, G-1 packed int16x2
    int16_t *sinc = nullptr;           // 256 x 32, [tap][phase]
    uint16_t *sinc_pm = nullptr;       // the same taps [phase][tap] (runs of outputs)
    bool p1_runs = false;              // pass 1 may form its sinc outputs in runs (job)
    double p1_ratio = 1.0;             // widest output spacing of pass 1 in source samples (job)
    bool p2_runs = false;              // pass 2 resamples in a kernel of its own (job)
    int p2_pitch = 0, p2_tlen = 0, p2_slack = 0;   // its window pitch, tan segment, slack of the affine guess (job)
    uint32_t *sq = nullptr;            // [m][n] Q0-quantised signal, packed int16x2, in y1's memory (range sinc; else null)
    int sms = 0;                       // SM count of the plan's device
    int probe = 0;                     // test hook: polls of a wait on an unarmed barrier (passes in runs)
    bool clear_err = false;            // the next frame clears ctrl[kFixedErrWord]
    // workspace (device)
    uint32_t *p1 = nullptr;            // [n][mpad] pass-1 output, packed int16x2
    uint32_t *y1 = nullptr;            // [n][G] FFT-1 output (range-bin rows)
    uint32_t *y2 = nullptr;            // [G][G] FFT-2 output (cross-bin rows)
    int32_t *e1 = nullptr;             // [G]
    int32_t *e2 = nullptr;             // [G]
    int32_t *ctrl = nullptr;           // [0] q0 max bits (0: quantised input), [1] emax1, [2] emax2, [kFixedErrWord]
    Blocks blocks;                     // the plan's device memory
    void *job_block = nullptr;         // the job vectors above (f0 .. sinc_pm)
    size_t job_bytes = 0;
    int32_t *each = nullptr;           // [2] (job): nonzero where passes 1 and 2 may not run in runs
};

struct FloatDev {
    int m = 0, n = 0, m2 = 0, n2 = 0, Lm = 0, Ln = 0, mpad = 0, npad = 0;
    int range_sinc = 0, az_sinc = 0, sgn = -1, layout = 0;
    Blocks blocks;                              // the plan's device memory; the job's vectors lie at its start
    size_t job_bytes = 0;
    double *f0 = nullptr, *df = nullptr, *flast = nullptr, *pr = nullptr, *tan_s = nullptr, *kr = nullptr, *kc = nullptr;
    float *ham_m = nullptr, *ham_n = nullptr;   // unused when window is off
    double *ham_m64 = nullptr, *ham_n64 = nullptr;
    int32_t *order = nullptr;
    float2 *twm = nullptr, *twn = nullptr;      // twiddle tables of m2- and n2-point lines (fft_f32.cuh)
    int16_t *tabq = nullptr;                    // sinc table (Q15 taps), [phase][tap] rows of 40 int16
    uint16_t *tabr = nullptr;                   // the same taps as uint16 tap + 32768, [phase][32] (sinc_run)
    bool consts_ready = false;                  // twm, twn and the tap tables (plan constants) uploaded
    double p1_ratio = 1.0;                      // widest output spacing of pass 1 in source samples (job)
    bool p1_runs = false;                       // pass 1 may form its sinc outputs in runs (job)
    int window = 1;
    float2 *p1 = nullptr;              // [n][mpad] pass-1 output (range-bin rows, sorted pulses)
    CUtensorMap p1_map;                // TMA map of p1: 8-byte elements, boxes of 256 x 1
    float2 *g2 = nullptr;              // [n][mpad] pass-2 resampled rows (azimuth sinc or mixed mode; autofocus: without the window)
    bool p2_runs = false;              // pass 2 resamples in a kernel of its own (job)
    int p2_pitch = 0, p2_tlen = 0, p2_slack = 0;   // its window pitch, tan segment, slack of the affine guess (job)
    float2 *y1 = nullptr;              // [m2][npad] cross FFT output, transposed (cross-bin rows)
    int ept_cross = 0, ept_range = 0;    // FFT register tile (complex values per thread; 0 = automatic)
    Blocks af_blocks;                  // the autofocus workspace below (af_acc .. af_pk)
    float2 *af_zadj = nullptr;         // [n][m2] autofocus: adjoint of the range FFT (range-bin rows)
    double *af_acc = nullptr;          // [2] sum I, sum I log I
    float *af_dacc = nullptr;          // [mpad] per-slot gradient accumulators
    uint32_t *af_pk = nullptr;         // [n][mpad] autofocus: packed pass-2 brackets of the forward pass
    uint32_t *pk_out = nullptr;        // where pass 2 stores its packed brackets for the adjoint (or nullptr)
    float2 *af_rp = nullptr;           // [n][mpad] autofocus, float-sinc plans: the forward's resampled rows R2 p1 (g2 where the plan
                                       // has it)
    float2 *rp_out = nullptr;          // where a float-sinc pass 2 stores R2 p1 for the adjoint (or nullptr)
    // split-precision (mixed) mode: tensor-core FFTs for lines of 2048..8192 points
    int mixed = 0;
    uint4 *mx_f128 = nullptr;          // F_128 TMEM image [128 lanes][256 columns] of fp16 pairs
    uint4 *mx_fn2m = nullptr, *mx_fn2n = nullptr;   // F_{m2/128}, F_{n2/128} shared-memory images
    int *wait_err = nullptr;           // device flag: a bounded wait ran out (TMA row load, tensor-core completion)
    int mx_clusters = 0;               // resident 4-CTA clusters of the mixed pass 2
    int mx_probe = 0;                  // test hook: polls of a wait on an unarmed barrier (pass 1 in runs; FP32: pass 2's
                                       // loads; mixed: the tensor-core range FFT)
    int sms = 0;                       // SM count of the plan's device
    int32_t *each = nullptr;           // [2] (job): nonzero where passes 1 and 2 may not run in runs
};

}  // namespace pfa

namespace pfa {
// Stage events recorded between kernels when profiling is on.
struct StageProf {
    static constexpr int kMax = 12;
    bool on = false;
    int count = 0;                      // events recorded in the last frame
    cudaEvent_t ev[kMax] = {};
    const char *names[kMax] = {};
    cudaError_t mark(cudaStream_t st, const char *name) {
        if (!on || count >= kMax) return cudaSuccess;
        names[count] = name;
        return cudaEventRecord(ev[count++], st);
    }
};
}  // namespace pfa

struct pfa_plan {
    pfa_config cfg{};
    int device = 0;
    bool job_ready = false;
    size_t ws_bytes = 0;
    pfa::FixedDev fx;
    pfa::FloatDev fl;
    float *staging_in = nullptr;       // device copy of the host signal (host entry points)
    void *staging_out = nullptr;
    size_t staging_in_bytes = 0, staging_out_bytes = 0;
    cudaStream_t host_stream = nullptr;
    // pipelined host frames: upload / compute / download streams, double-buffered staging
    cudaStream_t pipe_up = nullptr, pipe_comp = nullptr, pipe_down = nullptr;
    void *pipe_in[2] = {nullptr, nullptr}, *pipe_out[2] = {nullptr, nullptr};
    size_t pipe_in_bytes = 0, pipe_out_bytes = 0;
    cudaEvent_t pipe_ev[6] = {};      // uploaded[2], computed[2], downloaded[2]
    // fixed job staging: the host image of FixedDev::job_block (one upload per job) and the inputs the
    // grid-dependent tables were last derived from (rebuilt only when those change)
    std::vector<unsigned char> job_host;
    std::vector<int16_t> last_tw_in, last_sinc_in;
    int last_tw_builtin = -1, last_sinc_builtin = -1;
    pfa::StageProf prof;
    std::string err;
};

namespace pfa {

// Kernel launchers (pfa_fixed.cu / pfa_float.cu). They return a cudaError_t from the launches.
cudaError_t fixed_form(const FixedDev &d, const float *sig_c64, const uint32_t *sig_iq, uint16_t *img,
                       cudaStream_t st, StageProf *prof);
// pass 1 in runs (pfa_fixed_runs.cu): quantises the complex64 signal into d.sq first (sig_iq: already quantised)
cudaError_t fixed_pass1_runs(const FixedDev &d, const float *sig_c64, const uint32_t *sig_iq, cudaStream_t st);
// pass 2's resample in runs into g2 ([n][mpad]), and the shape it needs for a job (pfa_fixed_runs.cu)
cudaError_t fixed_resample2(const FixedDev &d, uint32_t *g2, cudaStream_t st);
bool fixed_resample2_shape(double ratio, int slack, double spread, int *pitch, int *tlen);
size_t fixed_workspace_bytes(int m, int n, int G);
cudaError_t fixed_alloc(FixedDev &d, int m, int n, int G, bool range_sinc);
void fixed_free(FixedDev &d);

// theta (device, [m], or nullptr): per-pulse phase correction exp(-j theta_i) applied in pass 1
cudaError_t float_form(const FloatDev &d, const float2 *sig, void *out, int detect, cudaStream_t st,
                       StageProf *prof, const float *theta = nullptr);
cudaError_t float_pass1(const FloatDev &d, const float2 *sig, const float *theta, cudaStream_t st);   // pfa_pass1.cu
cudaError_t float_resample2(const FloatDev &d, cudaStream_t st);                                      // pfa_resample2.cu
cudaError_t float_row_fft(const FloatDev &d, cudaStream_t st);                                        // pfa_resample2.cu
// window pitch and tan segment of the pass-2 resample for a job; false when they do not fit       (pfa_resample2.cu)
bool resample2_shape(bool sinc, double ratio, int slack, double spread, int *pitch, int *tlen);
cudaError_t float_pass2(const FloatDev &d, cudaStream_t st);                                          // pfa_pass2.cu
cudaError_t float_fft2(const FloatDev &d, void *out, int detect, float scale, cudaStream_t st);       // pfa_fft2.cu
size_t float_workspace_bytes(int m, int n, bool rows);
cudaError_t float_alloc(FloatDev &d, int m, int n, bool rows);   // rows: with g2
void float_free(FloatDev &d);

// Split-precision tensor-core FFT mode (pfa_mixed.cu).
bool mixed_axis(int L);                                  // 2^L-point lines run on the tensor cores
cudaError_t mixed_prepare(FloatDev &d);                  // tables, SM/cluster occupancy (plan creation)
void mixed_free(FloatDev &d);
cudaError_t mixed_pass2(const FloatDev &d, cudaStream_t st);
cudaError_t mixed_fft2(const FloatDev &d, void *out, int detect, float scale, cudaStream_t st);

// Pipelined host frames (pfa_capi.cu): form(plan, in_dev, out_dev, stream, arg) runs one frame.
typedef pfa_status (*FrameFn)(pfa_plan *p, const void *in_dev, void *out_dev, cudaStream_t st, int32_t arg);
pfa_status run_host_frames(pfa_plan *p, const void *const *ins, void *const *outs, int32_t nframes, size_t in_bytes,
                           size_t out_bytes, FrameFn form, int32_t arg);

// Host-side table builders used when the caller passes NULL for a table (libm based).
void build_sinc_table(int16_t *tab);   // table from the exact-rational recipe, [phase][tap]
// True when every phase of a [phase][tap] Q15 table has sum |tap| <= 65535 over taps 0-15 and over
// taps 16-31: the condition for the fixed-point sinc's int32 half-sum accumulation to be exact.
bool sinc_table_fits_int32(const int16_t *tab);
void build_twiddles_q15(int G, int16_t *tw2);   // [G/2][2]
void build_hamming_q15(int len, int size, int32_t *out);

}  // namespace pfa
