// Display scaling of the detected image, the quantiser of save_detected_geotiff
// (src/form_image_pfa.py:287-292):
//
//     amp  = |img| (float32)
//     hi   = np.percentile(amp, 99.7)
//     data = np.clip(amp / (hi + 1e-12) * 255.0, 0, 255).astype(np.uint8)
//
// bit-exact on the device, for non-negative magnitudes (the bit-pattern order below needs x >= 0).  np.percentile of a float32 array computes in float32 (NumPy 2 promotion):
// q = f32(99.7) / 100, virtual index v = f32(n - 1) * q, k = floor(v), gamma = v - k, and the lerp of the
// order statistics a = s[k], b = s[k + 1] is a + (b - a) gamma (gamma < 0.5) or b - (b - a)(1 - gamma),
// each a separate float32 operation.  The host evaluates k and gamma; the device finds the two order
// statistics on the float bit patterns (|z| >= 0, so the uint32 patterns sort like the values).
//
// The image (268 MB at 8192^2) is larger than L2, so what bounds the call is the number of sweeps over it.
// Two suffice: a stratified sample of 32768 elements gives a window [lo, hi] of bit patterns that holds both order
// statistics unless the sample is an outlier: 6 standard deviations of as many independent draws.  (They come in
// groups of four neighbours, which a zero-padded image correlates: for focused speckle the deviation of the count is
// 1.1 to 1.3 times that at 99.7 %, 1.4 times at the median, i.e. 4.2 to 5.6 sigma; 3 sigma if the four were equal.)
// One sweep counts what lies below the window, counts its two end values and collects what lies strictly inside
// (about 0.4 % of the image at 99.7 %); one cluster selects from those; the second sweep writes the bytes, back to
// front, so that its first reads find the end of the image in L2.  8192^2 image: 299 us with five sweeps (three radix
// histograms, the next order statistic, the bytes), 157 us now (a focused zero-padded one: 153); the two sweeps take
// 115 of them (floor at the measured copy rate: 92).
//
// When the window misses the rank or overflows the candidate buffer (an image that the sample does not represent),
// the selection takes the image itself instead of the list (up to 2^21 elements), or three gated radix sweeps
// (11 + 11 + 10 bits) by all SMs find the order statistics, launches that otherwise return at once.  Where the
// sample already says that the candidates would come near the buffer's size (a middle percentile of a very large
// image: the median of 8192^2 speckle) the radix sweeps run straight away: 406 us through the window that overflowed,
// 251 without it, 254 with the five sweeps.  Up to 4096 elements the sample is the whole image and the answer exact at once.  All of it is
// stream-ordered in a caller-provided workspace: no allocation, no host synchronisation.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>

#include "pfa_internal.h"
#include "pdl.cuh"

namespace pfa {
namespace {

constexpr int kBins = 2048;
// sample sizes: a larger sample narrows the window (6 sigma of 32768 hold 0.4 % of the image at 99.7 %, of 4096
// 1.4 %), which pays when the candidates of a large image would cost more than the larger sample does
constexpr int kSampleSmall = 4096, kSampleLarge = 32768;
constexpr long long kLargeImage = 1LL << 23;
constexpr unsigned int kCandCap = 1u << 21;
constexpr int kWarpCand = 256;          // candidates a warp of the collecting sweep buffers in shared memory
constexpr int kSelectCtas = 8;          // cluster of the selection
// up to here the selection's cluster itself reads the image when the window missed (a sweep of 8 MB by eight SMs: some
// 10 us); the gated launches would cost 5 us of a call that takes 30
constexpr long long kSelectImage = 1LL << 21;
constexpr unsigned int kNone = 0xffffffffu;

struct DispCtrl {
    unsigned long long rank;     // k (radix sweeps: among the elements that match the prefix so far)
    unsigned long long below;    // elements below lo
    unsigned long long n_lo;     // elements equal to lo
    unsigned long long n_hi;     // elements equal to hi (0 when hi == lo)
    unsigned int lo, hi;         // the window
    unsigned long long cand;     // elements strictly inside it (counted past the buffer's capacity too)
    unsigned int above;          // the smallest element above hi (kNone: none)
    unsigned int above_radix;    // radix sweeps: the smallest element above the prefix's range
    unsigned int prefix;         // radix sweeps: value bits fixed so far
    unsigned int ticket;         // blocks of a radix sweep that are done
    int fallback;                // the radix sweeps run
    float h;                     // hi + 1e-12 in float32
};

struct DispWs {
    DispCtrl ctrl;
    unsigned int hist[kBins];
    unsigned int list[kCandCap];
};

// hi = lerp(s[k], s[k+1], gamma) in float32 as NumPy evaluates it, and h = hi + 1e-12 (float32)
__device__ void disp_hi(DispCtrl &c, unsigned int ak, unsigned int bk, float gamma, float *hi_out) {
    const float a = __uint_as_float(ak), b = __uint_as_float(bk);
    const float d = __fsub_rn(b, a);
    const float r = gamma < 0.5f ? __fadd_rn(a, __fmul_rn(d, gamma)) : __fsub_rn(b, __fmul_rn(d, __fsub_rn(1.0f, gamma)));
    c.h = __fadd_rn(r, 1e-12f);
    if (hi_out) *hi_out = r;
}

// smallest shift that maps [0, width] onto the bins
__device__ __forceinline__ int bin_shift(unsigned int width) {
    return width < (unsigned)kBins ? 0 : 32 - __clz(width) - 11;
}

// The bin of a block histogram (2048 bins, 1024 threads) that holds `rank`, and the count before it.  Counts
// are summed in 64 bits: an image may hold more than 2^32 elements.  Ends with a barrier.
__device__ __forceinline__ void find_bin(const unsigned int *h, unsigned long long rank, unsigned long long *scratch,
                                         unsigned int *bin, unsigned long long *before) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned long long a = h[2 * threadIdx.x], b = h[2 * threadIdx.x + 1];
    unsigned long long inc = a + b;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) scratch[warp] = inc;
    __syncthreads();
    unsigned long long s = scratch[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long t = __shfl_up_sync(0xffffffffu, s, o);
        if (lane >= o) s += t;
    }
    const unsigned long long pw = __shfl_sync(0xffffffffu, s, (warp + 31) & 31);
    const unsigned long long e = (warp ? pw : 0ull) + inc - (a + b);
    if (rank >= e && rank < e + a + b) {
        const bool second = rank >= e + a;
        *bin = 2 * threadIdx.x + (second ? 1u : 0u);
        *before = second ? e + a : e;
    }
    __syncthreads();
}

// One block of 1024 threads, V values each.  n > S = 1024 V: the window [lo, hi] between the sample's order
// statistics r_lo and r_hi; one 16-byte group of elements at a hashed place of each of S / 4 strata (a single SM
// fetches about one scattered sector per clock: 32768 single elements took 33 us, the groups take 18).
// n <= S: the sample is the image, lo and hi are s[k] and s[k + 1], and nothing else has to read the image before the
// writing sweep.  The two order statistics are found by their own descents over 2048 bins of their current
// range (at most three steps, exact), their counts in the two halves of one word; the first range is [min, max], which
// spreads the elements over the bins.
template <int V>
__global__ void __launch_bounds__(1024) k_disp_sample(const float *v, long long n, DispWs *ws,
                                                      unsigned long long rank, unsigned int r_lo, unsigned int r_hi,
                                                      float gamma, float *hi_out) {
    pdl_wait();
    constexpr int S = 1024 * V, LG = V == 32 ? 13 : 10;
    static_assert(S / 4 == 1 << LG, "a power-of-two number of groups");
    __shared__ unsigned int h[kBins], mn, mx, scratch[32], bin[2], before[2];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned int cnt = n < S ? (unsigned int)n : (unsigned int)S;
    if (tid == 0) { mn = kNone; mx = 0u; }
    unsigned int x[V];
    if (n > S) {
        const float4 *v4 = reinterpret_cast<const float4 *>(v);
        const unsigned long long n4 = (unsigned long long)n >> 2;          // >= the number of groups
#pragma unroll
        for (int i = 0; i < V / 4; ++i) {
            const unsigned int g = tid + 1024u * i;
            const unsigned long long a0 = (g * n4) >> LG, a1 = ((g + 1) * n4) >> LG;
            unsigned int r = g * 2654435761u;
            r ^= r >> 15;
            r *= 2246822519u;
            r ^= r >> 13;
            const float4 q = *(v4 + (a0 + (((a1 - a0) * r) >> 32)));
            x[4 * i] = __float_as_uint(q.x); x[4 * i + 1] = __float_as_uint(q.y);
            x[4 * i + 2] = __float_as_uint(q.z); x[4 * i + 3] = __float_as_uint(q.w);
        }
    } else {
#pragma unroll
        for (int i = 0; i < V; ++i) x[i] = tid + 1024u * i < cnt ? __float_as_uint(v[tid + 1024 * i]) : kNone;
    }
    unsigned int lmn = kNone, lmx = 0u;
#pragma unroll
    for (int i = 0; i < V; ++i)
        if (tid + 1024u * i < cnt) { lmn = min(lmn, x[i]); lmx = max(lmx, x[i]); }
    lmn = __reduce_min_sync(0xffffffffu, lmn);
    lmx = __reduce_max_sync(0xffffffffu, lmx);
    __syncthreads();
    if (lane == 0) { atomicMin(&mn, lmn); atomicMax(&mx, lmx); }
    __syncthreads();
    unsigned int lo[2] = {mn, mn}, hi[2] = {mx, mx}, r[2] = {r_lo, r_hi};
    while (lo[0] < hi[0] || lo[1] < hi[1]) {             // block-uniform; a width below 2^32 is one value after three
        const int sh[2] = {bin_shift(hi[0] - lo[0]), bin_shift(hi[1] - lo[1])};
        const bool one = lo[0] == lo[1] && hi[0] == hi[1];
        for (int i = tid; i < kBins; i += 1024) h[i] = 0u;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < V; ++i) {
            if (tid + 1024u * i < cnt) {
                if (x[i] >= lo[0] && x[i] <= hi[0]) atomicAdd(&h[(x[i] - lo[0]) >> sh[0]], one ? 0x10001u : 1u);
                if (!one && x[i] >= lo[1] && x[i] <= hi[1]) atomicAdd(&h[(x[i] - lo[1]) >> sh[1]], 0x10000u);
            }
        }
        __syncthreads();
        // block scan of the packed counts (each sum is at most S <= 32768: no carry into the upper half)
        const unsigned int ha = h[2 * tid], hb = h[2 * tid + 1];
        unsigned int inc = ha + hb;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned int t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        if (lane == 31) scratch[warp] = inc;
        __syncthreads();
        unsigned int sc = scratch[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned int t = __shfl_up_sync(0xffffffffu, sc, o);
            if (lane >= o) sc += t;
        }
        const unsigned int pw = __shfl_sync(0xffffffffu, sc, (warp + 31) & 31);
        const unsigned int ex = (warp ? pw : 0u) + inc - (ha + hb);
#pragma unroll
        for (int w = 0; w < 2; ++w) {
            const unsigned int e = (ex >> (16 * w)) & 0xffffu, a = (ha >> (16 * w)) & 0xffffu, b = (hb >> (16 * w)) & 0xffffu;
            if (r[w] >= e && r[w] < e + a + b) {
                const bool second = r[w] >= e + a;
                bin[w] = 2 * tid + (second ? 1u : 0u);
                before[w] = second ? e + a : e;
            }
        }
        __syncthreads();
#pragma unroll
        for (int w = 0; w < 2; ++w) {
            r[w] -= before[w];
            const unsigned int off = bin[w] << sh[w], end = off + ((1u << sh[w]) - 1u);
            if (end < hi[w] - lo[w]) hi[w] = lo[w] + end;
            lo[w] += off;
        }
        __syncthreads();
    }
    for (int i = tid; i < kBins; i += 1024) ws->hist[i] = 0u;
    // a bound at the sample's end does not bound the image
    const unsigned int win_lo = r_lo == 0u && n > S ? 0u : lo[0], win_hi = r_hi == cnt - 1u && n > S ? kNone : lo[1];
    unsigned int inside = 0;
#pragma unroll
    for (int i = 0; i < V; ++i) inside += tid + 1024u * i < cnt && x[i] > win_lo && x[i] < win_hi ? 1u : 0u;
    inside = __reduce_add_sync(0xffffffffu, inside);
    if (lane == 0) scratch[warp] = inside;
    __syncthreads();
    if (tid < 32) inside = __reduce_add_sync(0xffffffffu, scratch[lane]);
    if (tid == 0) {
        DispCtrl c{};
        c.rank = rank;
        c.lo = win_lo;
        c.hi = win_hi;
        // the candidates to expect, with a quarter to spare (the sample's spacings vary by 5 to 10 %)
        c.fallback = 1.25 * inside / S * (double)n > (double)kCandCap;
        c.above = c.above_radix = kNone;
        if (n <= S) disp_hi(c, lo[0], lo[1], gamma, hi_out);
        ws->ctrl = c;
    }
}

// The collecting sweep: counts below / equal to the window's ends, the smallest element above it, and the
// elements strictly inside.  The common element costs three compares and a
// minimum; a warp enters the slow path when one of its 128 loaded elements lies in the window (40 % of the loads
// at 99.7 %), where ballots give each candidate its place in the warp's buffer, without atomics.  One
// reservation of the global list per block (and per full buffer).  The counters are summed over the block before
// the one atomic each: 9472 warps on one address cost more than 30 us.  Reads the image once; what it reads last
// stays in L2 for the writing sweep.
__global__ void __launch_bounds__(512) k_disp_collect(const float *v, long long n, DispWs *ws) {
    pdl_wait();
    __shared__ unsigned int buf_s[16][kWarpCand], sum_s[4][16], min_s[16];
    __shared__ unsigned long long base_s;
    DispCtrl &c = ws->ctrl;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned int *buf = buf_s[threadIdx.x >> 5];
    if (c.fallback) return;                                  // uniform over the grid
    const unsigned int lo = c.lo, hi = c.hi, width = hi - lo;
    unsigned int below = 0, n_lo = 0, n_hi = 0, nbuf = 0;    // the last three are the warp's
    unsigned int best = kNone;                               // min of b - (hi + 1): wraps past the rest for b <= hi
    auto write_out = [&](unsigned long long g) {
        for (unsigned int k = lane; k < nbuf; k += 32) {
            if (g + k < kCandCap) ws->list[g + k] = buf[k];
        }
    };
    auto flush = [&]() {
        __syncwarp();
        unsigned long long g = 0;
        if (lane == 0) g = atomicAdd(&c.cand, (unsigned long long)nbuf);
        write_out(__shfl_sync(0xffffffffu, g, 0));
        __syncwarp();
        nbuf = 0;
    };
    auto slow = [&](const unsigned int (&b)[4], const bool (&live)[4]) {
        if (nbuf > (unsigned)kWarpCand - 128u) flush();
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const unsigned int d = b[e] - lo;
            n_lo += __popc(__ballot_sync(0xffffffffu, live[e] && d == 0u));
            n_hi += __popc(__ballot_sync(0xffffffffu, live[e] && d == width && width));
            const bool in = live[e] && d != 0u && d < width;
            const unsigned int mk = __ballot_sync(0xffffffffu, in);
            if (in) buf[nbuf + __popc(mk & ((1u << lane) - 1u))] = b[e];
            nbuf += __popc(mk);
        }
    };
    auto take = [&](float4 q, bool any) {                    // warp-uniform call; any: this lane holds elements
        const unsigned int b[4] = {__float_as_uint(q.x), __float_as_uint(q.y), __float_as_uint(q.z), __float_as_uint(q.w)};
        const bool live[4] = {any, any, any, any};
        bool in = false;
        if (any) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                below += b[e] < lo ? 1u : 0u;
                best = min(best, b[e] - hi - 1u);
                in |= b[e] - lo <= width;
            }
        }
        if (__any_sync(0xffffffffu, in)) slow(b, live);
    };
    const long long n4 = n >> 2;
    const float4 *v4 = reinterpret_cast<const float4 *>(v);
    const long long stride = (long long)gridDim.x * blockDim.x;
    const long long i0 = blockIdx.x * (long long)blockDim.x + (threadIdx.x & ~31);     // the warp's first element
    long long i = i0;
    for (; i + 31 + 3 * stride < n4; i += 4 * stride) {      // four independent loads in flight
        float4 q[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) q[u] = v4[i + lane + u * stride];
#pragma unroll
        for (int u = 0; u < 4; ++u) take(q[u], true);
    }
    for (; i < n4; i += stride) {
        const bool any = i + lane < n4;
        take(any ? v4[i + lane] : make_float4(0.f, 0.f, 0.f, 0.f), any);
    }
    if (blockIdx.x == 0 && threadIdx.x < 32 && (n & 3)) {    // the last one to three elements
        const bool any = lane < (int)(n & 3);
        const unsigned int b[4] = {any ? __float_as_uint(v[4 * n4 + lane]) : 0u, 0u, 0u, 0u};
        const bool live[4] = {any, false, false, false};
        if (any) {
            below += b[0] < lo ? 1u : 0u;
            best = min(best, b[0] - hi - 1u);
        }
        slow(b, live);
    }
    below = __reduce_add_sync(0xffffffffu, below);
    best = __reduce_min_sync(0xffffffffu, best);
    if (lane == 0) {
        sum_s[0][warp] = below;
        sum_s[1][warp] = n_lo;
        sum_s[2][warp] = n_hi;
        sum_s[3][warp] = nbuf;
        min_s[warp] = best;
    }
    __syncthreads();
    if (threadIdx.x < 16) {                                  // warp 0, lanes 0..15: one warp's values each
        unsigned int t[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) t[k] = __reduce_add_sync(0xffffu, sum_s[k][lane]);
        const unsigned int bm = __reduce_min_sync(0xffffu, min_s[lane]);
        if (lane == 0) {
            if (t[3]) base_s = atomicAdd(&c.cand, (unsigned long long)t[3]);
            if (t[0]) atomicAdd(&c.below, (unsigned long long)t[0]);
            if (t[1]) atomicAdd(&c.n_lo, (unsigned long long)t[1]);
            if (t[2]) atomicAdd(&c.n_hi, (unsigned long long)t[2]);
            if (hi != kNone && bm <= kNone - 1u - hi) atomicMin(&c.above, bm + hi + 1u);
        }
    }
    __syncthreads();
    unsigned long long g = base_s;
    for (int w = 0; w < warp; ++w) g += sum_s[3][w];
    write_out(g);
}

// One cluster: s[k] and s[k + 1] from the window's counts and candidates; where the window missed, from the image, or the
// fallback flag.  Each CTA takes a share of
// the list (L2 resident: 1.1 MB at 8192^2), and every descent over 2048 bins of the current range adds up the
// CTAs' shared-memory histograms through distributed shared memory; three descents end at one value.  (A single
// block took 53 us for 275 000 candidates, bound by one SM's loads; a histogram in global memory, added to by the
// collecting sweep, cost that sweep 40 us where bright responses stretch the window and crowd its bins.)
__global__ void __cluster_dims__(kSelectCtas, 1, 1) __launch_bounds__(1024) k_disp_select(const float *v, long long n, DispWs *ws, int top_only,
                                                                                           float gamma, float *hi_out) {
    pdl_wait();
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    __shared__ unsigned int h[kBins], tot[kBins];
    __shared__ unsigned long long scratch[32], before;
    __shared__ unsigned int bin, next;
    DispCtrl &c = ws->ctrl;
    if (c.fallback) return;                                  // uniform over the cluster
    const int tid = threadIdx.x;
    const unsigned int r = cluster.block_rank();
    const unsigned long long r0 = c.rank - c.below;          // rank inside the window
    const unsigned long long in_end = c.n_lo + c.cand;
    const bool hit = c.rank >= c.below && r0 < in_end + c.n_hi && c.cand <= kCandCap;
    if (!hit && n > kSelectImage) {                          // uniform over the cluster
        if (r == 0 && tid == 0) c.fallback = 1;              // (the radix sweeps find their words zero)
        return;
    }
    // the elements to select from: the candidates, or the image where the window missed
    const unsigned int *src = hit ? ws->list : reinterpret_cast<const unsigned int *>(v);
    const unsigned int cand = (unsigned int)(hit ? c.cand : (unsigned long long)n);
    unsigned int lo = c.lo, hi = c.lo, rank = 0, cnt = 0;
    if (tid == 0) next = kNone;
    const bool inner = !hit || (r0 >= c.n_lo && r0 < in_end);
    auto each = [&](auto &&f) {                              // this CTA's candidates, eight loads in flight
        constexpr unsigned int ST = kSelectCtas * 1024;
        unsigned int i = r * 1024u + tid;
        for (; i + 7 * ST < cand; i += 8 * ST) {
            unsigned int x[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) x[u] = src[i + ST * u];
#pragma unroll
            for (int u = 0; u < 8; ++u) f(x[u]);
        }
        for (; i < cand; i += ST) f(src[i]);
    };
    if (inner) {
        rank = (unsigned int)(hit ? r0 - c.n_lo : c.rank);
        lo = hit ? c.lo : 0u;
        hi = hit ? c.hi : kNone;
        do {
            const int sh = bin_shift(hi - lo);
            for (int i = tid; i < kBins; i += 1024) h[i] = 0u;
            __syncthreads();
            each([&](unsigned int x) { if (x >= lo && x <= hi) atomicAdd(&h[(x - lo) >> sh], 1u); });
            cluster.sync();
            for (int i = tid; i < kBins; i += 1024) {
                unsigned int t = 0;
#pragma unroll
                for (int q = 0; q < kSelectCtas; ++q) t += cluster.map_shared_rank(h, q)[i];
                tot[i] = t;
            }
            cluster.sync();                                  // the histograms have been read
            find_bin(tot, rank, scratch, &bin, &before);
            const unsigned int off = bin << sh, end = off + ((1u << sh) - 1u);
            cnt = tot[bin];
            rank -= (unsigned int)before;
            if (end < hi - lo) hi = lo + end;
            lo += off;
            __syncthreads();
        } while (lo < hi);
    }
    // lo == s[k] where it is a candidate (cnt of them, rank: its place among them) or the window's lower end
    unsigned int up = kNone;                                 // the smallest candidate above it
    if (!hit || r0 < in_end) each([&](unsigned int x) { if (x > lo) up = min(up, x); });
    up = __reduce_min_sync(0xffffffffu, up);
    __syncthreads();
    if ((tid & 31) == 0) atomicMin(&next, up);
    cluster.sync();
    if (r == 0 && tid == 0) {
        unsigned int nx = kNone;
        for (int q = 0; q < kSelectCtas; ++q) nx = min(nx, *cluster.map_shared_rank(&next, q));
        const bool again = inner ? rank + 1 < cnt : r0 + 1 < c.n_lo;                     // s[k + 1] == s[k]
        unsigned int a = lo, b = again ? lo : nx != kNone || !hit ? nx : (c.n_hi ? c.hi : c.above);
        if (hit && r0 >= in_end) {
            a = c.hi;
            b = r0 + 1 < in_end + c.n_hi ? c.hi : c.above;
        }
        disp_hi(c, a, top_only ? a : b, gamma, hi_out);
    }
    cluster.sync();                                          // the peers' shared memory stays until it has been read
}

// The radix sweeps over the whole image, one launch each (bits 31..21, 20..10, 9..0 of the elements whose bits above equal
// the prefix).  The block that adds its histogram last picks the bin that holds the rank and clears the histogram for
// the next sweep.  The last sweep also keeps the smallest element above the prefix's range, so that s[k + 1] needs no
// sweep of its own.  Gated: launches that do nothing when the window held (the three cost 1.4 us at 4096^2 against one cooperative launch
// with grid barriers, but that one has to wait until every SM has room for it at once, behind another stream's
// frame as well, and a context that is limited to some of the SMs refuses it).
__global__ void __launch_bounds__(1024, 2) k_disp_radix(const float *v, long long n, DispWs *ws, int pass, int top_only,
                                                     float gamma, float *hi_out) {
    pdl_wait();
    DispCtrl &c = ws->ctrl;
    if (!c.fallback) return;                                 // uniform over the grid
    __shared__ unsigned int h[2 * kBins];                    // a histogram for each half of the block: fewer threads on one word
    __shared__ unsigned long long scratch[32], before;
    __shared__ unsigned int bin, nxt;
    __shared__ int mine;
    const int tid = threadIdx.x;
    const long long n4 = n >> 2;
    const float4 *v4 = reinterpret_cast<const float4 *>(v);
    const long long stride = (long long)gridDim.x * blockDim.x;
    const int shift = pass == 0 ? 21 : pass == 1 ? 10 : 0, width = pass == 2 ? 10 : 11, top = shift + width;
    const bool last = pass == 2;
    unsigned int *mine_h = h + (tid < 512 ? 0 : kBins);
    for (int i = tid; i < 2 * kBins; i += 1024) h[i] = 0u;
    __syncthreads();
    const unsigned int prefix = c.prefix;
    const unsigned int mask = (1u << width) - 1u;
    unsigned int best = kNone;
    auto add = [&](float x) {                                // (increments by one: equal words of a warp are counted together)
        const unsigned int b = __float_as_uint(x);
        if (top >= 32 || (b >> top) == prefix) atomicAdd(&mine_h[(b >> shift) & mask], 1u);
        else if (last && (b >> top) > prefix) best = min(best, b);
    };
    auto add4 = [&](float4 q) { add(q.x); add(q.y); add(q.z); add(q.w); };
    long long i = blockIdx.x * (long long)blockDim.x + tid;
    for (; i + 3 * stride < n4; i += 4 * stride) {           // four independent loads in flight
        float4 q[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) q[u] = __ldcs(v4 + i + u * stride);
#pragma unroll
        for (int u = 0; u < 4; ++u) add4(q[u]);
    }
    for (; i < n4; i += stride) add4(__ldcs(v4 + i));
    if (blockIdx.x == 0)
        for (long long k = 4 * n4 + tid; k < n; k += 1024) add(v[k]);
    __syncthreads();
    for (int k = tid; k < (1 << width); k += 1024) {
        const unsigned int t = h[k] + h[kBins + k];
        if (t) atomicAdd(&ws->hist[k], t);
    }
    best = __reduce_min_sync(0xffffffffu, best);
    if ((tid & 31) == 0 && best != kNone) atomicMin(&c.above_radix, best);
    __threadfence();
    __syncthreads();
    if (tid == 0) mine = atomicAdd(&c.ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!mine) return;
    __threadfence();
    for (int k = tid; k < kBins; k += 1024) {
        h[k] = __ldcg(&ws->hist[k]);
        ws->hist[k] = 0u;
    }
    if (tid == 0) nxt = kNone;
    const unsigned long long rank = c.rank;
    __syncthreads();
    find_bin(h, rank, scratch, &bin, &before);
    const unsigned int b = bin;
    if (last) {
        for (int k = tid; k < kBins; k += 1024)
            if ((unsigned)k > b && h[k]) atomicMin(&nxt, (unsigned)k);
        __syncthreads();
    }
    if (tid == 0) {
        const unsigned long long r = rank - before;
        c.rank = r;
        c.prefix = (prefix << width) | b;
        c.ticket = 0u;
        if (last) {
            const unsigned int a = (prefix << width) | b;
            const unsigned int up = nxt != kNone ? ((prefix << width) | nxt) : __ldcg(&c.above_radix);
            disp_hi(c, a, (top_only || r + 1 < h[b]) ? a : up, gamma, hi_out);
        }
    }
}

// data = uint8(clip(amp / h * 255, 0, 255)) (truncation toward zero; a NaN quotient gives 0)
__global__ void __launch_bounds__(256) k_disp_quant(const float *v, long long n, const DispWs *ws,
                                                    uint8_t *__restrict__ out) {
    pdl_wait();
    const float h = ws->ctrl.h;
    auto q8 = [&](float x) -> uint32_t {
        const float y = __fmul_rn(__fdiv_rn(x, h), 255.0f);
        const float c = fminf(fmaxf(y, 0.0f), 255.0f);     // NaN -> 0 (fmaxf returns the number)
        return (uint32_t)c;
    };
    // t = x (255 / h) is within 4 ulp (1e-4 below 256) of the two-step quotient y, so trunc(min(t, 255)) is the byte unless t
    // lies that close to one of the integers 1..255 (a byte that t < 1 - 2^-12 cannot leave is 0): those, and
    // anything that is not an ordinary number, take the exact steps.  The division costs a third of the sweep's time otherwise.
    const float s255 = 255.0f / h;
    const bool plain = s255 > 1e-30f && s255 < 1e30f;
    auto q84 = [&](float4 q) -> uint32_t {
        const float t[4] = {q.x * s255, q.y * s255, q.z * s255, q.w * s255};
        uint32_t r = 0;
        bool sure = plain;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float c = fminf(t[e], 255.5f);           // NaN -> 255.5, and not sure below
            const uint32_t k = (uint32_t)c;
            const float f = c - (float)k;
            sure = sure && t[e] >= 0.0f && f < 1.0f - 0x1p-12f && (f > 0x1p-12f || k == 0u);
            r |= k << (8 * e);
        }
        return sure ? r : q8(q.x) | (q8(q.y) << 8) | (q8(q.z) << 16) | (q8(q.w) << 24);
    };
    const long long n4 = n >> 2;
    const float4 *v4 = reinterpret_cast<const float4 *>(v);
    uint32_t *o4 = reinterpret_cast<uint32_t *>(out);
    const long long stride = (long long)gridDim.x * blockDim.x;
    // back to front: the sweep before this one left the end of the image in L2; four loads in flight
    long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    for (; r + 3 * stride < n4; r += 4 * stride) {
        float4 q[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) q[u] = __ldcs(v4 + (n4 - 1 - r - u * stride));
#pragma unroll
        for (int u = 0; u < 4; ++u)
            __stcs(o4 + (n4 - 1 - r - u * stride), q84(q[u]));
    }
    for (; r < n4; r += stride) {
        const float4 q = __ldcs(v4 + (n4 - 1 - r));
        o4[n4 - 1 - r] = q84(q);
    }
    if (blockIdx.x == 0)
        for (long long i = 4 * n4 + threadIdx.x; i < n; i += blockDim.x) out[i] = (uint8_t)q8(v[i]);
}

}  // namespace
}  // namespace pfa

extern "C" {

size_t pfa_display_workspace_bytes(void) { return sizeof(pfa::DispWs); }

pfa_status pfa_display_u8(const float *mag_dev, int64_t count, float percentile, void *workspace_dev, uint8_t *out_dev,
                          float *hi_dev, void *stream) {
    using namespace pfa;
    if (!mag_dev || !workspace_dev || !out_dev || count < 1) return PFA_ERR_BAD_ARG;
    if ((reinterpret_cast<uintptr_t>(mag_dev) & 15) || (reinterpret_cast<uintptr_t>(out_dev) & 3) ||
        (reinterpret_cast<uintptr_t>(workspace_dev) & 7))
        return PFA_ERR_BAD_ARG;
    if (!(percentile >= 0.0f && percentile <= 100.0f)) return PFA_ERR_BAD_ARG;
    // np.percentile's index arithmetic, float32 throughout (q = f32(pct) / f32(100), v = f32(n - 1) * q)
    volatile float q = percentile / 100.0f;
    volatile float vi = (float)(count - 1) * q;
    const float prev = floorf(vi);
    const bool top = vi >= (float)(count - 1);          // at or above the last index: the maximum
    const unsigned long long rank = top ? (unsigned long long)(count - 1) : (unsigned long long)prev;
    const float gamma = top ? 0.0f : (float)(vi - prev);
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    DispWs *ws = static_cast<DispWs *>(workspace_dev);
    int sms = 148;
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const bool large = count >= kLargeImage;
    const int S = large ? kSampleLarge : kSampleSmall;
    auto sample = large ? k_disp_sample<kSampleLarge / 1024> : k_disp_sample<kSampleSmall / 1024>;
    if (count <= S) {
        (void)launch(sample, 1, 1024, 0, st, mag_dev, count, ws, rank, (unsigned)rank, (unsigned)(top ? rank : rank + 1), gamma, hi_dev);
    } else {
        // sample ranks 6 standard deviations (of the binomial count) and a few elements around the image's rank
        const double p = (double)rank / (double)count, at = p * S;
        const double dr = 6.0 * std::sqrt((double)S * p * (1.0 - p)) + 8.0;
        const unsigned r_lo = (unsigned)std::max(0.0, std::floor(at - dr));
        const unsigned r_hi = (unsigned)std::min((double)(S - 1), std::ceil(at + dr));
        (void)launch(sample, 1, 1024, 0, st, mag_dev, count, ws, rank, r_lo, r_hi, gamma, hi_dev);
        (void)launch(k_disp_collect, sms * 4, 512, 0, st, mag_dev, count, ws);
        (void)launch(k_disp_select, kSelectCtas, 1024, 0, st, mag_dev, count, ws, top ? 1 : 0, gamma, hi_dev);
        for (int pass = 0; pass < 3 && count > kSelectImage; ++pass)
            (void)launch(k_disp_radix, sms * 2, 1024, 0, st, mag_dev, count, ws, pass, top ? 1 : 0, gamma, hi_dev);
    }
    (void)launch(k_disp_quant, sms * 8, 256, 0, st, mag_dev, count, ws, out_dev);
    return cudaGetLastError() == cudaSuccess ? PFA_OK : PFA_ERR_CUDA;
}

}  // extern "C"
