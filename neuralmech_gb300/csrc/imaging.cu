// Total focusing method on full-matrix-capture traces (sm_103a): the consumer
// of the wave path's traces in projects/18_fwi/2D_tfm.py.
//
// analytic_kernel: the analytic signal h = x + i H[x] of every trace, with H the
// periodic discrete Hilbert transform. The transform is a circular
// convolution with the kernel g (g = ifft(-i sign(k)) with the Nyquist bin
// zeroed for even N, the transform scipy.signal.hilbert applies through its
// FFT). One CTA per trace: the trace and two periods of g sit in shared
// memory, and each thread accumulates 8 output samples over the N inputs
// (O(N^2) per trace) from registers. Bound by the FP32 pipe: 1024 traces of 1500
// samples take 2.4 G fused multiply-adds, 61 us at the chip's rate; 409 -> 160 us a call
// (the one-output form read two shared-memory words per multiply-add).
//
// tfm_kernel: delay and sum, one thread per pixel:
//   image[p] = | sum_{e <= r} w_er h_er((t0 + tau_e(p) + tau_r(p)) / dt) |,
// tau_e = |p - x_e| / c, w_er = 2 for r > e (reciprocity), linear interpolation
// in time, pairs past the end of the trace skipped
// (projects/18_fwi/tfm.py:12-36). Without reciprocity every ordered pair
// counts once. A pixel's times of flight sit in a shared-memory column of
// its own (any element count up to 256). The complex traces are read through
// the read-only path; they are L2-resident for the array sizes of the
// reference drivers.
#include <algorithm>
#include <atomic>

#include "common.cuh"
#include "internal.h"

namespace wfd {
namespace {

// Outputs of a thread: 8 consecutive samples n = 8 t + i, against blocks of 8 inputs
// k = 8 b + j. The 15 values g[n - k] of a block are two aligned groups of 8, A below
// and B from q0 on, of the staged kernel P; the next block's B is this block's A, so a
// block costs two 16-byte loads of g per thread and two broadcast ones of x for 64
// fused multiply-adds. One output's sum runs over k in ascending order.
//   P[q] = g[(q + r - 8) mod nt] for 0 <= q + r - 8 < 2 nt (else 0), r = nt mod 8, so that
//   g[(n - k) mod nt] = P[q0 + i - j], q0 = 8 (t - b) + nt - r + 8.
// P is stored with one 16-byte unit of padding per 8 (pad = 3), which makes the lanes'
// loads, 32 bytes apart, free of bank conflicts; very long traces that leave no room for
// the padding (pad = 31) go without.
__global__ void analytic_kernel(const float* __restrict__ x, const float* __restrict__ g, int nt, int pad,
                                float2* __restrict__ h) {
    extern __shared__ __align__(16) float sm[];
    const int nb = (nt + 7) / 8, r = nt & 7;
    float* xs = sm;            // [8 nb], zero past nt
    float* P = sm + 8 * nb;    // [2 nt + 24] in units of 4, padded
    auto at = [&](int q) { const int u = q >> 2; return ((u + (u >> pad)) << 2) + (q & 3); };
    const float* xt = x + blockIdx.x * (long long)nt;
    for (int i = threadIdx.x; i < 8 * nb; i += blockDim.x) xs[i] = i < nt ? xt[i] : 0.f;
    for (int q = threadIdx.x; q < 2 * nt + 24; q += blockDim.x) {
        int m = q + r - 8;
        const bool in = m >= 0 && m < 2 * nt;
        if (m >= nt) m -= nt;
        P[at(q)] = in ? g[m] : 0.f;
    }
    __syncthreads();
    auto load8 = [&](int q, float (&v)[8]) {  // q a multiple of 8
        const float4 a = *reinterpret_cast<const float4*>(P + at(q)), b = *reinterpret_cast<const float4*>(P + at(q + 4));
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
        v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    };
    float2* ht = h + blockIdx.x * (long long)nt;
    for (int t = threadIdx.x; t < nb; t += blockDim.x) {
        float acc[8], A[8], B[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] = 0.f;
        int q = 8 * t + nt - r + 8;
        load8(q, B);
        for (int b = 0; b < nb; ++b) {
            q -= 8;
            load8(q, A);
            const float4 x0 = *reinterpret_cast<const float4*>(xs + 8 * b), x1 = *reinterpret_cast<const float4*>(xs + 8 * b + 4);
            const float xk[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
#pragma unroll
            for (int j = 0; j < 8; ++j)
#pragma unroll
                for (int i = 0; i < 8; ++i) acc[i] = fmaf(xk[j], i >= j ? B[i >= j ? i - j : 0] : A[i < j ? 8 + i - j : 0], acc[i]);
#pragma unroll
            for (int i = 0; i < 8; ++i) B[i] = A[i];
        }
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (8 * t + i < nt) ht[8 * t + i] = make_float2(xs[8 * t + i], acc[i]);
    }
}

constexpr int TFM_THREADS = 128;
constexpr int TFM_MAX_ELEMENTS = 256;  // (wfd_tfm checks)
// How a time becomes a sample index (see tfm_index).
enum TfmIndex : int { TFM_LATE, TFM_EARLY, TFM_ANY };
constexpr int TFM_PAIRS = 4;
template <int N>
struct Count {
    static constexpr int value = N;
};
constexpr int TFM_COLS = 16, TFM_ROWS = TFM_THREADS / TFM_COLS;  // pixels of a CTA on a grid of pixels

// The length of the rows that the pixel list is made of: the first pixel after which
// the coordinate that all pixels before it share changes; P where the list is none of a
// grid's (or its rows are longer than 4096 pixels), or where blocks would leave more than a
// lane in 32 idle, which costs more than they give. us a call, blocks / list, 32 elements, 512^2
// pixels in rows of 2 1344 / 272, 17 580 / 385, 28 440 / 383, 200 299 / 278, 32 368 / 393,
// 127 274 / 288, 512 247 / 260. Called by a whole CTA.
__device__ int row_length(const float* xp, const float* yp, int P) {
    __shared__ int fx, fy;
    if (threadIdx.x == 0) fx = fy = P;
    __syncthreads();
    const float x0 = xp[0], y0 = yp[0];
    for (int i = threadIdx.x + 1; i < min(P, 4097) && (i <= fx || i <= fy); i += TFM_THREADS) {
        if (xp[i] != x0) atomicMin(&fx, i);
        if (yp[i] != y0) atomicMin(&fy, i);
    }
    __syncthreads();
    const int w = max(fx, fy);
    const int idle = (w + TFM_COLS - 1) / TFM_COLS * TFM_COLS - w;  // lanes of a row of blocks
    return w < 4097 && w >= TFM_COLS && 32 * idle <= w ? w : P;
}

// Bound by the latency of the gathers (87% of their sectors hit L1) and the instructions of a
// pair: so TFM_PAIRS pairs have their samples in flight at once, the sample index takes no
// integer conversion where t + 2^23 holds it, and no test for a time before the first sample
// unless t0 < 0 (INDEX, see tfm_index), half of an SM's on-chip memory is left to L1 (see the launch), and where the list is a
// grid's, a CTA takes a block of 16 x 8 pixels, whose samples of a trace lie closer together
// than a row's. 32 elements, 1500 samples, 512^2 pixels: 340 -> 250 us a call (one pair at a
// time, 128 pixels of a row, all of the memory to tau).
template <TfmIndex INDEX>
__global__ void __launch_bounds__(TFM_THREADS)
    tfm_kernel(const float2* __restrict__ h, int E, const float* __restrict__ xe,
               const float* __restrict__ ye, int nt, float inv_dt, float t0, float inv_c,
               const float* __restrict__ xp, const float* __restrict__ yp, int P, int reciprocity,
               float* __restrict__ image) {
    extern __shared__ float tau_s[];  // [E][TFM_THREADS]: the pixel's times of flight
    const int W = row_length(xp, yp, P), H = (P + W - 1) / W;
    const bool grid = W < P;
    const int across = grid ? (W + TFM_COLS - 1) / TFM_COLS : 1;
    const int blocks = grid ? across * ((H + TFM_ROWS - 1) / TFM_ROWS) : (P + TFM_THREADS - 1) / TFM_THREADS;
    const float last = float(nt - 1);
    float* tau = tau_s + threadIdx.x;
    for (int blk = blockIdx.x; blk < blocks; blk += gridDim.x) {
        int p = blk * TFM_THREADS + threadIdx.x;
        if (grid) {
            const int c = blk % across * TFM_COLS + threadIdx.x % TFM_COLS;
            const long long q = (long long)(blk / across * TFM_ROWS + threadIdx.x / TFM_COLS) * W + c;
            p = c < W && q < P ? int(q) : P;
        }
        if (p >= P) continue;  // no barrier below: each thread reads only its own column
        const float px = xp[p], py = yp[p];
        float all = 0.f;
        for (int e = 0; e < E; ++e) {
            const float f = hypotf(px - __ldg(xe + e), py - __ldg(ye + e)) * inv_c;
            tau[e * TFM_THREADS] = f;
            all = fmaxf(all, f != f ? __int_as_float(0x7f800000) : 0.f);
        }
        float sx = 0.f, sy = 0.f;
        for (int e = 0; e < E; ++e) {
            const float te = t0 + tau[e * TFM_THREADS];
            const int r0 = reciprocity ? e : 0;
            const float2* hr = h + ((long long)e * E + r0) * nt;
            const float* tr = tau + r0 * TFM_THREADS;
            // N pairs at a time, all their samples in flight before the first is used
            auto pairs = [&](auto n, float scale) {
                constexpr int N = decltype(n)::value;
                float w[N];
                float2 a[N], c[N];
                bool in[N];
#pragma unroll
                for (int i = 0; i < N; ++i) {
                    const float t = (te + tr[i * TFM_THREADS]) * inv_dt;
                    int k;
                    float kf;
                    if (INDEX == TFM_ANY) {
                        k = int(t);
                        kf = float(k);
                        in[i] = k < nt - 1;
                    } else {
                        in[i] = t < last;
                        // int(t) and its float without conversions: t + 2^23 rounded down holds floor(t)
                        // in its low bits (a time before the first sample truncates towards 0 instead)
                        const float b = __fadd_rd(t, 8388608.f);
                        k = __float_as_int(b) - 0x4B000000;
                        kf = b - 8388608.f;
                        if (INDEX == TFM_EARLY && t < 0.f) {
                            k = int(t);
                            kf = float(k);
                        }
                    }
                    w[i] = (t - kf) * scale;
                    const float2* hp = hr + (in[i] ? k : 0);
                    asm volatile("ld.global.nc.v2.f32 {%0, %1}, [%2];" : "=f"(a[i].x), "=f"(a[i].y) : "l"(hp));
                    asm volatile("ld.global.nc.v2.f32 {%0, %1}, [%2];" : "=f"(c[i].x), "=f"(c[i].y) : "l"(hp + 1));
                    hr += nt;
                }
#pragma unroll
                for (int i = 0; i < N; ++i) {
                    const float v = scale - w[i];
                    float nx = sx, ny = sy;
                    nx += v * a[i].x + w[i] * c[i].x;
                    ny += v * a[i].y + w[i] * c[i].y;
                    sx = in[i] ? nx : sx;
                    sy = in[i] ? ny : sy;
                }
                tr += N * TFM_THREADS;
            };
            int r = r0;
            if (reciprocity) {
                pairs(Count<1>{}, 1.f);
                ++r;
            }
            const float scale = reciprocity ? 2.f : 1.f;
            for (; r + TFM_PAIRS <= E; r += TFM_PAIRS) pairs(Count<TFM_PAIRS>{}, scale);
            for (; r < E; ++r) pairs(Count<1>{}, scale);
        }
        // (a pixel or an element that is not a number leaves no image)
        image[p] = all > 0.f ? __int_as_float(0x7fffffff) : hypotf(sx, sy);
    }
}

}  // namespace

cudaError_t launch_analytic(const float* traces, long long ntr, int nt, const float* g, float2* h,
                            cudaStream_t s) {
    const size_t xs = (size_t)((nt + 7) / 8) * 8, P = (size_t)2 * nt + 24;
    int pad = 3;
    size_t smem = (xs + P + P / 8 + 8) * sizeof(float);
    if (smem > 227 * 1024) {
        pad = 31;
        smem = (xs + P + 8) * sizeof(float);
    }
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(analytic_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)smem);
        if (e != cudaSuccess) return e;
    }
    const int threads = std::min(256, ((nt + 7) / 8 + 31) / 32 * 32);
    analytic_kernel<<<(unsigned)ntr, threads, smem, s>>>(traces, g, nt, pad, h);
    count_launch();
    return cudaGetLastError();
}

// The bits of t + 2^23 count samples while t < 2^23 (from there on floats lie 2 apart and
// more): so for traces of up to 2^23 samples, and times that are numbers, which they are
// unless t0 is none, or 1 / dt is 0 or infinite. The rest takes int(t) (TFM_ANY), in which a
// time that is no number reads sample 0 and leaves no image.
static TfmIndex tfm_index(int nt, float inv_dt, float t0) {
    if (nt > (1 << 23) || !(inv_dt > 0.f && inv_dt <= 3.402823466e38f)) return TFM_ANY;
    return t0 >= 0.f ? TFM_LATE : t0 < 0.f ? TFM_EARLY : TFM_ANY;
}

// Share of an SM's on-chip memory for tau. The gathers need L1 more than they need the last
// CTAs, so half, unless that leaves only three CTAs where a little more gives four, or one where
// all of it gives two. us a call, half / the share taken, pixels of a grid (scattered ones):
// 64 elements, 65536 pixels 526 / 329 (772 / 515); 56, 262144 776 / 627 (1387 / 1260); 200, 65536
// 8384 / 4325 (17198 / 8982). 32, 262144 with half / three quarters 242 / 242 (546 / 654); 96, 262144
// with half / all 3430 / 1998 (4206 / 6692).
static int tfm_carveout(int E) { return E > 128 ? 100 : E > 48 && E <= 64 ? 60 : 50; }

cudaError_t launch_tfm(const float2* h, int E, const float* xe, const float* ye, int nt, float dt,
                       float t0, float c, const float* xp, const float* yp, int P, int reciprocity,
                       float* image, cudaStream_t s) {
    const size_t smem = (size_t)E * TFM_THREADS * sizeof(float);
    const TfmIndex index = tfm_index(nt, 1.f / dt, t0);
    const auto kernel = index == TFM_LATE    ? tfm_kernel<TFM_LATE>
                        : index == TFM_EARLY ? tfm_kernel<TFM_EARLY>
                                             : tfm_kernel<TFM_ANY>;
    // What the launch wants of the kernel; asked for when it is another than the last launch's
    // on the device (two calls of the runtime are 5% of a small image's). The limit of shared
    // memory is the one for the most elements, whatever this call has: with row_length's two
    // words 48 KB of tau, 96 elements, are past the default one too.
    static std::atomic<int> set[3][64];
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const int carveout = tfm_carveout(E);
    if (set[index][dev & 63].load(std::memory_order_relaxed) != carveout) {
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 int(TFM_MAX_ELEMENTS * TFM_THREADS * sizeof(float)));
        if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, carveout);
        if (e != cudaSuccess) return e;
        set[index][dev & 63].store(carveout, std::memory_order_relaxed);
    }
    // (blocks at the edges of a grid of pixels are partly empty: a CTA takes another one)
    kernel<<<(P + TFM_THREADS - 1) / TFM_THREADS, TFM_THREADS, smem, s>>>(
        h, E, xe, ye, nt, 1.f / dt, t0, 1.f / c, xp, yp, P, reciprocity, image);
    count_launch();
    return cudaGetLastError();
}

}  // namespace wfd
