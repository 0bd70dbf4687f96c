// Drop-ins for the reference's order-2 step kernels that store the field in
// reduced precision or in 1D (sm_103a): the same arguments, cells and storage
// formats as
//   mixed_step  (projects/18_simple_wave_fd/step2D_wave.cu:85-124): FP16 storage,
//   scaled_step (step2D_wave.cu:128-183): int16 with one FP32 scale per block of
//               32 values along a row, scale = block max / 32767,
//   step1D      (step1D_wave.cu:4-17): the 1D 3-point step.
// The arithmetic of every cell is the reference's expression in its operation
// order, in explicitly rounded IEEE operations (no contraction into FMAs, IEEE
// division), so the results equal a plain IEEE evaluation of the reference
// source value for value.
//
// The reference's row index i runs with dx and its column index j (fastest,
// M of them, padded to M_padded) with dy. Rows 0 and N - 1 and columns 0 and
// M - 1 are the fixed boundary.
#include <algorithm>

#include "../../include/wavefd.h"
#include "common.cuh"
#include "internal.h"

namespace wfd {
namespace {

// u2 = -u0 + 2 u1 + k (lap_i / (dx dx) + lap_j / (dy dy)), k = dt dt c c, with
// lap = (a - 2 c) + b, evaluated left to right as the reference writes it.
__device__ __forceinline__ float update2d(float u0, float u1, float il, float ir, float jl, float jr,
                                          float k, float dx2, float dy2) {
    const float two_c = __fmul_rn(2.f, u1);
    const float li = __fadd_rn(__fsub_rn(il, two_c), ir);
    const float lj = __fadd_rn(__fsub_rn(jl, two_c), jr);
    const float lap = __fadd_rn(__fdiv_rn(li, dx2), __fdiv_rn(lj, dy2));
    return __fadd_rn(__fadd_rn(-u0, two_c), __fmul_rn(k, lap));
}

// 1D: one thread per cell of 0 < i < N - 1.
__global__ void step1d_kernel(const float* __restrict__ u0, const float* __restrict__ u1,
                              float* __restrict__ u2, float k, float dx2, int N) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i <= 0 || i >= N - 1) return;
    const float c = u1[i];
    const float lap = __fdiv_rn(__fadd_rn(__fsub_rn(u1[i - 1], __fmul_rn(2.f, c)), u1[i + 1]), dx2);
    u2[i] = __fadd_rn(__fadd_rn(-u0[i], __fmul_rn(2.f, c)), __fmul_rn(k, lap));
}

// FP32 storage with any row stride (padded_step / shared_step with M_padded,
// basic_step / coalesced_step with M_padded = M): a thread owns 4 consecutive
// cells j .. j + 3 of row i, read and written as scalars (rows need not be
// 16-byte aligned).
__global__ void exact_kernel(const float* __restrict__ u0, const float* __restrict__ u1,
                             float* __restrict__ u2, float k, float dx2, float dy2, int N, int M, int Mp) {
    const int j = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
    const int i = blockIdx.y * blockDim.y + threadIdx.y;
    if (i <= 0 || i >= N - 1 || j >= M - 1) return;
    const size_t c = (size_t)i * Mp + j;
    float w[6];  // u1 at j - 1 .. j + 4 of row i
#pragma unroll
    for (int e = 0; e < 6; ++e) w[e] = (j - 1 + e >= 0 && j - 1 + e < M) ? u1[c - 1 + e] : 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const int je = j + e;
        if (je == 0 || je >= M - 1) continue;  // the boundary columns (and beyond) stay untouched
        u2[c + e] = update2d(u0[c + e], w[e + 1], u1[c + e - Mp], u1[c + e + Mp], w[e], w[e + 2], k, dx2, dy2);
    }
}

// FP16 storage: a thread owns the pair (j, j + 1), j even, of row i, loaded and
// stored as one __half2.
__global__ void mixed_kernel(const __half* __restrict__ u0, const __half* __restrict__ u1,
                             __half* __restrict__ u2, float k, float dx2, float dy2, int N, int M,
                             int Mp) {
    const int j = 2 * (blockIdx.x * blockDim.x + threadIdx.x);
    const int i = blockIdx.y * blockDim.y + threadIdx.y;
    if (i <= 0 || i >= N - 1 || j >= M) return;
    const size_t c = (size_t)i * Mp + j;
    const float2 a = __half22float2(*reinterpret_cast<const __half2*>(u0 + c));
    const float2 b = __half22float2(*reinterpret_cast<const __half2*>(u1 + c));
    const float2 up = __half22float2(*reinterpret_cast<const __half2*>(u1 + c - Mp));
    const float2 dn = __half22float2(*reinterpret_cast<const __half2*>(u1 + c + Mp));
    const float left = j > 0 ? __half2float(u1[c - 1]) : 0.f;
    const float right = __half2float(u1[c + 2]);
    const float v0 = update2d(a.x, b.x, up.x, dn.x, left, b.y, k, dx2, dy2);
    const float v1 = update2d(a.y, b.y, up.y, dn.y, b.x, right, k, dx2, dy2);
    if (j > 0 && j + 1 < M - 1) {
        *reinterpret_cast<__half2*>(u2 + c) = __floats2half2_rn(v0, v1);
    } else {
        if (j > 0 && j < M - 1) u2[c] = __float2half_rn(v0);
        if (j + 1 < M - 1) u2[c + 1] = __float2half_rn(v1);
    }
}

// FP16 storage with pre-divided weights (the mixed_step update within FP32
// rounding, as the reference's --use_fast_math build computes it): a thread
// owns 8 consecutive values j .. j + 7 (j a multiple of 8) of row i, loaded
// and stored as 16 bytes; the left and right neighbours of the octet are two
// scalar loads. u2 = (2u - u0) + cx (u_{i-1} - 2u + u_{i+1}) + cy (u_{j-1} -
// 2u + u_{j+1}), cx = k / dx^2, cy = k / dy^2, rounded to FP16 once.
__global__ void mixed_fast_kernel(const __half* __restrict__ u0, const __half* __restrict__ u1,
                                  __half* __restrict__ u2, float cx, float cy, int N, int M, int Mp) {
    const int j = 8 * (blockIdx.x * blockDim.x + threadIdx.x);
    const int i = blockIdx.y * blockDim.y + threadIdx.y;
    if (i <= 0 || i >= N - 1 || j >= M - 1) return;
    const size_t c = (size_t)i * Mp + j;
    const uint4 ra = *reinterpret_cast<const uint4*>(u0 + c);
    const uint4 rb = *reinterpret_cast<const uint4*>(u1 + c);
    const uint4 ru = *reinterpret_cast<const uint4*>(u1 + c - Mp);
    const uint4 rd = *reinterpret_cast<const uint4*>(u1 + c + Mp);
    float w[10];  // u1 at j - 1 .. j + 8 of row i
    w[0] = j > 0 ? __half2float(u1[c - 1]) : 0.f;
    w[9] = j + 8 < Mp ? __half2float(u1[c + 8]) : 0.f;  // (row i + 1 starts after the padding)
    const __half2* hb = reinterpret_cast<const __half2*>(&rb);
    const __half2* ha = reinterpret_cast<const __half2*>(&ra);
    const __half2* hu = reinterpret_cast<const __half2*>(&ru);
    const __half2* hd = reinterpret_cast<const __half2*>(&rd);
    float a[8], up[8], dn[8];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const float2 vb = __half22float2(hb[q]), va = __half22float2(ha[q]);
        const float2 vu = __half22float2(hu[q]), vd = __half22float2(hd[q]);
        w[1 + 2 * q] = vb.x;
        w[2 + 2 * q] = vb.y;
        a[2 * q] = va.x;
        a[2 * q + 1] = va.y;
        up[2 * q] = vu.x;
        up[2 * q + 1] = vu.y;
        dn[2 * q] = vd.x;
        dn[2 * q + 1] = vd.y;
    }
    float v[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const float two_c = 2.f * w[e + 1];
        v[e] = fmaf(cx, (up[e] - two_c) + dn[e], fmaf(cy, (w[e] - two_c) + w[e + 2], two_c - a[e]));
    }
    if (j > 0 && j + 7 < M - 1) {
        uint4 o;
        __half2* ho = reinterpret_cast<__half2*>(&o);
#pragma unroll
        for (int q = 0; q < 4; ++q) ho[q] = __floats2half2_rn(v[2 * q], v[2 * q + 1]);
        *reinterpret_cast<uint4*>(u2 + c) = o;
    } else {
#pragma unroll
        for (int e = 0; e < 8; ++e)
            if (j + e > 0 && j + e < M - 1) u2[c + e] = __float2half_rn(v[e]);
    }
}

// Block-scaled int16: a thread owns 4 values (j .. j + 3, j a multiple of 4) of
// row i; the 8 lanes of an aligned lane octet hold one 32-value block and
// share its scale. Rows of the warp: a warp covers 128 columns of one row.
__global__ void scaled_kernel(const short* __restrict__ q0, const float* __restrict__ s0,
                              const short* __restrict__ q1, const float* __restrict__ s1,
                              short* __restrict__ q2, float* __restrict__ s2, float k, float dx2,
                              float dy2, int N, int M, int Mp) {
    const int j = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
    const int i = blockIdx.y * blockDim.y + threadIdx.y;
    if (i <= 0 || i >= N - 1) return;  // whole warps: blockDim.x is a multiple of 32
    const bool live = j < Mp;           // (Mp % 64 == 0: a lane octet is all live or all not)
    const int S = Mp / 32;              // blocks per row
    const size_t c = (size_t)i * Mp + j;
    const size_t b = (size_t)i * S + j / 32;
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    if (live) {
        const short4 p0 = *reinterpret_cast<const short4*>(q0 + c);
        const short4 p1 = *reinterpret_cast<const short4*>(q1 + c);
        const short4 pu = *reinterpret_cast<const short4*>(q1 + c - Mp);
        const short4 pd = *reinterpret_cast<const short4*>(q1 + c + Mp);
        const float a0 = s0[b], a1 = s1[b], au = s1[b - S], ad = s1[b + S];
        const float u0v[4] = {a0 * p0.x, a0 * p0.y, a0 * p0.z, a0 * p0.w};
        const float u1v[4] = {a1 * p1.x, a1 * p1.y, a1 * p1.z, a1 * p1.w};
        const float uu[4] = {au * pu.x, au * pu.y, au * pu.z, au * pu.w};
        const float ud[4] = {ad * pd.x, ad * pd.y, ad * pd.z, ad * pd.w};
        // the neighbours j - 1 and j + 4, each decoded with its own block's scale
        const float left = j > 0 ? s1[(size_t)i * S + (j - 1) / 32] * q1[c - 1] : 0.f;
        const float right = j + 4 < Mp ? s1[(size_t)i * S + (j + 4) / 32] * q1[c + 4] : 0.f;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float jl = e > 0 ? u1v[e - 1] : left;
            const float jr = e < 3 ? u1v[e + 1] : right;
            const int je = j + e;
            v[e] = (je == 0 || je >= M - 1) ? 0.f  // boundary and padding stay zero
                                            : update2d(u0v[e], u1v[e], uu[e], ud[e], jl, jr, k, dx2, dy2);
        }
    }
    // encode: the largest magnitude of the block sets its scale
    float m = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));
#pragma unroll
    for (int o = 1; o < 8; o *= 2) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (!live) return;
    const float inv = m > 0.f ? __fdiv_rn(32767.f, m) : 0.f;
    *reinterpret_cast<short4*>(q2 + c) =
        make_short4(short(__float2int_rn(v[0] * inv)), short(__float2int_rn(v[1] * inv)),
                    short(__float2int_rn(v[2] * inv)), short(__float2int_rn(v[3] * inv)));
    if ((threadIdx.x & 7) == 0) s2[b] = __fdiv_rn(m, 32767.f);
}

float kcoef(float c, float dt) { return dt * dt * c * c; }  // as the reference: ((dt dt) c) c

// Eight steps per launch (temporal_step): a CTA stages both levels of a
// 160 x 48 window (a 144 x 32 output tile plus an 8-cell halo on every side)
// by TMA, advances them in shared memory, and writes the tile of both final
// levels. The cells a step can update shrink by one per step from the window
// edges (the halo is the step count); global boundary cells and cells outside
// the grid are never updated, exactly as eight padded_step launches.
constexpr int TT_TX = 144, TT_TZ = 32, TT_H = 8, TT_STEPS = 8;
constexpr int TT_W = TT_TX + 2 * TT_H;   // 160 staged columns (40 float4)
constexpr int TT_WZ = TT_TZ + 2 * TT_H;  // 48 staged rows
constexpr int TT_THREADS = 320;  // 8 rows x 40 float4 columns per pass
constexpr int TT_PASSES = TT_WZ / 8;  // 6 row passes per step
constexpr int TT_LEVEL = TT_WZ * TT_W * 4;  // bytes of one staged level
constexpr int TT_BYTES = 2 * TT_LEVEL + 16 + 128;

__global__ void __launch_bounds__(TT_THREADS)
    temporal_kernel(const __grid_constant__ CUtensorMap map_u0, const __grid_constant__ CUtensorMap map_u1,
                    float* __restrict__ v0, float* __restrict__ v1, float k, float dx2, float dy2, int N,
                    int M, int Mp) {
    extern __shared__ unsigned char smem_raw[];
    float* base = reinterpret_cast<float*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
    float* lev[2] = {base, base + TT_WZ * TT_W};
    uint64_t* bar = reinterpret_cast<uint64_t*>(base + 2 * TT_WZ * TT_W);
    const int tid = threadIdx.x;
    const int j0 = blockIdx.x * TT_TX - TT_H, i0 = blockIdx.y * TT_TZ - TT_H;  // window origin

    if (tid == 0) {
        mbar_init(bar, 1);
        fence_mbar_init();
    }
    __syncthreads();  // no thread polls the barrier before it is initialised
    grid_dependency_wait();
    if (tid == 0) {
        mbar_arrive_expect_tx(bar, 2u * TT_LEVEL);
        // (the maps are rank 3: x, rows, shot; one shot here)
        tma_load_3d(lev[0], &map_u0, j0, i0, 0, bar);  // cells outside the grid arrive as 0
        tma_load_3d(lev[1], &map_u1, j0, i0, 0, bar);
        launch_dependents();
    }
    mbar_wait(bar, 0);  // bounded; every thread goes on to the same barriers either way

    // a thread owns the float4 column tj of rows r0, r0 + 8, ..., r0 + 40
    const int tj = 4 * (tid % (TT_W / 4)), r0 = tid / (TT_W / 4);
    for (int st = 0; st < TT_STEPS; ++st) {
        float* old = lev[st & 1];              // u_{n-1}, overwritten by u_{n+1}
        const float* cur = lev[1 - (st & 1)];  // u_n
#pragma unroll 3
        for (int ps = 0; ps < TT_PASSES; ++ps) {
            const int ti = r0 + 8 * ps;
            const int i = i0 + ti;
            if (ti <= st || ti >= TT_WZ - 1 - st || i <= 0 || i >= N - 1) continue;
            const float* c = cur + ti * TT_W + tj;
            const float4 cv = *reinterpret_cast<const float4*>(c);
            const float4 up = *reinterpret_cast<const float4*>(c - TT_W);
            const float4 dn = *reinterpret_cast<const float4*>(c + TT_W);
            const float left = tj > 0 ? c[-1] : 0.f, right = tj + 4 < TT_W ? c[4] : 0.f;
            float4 ov = *reinterpret_cast<const float4*>(old + ti * TT_W + tj);
            const float cc[6] = {left, cv.x, cv.y, cv.z, cv.w, right};
            const float uu[4] = {up.x, up.y, up.z, up.w}, dd[4] = {dn.x, dn.y, dn.z, dn.w};
            float o[4] = {ov.x, ov.y, ov.z, ov.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int te = tj + e, j = j0 + te;
                if (te > st && te < TT_W - 1 - st && j > 0 && j < M - 1)
                    o[e] = update2d(o[e], cc[e + 1], uu[e], dd[e], cc[e], cc[e + 2], k, dx2, dy2);
            }
            *reinterpret_cast<float4*>(old + ti * TT_W + tj) = make_float4(o[0], o[1], o[2], o[3]);
        }
        __syncthreads();
    }

    // after the eight steps lev[0] holds u_{n+7} and lev[1] u_{n+8}
    for (int g = tid; g < TT_TZ * (TT_TX / 4); g += TT_THREADS) {
        const int r = g / (TT_TX / 4), q = 4 * (g - r * (TT_TX / 4));
        const int i = i0 + TT_H + r, j = j0 + TT_H + q;
        if (i >= N || j >= M) continue;
        const float* a = lev[0] + (TT_H + r) * TT_W + TT_H + q;
        const float* b = lev[1] + (TT_H + r) * TT_W + TT_H + q;
        const size_t o = (size_t)i * Mp + j;
        if (j + 3 < M) {
            *reinterpret_cast<float4*>(v0 + o) = *reinterpret_cast<const float4*>(a);
            *reinterpret_cast<float4*>(v1 + o) = *reinterpret_cast<const float4*>(b);
        } else {
            for (int e = 0; j + e < M; ++e) {
                v0[o + e] = a[e];
                v1[o + e] = b[e];
            }
        }
    }
}

// Eight steps per launch as a stream of rows (temporal_step's arguments and results,
// pre-divided weights and fused multiply-adds).
//
// A warp marches down a strip of 128 columns, 4 per lane, and carries all eight steps
// along: at row t it takes u_n there and u_{n-1}, forms u_{n+1} of row t - 1, from that
// u_{n+2} of row t - 2, and so on to u_{n+8} of row t - 8. Per step it keeps the row
// above (prev) and the two parts of the next row's result that do not need the row below:
//   u = Q + cx (S + v),                                           (row t - s - 1 done)
//   Q = (2 v - old) + cy ((l - 2 v) + r),  S = prev - 2 v,        (row t - s begun)
// with old the level two before at row t - s, which is the prev that the step before has
// just replaced. The neighbours l and r of a lane's 4 cells are two shuffles; nothing is
// exchanged between warps, so there is neither shared state nor a barrier. A step spreads
// what a strip's edge does not know by one column and one row: the stored columns lie
// TS_HALO inside the strip, and a warp starts TS_HALO rows above its first stored row.
//
// Why this form: the window kernel it replaces (256 x 40 cells in registers, 240 x 24 of
// them stored) computed 1.8 times the cells stored and met at a CTA barrier per step. Here
// it is 128 / 112 in x and (rows + 16) / rows in z. Rows come through a ring of 16-byte
// asynchronous copies that only the copying lane reads. 8000 x 16000: 1243 -> 463 us a
// launch (823 -> 2210 G updates/s, 4.4 TB/s of the 16 bytes a launch moves per cell), the
// same values; what bounds it now is issue at 12 warps per SM (the state of eight steps,
// 96 registers, leaves no room for more; folding S into Q saves 32 of them and 40 us, for
// 18% more rounding error).
//
// The fixed cells (rows 0 and N - 1, columns 0 and M - 1, and what lies outside) keep the
// value of two levels before; only warps that meet them (EDGE) look.
constexpr int TS_STEPS = 8, TS_HALO = 8;
constexpr int TS_COLS = 128 - 2 * TS_HALO;  // stored columns of a strip
constexpr int TS_WARPS = 4;                 // warps of a CTA (independent)
constexpr int TS_RING = 6;                  // rows in flight per warp

template <bool VEC, bool CHECK>
__device__ __forceinline__ void copy_row(float* dst, const float* src, bool row_in, int j, int M) {
    const unsigned d = smem_addr(dst);
    if (VEC) {  // (j is a multiple of 4 and the rows are whole groups of 4: inside the row for j < M)
        const int n = !CHECK || (row_in && j >= 0 && j < M) ? 16 : 0;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
    } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int n = !CHECK || (row_in && j + e >= 0 && j + e < M) ? 4 : 0;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d + 4 * e), "l"(src + e), "r"(n) : "memory");
        }
    }
}

template <bool VEC>
__global__ void __launch_bounds__(32 * TS_WARPS, 3)
    temporal_stream_kernel(const float* __restrict__ u0, const float* __restrict__ u1, float* __restrict__ v0,
                           float* __restrict__ v1, float cx, float cy, int N, int M, int Mp, int strips, int rows) {
    __shared__ __align__(16) float ring[TS_WARPS][TS_RING][2][128];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int id = blockIdx.x * TS_WARPS + warp;
    const int j = id % strips * TS_COLS - TS_HALO + 4 * lane;
    const int z0 = id / strips * rows, z1 = min(N, z0 + rows);
    if (z0 >= N) return;
    float* own = &ring[warp][0][0][4 * lane];
    auto march = [&](auto edge_c) {
        constexpr bool EDGE = decltype(edge_c)::value;
        bool fixed[4];  // columns that keep their values
#pragma unroll
        for (int e = 0; e < 4; ++e) fixed[e] = j + e <= 0 || j + e >= M - 1;
        const float2 cx2 = make_float2(cx, cx), cy2 = make_float2(cy, cy);
        const float2 mone = make_float2(-1.f, -1.f), mtwo = make_float2(-2.f, -2.f);
        float4 Q[TS_STEPS], S[TS_STEPS], prev[TS_STEPS];
#pragma unroll
        for (int s = 0; s < TS_STEPS; ++s) Q[s] = S[s] = prev[s] = make_float4(0.f, 0.f, 0.f, 0.f);
        const int first = z0 - TS_HALO, last = z1 - 1 + TS_STEPS;
        // row t into the ring; what lies outside the grid (only EDGE warps meet it) as zeros
        const float *p0 = u0 + ((long long)first * Mp + j), *p1 = u1 + ((long long)first * Mp + j);
        int next = first;
        auto fetch = [&](int slot) {
            if (EDGE) {
                const bool in = next >= 0 && next < N;
                copy_row<VEC, true>(own + slot * 256, in && j < M ? p0 : u0, in, j, M);
                copy_row<VEC, true>(own + slot * 256 + 128, in && j < M ? p1 : u1, in, j, M);
            } else if (next <= last) {
                copy_row<VEC, false>(own + slot * 256, p0, true, j, M);
                copy_row<VEC, false>(own + slot * 256 + 128, p1, true, j, M);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            ++next;
            p0 += Mp;
            p1 += Mp;
        };
        for (int k = 0; k < TS_RING; ++k) fetch(k);
        float *o0 = v0 + ((long long)(first - 7) * Mp + j), *o1 = v1 + ((long long)(first - 8) * Mp + j);
        const bool stores = lane >= TS_HALO / 4 && lane < 32 - TS_HALO / 4;
        int slot = 0;
        // (four rows per turn: the values handed from a step to the next then change registers by name)
#pragma unroll 4
        for (int t = first; t <= last; ++t) {
            asm volatile("cp.async.wait_group %0;" ::"n"(TS_RING - 1) : "memory");
            float4 old = *reinterpret_cast<const float4*>(own + slot * 256);
            float4 v = *reinterpret_cast<const float4*>(own + slot * 256 + 128);
            fetch(slot);
            slot = slot + 1 == TS_RING ? 0 : slot + 1;
            float4 seventh;
#pragma unroll
            for (int s = 0; s < TS_STEPS; ++s) {
                // (differences as multiply-adds by -1 and -2, which are exact: a packed add
                // would negate its operand first)
                const float4 p = prev[s], q = Q[s], c = S[s];
                const float2 vl = make_float2(v.x, v.y), vh = make_float2(v.z, v.w);
                float2 ul = __ffma2_rn(cx2, __fadd2_rn(make_float2(c.x, c.y), vl), make_float2(q.x, q.y));
                float2 uh = __ffma2_rn(cx2, __fadd2_rn(make_float2(c.z, c.w), vh), make_float2(q.z, q.w));
                const float l = __shfl_up_sync(0xffffffffu, v.w, 1), r = __shfl_down_sync(0xffffffffu, v.x, 1);
                const float2 dl = __fadd2_rn(__ffma2_rn(mtwo, vl, make_float2(l, v.x)), make_float2(v.y, v.z));
                const float2 dh = __fadd2_rn(__ffma2_rn(mtwo, vh, make_float2(v.y, v.z)), make_float2(v.w, r));
                float2 ql = __ffma2_rn(cy2, dl, __ffma2_rn(mone, make_float2(old.x, old.y), __fadd2_rn(vl, vl)));
                float2 qh = __ffma2_rn(cy2, dh, __ffma2_rn(mone, make_float2(old.z, old.w), __fadd2_rn(vh, vh)));
                const float2 sl = __ffma2_rn(mtwo, vl, make_float2(p.x, p.y)), sh = __ffma2_rn(mtwo, vh, make_float2(p.z, p.w));
                if (EDGE) {
                    // fixed cells: Q holds old, and the finished row takes Q as it is
                    const bool row = t - s <= 0 || t - s >= N - 1, above = t - s - 1 <= 0 || t - s - 1 >= N - 1;
                    ql.x = row || fixed[0] ? old.x : ql.x;
                    ql.y = row || fixed[1] ? old.y : ql.y;
                    qh.x = row || fixed[2] ? old.z : qh.x;
                    qh.y = row || fixed[3] ? old.w : qh.y;
                    ul.x = above || fixed[0] ? q.x : ul.x;
                    ul.y = above || fixed[1] ? q.y : ul.y;
                    uh.x = above || fixed[2] ? q.z : uh.x;
                    uh.y = above || fixed[3] ? q.w : uh.y;
                }
                Q[s] = make_float4(ql.x, ql.y, qh.x, qh.y);
                S[s] = make_float4(sl.x, sl.y, sh.x, sh.y);
                prev[s] = v;
                old = p;
                v = make_float4(ul.x, ul.y, uh.x, uh.y);
                if (s == TS_STEPS - 2) seventh = v;  // u_{n+7} of row t - 7; v ends as u_{n+8} of row t - 8
            }
            auto put = [&](float* o, const float4& u) {
                if (VEC && (!EDGE || j + 3 < M)) {
                    __stcs(reinterpret_cast<float4*>(o), u);
                } else {
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (j + e < M) o[e] = comp(u, e);
                }
            };
            if (stores && t >= z0 + 7 && t < z1 + 7) put(o0, seventh);
            if (stores && t >= z0 + 8) put(o1, v);
            o0 += Mp;
            o1 += Mp;
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    };
    const int j0 = id % strips * TS_COLS - TS_HALO;
    if (j0 <= 0 || j0 + 128 >= M || z0 - TS_HALO <= 0 || z1 + TS_HALO >= N)
        march(Flag<true>{});
    else
        march(Flag<false>{});
}

}  // namespace

// the staged window of temporal_kernel: TMA box (columns, rows)
void temporal_box(unsigned* cols, unsigned* rows) {
    *cols = TT_W;
    *rows = TT_WZ;
}

cudaError_t launch_temporal_stream(const float* u0, const float* u1, float* v0, float* v1, float wavespeed, float dt,
                                   float dx, float dy, int N, int M, int Mp, cudaStream_t s) {
    const int strips = (M + TS_COLS - 1) / TS_COLS;
    // Rows per warp. A warp spends 16 rows on its first and last results. A row takes it
    // 0.33 us alone and 0.045 more for each warp of its SM, up to the 12 that are resident;
    // beyond them, more and shorter strips even out the SMs. Measured, us (the rule's choice
    // first): 256^2 4 rows 14.4, 8 rows 17.1, 32 rows 31.2; 1000^2 10 rows 23.6, 24 rows 27.1; 2048^2
    // 26 rows 43.8, 32 rows 37.5, 64 rows 49.7; 4000^2 44 rows 95.6, 80 rows 91.6, 128 rows 107.3;
    // 8000 x 16000 127 rows 463, 250 rows 484, 471 rows 589, 1000 rows 735.
    int rows = N;
    double least = 0;
    for (int q = 1; q <= 64; ++q) {
        const int n = std::max(1, std::min(304 * q / strips, (N + 3) / 4));
        const int r = (N + n - 1) / n;
        const double warps = double(strips) * ((N + r - 1) / r);
        const double row = warps <= 1824 ? 0.33 + 0.045 * warps / 152 : 0.53 * (warps / 1824 + 0.63);
        const double cost = row * (r + 16);
        if (least == 0 || cost < least) {
            least = cost;
            rows = r;
        }
    }
    const long long warps = (long long)strips * ((N + rows - 1) / rows);
    const unsigned ctas = unsigned((warps + TS_WARPS - 1) / TS_WARPS);
    const float k = kcoef(wavespeed, dt), cx = k / (dx * dx), cy = k / (dy * dy);
    auto a16 = [](const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; };
    // a plain launch: the copies of u0 and u1, the previous launch's output, are ordered
    // after it by the kernel boundary
    if (Mp % 4 == 0 && a16(u0) && a16(u1) && a16(v0) && a16(v1))
        temporal_stream_kernel<true><<<ctas, 32 * TS_WARPS, 0, s>>>(u0, u1, v0, v1, cx, cy, N, M, Mp, strips, rows);
    else
        temporal_stream_kernel<false><<<ctas, 32 * TS_WARPS, 0, s>>>(u0, u1, v0, v1, cx, cy, N, M, Mp, strips, rows);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_temporal(const CUtensorMap& m0, const CUtensorMap& m1, float* v0, float* v1, float wavespeed,
                            float dt, float dx, float dy, int N, int M, int Mp, cudaStream_t s) {
    static int configured_device = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (configured_device != dev) {
        const cudaError_t e =
            cudaFuncSetAttribute(temporal_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, TT_BYTES);
        if (e != cudaSuccess) return e;
        configured_device = dev;
    }
    const dim3 grid((M + TT_TX - 1) / TT_TX, (N + TT_TZ - 1) / TT_TZ);
    const cudaError_t e = launch_pdl(temporal_kernel, grid, dim3(TT_THREADS), TT_BYTES, s, m0, m1, v0, v1,
                                     kcoef(wavespeed, dt), dx * dx, dy * dy, N, M, Mp);
    count_launch();
    return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace wfd

using namespace wfd;

extern "C" {

int wfd_step1d(const float* u0, const float* u1, float* u2, float wavespeed, float dt, float dx,
               int N, void* stream) {
    if (!u0 || !u1 || !u2) return set_error(WFD_ERR_INVALID, "NULL field");
    if (N < 3) return set_error(WFD_ERR_INVALID, "need N >= 3");
    const int blocks = (N + 255) / 256;
    step1d_kernel<<<blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(u0, u1, u2, kcoef(wavespeed, dt),
                                                                          dx * dx, N);
    count_launch();
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? WFD_OK : set_error(WFD_ERR_CUDA, cudaGetErrorString(e));
}

int wfd_step2d_exact(const float* u0, const float* u1, float* u2, float wavespeed, float dt, float dx,
                     float dy, int N, int M, int M_padded, void* stream) {
    if (!u0 || !u1 || !u2) return set_error(WFD_ERR_INVALID, "NULL field");
    if (N < 3 || M < 3 || M_padded < M) return set_error(WFD_ERR_INVALID, "need N, M >= 3 and M_padded >= M");
    if ((long long)N * M_padded >= (1ll << 31)) return set_error(WFD_ERR_INVALID, "grid too large");
    if ((N + 3) / 4 > 65535) return set_error(WFD_ERR_INVALID, "N too large (more than 262140 rows)");
    const dim3 block(64, 4), grid(((M + 3) / 4 + 63) / 64, (N + 3) / 4);
    exact_kernel<<<grid, block, 0, static_cast<cudaStream_t>(stream)>>>(u0, u1, u2, kcoef(wavespeed, dt), dx * dx,
                                                                        dy * dy, N, M, M_padded);
    count_launch();
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? WFD_OK : set_error(WFD_ERR_CUDA, cudaGetErrorString(e));
}

int wfd_step2d_mixed(const void* u0, const void* u1, void* u2, float wavespeed, float dt, float dx,
                     float dy, int N, int M, int M_padded, void* stream) {
    if (!u0 || !u1 || !u2) return set_error(WFD_ERR_INVALID, "NULL field");
    if (N < 3 || M < 3 || M_padded < M + 1 || M_padded % 2)
        return set_error(WFD_ERR_INVALID, "need N, M >= 3 and an even M_padded > M");
    if (reinterpret_cast<uintptr_t>(u0) % 4 || reinterpret_cast<uintptr_t>(u1) % 4 ||
        reinterpret_cast<uintptr_t>(u2) % 4)
        return set_error(WFD_ERR_INVALID, "fields must be 4-byte aligned");
    if ((long long)N * M_padded >= (1ll << 31)) return set_error(WFD_ERR_INVALID, "grid too large");
    if ((N + 3) / 4 > 65535) return set_error(WFD_ERR_INVALID, "N too large (more than 262140 rows)");
    const dim3 block(128, 4), grid((M_padded / 2 + 127) / 128, (N + 3) / 4);
    mixed_kernel<<<grid, block, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const __half*>(u0), static_cast<const __half*>(u1), static_cast<__half*>(u2),
        kcoef(wavespeed, dt), dx * dx, dy * dy, N, M, M_padded);
    count_launch();
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? WFD_OK : set_error(WFD_ERR_CUDA, cudaGetErrorString(e));
}

int wfd_step2d_mixed_fast(const void* u0, const void* u1, void* u2, float wavespeed, float dt, float dx,
                          float dy, int N, int M, int M_padded, void* stream) {
    if (!u0 || !u1 || !u2) return set_error(WFD_ERR_INVALID, "NULL field");
    if (N < 3 || M < 3 || M_padded < M || M_padded % 8)
        return set_error(WFD_ERR_INVALID, "need N, M >= 3 and M_padded >= M, a multiple of 8");
    for (const void* p : {u0, u1, (const void*)u2})
        if (reinterpret_cast<uintptr_t>(p) % 16) return set_error(WFD_ERR_INVALID, "fields must be 16-byte aligned");
    if ((long long)N * M_padded >= (1ll << 31)) return set_error(WFD_ERR_INVALID, "grid too large");
    if ((N + 3) / 4 > 65535) return set_error(WFD_ERR_INVALID, "N too large (more than 262140 rows)");
    const float k = kcoef(wavespeed, dt);
    const dim3 block(64, 4), grid((M_padded / 8 + 63) / 64, (N + 3) / 4);
    mixed_fast_kernel<<<grid, block, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const __half*>(u0), static_cast<const __half*>(u1), static_cast<__half*>(u2), k / (dx * dx),
        k / (dy * dy), N, M, M_padded);
    count_launch();
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? WFD_OK : set_error(WFD_ERR_CUDA, cudaGetErrorString(e));
}

int wfd_step2d_scaled(const int16_t* q0, const float* s0, const int16_t* q1, const float* s1,
                      int16_t* q2, float* s2, float wavespeed, float dt, float dx, float dy, int N,
                      int M, int M_padded, void* stream) {
    if (!q0 || !s0 || !q1 || !s1 || !q2 || !s2) return set_error(WFD_ERR_INVALID, "NULL field");
    if (N < 3 || M < 3 || M_padded < M || M_padded % 64)
        return set_error(WFD_ERR_INVALID, "need N, M >= 3 and M_padded >= M, a multiple of 64");
    for (const void* p : {(const void*)q0, (const void*)q1, (const void*)q2})
        if (reinterpret_cast<uintptr_t>(p) % 8) return set_error(WFD_ERR_INVALID, "q fields must be 8-byte aligned");
    if ((long long)N * M_padded >= (1ll << 31)) return set_error(WFD_ERR_INVALID, "grid too large");
    if ((N + 3) / 4 > 65535) return set_error(WFD_ERR_INVALID, "N too large (more than 262140 rows)");
    const dim3 block(64, 4), grid((M_padded / 4 + 63) / 64, (N + 3) / 4);
    scaled_kernel<<<grid, block, 0, static_cast<cudaStream_t>(stream)>>>(
        q0, s0, q1, s1, q2, s2, kcoef(wavespeed, dt), dx * dx, dy * dy, N, M, M_padded);
    count_launch();
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? WFD_OK : set_error(WFD_ERR_CUDA, cudaGetErrorString(e));
}

}  // extern "C"
