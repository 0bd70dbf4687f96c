// Resident 2D kernel of the acoustic wave path (sm_103a): the whole field of
// one or more shots stays on the chip for many time steps.
//
// The streaming kernels (stencil2d.cu, stencil2d_k2.cu) read and write every
// level through L2 or HBM once per launch. A GB300 has 152 x 227 KB of shared
// memory and 152 x 256 KB of registers: up to 4.3 M cells of (u, u_old) and m
// fit on the chip together. One cooperative launch then advances them by as
// many steps as the caller asks (a checkpoint segment, or the whole forward),
// and only what leaves the recursion touches memory: halos between tiles,
// receiver samples, and L u_n of the levels a gradient keeps.
//
// Work split. A CTA runs `ng` groups of `nwg` warps. A group owns one tile
// (128 x tz cells, tz = RB nwg) of one shot: lane l of a warp owns columns
// 4 l .. 4 l + 3, a warp RB consecutive rows. u_n sits in shared memory with a
// halo of R rows and 4 columns; the second level (u_{n-1}, or d_n in the
// summed form) sits in the owning thread's registers, as does the gradient
// sum; m sits in shared memory. Groups synchronise on their own named
// barriers, so while one waits for its halo the others of the SM compute.
//
// Halo exchange. After a step each tile writes its R outer rows and 4 outer
// columns to its neighbours' mailboxes in global memory (L2): packets of 16
// bytes holding two cells, each next to the tag of its level in one 8-byte
// word. An 8-byte access is single-copy atomic, so a packet whose tags match is
// complete: no fence, flag or grid barrier is needed, and the latency of a step
// is one L2 write and one L2 read. Two mailboxes per tile alternate by level: a
// tile writes level n + 2 only after it has received its neighbour's level
// n + 1, which the neighbour wrote after its CTA barrier behind the read of
// level n. The launch is cooperative, so every tile is resident. Every wait is
// bounded; one that gives up records DEV_ERR_TMA_TIMEOUT, and its CTA goes on
// without further waiting, which overtakes its neighbours' tags: theirs give up in
// turn, each CTA once, and the launch runs to its end.
//
// Arithmetic. The cell updates are those of the streaming kernels, operation
// for operation (lap_row, lap_row_diff, the update with its sponge factors),
// so levels, traces and misfits come out the same bit for bit.
#pragma once
#include <atomic>

#include "common.cuh"
#include "internal.h"

namespace wfd {
namespace res {

constexpr int W = RES_TX + 8;  // staged row: 4 columns of halo on each side
// polls of one halo wait: a poll is one L2 round trip, so seconds in all
constexpr unsigned kMaxPolls = 1u << 22;

struct Packet {
    unsigned long long a, b;  // {tag, cell} twice: the tag in the high word
};

__device__ __forceinline__ Packet ld_packet(const Packet* p) {
    Packet v;
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(v.a), "=l"(v.b) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_packet(Packet* p, float x, float y, unsigned tag) {
    const unsigned long long t = (unsigned long long)tag << 32;
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(t | __float_as_uint(x)),
                 "l"(t | __float_as_uint(y))
                 : "memory");
}
__device__ __forceinline__ bool has_tag(const Packet& v, unsigned tag) {
    return unsigned(v.a >> 32) == tag && unsigned(v.b >> 32) == tag;
}
__device__ __forceinline__ float2 cells(const Packet& v) {
    return make_float2(__uint_as_float(unsigned(v.a)), __uint_as_float(unsigned(v.b)));
}
__device__ __forceinline__ void bar_group(int g, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(g + 1), "r"(threads) : "memory");
}
__device__ __forceinline__ float4 f4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void add_to(float4& v, int e, float x) {
    if (e == 0) v.x += x;
    if (e == 1) v.y += x;
    if (e == 2) v.z += x;
    if (e == 3) v.w += x;
}

__device__ __forceinline__ float keep(float v, int mask) { return __int_as_float(__float_as_int(v) & mask); }

// The streaming kernels' update with sponge factors, two cells at a time:
// u_{n+1} = g (m L u + 2 u) - g^2 u_{n-1}, or d_{n+1} = g m L u + (g^2 d - (1 - g)^2 u).
template <bool SUM>
__device__ __forceinline__ float2 damped(float2 g, float2 m, float2 l, float2 c, float2 o) {
    const float2 nc = make_float2(-c.x, -c.y), no = make_float2(-o.x, -o.y), ng = make_float2(-g.x, -g.y);
    if constexpr (SUM) {
        const float2 omg = __fadd2_rn(make_float2(1.f, 1.f), ng);
        return __ffma2_rn(__fmul2_rn(g, m), l, __ffma2_rn(__fmul2_rn(g, g), o, __fmul2_rn(__fmul2_rn(omg, omg), nc)));
    } else {
        const float2 A = __ffma2_rn(m, l, __fadd2_rn(c, c));
        return __ffma2_rn(g, A, __fmul2_rn(__fmul2_rn(g, g), no));
    }
}

// The stencil weights as duplicated pairs, staged in shared memory and read once per
// step: kept in registers across the halo wait they would push the state out of them.
template <int R>
struct Weights {
    float2 c0p, cxp[R], czp[R];
};

// What a group looks up in shared memory instead of keeping it in registers across steps.
struct Group {
    long long so;            // offset of the shot in a field
    int ilo, nlink, ihi;     // its tile's injected points: ent[ilo .. ihi), the first nlink linked
                             // (-1: too many, add_points)
    int slo, shi;            // its tile's sampled points
    int pad;
};

// The points injected into a group's tile, linked per owning thread.
struct Points {
    float v[RES_PTS];             // the step's values, g scale w
    int cell[RES_PTS], p[RES_PTS];  // the list's entries
    int2 smp[RES_PTS];              // sampled points: place in U, number
    unsigned short next[RES_PTS];
    unsigned short at[RES_PTS];   // 4 r + e within the owner's rows
};
// (behind it, per thread of the group: its first point)
constexpr unsigned NONE = 0xffffu;

// A point's step value: g scale w (times m for a residual).
__device__ __forceinline__ float point_value(const StepArgs& a, int cell, float w) {
    float v = w * a.inj_scale;
    if (a.inj_times_m) v *= __ldg(a.m + cell);
    const int z = cell / a.ld, xx = cell - z * a.ld;
    const float g = (a.gz ? __ldg(a.gz + z) : 1.f) * (a.gx ? __ldg(a.gx + xx) : 1.f);
    return __fmul_rn(g, v);
}

// Injection into a tile that holds many more points than are linked: all of them over all
// threads of the group, by shared-memory atomics. (By a walk of every thread past the linked
// points for its own cells: the gradient of 60 steps on 256^2 with a receiver in every cell
// 6486 us, on 1024^2 16421; this way 1206 and 2566, streaming kernels 1856 and 3070.)
__device__ __forceinline__ void add_points(const StepArgs& a, const Group& gr, float* U, int z0, int x0, int R,
                                           const float* ival, int grp, int gt, int GT) {
    bar_group(grp, GT);
#pragma unroll 2
    for (int j = gr.ilo + gt; j < gr.ihi; j += GT) {
        const int2 en = __ldg(a.inj.ent + j);
        const int z = en.x / a.ld, xx = en.x - z * a.ld;
        atomicAdd(U + (z - z0 + R) * W + (xx - x0 + 4), point_value(a, en.x, __ldg(ival + en.y)));
    }
    bar_group(grp, GT);
}

// MANY: a shot has so many points to inject that the walk past a tile's linked ones may be
// long (RES_WALK). An instance of its own: in the one kernel add_points costs the others' steps
// 1 to 7%, by registers and by its place in the loop (and without the walk in its place the
// order-8 forward at 2048^2 is 2% slower too).
template <int R, int MODE, int RB, bool MANY>
__global__ void __launch_bounds__(res_threads(MODE, RB), 1) res_kernel(const __grid_constant__ ResArgs p) {
    constexpr bool ADJ = MODE == RES_ADJOINT;
    constexpr bool SUM = MODE == RES_SUMMED || MODE == RES_SUMMED_DIFF;
    // rows of m read from L2 instead of shared memory (the largest tiles only)
    constexpr bool LM = res_l2_rows(RB) > 0;
    constexpr int NS = R;                // halo-row packets per thread: 4 R rows x half over nwg >= 4 warps
    constexpr int WE = (RB + 7) / 8;     // halo-column packets per thread
    const StepArgs& a = p.a;
    extern __shared__ __align__(128) unsigned char smem[];

    // (the broadcast tells the compiler that everything derived from the warp is uniform)
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int nwg = p.nwg, GT = nwg * 32, tz = p.tz;
    const int grp = warp / nwg, wl = warp - grp * nwg, gt = tid - grp * GT;
    int tile, slot;
    if (p.share_m) {
        tile = blockIdx.x % p.ntiles;
        slot = (blockIdx.x / p.ntiles) * p.ng + grp;
    } else {
        const int item = blockIdx.x * p.ng + grp;
        tile = item % p.ntiles;
        slot = item / p.ntiles;
    }
    const bool active = slot < p.nshots;
    const int s = p.shot0 + slot;
    const int tx = tile % a.tiles_x, tzi = tile / a.tiles_x;
    const int x0 = tx * RES_TX, z0 = tzi * tz;
    const int x = x0 + 4 * lane, tr0 = wl * RB, zb = z0 + tr0;

    const int ubytes = W * (tz + 2 * R) * 4, lm = LM ? p.lm : 0, mrow = RB - lm, mbytes = RES_TX * nwg * mrow * 4;
    const int gbytes = ubytes + (p.share_m ? 0 : mbytes) + res_group_bytes(nwg, tz);
    unsigned char* gs = smem + 128 + (p.share_m ? mbytes : 0) + grp * gbytes;
    float* U = reinterpret_cast<float*>(gs);
    float* M = reinterpret_cast<float*>(p.share_m ? smem + 128 : gs + ubytes);
    unsigned char* gend = gs + ubytes + (p.share_m ? 0 : mbytes);
    float* GX = reinterpret_cast<float*>(gend);  // sponge factors of the tile's columns and rows
    float* GZ = GX + RES_TX;
    Points& pt = *reinterpret_cast<Points*>(GZ + (tz + 3) / 4 * 4);
    Group& gr = *reinterpret_cast<Group*>(&pt + 1);
    unsigned* owned = reinterpret_cast<unsigned*>(&gr + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem);
    Weights<R>* weights = reinterpret_cast<Weights<R>*>(smem + 32);

    if (tid == 0) {
        *abort_flag = 0;
        weights->c0p = a.c0p;
        for (int k = 0; k < R; ++k) {
            weights->cxp[k] = a.cxp[k];
            weights->czp[k] = a.czp[k];
        }
    }
    owned[gt] = NONE;
    // ---- u_n with its halo, m, and the second level
    const long long so = (long long)s * a.shot_stride;
    auto state = [&](const float* from, long long off) {  // 4 cells of u_in or x_in
        if (MODE == RES_LEAP && p.in_bf16) return unpack_bf16x4(reinterpret_cast<const uint2*>(from)[off / 4]);
        return f4(from + off);
    };
    if (active) {
        for (int k = gt; k < (tz + 2 * R) * (W / 4); k += GT) {
            const int row = k / (W / 4), c = k - row * (W / 4);
            const int z = z0 - R + row, xx = x0 - 4 + 4 * c;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (p.u_in && z >= 0 && z < a.nz && xx >= 0 && xx < a.ld) v = state(p.u_in, so + (long long)z * a.ld + xx);
            *reinterpret_cast<float4*>(U + row * W + 4 * c) = v;
        }
    }
    const bool x_ok = x < a.ld;
    if (active || p.share_m) {  // (a shared m is written by every group: the same values)
#pragma unroll
        for (int r = 0; r < RB; ++r) {
            const int rm = r - lm;
            if (rm < 0) continue;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (zb + r < a.nz && x_ok) v = __ldg(reinterpret_cast<const float4*>(a.m + (long long)(zb + r) * a.ld + x));
            *reinterpret_cast<float4*>(M + (wl * mrow + rm) * RES_TX + 4 * lane) = v;
        }
    }
    float4 X[RB];
#pragma unroll
    for (int r = 0; r < RB; ++r) {
        X[r] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (active && p.x_in && zb + r < a.nz && x_ok) {
            const long long off = so + (long long)(zb + r) * a.ld + x;
            X[r] = state(p.x_in, off);
            if (MODE == RES_LEAP && p.x_is_diff) {
                const float4 u = state(p.u_in, off);
                X[r] = make_float4(u.x - X[r].x, u.y - X[r].y, u.z - X[r].z, u.w - X[r].w);
            }
        }
    }
    float4 G[ADJ ? RB : 1];
#pragma unroll
    for (int r = 0; r < (ADJ ? RB : 1); ++r) G[r] = make_float4(0.f, 0.f, 0.f, 0.f);

    // ---- sponge factors; a warp whose cells are all interior and undamped takes the plain update
    for (int k = gt; k < RES_TX; k += GT) GX[k] = (a.gx && x0 + k < a.nx) ? __ldg(a.gx + x0 + k) : 1.f;
    for (int k = gt; k < tz; k += GT) GZ[k] = (a.gz && z0 + k < a.nz) ? __ldg(a.gz + z0 + k) : 1.f;
    __syncthreads();
    bool mine = x >= R && x + 3 < a.nx - R && zb >= R && zb + RB <= a.nz - R;
#pragma unroll
    for (int e = 0; e < 4; ++e) mine = mine && GX[4 * lane + e] == 1.f;
#pragma unroll
    for (int r = 0; r < RB; ++r) mine = mine && GZ[tr0 + r] == 1.f;
    const bool plain = __all_sync(0xffffffffu, mine);

    // ---- this tile's points
    if (gt == 0) {
        const long long key = (long long)s * p.ntiles + tile;
        gr.so = so;
        gr.ilo = active && a.inj.off ? a.inj.off[key] : 0;
        gr.ihi = active && a.inj.off ? a.inj.off[key + 1] : 0;
        gr.slo = active && a.smp.off ? a.smp.off[key] : 0;
        gr.shi = active && a.smp.off ? a.smp.off[key + 1] : 0;
        gr.nlink = !MANY || gr.ihi - gr.ilo <= RES_PTS ? min(gr.ihi - gr.ilo, RES_PTS) : -1;
    }
    __syncthreads();
    auto owner_at = [&](int cell, int& own, int& at) {  // the owning thread of a cell of the tile
        const int z = cell / a.ld - z0, xx = cell % a.ld - x0;
        const int w = z / RB;
        own = w * 32 + (xx >> 2);
        at = 4 * (z - w * RB) + (xx & 3);
    };
    for (int j = gt; j < gr.nlink; j += GT) {
        int own, at;
        const int2 en = a.inj.ent[gr.ilo + j];
        pt.cell[j] = en.x;
        pt.p[j] = en.y;
        owner_at(en.x, own, at);
        pt.at[j] = (unsigned short)at;
        pt.next[j] = (unsigned short)atomicExch(&owned[own], unsigned(j));
    }
    auto staged_at = [&](int cell) {  // a cell of the tile in U
        const int z = cell / a.ld, xx = cell - z * a.ld;
        return (z - z0 + R) * W + (xx - x0 + 4);
    };
    for (int j = gt; j < min(gr.shi - gr.slo, RES_PTS); j += GT) {
        const int2 en = a.smp.ent[gr.slo + j];
        pt.smp[j] = make_int2(staged_at(en.x), en.y);
    }
    __syncthreads();
    if (!active) return;
    const int nlink = gr.nlink, nsmp = gr.shi - gr.slo;
    // ---- mailboxes: [tile item][parity][2 R rows x 64 + 4 tz packets]
    const int per = 2 * R * 64 + 4 * tz;
    const bool nb_n = tzi > 0, nb_s = tzi + 1 < a.tiles_z, nb_w = tx > 0, nb_e = tx + 1 < a.tiles_x;
    Packet* mail = reinterpret_cast<Packet*>(p.mail) + 2ll * per * ((long long)slot * p.ntiles + tile);
    for (int it = 0; it < p.steps; ++it) {
        // the thread's first row, opaque to the compiler: it would otherwise compute every
        // row's addresses and tests once before this loop and keep them in registers
        int row0 = tr0;
        asm volatile("" : "+r"(row0));
        const int zr = z0 + row0;
        const int inj_t = p.inj_t0 + it * p.dir, smp_t = p.smp_t0 + it * p.dir;
        // (read before the halo wait, which hides its latency)
        float iv = 0.f;
        const float* ival = a.inj_val + ((long long)s * a.inj_nt + inj_t) * a.inj_np;
        if (gt < nlink) iv = __ldg(ival + pt.p[gt]);
        // ------------------------------------------------ the halo of level n
        if (it > 0) {
            const unsigned tag = p.tag0 + unsigned(it);
            const Packet* in = mail + (it & 1) * per;
            constexpr int N = NS + WE;
            unsigned need = 0;
            int dst[N], from[N];
#pragma unroll
            for (int i = 0; i < N; ++i) {
                if (i < NS) {  // half rows of 32 packets, one per warp
                    const int h = wl + nwg * i, row = h >> 1;
                    if (h < 4 * R && (row < R ? nb_n : nb_s)) need |= 1u << i;
                    from[i] = h * 32 + lane;
                    dst[i] = (row < R ? row : tz + row) * W + 4 + (h & 1) * 64 + 2 * lane;
                } else {
                    const int q = gt + GT * (i - NS), east = q >= 2 * tz, rr = (q - (east ? 2 * tz : 0)) >> 1;
                    if (q < 4 * tz && (east ? nb_e : nb_w)) need |= 1u << i;
                    from[i] = 2 * R * 64 + q;
                    dst[i] = (rr + R) * W + (east ? 4 + RES_TX : 0) + 2 * (q & 1);
                }
            }
            for (unsigned polls = 0; need; ++polls) {
                Packet v[N];
#pragma unroll
                for (int i = 0; i < N; ++i) {
                    // (defined on every path: an undefined one would hold its registers
                    // through the whole time loop)
                    v[i].a = v[i].b = 0;
                    if (need >> i & 1) v[i] = ld_packet(in + from[i]);
                }
#pragma unroll
                for (int i = 0; i < N; ++i)
                    if ((need >> i & 1) && has_tag(v[i], tag)) {
                        *reinterpret_cast<float2*>(U + dst[i]) = cells(v[i]);
                        need &= ~(1u << i);
                    }
                if (need && (polls >= kMaxPolls || *abort_flag)) {
                    if (!*abort_flag) report(a.err, DEV_ERR_TMA_TIMEOUT);
                    *abort_flag = 1;
                    break;
                }
            }
        }
        bar_group(grp, GT);  // level n complete in U
        // samples of level n
        if (nsmp > 0 && smp_t >= 0 && smp_t < a.smp_nt) {
            float* out = a.smp_out + ((long long)s * a.smp_nt + smp_t) * a.smp_np;
            for (int j = gt; j < nsmp; j += GT) {
                int2 at;
                if (j < RES_PTS) {
                    at = pt.smp[j];
                } else {
                    at = __ldg(a.smp.ent + gr.slo + j);
                    at.x = staged_at(at.x);
                }
                float v = U[at.x] * a.smp_scale;
                if (a.smp_div_m) v /= __ldg(a.m + __ldg(&a.smp.ent[gr.slo + j].x));
                out[at.y] = v;
            }
        }
        // the step's injected values
        if (gt < nlink) pt.v[gt] = point_value(a, pt.cell[gt], iv);
        for (int j = gt + GT; j < nlink; j += GT) pt.v[j] = point_value(a, pt.cell[j], __ldg(ival + pt.p[j]));

        // ------------------------------------------------ the update, into X
        float* lap = p.lap && it >= p.lap_from ? p.lap + gr.so + (long long)it * p.lap_stride : nullptr;
        auto rows = [&](auto plain_c) {
            constexpr bool PLAIN = decltype(plain_c)::value;
            const Weights<R> wt = *weights;
            float4 V[RB + 2 * R];
            const float* urow = U + row0 * W + 4 + 4 * lane;  // V[j] = staged row row0 + j
#pragma unroll
            for (int j = 0; j < 2 * R; ++j) V[j] = f4(urow + j * W);
            const float4 gx = PLAIN ? make_float4(1.f, 1.f, 1.f, 1.f) : f4(GX + 4 * lane);
            int xm[4];  // all bits set in the interior's columns
            if constexpr (!PLAIN) {
                int xr = x;  // (opaque, as row0)
                asm volatile("" : "+r"(xr));
#pragma unroll
                for (int e = 0; e < 4; ++e) xm[e] = xr + e >= R && xr + e < a.nx - R ? -1 : 0;
            }
            float4 ML[LM ? RB : 1];
            auto load_m = [&](int r) {
                ML[r] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (r < lm && zr + r < a.nz && x_ok)
                    ML[r] = __ldg(reinterpret_cast<const float4*>(a.m + (unsigned)((zr + r) * a.ld + x)));
            };
            if constexpr (LM) {
                load_m(0);
                load_m(1);
            }
            float4 LU[ADJ ? RB + 2 : 1];
            auto load_lu = [&](int r) {
                LU[r] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (lap && zr + r < a.nz && x_ok)
                    LU[r] = __ldcs(reinterpret_cast<const float4*>(lap + (unsigned)((zr + r) * a.ld + x)));
            };
            if constexpr (ADJ) {
                load_lu(0);
                if (RB > 1) load_lu(1);
            }
#pragma unroll
            for (int r = 0; r < RB; ++r) {
                V[r + 2 * R] = f4(urow + (r + 2 * R) * W);
                if constexpr (ADJ)
                    if (r + 2 < RB) load_lu(r + 2);
                if constexpr (LM)
                    if (r + 2 < res_l2_rows(RB)) load_m(r + 2);
                const float* row = urow + (r + R) * W;
                const float4 lv = f4(row - 4), cv = V[r + R], rv = f4(row + 4);
                float4 mv;
                if (LM && r < res_l2_rows(RB) && r < lm)
                    mv = ML[LM ? r : 0];
                else
                    mv = f4(M + (wl * mrow + r - lm) * RES_TX + 4 * lane);
                const float4 l = MODE == RES_SUMMED_DIFF ? lap_row_diff<R>(lv, cv, rv, V, r + R, wt)
                                                         : lap_row<R>(lv, cv, rv, V, r + R, wt);
                if (!ADJ && lap && zr + r < a.nz && x_ok)
                    __stcs(reinterpret_cast<float4*>(lap + (unsigned)((zr + r) * a.ld + x)), l);
                if constexpr (ADJ) {
                    if (PLAIN) {
                        const float2 lo = __ffma2_rn(make_float2(cv.x, cv.y), make_float2(LU[r].x, LU[r].y),
                                                     make_float2(G[r].x, G[r].y));
                        const float2 hi = __ffma2_rn(make_float2(cv.z, cv.w), make_float2(LU[r].z, LU[r].w),
                                                     make_float2(G[r].z, G[r].w));
                        G[r] = make_float4(lo.x, lo.y, hi.x, hi.y);
                    } else {
                        G[r].x += cv.x * LU[r].x;
                        G[r].y += cv.y * LU[r].y;
                        G[r].z += cv.z * LU[r].z;
                        G[r].w += cv.w * LU[r].w;
                    }
                }
                if constexpr (PLAIN) {
                    if constexpr (SUM) {  // d_{n+1} = m L u + d_n
                        const float2 lo = __ffma2_rn(make_float2(mv.x, mv.y), make_float2(l.x, l.y),
                                                     make_float2(X[r].x, X[r].y));
                        const float2 hi = __ffma2_rn(make_float2(mv.z, mv.w), make_float2(l.z, l.w),
                                                     make_float2(X[r].z, X[r].w));
                        X[r] = make_float4(lo.x, lo.y, hi.x, hi.y);
                    } else {
                        X[r] = leap_plain(mv, l, cv, X[r]);
                    }
                } else {
                    const float gz = GZ[row0 + r];
                    const float2 gl = __fmul2_rn(make_float2(gz, gz), make_float2(gx.x, gx.y));
                    const float2 gh = __fmul2_rn(make_float2(gz, gz), make_float2(gx.z, gx.w));
                    const float2 lo = damped<SUM>(gl, make_float2(mv.x, mv.y), make_float2(l.x, l.y),
                                                  make_float2(cv.x, cv.y), make_float2(X[r].x, X[r].y));
                    const float2 hi = damped<SUM>(gh, make_float2(mv.z, mv.w), make_float2(l.z, l.w),
                                                  make_float2(cv.z, cv.w), make_float2(X[r].z, X[r].w));
                    const int zm = zr + r >= R && zr + r < a.nz - R ? -1 : 0;
                    X[r] = make_float4(keep(lo.x, xm[0] & zm), keep(lo.y, xm[1] & zm), keep(hi.x, xm[2] & zm),
                                       keep(hi.y, xm[3] & zm));
                }
            }
        };
        if (plain)
            rows(Flag<true>{});
        else
            rows(Flag<false>{});
        bar_group(grp, GT);  // every read of level n done

        // ------------------------------------------------ level n + 1 into U
#pragma unroll
        for (int r = 0; r < RB; ++r) {
            float* cell = U + (row0 + r + R) * W + 4 + 4 * lane;
            const float4 c = f4(cell);
            if constexpr (SUM) {
                const float2 lo = __fadd2_rn(make_float2(c.x, c.y), make_float2(X[r].x, X[r].y));
                const float2 hi = __fadd2_rn(make_float2(c.z, c.w), make_float2(X[r].z, X[r].w));
                *reinterpret_cast<float4*>(cell) = make_float4(lo.x, lo.y, hi.x, hi.y);
            } else {
                *reinterpret_cast<float4*>(cell) = X[r];
                X[r] = c;
            }
        }
        if (nlink > 0) {  // the points of this thread's cells
            auto add = [&](int at, float v) {
                U[(row0 + (at >> 2) + R) * W + 4 + 4 * lane + (at & 3)] += v;
                if constexpr (SUM) {
#pragma unroll
                    for (int r = 0; r < RB; ++r)
                        if ((at >> 2) == r) add_to(X[r], at & 3, v);
                }
            };
            for (unsigned k = owned[gt]; k != NONE; k = pt.next[k]) add(pt.at[k], pt.v[k]);
            for (int j = gr.ilo + RES_PTS; !MANY && j < gr.ihi; ++j) {  // (at most RES_WALK)
                const int2 en = a.inj.ent[j];
                int owner, at;
                owner_at(en.x, owner, at);
                if (owner == gt) add(at, point_value(a, en.x, __ldg(ival + en.y)));
            }
        }
        if (MANY && nlink < 0) {
#pragma unroll 1
            for (int k = 0; k < (SUM ? 2 : 1); ++k) {  // u and, in the summed form, d in its place in U
                add_points(a, gr, U, z0, x0, R, ival, grp, gt, GT);
                if constexpr (SUM) {
#pragma unroll
                    for (int r = 0; r < RB; ++r) {
                        float* cell = U + (row0 + r + R) * W + 4 + 4 * lane;
                        const float4 c = f4(cell);
                        *reinterpret_cast<float4*>(cell) = X[r];
                        X[r] = c;
                    }
                }
            }
        }
        // ------------------------------------------------ and to the neighbours, from this warp's rows
        if (it + 1 < p.steps) {
            __syncwarp();
            const unsigned tag = p.tag0 + unsigned(it) + 1;
            Packet* out = mail + ((it + 1) & 1) * per;
            auto send_row = [&](int tr, Packet* q) {
                const float4 u = f4(U + (tr + R) * W + 4 + 4 * lane);
                q += (lane >> 4) * 32 + 2 * (lane & 15);
                st_packet(q, u.x, u.y, tag);
                st_packet(q + 1, u.z, u.w, tag);
            };
            // columns: packet k of a side holds half k & 1 of row k >> 1; this tile's west
            // columns are the west neighbour's east halo
#pragma unroll
            for (int j = 0; j < (4 * RB + 31) / 32; ++j) {
                const int k = lane + 32 * j, east = k >= 2 * RB, kk = k - (east ? 2 * RB : 0);
                const int tr = row0 + (kk >> 1);
                if (k < 4 * RB && (east ? nb_e : nb_w)) {
                    const float2 u = *reinterpret_cast<const float2*>(U + (tr + R) * W + (east ? RES_TX : 4) + 2 * (kk & 1));
                    st_packet(out + 128 * R + (east ? 2 * per : 2 * tz - 2 * per) + 2 * tr + (kk & 1), u.x, u.y, tag);
                }
            }
            if (nb_n)  // the north neighbour's rows below it
                for (int tr = row0; tr < min(R, row0 + RB); ++tr) send_row(tr, out - 2 * per * a.tiles_x + 64 * (R + tr));
            if (nb_s)
                for (int tr = max(tz - R, row0); tr < row0 + RB; ++tr)
                    send_row(tr, out + 2 * per * a.tiles_x + 64 * (tr - (tz - R)));
        }
    }

    // ---- the state and the gradient sum
#pragma unroll
    for (int r = 0; r < RB; ++r) {
        const int z = zb + r;
        if (z >= a.nz || !x_ok) continue;
        const long long at = gr.so + (long long)z * a.ld + x;
        if (p.u_out) *reinterpret_cast<float4*>(p.u_out + at) = f4(U + (tr0 + r + R) * W + 4 + 4 * lane);
        if (p.x_out) *reinterpret_cast<float4*>(p.x_out + at) = X[r];
        if (!ADJ && p.u_bf16) {
            p.u_bf16[at / 4] = pack_bf16x4(f4(U + (tr0 + r + R) * W + 4 + 4 * lane));
            p.x_bf16[at / 4] = pack_bf16x4(X[r]);
        }
        if constexpr (ADJ) {
            if (z < R || z >= a.nz - R) continue;
            float* gp = a.grad + (long long)z * a.ld + x;
            if (x >= R && x + 3 < a.nx - R) {
                atomicAdd(reinterpret_cast<float4*>(gp), G[r]);
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (x + e >= R && x + e < a.nx - R) atomicAdd(gp + e, comp(G[r], e));
            }
        }
    }
}

template <int R, int MODE, int RB, bool MANY>
cudaError_t launch_one(const ResArgs& q, size_t smem, int ctas, cudaStream_t s) {
    static std::atomic<unsigned long long> configured{0};  // bit d: done on device d
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const unsigned long long bit = 1ull << (dev & 63);
    if (!(configured.load(std::memory_order_relaxed) & bit)) {
        e = cudaFuncSetAttribute(res_kernel<R, MODE, RB, MANY>, cudaFuncAttributeMaxDynamicSharedMemorySize, RES_SMEM);
        if (e != cudaSuccess) return e;
        configured.fetch_or(bit, std::memory_order_relaxed);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(32 * q.nwg * q.ng);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    e = cudaLaunchKernelEx(&cfg, res_kernel<R, MODE, RB, MANY>, q);
    count_launch();
    return e != cudaSuccess ? e : cudaGetLastError();
}

template <int R, int MODE, bool MANY>
cudaError_t launch_points(int rb, const ResArgs& q, size_t smem, int ctas, cudaStream_t s) {
    switch (rb) {
        case 2: return launch_one<R, MODE, 2, MANY>(q, smem, ctas, s);
        case 4: return launch_one<R, MODE, 4, MANY>(q, smem, ctas, s);
        case 7: return launch_one<R, MODE, 7, MANY>(q, smem, ctas, s);
        case 10:
            if constexpr (MODE != RES_ADJOINT) return launch_one<R, MODE, 10, MANY>(q, smem, ctas, s);
            return cudaErrorInvalidValue;
        case 14: return launch_one<R, MODE, 14, MANY>(q, smem, ctas, s);
        case 19:
            if constexpr (MODE != RES_ADJOINT) return launch_one<R, MODE, 19, MANY>(q, smem, ctas, s);
            return cudaErrorInvalidValue;
        default: return cudaErrorInvalidValue;
    }
}

template <int R, int MODE>
cudaError_t launch_rb(int rb, const ResArgs& q, size_t smem, int ctas, cudaStream_t s) {
    return q.a.inj_np > RES_PTS + RES_WALK ? launch_points<R, MODE, true>(rb, q, smem, ctas, s)
                                : launch_points<R, MODE, false>(rb, q, smem, ctas, s);
}

}  // namespace res
}  // namespace wfd
