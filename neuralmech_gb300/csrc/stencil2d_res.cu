// Plans and launches of the resident 2D kernel (stencil2d_res.cuh). Host code.
#include <algorithm>

#include "common.cuh"
#include "internal.h"

namespace wfd {

cudaError_t launch_resident_r1(ResMode, int, const ResArgs&, size_t, int, cudaStream_t);
cudaError_t launch_resident_r2(ResMode, int, const ResArgs&, size_t, int, cudaStream_t);
cudaError_t launch_resident_r4(ResMode, int, const ResArgs&, size_t, int, cudaStream_t);

namespace {
// A split's time per step, in microseconds: a latency of 2.2 (halo packets through
// L2: about 1; two barriers; the send) plus the rows of a warp times what one row
// costs at n warps per scheduler. It orders the splits by their rows and warps; as a time
// it is high, most of all at orders 2 and 4, so that some grids stream which would be
// faster resident, and none the other way round. us a step, estimate / measured, order 8
// (order 2): 256^2 2.45 / 1.56 (1.27); 1024^2 3.6 / 2.6 (1.9); 2040^2 7.8 / 6.3 (5.5); 24 shots of 401 x 1203
// 25.3 / 19.3 (14.2); 6 of 700^2 7.8 / 6.7 (5.7). The adjoint reads L u from HBM and sums
// the gradient.
double step_us(int rb, int warps, bool adjoint) {
    static const double row[5] = {0.0, 0.125, 0.2, 0.295, 0.5};
    const double t = rb * row[(warps + 3) / 4];
    return adjoint ? 2.5 + 1.3 * t : 2.2 + t;
}
}  // namespace

bool plan_resident(int nz, int nx, int R, int nshot, ResMode mode, ResPlan* out) {
    const bool adj = mode == RES_ADJOINT;
    const int tiles_x = (nx + RES_TX - 1) / RES_TX;
    ResPlan best;
    for (const int rb : {2, 4, 7, 10, 14, 19}) {
        if (adj && (rb == 10 || rb == 19)) continue;
        const int warps = res_threads(mode, rb) / 32;
        for (int nwg = 4; nwg <= warps; ++nwg)
            for (int ng = 1; ng * nwg <= warps; ++ng)
                for (int share = 0; share <= (ng > 1 ? 1 : 0); ++share) {
                    ResPlan p;
                    p.rb = rb;
                    p.nwg = nwg;
                    p.ng = ng;
                    p.share_m = share;
                    p.tz = rb * nwg;
                    p.tiles_x = tiles_x;
                    p.tiles_z = (nz + p.tz - 1) / p.tz;
                    const long long nt = (long long)p.tiles_z * tiles_x;
                    if (nt > (long long)RES_SMS * ng) continue;
                    p.ntiles = int(nt);
                    p.shots = std::min(nshot, share ? RES_SMS / p.ntiles * ng : RES_SMS * ng / p.ntiles);
                    if (p.shots < 1) continue;
                    const size_t u = size_t(RES_TX + 8) * (p.tz + 2 * R) * 4, rest = res_group_bytes(nwg, p.tz);
                    bool fits = false;
                    for (int lm = 0; lm <= res_l2_rows(rb) && !fits; ++lm) {
                        p.lm = lm;
                        p.smem = 128 + ng * (u + rest) + (share ? 1 : ng) * size_t(RES_TX) * nwg * (rb - lm) * 4;
                        fits = p.smem <= size_t(RES_SMEM);
                    }
                    if (!fits) continue;
                    p.mail_bytes = size_t(2) * 16 * (2 * R * 64 + 4 * p.tz) * p.ntiles * p.shots;
                    p.passes = (nshot + p.shots - 1) / p.shots;
                    p.step_us = p.passes * step_us(rb, ng * nwg, adj);
                    if (best.rb == 0 || p.step_us < best.step_us) best = p;
                }
    }
    if (best.rb == 0) return false;
    *out = best;
    return true;
}

cudaError_t launch_resident(int R, ResMode mode, const ResPlan& plan, const ResArgs& q_in, cudaStream_t s) {
    ResArgs q = q_in;
    q.a = with_weight_pairs(q_in.a);
    q.nwg = plan.nwg;
    q.ng = plan.ng;
    q.lm = plan.lm;
    q.share_m = plan.share_m;
    q.tz = plan.tz;
    q.ntiles = plan.ntiles;
    const int ctas = plan.ctas(q.nshots);
    switch (R) {
        case 1: return launch_resident_r1(mode, plan.rb, q, plan.smem, ctas, s);
        case 2: return launch_resident_r2(mode, plan.rb, q, plan.smem, ctas, s);
        case 4: return launch_resident_r4(mode, plan.rb, q, plan.smem, ctas, s);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace wfd
