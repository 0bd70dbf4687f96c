// The resident 2D kernel at order 4 (stencil2d_res.cuh).
#include "stencil2d_res.cuh"

namespace wfd {
cudaError_t launch_resident_r2(ResMode mode, int rb, const ResArgs& q, size_t smem, int ctas, cudaStream_t s) {
    switch (mode) {
        case RES_LEAP: return res::launch_rb<2, RES_LEAP>(rb, q, smem, ctas, s);
        case RES_SUMMED: return res::launch_rb<2, RES_SUMMED>(rb, q, smem, ctas, s);
        case RES_SUMMED_DIFF: return res::launch_rb<2, RES_SUMMED_DIFF>(rb, q, smem, ctas, s);
        case RES_ADJOINT: return res::launch_rb<2, RES_ADJOINT>(rb, q, smem, ctas, s);
        default: return cudaErrorInvalidValue;
    }
}
}  // namespace wfd
