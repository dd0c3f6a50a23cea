// gr_batch_classes.cu -- the batched trace grids specialised by scene class: clear
// isotropic stones and the general (birefringent or absorbing) ones, each per
// environment kind, as the single-scene kernels are (gr_single_clear.cu,
// gr_single_general.cu).  A batched launch holds segments of one class only.
#include "gr_batch.cuh"
#include "gr_ctx.h"

// Resident blocks per SM (in blocks of 128 threads) of the class-specialised batched grids:
// 64 random stones of 16 to 64 pixels a side, 9 / 12 / 16 blocks: 28.3 / 27.9 / 32.4 ms.  Class
// K_FULL, whose loops take all channels, at 9 where it is not clear and isotropic (16 absorbing
// stones of index 1.0002 at 48 x 48 and 32 spp, 9 / 12 blocks: 0.78 / 1.06 ms).
constexpr int kBatchBlocks = 12;

namespace grh {

gr_status launch_batch_class(int K, const grd::BatchLaunch &L, cudaStream_t s) {
    constexpr int IC = grd::K_ISO | grd::K_CLEAR;
#define GR_BATCH_CASE(KK)                                       \
    case KK:                                                    \
        grd::launch_batch_grids<false, KK, kBatchBlocks>(L, s); \
        break;
    switch (K) {
        GR_BATCH_CASE(IC | grd::k_env(GR_ENV_UNIFORM))
        GR_BATCH_CASE(IC | grd::k_env(GR_ENV_STUDIO))
        GR_BATCH_CASE(IC | grd::k_env(GR_ENV_LATLONG))
        GR_BATCH_CASE(grd::k_env(GR_ENV_UNIFORM))
        GR_BATCH_CASE(grd::k_env(GR_ENV_STUDIO))
        GR_BATCH_CASE(grd::k_env(GR_ENV_LATLONG))
        GR_BATCH_CASE(IC | grd::K_FULL)
    case grd::K_FULL: grd::launch_batch_grids<false, grd::K_FULL, GR_TRACE_MIN_BLOCKS>(L, s); break;
    default: return fail(GR_EINVAL, "scene class %d has no batched kernels", K);
    }
#undef GR_BATCH_CASE
    GR_CUDA(cudaGetLastError());
    return GR_OK;
}

}  // namespace grh
