// Rooted product kernels of the shapes in SG_BLK_SHAPES_E.
#include "rooted_ema.cuh"

namespace sg {
namespace rt {

bool launch_ema_e(const EmaArgs &a, size_t smem, cudaStream_t st)
{
#define SG_EMA_LAUNCH(NN, PP) \
    if (a.blk_shape == blk::shape_id(NN, PP)) { launch_ema_shape<NN, PP>(a, smem, st); return true; }
    SG_BLK_SHAPES_E(SG_EMA_LAUNCH)
#undef SG_EMA_LAUNCH
    return false;
}

}  // namespace rt
}  // namespace sg
