#include "rooted_gather.cuh"

namespace sg {
namespace rt {

void launch_gather_f32(const GatherArgs &a, int sm_count, cudaStream_t st) { launch_gather_t<float>(a, sm_count, st); }

}  // namespace rt
}  // namespace sg
