// Kernels on the packed scene for node records with 12 child slots: many scenes.
#include "pool_launch.cuh"

namespace bvhgpu {
namespace dev {
template <> cudaError_t launch_many_scenes<12>(ManyScenes& p, const PackedCfg& c, cudaStream_t s) {
  return launch_packed_width<12>(p, c, s);
}
}  // namespace dev
}  // namespace bvhgpu
