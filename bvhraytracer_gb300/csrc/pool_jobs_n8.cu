// Kernels on the packed scene for node records with 8 child slots: many scenes.
#include "pool_launch.cuh"

namespace bvhgpu {
namespace dev {
template <> cudaError_t launch_many_scenes<8>(ManyScenes& p, const PackedCfg& c, cudaStream_t s) {
  return launch_packed_width<8>(p, c, s);
}
}  // namespace dev
}  // namespace bvhgpu
