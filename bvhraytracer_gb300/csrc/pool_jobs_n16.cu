// Kernels on the packed scene for node records with 16 child slots: many scenes.
#include "pool_launch.cuh"

namespace bvhgpu {
namespace dev {
template <> cudaError_t launch_many_scenes<16>(ManyScenes& p, const PackedCfg& c, cudaStream_t s) {
  return launch_packed_width<16>(p, c, s);
}
}  // namespace dev
}  // namespace bvhgpu
