// Kernels on the packed scene for node records with 16 child slots: one scene.
#include "pool_launch.cuh"

namespace bvhgpu {
namespace dev {
template <> cudaError_t launch_one_scene<16>(OneScene& p, const PackedCfg& c, cudaStream_t s) {
  return launch_packed_width<16>(p, c, s);
}
template <> cudaError_t load_one_scene<16>(const PackedCfg& c) { return load_width<16>(c); }
template <> cudaError_t launch_counting<16>(OneScene& p, TraceArgs a, const PackedCfg& c, cudaStream_t s) {
  return launch_count_width<16>(p, a, c, s);
}
}  // namespace dev
}  // namespace bvhgpu
