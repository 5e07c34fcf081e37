// Kernels on the packed scene for node records with 12 child slots: one scene.
#include "pool_launch.cuh"

namespace bvhgpu {
namespace dev {
template <> cudaError_t launch_one_scene<12>(OneScene& p, const PackedCfg& c, cudaStream_t s) {
  return launch_packed_width<12>(p, c, s);
}
template <> cudaError_t load_one_scene<12>(const PackedCfg& c) { return load_width<12>(c); }
template <> cudaError_t launch_counting<12>(OneScene& p, TraceArgs a, const PackedCfg& c, cudaStream_t s) {
  return launch_count_width<12>(p, a, c, s);
}
}  // namespace dev
}  // namespace bvhgpu
