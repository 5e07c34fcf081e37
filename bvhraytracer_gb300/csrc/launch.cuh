// Host-side launch helpers: pick the kernel instance for a trace request.
#pragma once
#include <cuda_runtime.h>

#include "pool.cuh"
#include "traverse.cuh"

namespace bvhgpu {
namespace dev {

struct LaunchCfg {
  int kind = BVHGPU_CLOSEST;
  int scheme = BVHGPU_PER_RAY;
  int profile = BVHGPU_PROFILE_INSTRUMENTED;
  bool count = false;
  int block = 128;      // per-ray scheme threads per block
  int packet = 256;     // stream scheme rays per block
  int policy = 0;       // persistent scheme: 0 while-while, 1 if-if, 2 speculative any-hit,
                        // 3 the same with two leaves per lane, 4 as 3 with the leaves
                        // tested warp-wide
  int refill_min = 8;   // persistent scheme: idle lanes that trigger a refill
  unsigned long long* queue = nullptr;  // persistent scheme: queue head
  bool queue_cleared = false;  // true: the caller zeroed the head already
  // Packed scene: two words of device memory for this launch alone (null: it
  // may take them from the stream, see launch_pool).
  unsigned long long* pool_queue = nullptr;
  int sm_count = 152;
  int fmt = BVHGPU_NODES_FP32;  // node record format of the scene
  uint32_t top_nodes = 0;       // persistent scheme: inner records staged in shared memory
  uint32_t stall_bytes = 0;     // failure-detection tests (see bvhgpu_scene_inject_stall)
  bool save_distance = false;   // per-ray scheme: save-distance traversal (closest hits)
  int reorder = 0;              // > 0: group rays into 6 reorder^2 direction bins first
  bool stack_local = false;     // per-ray scheme: stacks in local memory (cap <= kLocalStack)
  bool any_order = false;       // any-hit rays without counters: child-index push order
};

constexpr int kLocalStack = 64;  // entries of the local-memory stack variant

template <typename K>
inline cudaError_t set_smem(K kernel, size_t bytes) {
  if (bytes <= 48 * 1024) return cudaSuccess;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

// Room for the block's visit histogram after `smem` bytes, if it is wanted and
// fits (else the kernel counts in global memory).
inline size_t add_block_hist(TraceArgs& a, bool count, size_t smem) {
  const size_t bytes = kHistBins * sizeof(uint32_t);
  a.block_hist = count && a.depth_hist != nullptr && smem + bytes <= 227 * 1024;
  return a.block_hist ? smem + bytes : smem;
}

template <int NM, int PROFILE, int KIND, bool COUNT, int FMT>
inline cudaError_t launch_one(const SceneDev& sc, TraceArgs a, const LaunchCfg& cfg,
                              cudaStream_t s) {
  if (a.n == 0) return cudaSuccess;
  if (cfg.scheme == BVHGPU_PER_RAY) {
    const int bs = cfg.block;
    // Any-hit rays never lower tMax, so a pushed entry (t0 <= t1 <= tMax) is
    // never dropped: save-distance any-hit traversal is the plain one.
    constexpr bool kDist = KIND == BVHGPU_CLOSEST;
    const bool dist = kDist && cfg.save_distance;
    const bool local = cfg.stack_local && !dist && !COUNT && a.stack_cap <= kLocalStack;
    const size_t smem =
        local ? 0 : add_block_hist(a, COUNT, (size_t)a.stack_cap * bs * 4 * (dist ? 2 : 1));
    auto k = dist ? trace_dfs_kernel<NM, PROFILE, KIND, COUNT, FMT, kDist>
             : local ? trace_dfs_kernel<NM, PROFILE, KIND, COUNT, FMT, false, (COUNT ? 0 : kLocalStack)>
                     : trace_dfs_kernel<NM, PROFILE, KIND, COUNT, FMT, false>;
    cudaError_t e = set_smem(k, smem);
    if (e != cudaSuccess) return e;
    const uint64_t grid = (a.n + bs - 1) / bs;
    k<<<(unsigned)grid, bs, smem, s>>>(sc, a);
  } else if (cfg.scheme == BVHGPU_PERSISTENT) {
    const int bs = 128;
    // Policies 2 to 4 change the order of leaf tests, which only any-hit
    // rays without counters may do; the others fall back to policy 0.
    constexpr bool kSpec = KIND == BVHGPU_ANY && !COUNT;
    const bool coop = cfg.policy == 4 && kSpec;
    const size_t smem = (size_t)a.stack_cap * bs * 4 +
                        ((size_t)cfg.top_nodes * NodeFmt<NM, FMT>::REC + 15) / 16 * 16 +
                        (coop ? (size_t)bs * kRayRecWords * 4 : 0);
    auto k = cfg.policy == 1 ? trace_persistent_kernel<NM, PROFILE, KIND, COUNT, 1, FMT>
             : (cfg.policy == 2 && kSpec)
                 ? trace_persistent_kernel<NM, PROFILE, KIND, COUNT, (kSpec ? 2 : 0), FMT>
             : (cfg.policy == 3 && kSpec)
                 ? trace_persistent_kernel<NM, PROFILE, KIND, COUNT, (kSpec ? 3 : 0), FMT>
             : coop ? trace_persistent_kernel<NM, PROFILE, KIND, COUNT, (kSpec ? 4 : 0), FMT>
                    : trace_persistent_kernel<NM, PROFILE, KIND, COUNT, 0, FMT>;
    cudaError_t e = set_smem(k, smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, bs, smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) per_sm = 1;
    uint64_t grid = (uint64_t)per_sm * cfg.sm_count;
    const uint64_t need = (a.n + bs - 1) / bs;
    if (grid > need) grid = need;
    QueueArgs q{cfg.queue, cfg.refill_min, cfg.top_nodes, cfg.top_nodes ? cfg.stall_bytes : 0u};
    if (!cfg.queue_cleared) {
      e = cudaMemsetAsync(cfg.queue, 0, sizeof(unsigned long long), s);
      if (e != cudaSuccess) return e;
    }
    k<<<(unsigned)grid, bs, smem, s>>>(sc, a, q);
  } else {
    if (FMT != kFmtFP32) return cudaErrorNotSupported;
    const int p = cfg.packet;
    const size_t smem = add_block_hist(
        a, COUNT, stream_smem_bytes(p, a.stack_cap, COUNT, COUNT && a.step_stats));
    auto k = trace_stream_kernel<NM, PROFILE, KIND, COUNT>;
    cudaError_t e = set_smem(k, smem);
    if (e != cudaSuccess) return e;
    const uint64_t grid = (a.n + p - 1) / p;
    k<<<(unsigned)grid, p, smem, s>>>(sc, a);
  }
  return cudaGetLastError();
}

template <int NM, int PROFILE, int KIND, bool COUNT>
inline cudaError_t launch_fmt(const SceneDev& sc, const TraceArgs& a, const LaunchCfg& c,
                              cudaStream_t s) {
  if (c.fmt == kFmtQ8) return launch_one<NM, PROFILE, KIND, COUNT, kFmtQ8>(sc, a, c, s);
  return launch_one<NM, PROFILE, KIND, COUNT, kFmtFP32>(sc, a, c, s);
}

template <int NM>
inline cudaError_t launch_for_width(const SceneDev& sc, const TraceArgs& a, const LaunchCfg& c,
                                    cudaStream_t s) {
  const int code = (c.profile << 2) | (c.kind << 1) | (c.count ? 1 : 0);
  switch (code) {
    case 0: return launch_fmt<NM, 0, 0, false>(sc, a, c, s);
    case 1: return launch_fmt<NM, 0, 0, true>(sc, a, c, s);
    case 2: return launch_fmt<NM, 0, 1, false>(sc, a, c, s);
    case 3: return launch_fmt<NM, 0, 1, true>(sc, a, c, s);
    case 4: return launch_fmt<NM, 1, 0, false>(sc, a, c, s);
    case 5: return launch_fmt<NM, 1, 0, true>(sc, a, c, s);
    case 6: return launch_fmt<NM, 1, 1, false>(sc, a, c, s);
    case 7: return launch_fmt<NM, 1, 1, true>(sc, a, c, s);
  }
  return cudaErrorInvalidValue;
}

// Shared memory of an SM that the pools may take; the rest of its 256 KB is
// L1, which the node records need.
#ifndef BVHGPU_POOL_SMEM
#define BVHGPU_POOL_SMEM (196 * 1024)
#endif
// Rays per resident warp from which a warp takes kPoolRays rays at once.
#ifndef BVHGPU_POOL_FULL
#define BVHGPU_POOL_FULL 48
#endif
// Batches of more rays may run on the pool kernel. Solo / pool, us: unordered
// ambient-occlusion rays (N8L8, 251k triangles) 131k rays 110 / 115, 262k
// 172 / 146, 1M 558 / 365, 4.2M 1953 / 1134; primary rays, which stay
// together, 262k 124 / 148, 1M 253 / 290. The lines cross at about 200k rays
// for rays that part and nowhere for rays that do not.
#ifndef BVHGPU_POOL_MIN_RAYS
#define BVHGPU_POOL_MIN_RAYS (1u << 18)
#endif
inline bool pool_wants_queue(uint64_t n) { return n > BVHGPU_POOL_MIN_RAYS; }
constexpr int kSoloBlock = 64;

template <int NM, int PROFILE, int KIND, int FMT, bool ORDERED>
inline cudaError_t launch_packed(PoolArgs& p, const LaunchCfg& cfg, cudaStream_t s) {
  cudaError_t e;
  const bool large = pool_wants_queue(p.n) && p.queue != nullptr;
  // Rays in direction order are for the pool; otherwise the rays themselves
  // decide.
  const bool pool = large && p.out_index != nullptr;
  p.planned = large && !pool;
  if (p.planned) {
    plan_kernel<<<1, kPlanWarps * 32, 0, s>>>(p.rays, p.n, p.queue);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  }
  if (!pool) {
    auto k = trace_solo_kernel<NM, PROFILE, KIND, FMT, ORDERED>;
    const size_t smem = sizeof(typename PoolWord<NM>::T) * p.levels * kSoloBlock;
    const uint64_t grid = ((uint64_t)p.n + kSoloBlock - 1) / kSoloBlock;
    k<<<(unsigned)grid, kSoloBlock, smem, s>>>(p);
    if ((e = cudaGetLastError()) != cudaSuccess || !large) return e;
  }
  auto k = trace_pool_kernel<NM, PROFILE, KIND, FMT, ORDERED>;
  const size_t smem = kPoolWarps * pool_warp_bytes<NM>(p.levels);
  if ((e = set_smem(k, smem)) != cudaSuccess) return e;
  // Resident warps; blocks past them would find the queue empty.
  const size_t fit = BVHGPU_POOL_SMEM / smem;
  const uint64_t per_sm = fit < 1 ? 1 : fit > BVHGPU_POOL_MIN_BLOCKS ? BVHGPU_POOL_MIN_BLOCKS : fit;
  const uint64_t warps = (uint64_t)cfg.sm_count * per_sm * kPoolWarps;
  p.slots = p.n >= warps * BVHGPU_POOL_FULL ? kPoolRays : 32;
  const uint64_t need = ((uint64_t)p.n + kPoolWarps * 32 - 1) / (kPoolWarps * 32);
  const uint64_t grid = need < warps / kPoolWarps ? need : warps / kPoolWarps;
  if (!p.planned) {
    e = cudaMemsetAsync(p.queue, 0, sizeof(unsigned long long), s);
    if (e != cudaSuccess) return e;
  }
  k<<<(unsigned)grid, kPoolWarps * 32, smem, s>>>(p);
  return cudaGetLastError();
}

template <int NM, int FMT>
inline cudaError_t launch_pool_fmt(PoolArgs& p, const LaunchCfg& c, cudaStream_t s) {
  constexpr int F = BVHGPU_PROFILE_FAST, I = BVHGPU_PROFILE_INSTRUMENTED;
  if (c.kind == BVHGPU_CLOSEST)
    return c.profile == F ? launch_packed<NM, F, BVHGPU_CLOSEST, FMT, true>(p, c, s)
                          : launch_packed<NM, I, BVHGPU_CLOSEST, FMT, true>(p, c, s);
  if (c.profile == F) return launch_packed<NM, F, BVHGPU_ANY, FMT, false>(p, c, s);
  return c.any_order ? launch_packed<NM, I, BVHGPU_ANY, FMT, false>(p, c, s)
                     : launch_packed<NM, I, BVHGPU_ANY, FMT, true>(p, c, s);
}

template <int NM>
inline cudaError_t launch_pool_for_width(PoolArgs p, const LaunchCfg& c, cudaStream_t s) {
  if (p.n == 0) return cudaSuccess;
  return c.fmt == kFmtQ8 ? launch_pool_fmt<NM, kFmtQ8>(p, c, s)
                         : launch_pool_fmt<NM, kFmtFP32>(p, c, s);
}

cudaError_t launch_pool_n4(const PoolArgs&, const LaunchCfg&, cudaStream_t);
cudaError_t launch_pool_n8(const PoolArgs&, const LaunchCfg&, cudaStream_t);
cudaError_t launch_pool_n12(const PoolArgs&, const LaunchCfg&, cudaStream_t);
cudaError_t launch_pool_n16(const PoolArgs&, const LaunchCfg&, cudaStream_t);
cudaError_t launch_trace_n4(const SceneDev&, const TraceArgs&, const LaunchCfg&, cudaStream_t);
cudaError_t launch_trace_n8(const SceneDev&, const TraceArgs&, const LaunchCfg&, cudaStream_t);
cudaError_t launch_trace_n12(const SceneDev&, const TraceArgs&, const LaunchCfg&, cudaStream_t);
cudaError_t launch_trace_n16(const SceneDev&, const TraceArgs&, const LaunchCfg&, cudaStream_t);

}  // namespace dev
}  // namespace bvhgpu
