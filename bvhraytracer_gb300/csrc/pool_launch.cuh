// Host-side launch of the kernels on the packed scene (pool.cuh).
#pragma once
#include <cuda_runtime.h>

#include "pool.cuh"
#include "smem_limit.cuh"

namespace bvhgpu {
namespace dev {

// What a launch's rays have in common.
struct PackedCfg {
  int nm, fmt;  // node width and format
  int kind, profile;
  bool any_order;        // any-hit rays push in child-index order
  bool direction_order;  // the rays are sorted by direction
  int sm_count;
  uint64_t node_bytes;   // packed node records of the scenes together
};

// Width NM of one scene or many (pool_n*.cu, pool_jobs_n*.cu).
template <int NM> cudaError_t launch_one_scene(OneScene& p, const PackedCfg& c, cudaStream_t s);
template <int NM> cudaError_t launch_many_scenes(ManyScenes& p, const PackedCfg& c, cudaStream_t s);
// Loads the code of every kernel that launch_one_scene may choose for a ray
// kind, profile and format, whatever the batch's size and push order.
template <int NM> cudaError_t load_one_scene(const PackedCfg& c);
// The counting kernel for the rays of p, counters and histograms as in a.
template <int NM> cudaError_t launch_counting(OneScene& p, TraceArgs a, const PackedCfg& c, cudaStream_t s);

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
// FP32 nodes of more than 8 children in trees of more than so many bytes of
// records: unordered rays have a thread each at every batch size. A pool's 56
// rays are at as many nodes, 288 or 384 bytes of boxes each, and eight pools per SM
// leave the L1 too little room for them. Closest-hit rays on 251k triangles, 2M
// unordered, pool / solo, us: N12L8 (6.6 MB) 2694 / 1670, N16L4 (12 MB) 2013 / 1631,
// N16L1 (43 MB) 3483 / 1811, but N16L8 (4.9 MB) 1578 / 1641, N16L16 (3.5 MB) 1744 /
// 1849; N8L4 (7.5 MB) 1119 / 1421, N8L8 of 1M triangles (17 MB), 3.5M rays, 2496 / 2870;
// N12L8 with Q8 records 2760 / 4057.
constexpr uint64_t kPoolWideBytes = 5u << 20;
inline bool pool_wants_queue(const PackedCfg& c, uint64_t n) {
  return n > BVHGPU_POOL_MIN_RAYS && (c.direction_order || c.nm <= 8 || c.fmt != kFmtFP32 ||
                                      c.node_bytes <= kPoolWideBytes);
}
// Whether counting traces of n rays run on the packed scene. Smaller batches,
// whose time is the longest ray's, are faster in the general per-ray kernel, and so
// are all on Q8 nodes of more than 8 children. General / packed time, least and
// median over primary, shadow and random rays, 251k and 33k triangles, two leaf
// sizes, with histograms and without: FP32 1k rays 0.85 (median), 30k 0.90, 130k
// 0.87 1.01, 250k N4 1.08 1.12, N8 1.02 1.12, N12 0.94 1.03, N16 0.95 1.06, 1M 1.02
// 1.25; Q8 250k N4 1.03 1.11, N8 0.92 1.06, N12 0.88 0.98, N16 0.81 0.93, 1M N16 0.88
// 1.00.
constexpr uint64_t kCountRays = 3u << 16;
inline bool pool_counts(int nm, int fmt, uint64_t n) {
  return n > kCountRays && (fmt == kFmtFP32 || nm <= 8);
}
constexpr int kSoloBlock = 64;
// Batches of up to so many rays run with a team of lanes per ray (closest-hit /
// any-hit). Solo / team, us, of a call from Python, which itself takes 15-17
// (251k triangles): N8 primary rays 1k 25 / 25, 4k 60 / 36, 16k 58 / 43, 33k
// 60 / 61; N8 ambient-occlusion rays 1k 46 / 21, 4k 47 / 24, 16k 56 / 39, 33k
// 82 / 60, 66k 84 / 82; N16 primary rays 16k 57 / 41, 33k 59 / 76, any-hit rays
// 16k 61 / 37, 33k 86 / 61, 66k 97 / 91. Closest-hit rays, solo / team time, least
// and median over primary and random rays, 251k and 33k triangles, leaf sizes 1, 4
// and 8, both formats: 28k rays N4 0.74 0.93, N8 0.89 1.12, N12 0.89 1.10, N16 1.06
// 1.30; 33k N8 0.81 1.08, N12 0.79 1.07, N16 0.87 1.20; 18k N4 0.80 0.93.
template <int NM>
constexpr uint32_t kTeamMaxClosest = NM <= 4 ? 16384 : NM <= 12 ? 28672 : 32768;
#ifndef BVHGPU_TEAM_MAX_ANY
#define BVHGPU_TEAM_MAX_ANY 32768
#endif
// Warps per SM that the teams are spread over (N16 ambient-occlusion rays, 4k:
// 16 warps 25.6 us, 32 24.3; N4 8k 47.0 / 42.5).
#ifndef BVHGPU_TEAM_WARPS
#define BVHGPU_TEAM_WARPS 32
#endif
constexpr int kTeamBlock = 64;

// Batches of up to so many blocks' rays per SM run in the solo kernel of one wave,
// also those that need a little more than one (four blocks, 78k rays). The other
// solo kernel's time / its, least and median over primary and random rays: 80k
// rays N4 0.99 1.10, N8 0.97 1.04, FP32 N16 closest-hit 0.86 1.01, Q8 0.83 0.97;
// 100k N4 0.99 1.09, N8 0.82 1.01, N16 0.81 0.94; 131k N4 0.83 1.03, N8 0.80 0.99.
template <int NM, int KIND, int FMT>
constexpr int kFewLimit = NM <= 4 ? 6 : NM <= 8 || (KIND == BVHGPU_CLOSEST && FMT == kFmtFP32) ? 5 : 4;

// The traces of one launch: a team per ray, one thread per ray, pools, or both
// of these with the rays' own choice between them.
template <int NM, int PROFILE, int KIND, int FMT, bool ORDERED, typename SRC>
inline cudaError_t launch_packed(SRC& p, const PackedCfg& c, cudaStream_t s) {
  const int sm_count = c.sm_count;
  cudaError_t e;
  if (p.n <= (KIND == BVHGPU_ANY ? BVHGPU_TEAM_MAX_ANY : kTeamMaxClosest<NM>)) {
    auto k = trace_team_kernel<NM, PROFILE, KIND, FMT, ORDERED, SRC>;
    constexpr int kMost = 32 / kTeam<NM>;
    // As few rays per warp as keep the warps resident.
    const uint64_t warps = (uint64_t)sm_count * BVHGPU_TEAM_WARPS;
    const uint64_t per = (p.n + warps - 1) / warps;
    p.slots = per > kMost ? kMost : (int)per;
    const uint64_t need = (p.n + p.slots - 1) / p.slots;
    const size_t smem = sizeof(typename PoolWord<NM>::T) * p.levels * kTeamBlock;
    k<<<(unsigned)((need * 32 + kTeamBlock - 1) / kTeamBlock), kTeamBlock, smem, s>>>(p);
    return cudaGetLastError();
  }
  const bool large = pool_wants_queue(c, p.n) && p.queue != nullptr;
  // Rays in direction order are for the pool; otherwise the rays themselves
  // decide.
  const bool pool = large && c.direction_order;
  p.planned = large && !pool;
  if (p.planned) {
    plan_kernel<SRC><<<1, kPlanWarps * 32, 0, s>>>(p);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  }
  if (!pool) {
    auto k = p.n <= (uint64_t)sm_count * kFewLimit<NM, KIND, FMT> * 128
                 ? trace_solo_kernel<NM, PROFILE, KIND, FMT, ORDERED, true, SRC>
                 : trace_solo_kernel<NM, PROFILE, KIND, FMT, ORDERED, false, SRC>;
    // A planned launch takes blocks of twice the size: if the pool is chosen,
    // its blocks only start and return (half as many: a 1001 x 563 frame with 8
    // random rays per hit 1.54 -> 1.52 ms), and if not, fewer starts are as good
    // (2.1M primary rays on 251k triangles, N8 0.442 -> 0.437 ms, shadow rays
    // 0.337 -> 0.335).
    // Blocks of 256 hold their slots until the last warp ends: 0.449 and 0.347.
    // Closest-hit rays take them at every size (251k triangles, N8, 131k rays 89
    // -> 84 us; 32k triangles, N4, 262k rays 65 -> 62; 251k, N16, 262k 146 ->
    // 145), any-hit rays, which end sooner and less evenly, lose by it (N8 131k
    // rays 57 -> 60, N4 262k 90 -> 92).
    const int block = p.planned || KIND == BVHGPU_CLOSEST ? 2 * kSoloBlock : kSoloBlock;
    const size_t smem = sizeof(typename PoolWord<NM>::T) * p.levels * block;
    const uint64_t grid = (p.n + block - 1) / block;
    k<<<(unsigned)grid, block, smem, s>>>(p);
    if ((e = cudaGetLastError()) != cudaSuccess || !large) return e;
  }
  auto k = trace_pool_kernel<NM, PROFILE, KIND, FMT, ORDERED, SRC>;
  const size_t smem = kPoolWarps * pool_warp_bytes<NM>(p.levels);
  if ((e = allow_smem(k, smem)) != cudaSuccess) return e;
  // Resident warps; blocks past them would find the queue empty.
  const size_t fit = BVHGPU_POOL_SMEM / smem;
  const uint64_t per_sm = fit < 1 ? 1 : fit > BVHGPU_POOL_MIN_BLOCKS ? BVHGPU_POOL_MIN_BLOCKS : fit;
  const uint64_t warps = (uint64_t)sm_count * per_sm * kPoolWarps;
  p.slots = p.n >= warps * BVHGPU_POOL_FULL ? kPoolRays : 32;
  const uint64_t need = (p.n + kPoolWarps * 32 - 1) / (kPoolWarps * 32);
  const uint64_t grid = need < warps / kPoolWarps ? need : warps / kPoolWarps;
  if (!p.planned) {
    e = cudaMemsetAsync(p.queue, 0, sizeof(unsigned long long), s);
    if (e != cudaSuccess) return e;
  }
  k<<<(unsigned)grid, kPoolWarps * 32, smem, s>>>(p);
  return cudaGetLastError();
}

template <int NM, int FMT, typename SRC>
inline cudaError_t launch_packed_fmt(SRC& p, const PackedCfg& c, cudaStream_t s) {
  constexpr int F = BVHGPU_PROFILE_FAST, I = BVHGPU_PROFILE_INSTRUMENTED;
  constexpr int C = BVHGPU_CLOSEST, A = BVHGPU_ANY;
  if (c.kind == C)
    return c.profile == F ? launch_packed<NM, F, C, FMT, true>(p, c, s)
                          : launch_packed<NM, I, C, FMT, true>(p, c, s);
  // Any-hit rays of the fast profile push in child-index order always.
  if (c.profile == F) return launch_packed<NM, F, A, FMT, false>(p, c, s);
  return c.any_order ? launch_packed<NM, I, A, FMT, false>(p, c, s)
                     : launch_packed<NM, I, A, FMT, true>(p, c, s);
}

// A kernel's code is loaded when its attributes are first asked for.
template <typename K>
inline void load_kernel(K kernel, cudaError_t& e) {
  cudaFuncAttributes a;
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, kernel);
}
template <int NM, int PROFILE, int KIND, int FMT, bool ORDERED>
inline void load_order(cudaError_t& e) {
  load_kernel(trace_team_kernel<NM, PROFILE, KIND, FMT, ORDERED, OneScene>, e);
  load_kernel(trace_solo_kernel<NM, PROFILE, KIND, FMT, ORDERED, true, OneScene>, e);
  load_kernel(trace_solo_kernel<NM, PROFILE, KIND, FMT, ORDERED, false, OneScene>, e);
  load_kernel(trace_pool_kernel<NM, PROFILE, KIND, FMT, ORDERED, OneScene>, e);
}
template <int NM, int FMT>
inline cudaError_t load_fmt(const PackedCfg& c) {
  constexpr int F = BVHGPU_PROFILE_FAST, I = BVHGPU_PROFILE_INSTRUMENTED;
  constexpr int C = BVHGPU_CLOSEST, A = BVHGPU_ANY;
  cudaError_t e = cudaSuccess;
  load_kernel(plan_kernel<OneScene>, e);
  if (c.kind == C) {
    if (c.profile == F) load_order<NM, F, C, FMT, true>(e);
    else load_order<NM, I, C, FMT, true>(e);
  } else if (c.profile == F) {
    load_order<NM, F, A, FMT, false>(e);
  } else {
    load_order<NM, I, A, FMT, true>(e);
    load_order<NM, I, A, FMT, false>(e);
  }
  return e;
}
template <int NM>
inline cudaError_t load_width(const PackedCfg& c) {
  return c.fmt == kFmtQ8 ? load_fmt<NM, kFmtQ8>(c) : load_fmt<NM, kFmtFP32>(c);
}

template <int NM, int KIND, int FMT>
inline cudaError_t launch_count(OneScene& p, TraceArgs& a, cudaStream_t s) {
  constexpr int kBlock = 128;  // 64: 329 us against 326
  size_t smem = sizeof(typename PoolWord<NM>::T) * p.levels * kBlock;
  if (a.block_hist && a.depth_hist != nullptr) {
    a.hist_at = (uint32_t)(smem / 4);
    smem += kHistBins * sizeof(uint32_t);
  }
  auto k = trace_count_kernel<NM, KIND, FMT>;
  const cudaError_t e = allow_smem(k, smem);
  if (e != cudaSuccess) return e;
  k<<<(unsigned)((p.n + kBlock - 1) / kBlock), kBlock, smem, s>>>(p, a);
  return cudaGetLastError();
}
template <int NM>
inline cudaError_t launch_count_width(OneScene& p, TraceArgs& a, const PackedCfg& c, cudaStream_t s) {
  if (p.n == 0) return cudaSuccess;
  if constexpr (NM <= 8) {
    if (c.fmt == kFmtQ8)
      return c.kind == BVHGPU_CLOSEST ? launch_count<NM, BVHGPU_CLOSEST, kFmtQ8>(p, a, s)
                                      : launch_count<NM, BVHGPU_ANY, kFmtQ8>(p, a, s);
  }
  if (c.fmt != kFmtFP32) return cudaErrorNotSupported;  // see pool_counts
  return c.kind == BVHGPU_CLOSEST ? launch_count<NM, BVHGPU_CLOSEST, kFmtFP32>(p, a, s)
                                  : launch_count<NM, BVHGPU_ANY, kFmtFP32>(p, a, s);
}

template <int NM, typename SRC>
inline cudaError_t launch_packed_width(SRC& p, const PackedCfg& c, cudaStream_t s) {
  if (p.n == 0) return cudaSuccess;
  return c.fmt == kFmtQ8 ? launch_packed_fmt<NM, kFmtQ8>(p, c, s)
                         : launch_packed_fmt<NM, kFmtFP32>(p, c, s);
}

}  // namespace dev
}  // namespace bvhgpu
