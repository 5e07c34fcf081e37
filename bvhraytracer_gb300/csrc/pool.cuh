// Traces without counters, on the packed scene (pack.cuh): three kernels with
// the same node and leaf visits.
//
// trace_team_kernel: several lanes per ray, for small batches.
// trace_solo_kernel: one thread per ray. trace_pool_kernel: each warp owns a
// pool of kPoolRays rays in shared memory and three lists of them: rays whose
// next entry is an inner node, rays whose next entry is a leaf, and free
// slots. A step takes up to 32 rays of one list, so all lanes of the warp
// visit nodes, or all visit leaves, or all set up new rays from the launch's
// queue; the lists are kept by ballots, and no step needs a block barrier. A
// ray's own visits stay in depth-first order, so results are those of the
// scheme kernels in traverse.cuh (any-hit rays: occlusion does not depend on
// the order of their visits, tMax is fixed).
//
// A ray's stack holds one word per level instead of one entry per pushed
// child: the inner node and the set of its hit children still to visit (as
// positions in the ray's push sequence). Its depth is bounded by the tree's
// levels.
//
// What bounds them. Pool, ambient-occlusion rays in direction order (3.7M rays,
// 251k triangles, N8L8): the L1 data pipe is busy 82 % of the time (a node
// visit gathers 192 bytes of boxes, 40 of the 57 L1 cycles of a ray), issue
// 66 %; steps have 29 of 32 rays at nodes and 26 at leaves. 1.18 ms on the
// persistent kernel (17.4 lanes per instruction, a fifth of the L1 cycles lost
// to bank conflicts), 0.81 ms here; 8.3M such rays of the 1M-triangle frame
// 3.13 -> 2.04 ms; unordered, from the per-ray kernel (6.7 lanes), 4.5M rays,
// N4L8, 2.97 -> 1.33 ms. Solo, 2.1M primary rays of that frame 0.64 -> 0.46 ms,
// shadow rays 0.38 -> 0.24 ms: issue (70 %), latency and the longest rays (a
// third of the warps resident on average).
#pragma once
#include "pack.cuh"
#include "traverse.cuh"

namespace bvhgpu {
namespace dev {

// Rays per pool. More rays fill the steps better and take L1 from the node
// records (frame of the 1M-triangle scene / 4.5M unordered N4 rays: 48 rays
// 4.94 / 1.47 ms, 56 4.69 / 1.48, 64 4.74 / 1.58, 96 5.5 / 1.77).
#ifndef BVHGPU_POOL_RAYS
#define BVHGPU_POOL_RAYS 56
#endif
constexpr int kPoolRays = BVHGPU_POOL_RAYS;
constexpr int kPoolWarps = 4;  // per block
// Resident blocks per SM (64 registers per thread): same frame with 64 rays
// per pool, 8 blocks 4.80 ms, 7 4.95, 6 5.15, 5 5.4.
#ifndef BVHGPU_POOL_MIN_BLOCKS
#define BVHGPU_POOL_MIN_BLOCKS 8
#endif
// Free slots at which a warp takes new rays: a full step of them (same frame:
// 32 4.80 ms, 24 5.0, 16 5.15, 8 5.4).
#ifndef BVHGPU_POOL_REFILL
#define BVHGPU_POOL_REFILL 32
#endif

// Blocks of 128 threads per SM that the solo kernel's registers allow. Closest-hit
// rays, us: N8L8, primary rays of 12 scenes, 0.46M, 5 / 6 / 7 / 8 blocks 201 197
// 197 210, of one (251k triangles), 0.5M, 6 / 7 / 8 228 223 226; N16L8, 0.26M
// unordered, 6 / 7 285 255; N4L4, 131k unordered, 5 / 6 / 7 182 136 137. Q8 nodes,
// N8, 2.1M rays, ms, 4 / 6 / 7 / 8: primary 1.38 1.36 1.33 1.39, shadow 0.45 0.43
// 0.45 0.47.
template <int NM, int FMT>
constexpr int kSoloBlocks = NM > 4 && FMT == kFmtQ8 ? 6 : 7;
// The same for launches of no more rays than these blocks hold, or little more
// (FEW, kFewLimit): up to 128 registers. N16L8, 40k / 65k unordered closest-hit rays, us, 3 / 4 / 5 blocks: 92
// 96 98 / 112 105 108 (3 blocks hold 58k rays).
constexpr int kSoloFewBlocks = 4;

// PackView::leaves: no leaf has more than two triangles; none costs more than a
// node: no more triangles than child slots, or 8 with 4-wide Q8 nodes (see
// trace_solo_kernel).
constexpr int kSmallLeaves = 1, kLeavesInTurn = 2;

// What a ray's visits need of its scene, and where its result goes.
struct PackView {
  const uint8_t* nodes;  // packed node records (PackFmt)
  const float4* blocks;  // leaf blocks
  void* out;             // hits or occlusion bytes
  uint32_t root;         // stack entry of the root
  int16_t gang;
  int8_t nested;         // every box lies in its parent's, every triangle in its leaf's
  int8_t leaves;         // kSmallLeaves, kLeavesInTurn
};

// Common arguments of a launch.
struct PoolArgs {
  uint64_t n;   // rays
  int levels;   // inner levels of the deepest tree: words of a ray's stack
  // Two words of this launch's own: [0] next unclaimed ray of the pool kernel,
  // [1] the kernel chosen by plan_kernel. Null: one thread per ray.
  unsigned long long* queue;
  int planned;  // 1: a kernel other than the chosen one returns at once
  int slots;    // rays a warp takes at once (32 or kPoolRays)
};

// A batch of rays of one scene.
struct OneScene : PoolArgs {
  PackView scene;
  const bvhgpu_ray_t* rays;
  const uint32_t* out_index;  // as TraceArgs
  BVHGPU_DEV const PackView& view(uint32_t) const { return scene; }
  // The i-th ray of the launch, its result slot and its job.
  BVHGPU_DEV bvhgpu_ray_t ray(uint64_t i, uint32_t& slot, uint32_t& job) const {
    job = 0;
    slot = out_index ? __ldg(out_index + i) : (uint32_t)i;
    return load_ray(rays, slot);
  }
};

// Batches of several scenes, one after the other.
constexpr int kPoolMaxJobs = 192;
struct PoolJob {
  PackView scene;
  const bvhgpu_ray_t* rays;
  const uint32_t* out_index;
  uint64_t begin;  // the job's first ray in the launch
};
struct ManyScenes : PoolArgs {
  int n_jobs;
  PoolJob jobs[kPoolMaxJobs];
  BVHGPU_DEV const PackView& view(uint32_t job) const { return jobs[job].scene; }
  BVHGPU_DEV bvhgpu_ray_t ray(uint64_t i, uint32_t& slot, uint32_t& job) const {
    // The last job that begins at or before ray i.
    int lo = 0, hi = n_jobs - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (jobs[mid].begin <= i) lo = mid;
      else hi = mid - 1;
    }
    job = (uint32_t)lo;
    const PoolJob& J = jobs[lo];
    slot = (uint32_t)(i - J.begin);
    if (J.out_index) slot = __ldg(J.out_index + slot);
    return load_ray(J.rays, slot);
  }
};

// Which of the two kernels traces a batch.
constexpr unsigned long long kPlanSolo = 1, kPlanPool = 2;

// A level of a ray's stack: the node and the set of its children left, in one
// word for up to 8 children and 2^24 inner nodes.
template <int NM>
struct PoolWord {
  using T = uint32_t;
  static BVHGPU_DEV uint32_t make(uint32_t node, uint32_t left) { return node | (left << 24); }
  static BVHGPU_DEV uint32_t node(uint32_t w) { return w & 0xFFFFFFu; }
  static BVHGPU_DEV uint32_t left(uint32_t w) { return w >> 24; }
};
struct PoolWordWide {
  using T = uint2;
  static BVHGPU_DEV uint2 make(uint32_t node, uint32_t left) { return make_uint2(node, left); }
  static BVHGPU_DEV uint32_t node(const uint2& w) { return w.x; }
  static BVHGPU_DEV uint32_t left(const uint2& w) { return w.y; }
};
template <> struct PoolWord<12> : PoolWordWide {};
template <> struct PoolWord<16> : PoolWordWide {};
constexpr uint32_t pool_max_inner(int nm) { return nm <= 8 ? 1u << 24 : kLeafBit; }

// Shared memory of one warp: three float4 and a word pair per ray, the stacks
// and the lists.
template <int NM>
__host__ __device__ inline size_t pool_warp_bytes(int levels) {
  return (size_t)kPoolRays * (3 * 16 + 8 + sizeof(typename PoolWord<NM>::T) * (size_t)levels) +
         64 + (3 * kPoolRays + 15) / 16 * 16;
}

// max / min of three.
BVHGPU_DEV float max3f(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
BVHGPU_DEV float min3f(float a, float b, float c) {
  float d;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

struct PoolRay {
  float o[3], inv[3], tmax;
  uint32_t bits;  // code | reverse << 2 | exact << 3 | job << 4 | hit << 12 (closest-hit rays)
};

// The traversal's view of a ray record; c: its leaf constants and result slot.
constexpr float kMaxInv = 1152921504606846976.0f;  // 2^60
template <int PROFILE, bool LOOSE = false>
BVHGPU_DEV PoolRay pool_ray(const bvhgpu_ray_t& in, uint32_t slot, float4& c) {
  const Ray q = make_ray<PROFILE>(in);
  PoolRay r;
#pragma unroll
  for (int a = 0; a < 3; ++a) { r.o[a] = q.o[a]; r.inv[a] = q.inv[a]; }
  r.tmax = q.tmax;
  // 1 / direction = 0 (an infinite direction) takes the exact form too: it
  // would make NaNs of the empty slots' rows.
  bool exact = q.exact || q.inv[0] == 0.0f || q.inv[1] == 0.0f || q.inv[2] == 0.0f;
  if (LOOSE) {
    // So does one whose 1 / direction is clamped (q8_axis) where the planes
    // are not moved apart by more than the ray's length there.
#pragma unroll
    for (int a = 0; a < 3; ++a)
      exact = exact || (fabsf(q.inv[a]) > kMaxInv && !(fabsf(q.o[a]) * 1.0e12f > 2.0f * fabsf(q.tmax)));
  }
  r.bits = (uint32_t)q.code | ((q.reverse ? 1u : 0u) << 2) | ((exact ? 1u : 0u) << 3);
  c = PROFILE == BVHGPU_PROFILE_INSTRUMENTED
          ? make_float4(q.sx, q.sy, q.sz, __uint_as_float(slot))
          : make_float4(q.d[0], q.d[1], q.d[2], __uint_as_float(slot));
  return r;
}

// Slab test of four boxes given as rows (near and far plane of each axis,
// four floats each): bit k of the result is set where box k is missed. The
// booleans are slab_mm's for NaN-free rays and ordered boxes (see visit_node),
// t0 <= t1 taken from the sign of t1 - t0 (t1 is at most tMax, which is finite,
// and t0 at least 0, so the difference is no NaN; the +inf / -inf rows of empty
// slots give a miss).
BVHGPU_DEV uint32_t miss2(const float2& nx, const float2& ny, const float2& nz, const float2& fx,
                          const float2& fy, const float2& fz, float tmax, uint32_t miss) {
  const float t0x = fmaxf(max3f(nx.x, ny.x, nz.x), 0.0f), t0y = fmaxf(max3f(nx.y, ny.y, nz.y), 0.0f);
  const float t1x = fminf(min3f(fx.x, fy.x, fz.x), tmax), t1y = fminf(min3f(fx.y, fy.y, fz.y), tmax);
  // + 0 turns the -0 of t1 = -0, t0 = 0 (a hit) into +0.
  const float2 s = f2unpack(f2add(f2sub(f2pack(t1x, t1y), f2pack(t0x, t0y)), 0ull));
  miss = __funnelshift_l(__float_as_uint(s.y), miss, 1);
  return __funnelshift_l(__float_as_uint(s.x), miss, 1);
}
BVHGPU_DEV uint32_t miss4(const float4& nx, const float4& ny, const float4& nz, const float4& fx,
                          const float4& fy, const float4& fz, const PoolRay& r, uint32_t miss) {
  const uint64_t ox = f2splat(r.o[0]), oy = f2splat(r.o[1]), oz = f2splat(r.o[2]);
  const uint64_t ix = f2splat(r.inv[0]), iy = f2splat(r.inv[1]), iz = f2splat(r.inv[2]);
#pragma unroll
  for (int p = 1; p >= 0; --p) {
    const int k = 2 * p;
    miss = miss2(f2plane(f4get(nx, k), f4get(nx, k + 1), ox, ix),
                 f2plane(f4get(ny, k), f4get(ny, k + 1), oy, iy),
                 f2plane(f4get(nz, k), f4get(nz, k + 1), oz, iz),
                 f2plane(f4get(fx, k), f4get(fx, k + 1), ox, ix),
                 f2plane(f4get(fy, k), f4get(fy, k + 1), oy, iy),
                 f2plane(f4get(fz, k), f4get(fz, k + 1), oz, iz), r.tmax, miss);
  }
  return miss;
}

// The reference's comparison form for rays that can produce a NaN: same
// boolean as slab(), one child at a time.
BVHGPU_DEV bool slab_exact(float lx, float ly, float lz, float hx, float hy, float hz,
                           const PoolRay& r) {
  Ray q;
#pragma unroll
  for (int a = 0; a < 3; ++a) { q.o[a] = r.o[a]; q.inv[a] = r.inv[a]; }
  return slab(lx, ly, lz, hx, hy, hz, q, r.tmax);
}

// 1 / direction up to 2^60 in size.
BVHGPU_DEV float clamp_inv(float inv) { return fminf(fmaxf(inv, -kMaxInv), kMaxInv); }

// One axis of a Q8 node for q8_planes4: t = f * c + d for a byte q placed in
// f = 1 + q / 2^15; c = 2^15 step / direction, d for the near and the far
// planes moved apart by more than every rounding error between them and the
// exact chain (decoded plane - origin) / direction: each error is below 2^-22
// of one of the terms in s.
struct Q8Axis {
  uint64_t c, dn, df;
};
BVHGPU_DEV Q8Axis q8_axis(float org, float step, float o, float inv) {
  inv = clamp_inv(inv);
  const float b = (org - o) * inv, c = step * 32768.0f * inv;
  const float s = (fabsf(b) + fabsf(o * inv) + fabsf(c)) * 9.5367431640625e-7f;  // 2^-20
  const float d = b - c;
  return Q8Axis{f2splat(c), f2splat(d - s), f2splat(d + s)};
}
// Four bytes of a row, two planes per pair.
BVHGPU_DEV void q8_planes4(uint32_t w, uint64_t c, uint64_t d, float2& p01, float2& p23) {
  p01 = f2unpack(f2fma(f2pack(__uint_as_float(__byte_perm(w, 0x3F800000u, 0x7604u)),
                              __uint_as_float(__byte_perm(w, 0x3F800000u, 0x7614u))), c, d));
  p23 = f2unpack(f2fma(f2pack(__uint_as_float(__byte_perm(w, 0x3F800000u, 0x7624u)),
                              __uint_as_float(__byte_perm(w, 0x3F800000u, 0x7634u))), c, d));
}

// Children of node e that the ray hits, bit c for child c.
//
// LOOSE (Q8 records, any-hit rays of the instrumented profile): one fused
// multiply-add per plane instead of the decode and the slab's subtract and
// multiply, with the planes moved outward, so that some children are visited
// that the ray misses. That changes no result: a triangle counts only if the
// ray hits its own bounds (the leaf's pre-test), and then it hits every box
// around it, whose t0 and t1 enclose the triangle's (rounding is monotonic)
// with the same tMax. The scene's boxes must be nested.
template <int NM, int FMT, bool LOOSE>
BVHGPU_DEV uint32_t pool_node_hits(const uint8_t* rec, const PoolRay& r) {
  using F = PackFmt<NM, FMT>;
  const int nx = r.inv[0] >= 0.0f ? 0 : 3, ny = r.inv[1] >= 0.0f ? 1 : 4;
  const int nz = r.inv[2] >= 0.0f ? 2 : 5;
  const int fx = 3 - nx, fy = 5 - ny, fz = 7 - nz;
  uint32_t miss = 0;
  if (FMT == kFmtFP32) {
    if ((r.bits >> 3) & 1u) {
      const float* b = reinterpret_cast<const float*>(rec);
      const int count = (int)(ldgu(rec + F::COUNT) & 0xFFu);
      uint32_t hit = 0;
      for (int c = 0; c < count; ++c)
        if (slab_exact(__ldg(b + c), __ldg(b + NM + c), __ldg(b + 2 * NM + c),
                       __ldg(b + 3 * NM + c), __ldg(b + 4 * NM + c), __ldg(b + 5 * NM + c), r))
          hit |= 1u << c;
      return hit;
    }
#pragma unroll
    for (int q = NM / 4 - 1; q >= 0; --q)
      miss = miss4(ldg4(rec + (nx * NM + 4 * q) * 4), ldg4(rec + (ny * NM + 4 * q) * 4),
                   ldg4(rec + (nz * NM + 4 * q) * 4), ldg4(rec + (fx * NM + 4 * q) * 4),
                   ldg4(rec + (fy * NM + 4 * q) * 4), ldg4(rec + (fz * NM + 4 * q) * 4), r, miss);
    return ~miss & ((1u << NM) - 1u);
  } else {
    const uint4 h = ldgu4(rec);
    const float org[3] = {__uint_as_float(h.x), __uint_as_float(h.y), __uint_as_float(h.z)};
    const float st[3] = {exp2i((int)(int8_t)(h.w & 0xFFu)), exp2i((int)(int8_t)((h.w >> 8) & 0xFFu)),
                         exp2i((int)(int8_t)((h.w >> 16) & 0xFFu))};
    const int count = (int)(h.w >> 24);
    if ((r.bits >> 3) & 1u) {
      uint32_t hit = 0;
      for (int c = 0; c < count; ++c) {
        float v[6];
#pragma unroll
        for (int a = 0; a < 6; ++a) {
          const float q = (float)__ldg(rec + F::BOX + a * NM + c) * st[a % 3];
          v[a] = a < 3 ? __fadd_rd(org[a], q) : __fadd_ru(org[a % 3], q);
        }
        if (slab_exact(v[0], v[1], v[2], v[3], v[4], v[5], r)) hit |= 1u << c;
      }
      return hit;
    }
    const uint8_t* qb = rec + F::BOX;
    if constexpr (LOOSE) {
      const Q8Axis ax = q8_axis(org[0], st[0], r.o[0], r.inv[0]);
      const Q8Axis ay = q8_axis(org[1], st[1], r.o[1], r.inv[1]);
      const Q8Axis az = q8_axis(org[2], st[2], r.o[2], r.inv[2]);
#pragma unroll
      for (int q = NM / 4 - 1; q >= 0; --q) {
        float2 n[3][2], f[3][2];
        q8_planes4(ldgu(qb + nx * NM + 4 * q), ax.c, ax.dn, n[0][0], n[0][1]);
        q8_planes4(ldgu(qb + ny * NM + 4 * q), ay.c, ay.dn, n[1][0], n[1][1]);
        q8_planes4(ldgu(qb + nz * NM + 4 * q), az.c, az.dn, n[2][0], n[2][1]);
        q8_planes4(ldgu(qb + fx * NM + 4 * q), ax.c, ax.df, f[0][0], f[0][1]);
        q8_planes4(ldgu(qb + fy * NM + 4 * q), ay.c, ay.df, f[1][0], f[1][1]);
        q8_planes4(ldgu(qb + fz * NM + 4 * q), az.c, az.df, f[2][0], f[2][1]);
#pragma unroll
        for (int k = 1; k >= 0; --k)
          miss = miss2(n[0][k], n[1][k], n[2][k], f[0][k], f[1][k], f[2][k], r.tmax, miss);
      }
      return ~miss & ((1u << count) - 1u);
    }
#pragma unroll
    for (int q = NM / 4 - 1; q >= 0; --q) {
      float4 near[3], far[3];
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const bool up = (a == 0 ? nx : (a == 1 ? ny : nz)) >= 3;
        const float4 lo = q8_row(ldgu(qb + a * NM + 4 * q), org[a], st[a], false);
        const float4 hi = q8_row(ldgu(qb + (3 + a) * NM + 4 * q), org[a], st[a], true);
        near[a] = up ? hi : lo;
        far[a] = up ? lo : hi;
      }
      miss = miss4(near[0], near[1], near[2], far[0], far[1], far[2], r, miss);
    }
    return ~miss & ((1u << count) - 1u);
  }
}

// What pool_positions reads of a node's record: the child at each position of
// the push sequence of axis `code`, or for more than 8 children the position of
// each child.
template <int NM, int FMT>
BVHGPU_DEV typename PoolWord<NM>::T pool_sequence(const uint8_t* rec, uint32_t code) {
  using F = PackFmt<NM, FMT>;
  if constexpr (NM <= 8)
    return ldgu(rec + F::SEQ + 4 * code);
  else
    return make_uint2(ldgu(rec + F::INV + 8 * code), ldgu(rec + F::INV + 8 * code + 4));
}

// Hit children as positions in the push sequence of the ray's major axis.
template <int NM>
BVHGPU_DEV uint32_t pool_positions(const typename PoolWord<NM>::T seq, uint32_t hit) {
  if constexpr (NM <= 8) {
    // Each hit bit spread to a byte, the bytes permuted by the sequence (its
    // nibbles are the selectors of the byte permute), and gathered again.
    const uint32_t lo = ((hit & 15u) * 0x00204081u) & 0x01010101u;
    const uint32_t hi = NM > 4 ? ((hit >> 4) * 0x00204081u) & 0x01010101u : 0u;
    const uint32_t p0 = __byte_perm(lo, hi, seq & 0xFFFFu);
    uint32_t pm = (p0 * 0x01020408u) >> 24;
    if (NM > 4) {
      const uint32_t p1 = __byte_perm(lo, hi, seq >> 16);
      pm |= ((p1 * 0x01020408u) >> 24) << 4;
    }
    return pm;
  } else {
    const uint64_t inv = (uint64_t)seq.x | ((uint64_t)seq.y << 32);
    uint32_t pm = 0;
    while (hit) {
      const int c = __ffs(hit) - 1;
      hit &= hit - 1u;
      pm |= 1u << (uint32_t)((inv >> (4 * c)) & 15u);
    }
    return pm;
  }
}

// One lane's view of its warp's pool.
template <int NM>
struct Pool {
  float4 *a, *b, *c;  // origin, tMax | 1 / direction, bits | leaf constants, result slot
  uint2* state;       // next entry, stack words in use
  typename PoolWord<NM>::T* stack;  // [level][ray]
  uint16_t* pairs;    // pool_pairs: 32
  uint8_t* list;      // node rays, leaf rays, free slots: kPoolRays each
  BVHGPU_DEV PoolRay ray(int j) const {
    const float4 x = a[j], y = b[j];
    PoolRay r;
    r.o[0] = x.x; r.o[1] = x.y; r.o[2] = x.z; r.tmax = x.w;
    r.inv[0] = y.x; r.inv[1] = y.y; r.inv[2] = y.z;
    r.bits = __float_as_uint(y.w);
    return r;
  }
};

// Whether the child at push position k of a node lies behind the ray's tMax:
// its entry distance t0, as the slab test computes it.
template <int NM, int FMT>
BVHGPU_DEV bool pool_behind(const uint8_t* rec, const PoolRay& r, int k) {
  using F = PackFmt<NM, FMT>;
  const uint32_t code = r.bits & 3u;
  const uint32_t w = NM <= 8 ? ldgu(rec + F::SEQ + 4 * code) >> (4 * k)
                             : ldgu(rec + F::SEQ + 8 * code + (k >= 8 ? 4 : 0)) >> (4 * (k & 7));
  const int c = (int)(w & 15u);
  float t[3];
  uint4 h = make_uint4(0u, 0u, 0u, 0u);
  if (FMT == kFmtQ8) h = ldgu4(rec);
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const bool neg = !(r.inv[a] >= 0.0f);
    const int row = neg ? 3 + a : a;
    float x;
    if (FMT == kFmtFP32) {
      x = __ldg(reinterpret_cast<const float*>(rec) + row * NM + c);
    } else {
      const float org = __uint_as_float(a == 0 ? h.x : (a == 1 ? h.y : h.z));
      const float q = (float)__ldg(rec + F::BOX + row * NM + c) * exp2i((int)(int8_t)(h.w >> (8 * a)));
      x = neg ? __fadd_ru(org, q) : __fadd_rd(org, q);
    }
    t[a] = (x - r.o[a]) * r.inv[a];
  }
  return max3f(t[0], t[1], t[2]) > r.tmax;
}

// The first of a node's children `left`, as a position, and where its record
// holds their entries by position.
template <bool ORDERED>
BVHGPU_DEV int pool_first(const PoolRay& r, uint32_t left) {
  return ORDERED && ((r.bits >> 2) & 1u) ? 31 - __clz(left) : __ffs(left) - 1;
}
template <int NM, int FMT, bool ORDERED>
BVHGPU_DEV uint32_t pool_entries(const PoolRay& r) {
  using F = PackFmt<NM, FMT>;
  return ORDERED ? F::SORTED + (r.bits & 3u) * (4 * NM) : F::ENTRY;
}

// A ray's next entry: the first of `left` (children of `node` still to visit),
// the others back on the ray's stack (level l at stack[l * stride]). fresh:
// node is not on the stack yet; otherwise its word is the stack's top, and
// with left = 0 the top is read here. Returns false when nothing is left.
//
// CULL (closest-hit rays of the instrumented profile that have a hit, nested
// boxes): children behind tMax are dropped. A visit would find nothing there:
// every box and triangle inside starts at the same t0 or later (rounding is
// monotonic) and tMax does not change during the visit. Not for leaves of one or
// two triangles, which cost as much as the check. 1M-triangle N8L8 tree,
// primary rays: 18.8 -> 13.9 node visits per ray, solo kernel 0.53 -> 0.47 ms
// (2.1M rays); N16 0.76 -> 0.65 ms; N4, whose visits cost little more than the
// check, 0.46 -> 0.47. Pool kernel, bounced rays: N16 1.13 -> 1.06 ms, N8 1.15
// -> 1.19.
template <int NM, int FMT, bool ORDERED, bool CULL>
BVHGPU_DEV bool pool_take(const PackView& v, typename PoolWord<NM>::T* stack, int stride,
                          const PoolRay& r, uint32_t node, uint32_t left, bool fresh,
                          uint32_t& sp, uint32_t& e) {
  using F = PackFmt<NM, FMT>;
  using W = PoolWord<NM>;
  const bool cull = CULL && ((r.bits >> 12) & 1u) && !((r.bits >> 3) & 1u) && v.nested &&
                    !(v.leaves & kSmallLeaves);
  while (true) {
    if (!fresh) {
      if (sp == 0) return false;
      const typename W::T g = stack[(sp - 1) * stride];
      node = W::node(g);
      left = W::left(g);
    }
    const int k = pool_first<ORDERED>(r, left);
    left &= ~(1u << k);
    const uint8_t* rec = v.nodes + (size_t)node * F::REC;
    if (fresh) {
      if (left) stack[sp++ * stride] = W::make(node, left);
    } else {
      if (left) stack[(sp - 1) * stride] = W::make(node, left);
      else --sp;
      if (CULL && cull && pool_behind<NM, FMT>(rec, r, k)) continue;
    }
    e = ldgu(rec + pool_entries<NM, FMT, ORDERED>(r) + 4 * k);
    return true;
  }
}

template <bool MM>
BVHGPU_DEV bool pool_watertight(const float4& t0, const float4& t1, const float4& t2, const Ray& r,
                                float tmax, float& t, float& b1, float& b2) {
  // Vertices in the ray's permuted axes (kx, ky, code).
  float p[3][3];
  const float v[9] = {t0.x, t0.y, t0.z, t0.w, t1.x, t1.y, t1.z, t1.w, t2.x};
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const float x = v[3 * q], y = v[3 * q + 1], z = v[3 * q + 2];
    p[q][0] = r.code == 0 ? y : (r.code == 1 ? z : x);
    p[q][1] = r.code == 0 ? z : (r.code == 1 ? x : y);
    p[q][2] = r.code == 0 ? x : (r.code == 1 ? y : z);
  }
  return watertight<MM, !MM>(p, r, tmax, t, b1, b2);
}

// Whether Moller-Trumbore certainly rejects a triangle by its first
// barycentric b1 = n1 * (1 / div): of the other sign than it may have and far
// from underflow, or well above 1 (comparisons with a NaN are false, so it is
// left to the full test).
BVHGPU_DEV bool mt_rejects(float n1, float div) {
  const float an = fabsf(n1), ad = fabsf(div);
  const bool neg = (int)(__float_as_uint(n1) ^ __float_as_uint(div)) < 0;
  return an > ad * (neg ? 1e-30f : 1.0001f);
}

// The triangles of a leaf that a cheap test does not rule out, four at a time:
// the stored bounds (instrumented profile; all of them for rays that take the
// exact forms), or the first barycentric without its division.
//
// In the fast profile leaves of one or two triangles go straight to the full
// test, as the cheap one is half of it (0.26M unordered any-hit rays, N4L1, 149
// -> 143 us).
template <int PROFILE>
BVHGPU_DEV uint32_t leaf_candidates(const PackView& v, const float4* blk, int cnt, const PoolRay& r,
                                    const float4& c) {
  const uint32_t all = (1u << cnt) - 1u;
  uint32_t miss = 0;
  if (PROFILE == BVHGPU_PROFILE_INSTRUMENTED) {
    if ((r.bits >> 3) & 1u) return all;
    const int nx = r.inv[0] >= 0.0f ? 0 : 3, ny = r.inv[1] >= 0.0f ? 1 : 4;
    const int nz = r.inv[2] >= 0.0f ? 2 : 5;
    const int fx = 3 - nx, fy = 5 - ny, fz = 7 - nz;
    for (int g = (cnt - 1) >> 2; g >= 0; --g) {
      const float4* b = blk + g * kBlockWords;
      miss = miss4(__ldg(b + nx), __ldg(b + ny), __ldg(b + nz), __ldg(b + fx), __ldg(b + fy),
                   __ldg(b + fz), r, miss);
    }
    return ~miss & all;
  }
  if (v.leaves & kSmallLeaves) return all;
  for (int g = (cnt - 1) >> 2; g >= 0; --g) {
    const float4* tri = blk + g * kBlockWords + kBlockTris;
#pragma unroll
    for (int i = 3; i >= 0; --i) {
      const float4 t0 = __ldg(tri + 3 * i), t1 = __ldg(tri + 3 * i + 1), t2 = __ldg(tri + 3 * i + 2);
      // moller_trumbore()'s divisor and numerator of b1.
      const float e1x = t0.w - t0.x, e1y = t1.x - t0.y, e1z = t1.y - t0.z;
      const float e2x = t1.z - t0.x, e2y = t1.w - t0.y, e2z = t2.x - t0.z;
      const float s1x = c.y * e2z - c.z * e2y;
      const float s1y = c.z * e2x - c.x * e2z;
      const float s1z = c.x * e2y - c.y * e2x;
      const float div = s1x * e1x + s1y * e1y + s1z * e1z;
      const float n1 = (r.o[0] - t0.x) * s1x + (r.o[1] - t0.y) * s1y + (r.o[2] - t0.z) * s1z;
      miss = (miss << 1) | (mt_rejects(n1, div) ? 1u : 0u);
    }
  }
  return ~miss & all;
}

// What the full triangle tests read of a ray.
template <int PROFILE>
BVHGPU_DEV Ray leaf_ray(const PoolRay& pr, const float4& c) {
  Ray r;
#pragma unroll
  for (int a = 0; a < 3; ++a) { r.o[a] = pr.o[a]; r.inv[a] = pr.inv[a]; }
  r.code = (int)(pr.bits & 3u);
  r.kx = r.code == 2 ? 0 : r.code + 1;
  r.ky = r.code == 0 ? 2 : r.code - 1;
  if (PROFILE == BVHGPU_PROFILE_INSTRUMENTED) {
    r.sx = c.x; r.sy = c.y; r.sz = c.z;
  } else {
    r.d[0] = c.x; r.d[1] = c.y; r.d[2] = c.z;
  }
  return r;
}

// The full test of one triangle.
template <int PROFILE>
BVHGPU_DEV bool leaf_test(const float4* tri, const Ray& r, bool exact, float tmax, float& t,
                          float& b1, float& b2, float& prim) {
  const float4 t0 = __ldg(tri), t1 = __ldg(tri + 1), t2 = __ldg(tri + 2);
  prim = t2.y;
  if (PROFILE == BVHGPU_PROFILE_INSTRUMENTED)
    return exact ? pool_watertight<false>(t0, t1, t2, r, tmax, t, b1, b2)
                 : pool_watertight<true>(t0, t1, t2, r, tmax, t, b1, b2);
  const float q[3][3] = {{t0.x, t0.y, t0.z}, {t0.w, t1.x, t1.y}, {t1.z, t1.w, t2.x}};
  return moller_trumbore(q, r, tmax, t, b1, b2);
}

BVHGPU_DEV const float4* leaf_blocks(const PackView& v, uint32_t e) {
  return v.blocks + (size_t)(e & kLeafIndexMask) * kBlockWords;
}
BVHGPU_DEV int leaf_count(uint32_t e) { return (int)((e >> kLeafCountShift) & 15u) + 1; }
BVHGPU_DEV const float4* leaf_tri(const float4* blk, int i) {
  return blk + (i >> 2) * kBlockWords + kBlockTris + 3 * (i & 3);
}

// One leaf visit: returns whether any triangle was hit. Closest-hit rays
// lower tmax and write their hit record. First the cheap test of every
// triangle, then the full test of the few that pass, so that a warp runs as
// many full tests as one of its rays needs at most. With COUNT any-hit rays
// test all of these too, and hits grows by the triangles hit.
template <int PROFILE, int KIND, bool COUNT = false>
BVHGPU_DEV bool pool_leaf(const PackView& v, uint32_t e, const PoolRay pr, const float4 c,
                          float& tmax, uint32_t* hits = nullptr) {
  const float4* blk = leaf_blocks(v, e);
  const uint32_t slot = __float_as_uint(c.w);
  const bool exact = PROFILE == BVHGPU_PROFILE_INSTRUMENTED && ((pr.bits >> 3) & 1u);
  uint32_t pass = leaf_candidates<PROFILE>(v, blk, leaf_count(e), pr, c);
  const Ray r = leaf_ray<PROFILE>(pr, c);
  bool any = false;
  // Fast profile: the tie rule of triIntersect{L} as in visit_leaf_points.
  float leaf_best = 1000000.0f, wu = 0.f, wv = 0.f, wprim = 0.f;
  int winner = -1;
  uint32_t lanes_at_best = 0;
  while (pass) {
    const int i = __ffs(pass) - 1;
    pass &= pass - 1u;
    if (PROFILE == BVHGPU_PROFILE_INSTRUMENTED && KIND == BVHGPU_CLOSEST && !exact &&
        tmax != pr.tmax) {
      // tMax fell in this leaf: the pre-test's tMax condition again.
      const float* bf = reinterpret_cast<const float*>(blk + (i >> 2) * kBlockWords) + (i & 3);
      float m[3];
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const float lo = (__ldg(bf + 4 * a) - r.o[a]) * r.inv[a];
        const float hi = (__ldg(bf + 4 * (3 + a)) - r.o[a]) * r.inv[a];
        m[a] = fminf(lo, hi);
      }
      if (tmax < fmaxf(fmaxf(m[0], m[1]), m[2])) continue;
    }
    float t, b1, b2, prim;
    if (!leaf_test<PROFILE>(leaf_tri(blk, i), r, exact, tmax, t, b1, b2, prim)) continue;
    any = true;
    if (COUNT) ++*hits;
    if (KIND == BVHGPU_ANY) {
      if (COUNT) continue;
      break;
    }
    if (PROFILE == BVHGPU_PROFILE_INSTRUMENTED) {
      // Each accepted triangle overwrites the hit (triangle.cpp:243).
      tmax = t;
      static_cast<float4*>(v.out)[slot] = make_float4(prim, t, b1, b2);
      continue;
    }
    const uint32_t lane_bit = 1u << (i % v.gang);
    if (t < leaf_best || (winner >= 0 && t == leaf_best && !(lanes_at_best & lane_bit))) {
      // (a tie keeps the first one's t: it may be a zero of the other sign)
      lanes_at_best = t < leaf_best ? lane_bit : lanes_at_best | lane_bit;
      leaf_best = t < leaf_best ? t : leaf_best;
      winner = i;
      wu = b1;
      wv = b2;
      wprim = prim;
    }
  }
  if (PROFILE == BVHGPU_PROFILE_FAST && KIND == BVHGPU_CLOSEST && winner >= 0) {
    tmax = leaf_best;
    static_cast<float4*>(v.out)[slot] = make_float4(wprim, leaf_best, wu, wv);
  }
  return any;
}

// The full tests of a pool's any-hit leaf step: the (ray, triangle) pairs that
// passed the cheap test, 32 at a time, one per lane, whichever ray they belong
// to. About one triangle per leaf visit passes, so the step's up to 32 rays
// have about as many pairs, where a loop per ray runs as long as the ray with
// most of them (three to four, with 8 of 32 lanes busy). pass: the lane's
// candidates of pool ray j. Every lane of the warp calls it; returns whether
// the lane's ray was hit. Instrumented profile: 1M-triangle frame 4.54 -> 4.50
// ms, 12 scenes 711 -> 700 us, Q8 frame 3.03 -> 2.92 ms. The fast profile keeps
// the loop per ray (per-ray calls 1.55 against 1.59 ms: its cheap test leaves
// more triangles, and the pairs read every triangle a second time).
template <int PROFILE, typename SRC, typename POOL>
BVHGPU_DEV bool pool_pairs(const SRC& p, const POOL& P, int j, uint32_t pass, int lane) {
  constexpr unsigned FULL = 0xFFFFFFFFu;
  const int mine = __popc(pass);
  int incl = mine;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int x = __shfl_up_sync(FULL, incl, d);
    if (lane >= d) incl += x;
  }
  const int total = __shfl_sync(FULL, incl, 31), first = incl - mine;
  int at = first;
  bool hit = false;
  for (int base = 0; base < total; base += 32) {
    while (pass && at < base + 32) {
      const int i = __ffs(pass) - 1;
      pass &= pass - 1u;
      P.pairs[at - base] = (uint16_t)(j | (i << 8));
      ++at;
    }
    __syncwarp();
    bool h = false;
    if (base + lane < total) {
      const int q = P.pairs[lane];
      const PoolRay pr = P.ray(q & 0xFF);
      const float4 c = P.c[q & 0xFF];
      const PackView& v = p.view((pr.bits >> 4) & 0xFFu);
      const float4* blk = leaf_blocks(v, P.state[q & 0xFF].x);
      const bool exact = PROFILE == BVHGPU_PROFILE_INSTRUMENTED && ((pr.bits >> 3) & 1u);
      float t, b1, b2, prim;
      h = leaf_test<PROFILE>(leaf_tri(blk, q >> 8), leaf_ray<PROFILE>(pr, c), exact, pr.tmax, t, b1,
                             b2, prim);
    }
    const unsigned hits = __ballot_sync(FULL, h);
    const int lo = max(first - base, 0), hi = min(first + mine - base, 32);
    if (lo < hi && ((hits >> lo) & (FULL >> (32 - (hi - lo))))) hit = true;
    // Other lanes write these pairs, and the owners their rays, next.
    __syncwarp();
  }
  return hit;
}

template <int NM, int PROFILE, int KIND, int FMT, bool ORDERED, typename SRC>
__global__ void __launch_bounds__(kPoolWarps * 32, BVHGPU_POOL_MIN_BLOCKS)
    trace_pool_kernel(const __grid_constant__ SRC p) {
  using F = PackFmt<NM, FMT>;
  constexpr unsigned FULL = 0xFFFFFFFFu;
  constexpr int K = kPoolRays;
  constexpr bool kPairs = KIND == BVHGPU_ANY && PROFILE == BVHGPU_PROFILE_INSTRUMENTED;
  constexpr bool kLoose = FMT == kFmtQ8 && PROFILE == BVHGPU_PROFILE_INSTRUMENTED &&
                          KIND == BVHGPU_ANY;
  constexpr bool kCull =
      PROFILE == BVHGPU_PROFILE_INSTRUMENTED && KIND == BVHGPU_CLOSEST && NM >= 12;
  extern __shared__ __align__(16) uint8_t pool_smem[];
  if (p.planned && p.queue[1] != kPlanPool) return;
  const unsigned lane = threadIdx.x & 31u;
  const unsigned below = (1u << lane) - 1u;
  using W = PoolWord<NM>;
  Pool<NM> P;
  {
    uint8_t* w = pool_smem + pool_warp_bytes<NM>(p.levels) * (threadIdx.x >> 5);
    P.a = reinterpret_cast<float4*>(w);
    P.b = P.a + K;
    P.c = P.b + K;
    P.state = reinterpret_cast<uint2*>(P.c + K);
    P.stack = reinterpret_cast<typename W::T*>(P.state + K);
    P.pairs = reinterpret_cast<uint16_t*>(P.stack + (size_t)p.levels * K);
    P.list = reinterpret_cast<uint8_t*>(P.pairs + 32);
  }
  // Lists 0 node rays, 1 leaf rays, 2 free slots; each grows and shrinks at
  // its end, so rays that went together last stay together.
  for (int i = (int)lane; i < K; i += 32) P.list[2 * K + i] = (uint8_t)i;
  int n_node = 0, n_leaf = 0, n_free = p.slots;
  bool drained = false;
  __syncwarp();

  while (true) {
    // The step's rays: one per lane below m. next: the list this lane's ray
    // goes to (-1: no ray).
    int next = -1, j = 0, m = 0;
    if (!drained && n_free >= BVHGPU_POOL_REFILL &&
        (n_free >= 32 || (n_node < 32 && n_leaf < 32))) {
      // New rays into free slots.
      const int want = min(32, n_free);
      unsigned long long base = 0;
      if (lane == 0) base = atomicAdd(p.queue, (unsigned long long)want);
      base = __shfl_sync(FULL, base, 0);
      m = base >= p.n ? 0 : (int)min((unsigned long long)want, p.n - base);
      drained = base + want >= p.n;
      n_free -= m;
      if ((int)lane < m) {
        j = P.list[2 * K + n_free + lane];
        uint32_t slot, job;
        const bvhgpu_ray_t in = p.ray(base + lane, slot, job);
        const PackView& v = p.view(job);
        next = 2;
        if (KIND == BVHGPU_CLOSEST)
          static_cast<float4*>(v.out)[slot] = make_float4(__int_as_float(-1), in.tmax, 0.f, 0.f);
        if (!isnan(in.ox)) {
          float4 c;
          PoolRay r = pool_ray<PROFILE, kLoose>(in, slot, c);
          r.bits |= job << 4;
          P.a[j] = make_float4(r.o[0], r.o[1], r.o[2], r.tmax);
          P.b[j] = make_float4(r.inv[0], r.inv[1], r.inv[2], __uint_as_float(r.bits));
          P.c[j] = c;
          P.state[j] = make_uint2(v.root, 0u);
          next = (v.root & kLeafBit) ? 1 : 0;
        } else if (KIND == BVHGPU_ANY) {
          static_cast<uint8_t*>(v.out)[slot] = 0;
        }
      }
    } else if (n_node >= 32 || (n_node > 0 && n_node >= n_leaf)) {
      m = min(32, n_node);
      n_node -= m;
      if ((int)lane < m) {
        j = P.list[n_node + (int)lane];
        const PoolRay r = P.ray(j);
        const PackView& v = p.view((r.bits >> 4) & 0xFFu);
        const uint2 st = P.state[j];
        uint32_t sp = st.y, e;
        const uint8_t* rec = v.nodes + (size_t)st.x * F::REC;
        uint32_t left = pool_node_hits<NM, FMT, kLoose>(rec, r);
        const bool fresh = left != 0;
        if (ORDERED && fresh) left = pool_positions<NM>(pool_sequence<NM, FMT>(rec, r.bits & 3u), left);
        next = 2;
        if (pool_take<NM, FMT, ORDERED, kCull>(v, P.stack + j, K, r, st.x, left, fresh, sp, e)) {
          P.state[j] = make_uint2(e, sp);
          next = (int)(e >> 31);
        } else if (KIND == BVHGPU_ANY) {
          static_cast<uint8_t*>(v.out)[__float_as_uint(P.c[j].w)] = 0;
        }
      }
    } else if (n_leaf > 0) {
      m = min(32, n_leaf);
      n_leaf -= m;
      const bool on = (int)lane < m;
      uint32_t pass = 0;
      bool hit = false;
      if (on) j = P.list[K + n_leaf + (int)lane];
      if (kPairs) {
        if (on) {
          const PoolRay r = P.ray(j);
          const uint32_t e = P.state[j].x;
          const PackView& v = p.view((r.bits >> 4) & 0xFFu);
          pass = leaf_candidates<PROFILE>(v, leaf_blocks(v, e), leaf_count(e), r, P.c[j]);
        }
        hit = pool_pairs<PROFILE>(p, P, j, pass, (int)lane);
      }
      if (on) {
        PoolRay r = P.ray(j);
        const PackView& v = p.view((r.bits >> 4) & 0xFFu);
        const uint2 st = P.state[j];
        uint32_t sp = st.y, e;
        if (!kPairs) {
          float tmax = r.tmax;
          hit = pool_leaf<PROFILE, KIND>(v, st.x, r, P.c[j], tmax);
          if (KIND == BVHGPU_CLOSEST && hit) {
            r.tmax = tmax;
            r.bits |= 1u << 12;
            P.a[j].w = tmax;
            P.b[j].w = __uint_as_float(r.bits);
          }
        }
        next = 2;
        if (KIND == BVHGPU_ANY && hit) {
          static_cast<uint8_t*>(v.out)[__float_as_uint(P.c[j].w)] = 1;
        } else if (pool_take<NM, FMT, ORDERED, kCull>(v, P.stack + j, K, r, 0u, 0u, false, sp, e)) {
          P.state[j] = make_uint2(e, sp);
          next = (int)(e >> 31);
        } else if (KIND == BVHGPU_ANY) {
          static_cast<uint8_t*>(v.out)[__float_as_uint(P.c[j].w)] = 0;
        }
      }
    } else if (drained) {
      break;
    }
    // The step's rays onto their next lists.
    const unsigned mn = __ballot_sync(FULL, next == 0), ml = __ballot_sync(FULL, next == 1);
    const unsigned mf = (m == 32 ? FULL : (1u << m) - 1u) & ~(mn | ml);
    const unsigned mine = next == 0 ? mn : (next == 1 ? ml : mf);
    const int at = next == 0 ? n_node : (next == 1 ? K + n_leaf : 2 * K + n_free);
    // Every lane has read its own entry (votes alone order no memory).
    __syncwarp();
    if (next >= 0) P.list[at + __popc(mine & below)] = (uint8_t)j;
    n_node += __popc(mn);
    n_leaf += __popc(ml);
    n_free += __popc(mf);
    __syncwarp();
  }
}

// Chooses the kernel of a batch by its rays: 64 groups of 32 consecutive rays,
// spread over the launch, each lane compared with the group's first active ray.
// Rays that run alike (primary rays of a tile, shadow rays of neighbouring
// hits) start close to it and point the same way; then one thread per ray
// keeps most of a warp busy without the pool's lists. Also clears the pool's
// queue head.
constexpr int kPlanWarps = 8, kPlanGroups = 8;  // groups per warp
template <typename SRC>
__global__ void __launch_bounds__(kPlanWarps * 32) plan_kernel(const __grid_constant__ SRC p) {
  __shared__ int votes[2];  // lanes that agree with their group's first ray, active lanes
  constexpr unsigned FULL = 0xFFFFFFFFu;
  if (threadIdx.x < 2) votes[threadIdx.x] = 0;
  __syncthreads();
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  constexpr uint32_t kGroups = kPlanWarps * kPlanGroups;
  int agree = 0, active = 0;
#pragma unroll
  for (uint32_t k = 0; k < kPlanGroups; ++k) {
    const uint64_t first = p.n / kGroups * (warp * kPlanGroups + k);
    const uint64_t i = first + lane < p.n ? first + lane : p.n - 1u;
    uint32_t slot, job;
    const bvhgpu_ray_t q = p.ray(i, slot, job);
    const unsigned live = __ballot_sync(FULL, !isnan(q.ox));
    if (live == 0) continue;
    const int lead = __ffs(live) - 1;
    const float ox = q.ox - __shfl_sync(FULL, q.ox, lead), oy = q.oy - __shfl_sync(FULL, q.oy, lead);
    const float oz = q.oz - __shfl_sync(FULL, q.oz, lead);
    const float dx = __shfl_sync(FULL, q.dx, lead), dy = __shfl_sync(FULL, q.dy, lead);
    const float dz = __shfl_sync(FULL, q.dz, lead), tmax = __shfl_sync(FULL, q.tmax, lead);
    const float dd = dx * dx + dy * dy + dz * dz;
    const float qq = q.dx * q.dx + q.dy * q.dy + q.dz * q.dz;
    const float dot = q.dx * dx + q.dy * dy + q.dz * dz;
    // Within a twentieth of the ray's length and 18 degrees.
    const bool same = ox * ox + oy * oy + oz * oz <= 0.0025f * tmax * tmax * dd && dot > 0.0f &&
                      dot * dot >= 0.9f * dd * qq;
    agree += __popc(__ballot_sync(FULL, same) & live);
    active += __popc(live);
  }
  if (lane == 0) {
    atomicAdd(&votes[0], agree);
    atomicAdd(&votes[1], active);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    p.queue[0] = 0ull;
    p.queue[1] = 4 * votes[0] >= 3 * votes[1] ? kPlanSolo : kPlanPool;
  }
}

// One thread per ray on the packed scene, its stack in shared memory
// ([level][thread]). FEW: for launches whose rays all run at once, where the
// longest rays' latency counts and not the rate of visits; a visit then loads
// the push sequence (and the entries of 4 children) together with the boxes
// instead of after them. 40k unordered closest-hit rays (L8, 251k triangles), us,
// of the general per-ray kernel / this one without FEW / with it: N4 119 / 125 /
// 98, N8 103 / 112 / 96, N12 111 / 131 / 108, N16 103 / 116 / 96. Well beyond
// one wave of its blocks it loses: N8, 131k rays, 149 without / 189 with it.
//
// kLeavesInTurn: a lane that reaches a leaf visits it after the warp's current
// node step, instead of when every lane has a leaf. A leaf of few triangles
// costs less than a node, so waiting for company only idles lanes (N8L1: 16.4
// of 32 lanes against 19.8 of the general per-ray kernel). 0.5M primary rays
// (251k triangles), us, general / waiting / in turn: N4L1 335 / 349 / 235, N8L1 316
// / 363 / 239, N8L8 301 / 253 / 223. With leaves larger than nodes waiting is
// better: N4L8, 0.26M unordered any-hit rays of the fast profile, 172 waiting / 190
// in turn. On Q8 nodes, which are decoded first, 4-wide ones gain up to L8: 131k
// primary rays 258 / 317 / 223, random closest-hit rays of all sizes 0.90 to 1.17
// times as fast (median 1.01 to 1.04).
template <int NM, int PROFILE, int KIND, int FMT, bool ORDERED, bool FEW, typename SRC>
__global__ void __launch_bounds__(128, FEW ? kSoloFewBlocks : kSoloBlocks<NM, FMT>)
    trace_solo_kernel(const __grid_constant__ SRC p) {
  using F = PackFmt<NM, FMT>;
  using W = PoolWord<NM>;
  constexpr bool kLoose = FMT == kFmtQ8 && PROFILE == BVHGPU_PROFILE_INSTRUMENTED &&
                          KIND == BVHGPU_ANY;
  constexpr bool kCull =
      PROFILE == BVHGPU_PROFILE_INSTRUMENTED && KIND == BVHGPU_CLOSEST && NM >= 8;
  constexpr bool kRow = FEW && NM == 4;
  extern __shared__ __align__(16) uint8_t pool_smem[];
  if (p.planned && p.queue[1] != kPlanSolo) return;
  typename W::T* stack = reinterpret_cast<typename W::T*>(pool_smem) + threadIdx.x;
  const int stride = (int)blockDim.x;
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= p.n) return;
  uint32_t slot, job;
  const bvhgpu_ray_t in = p.ray(i, slot, job);
  const PackView v = p.view(job);
  if (KIND == BVHGPU_CLOSEST)
    static_cast<float4*>(v.out)[slot] = make_float4(__int_as_float(-1), in.tmax, 0.f, 0.f);
  bool hit = false;
  if (!isnan(in.ox)) {
    float4 c;
    PoolRay r = pool_ray<PROFILE, kLoose>(in, slot, c);
    uint32_t e = v.root, sp = 0;
    bool more = true;
    while (more) {
      while (more && !(e & kLeafBit)) {
        const uint8_t* rec = v.nodes + (size_t)e * F::REC;
        typename W::T seq{};
        uint4 row{};
        if (FEW && ORDERED) seq = pool_sequence<NM, FMT>(rec, r.bits & 3u);
        if (kRow) row = ldgu4(rec + pool_entries<NM, FMT, ORDERED>(r));
        uint32_t left = pool_node_hits<NM, FMT, kLoose>(rec, r);
        const bool fresh = left != 0;
        if (ORDERED && fresh)
          left = pool_positions<NM>(FEW ? seq : pool_sequence<NM, FMT>(rec, r.bits & 3u), left);
        if (kRow && fresh) {
          const int k = pool_first<ORDERED>(r, left);
          left &= ~(1u << k);
          if (left) stack[sp++ * stride] = W::make(e, left);
          e = (k & 2) ? ((k & 1) ? row.w : row.z) : ((k & 1) ? row.y : row.x);
        } else {
          more = pool_take<NM, FMT, ORDERED, kCull>(v, stack, stride, r, e, left, fresh, sp, e);
        }
        if (v.leaves & kLeavesInTurn) break;
      }
      if (!more) break;
      if (!(e & kLeafBit)) continue;
      float tmax = r.tmax;
      if (pool_leaf<PROFILE, KIND>(v, e, r, c, tmax)) {
        hit = true;
        if (KIND == BVHGPU_ANY) break;
        r.tmax = tmax;
        r.bits |= 1u << 12;
      }
      more = pool_take<NM, FMT, ORDERED, kCull>(v, stack, stride, r, 0u, 0u, false, sp, e);
    }
  }
  if (KIND == BVHGPU_ANY) static_cast<uint8_t*>(v.out)[slot] = hit ? 1 : 0;
}

// Counting traces of the instrumented profile on the packed scene: a thread per
// ray that visits what the per-ray kernel visits, in its order, and counts it
// in its counters and histograms. 640 x 360 primary and shadow rays on a
// 251k-triangle N16L16 tree: 370 us in the general kernel (128 registers, 39 KB
// of stacks and histogram: 4 blocks of 128 threads per SM), 326 here, bound by
// the traversal as without counters. Blocks per SM (registers): 4 341 us, 5 327,
// 6 and 7 323, 8 333. Several copies of the block's histogram change nothing.
template <int NM, int KIND, int FMT>
__global__ void __launch_bounds__(128, 6)
    trace_count_kernel(const __grid_constant__ OneScene p, const __grid_constant__ TraceArgs a) {
  using F = PackFmt<NM, FMT>;
  using W = PoolWord<NM>;
  constexpr int I = BVHGPU_PROFILE_INSTRUMENTED;
  extern __shared__ __align__(16) uint8_t pool_smem[];
  const int stride = (int)blockDim.x;
  typename W::T* stack = reinterpret_cast<typename W::T*>(pool_smem) + threadIdx.x;
  hist_clear(a);
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < p.n) {
    uint32_t slot, job;
    const bvhgpu_ray_t in = p.ray(i, slot, job);
    const PackView& v = p.scene;
    if (KIND == BVHGPU_CLOSEST)
      static_cast<float4*>(v.out)[slot] = make_float4(__int_as_float(-1), in.tmax, 0.f, 0.f);
    Counters ctr;
    bool hit = false;
    if (!isnan(in.ox)) {
      float4 c;
      PoolRay r = pool_ray<I>(in, slot, c);
      uint32_t e = v.root, sp = 0;
      uint32_t held = 0;  // entries that a stack of single children would hold
      bool more = true;
      while (more) {
        while (more && !(e & kLeafBit)) {
          const uint8_t* rec = v.nodes + (size_t)e * F::REC;
          uint32_t left = pool_node_hits<NM, FMT, false>(rec, r);
          const uint32_t info = ldgu(rec + F::COUNT), n = (uint32_t)__popc(left);
          ctr.node_visits++;
          ctr.box_tests += info & 0xFFu;
          ctr.box_hits += n;
          held += n;
          ctr.max_stack = max(ctr.max_stack, held);
          count_node<true>(a, (int)((info >> 8) | (info & 0xFFu) << 8));
          const bool fresh = left != 0;
          if (fresh) left = pool_positions<NM>(pool_sequence<NM, FMT>(rec, r.bits & 3u), left);
          more = pool_take<NM, FMT, true, false>(v, stack, stride, r, e, left, fresh, sp, e);
          --held;
        }
        if (!more) break;
        ctr.leaf_visits++;
        ctr.tri_tests += (uint32_t)leaf_count(e);
        count_leaf<true>(a, reinterpret_cast<const uint8_t*>(leaf_blocks(v, e) + kBlockWords - 1), e);
        float tmax = r.tmax;
        if (pool_leaf<I, KIND, true>(v, e, r, c, tmax, &ctr.tri_hits)) {
          hit = true;
          if (KIND == BVHGPU_ANY) break;
          r.tmax = tmax;
        }
        more = pool_take<NM, FMT, true, false>(v, stack, stride, r, 0u, 0u, false, sp, e);
        --held;
      }
    }
    if (KIND == BVHGPU_ANY) static_cast<uint8_t*>(v.out)[slot] = hit ? 1 : 0;
    store_counters(a, slot, ctr);
  }
  hist_flush(a);
}

// A team of lanes per ray, one child or triangle per lane, for batches too
// small to fill the GPU with a ray per thread, whose time is the longest
// ray's: a visit then costs one slab or triangle test instead of a loop over
// them, and few rays share a warp's control flow. Every lane of a team keeps
// the ray and its own copy of the stack.
template <int NM> constexpr int kTeam = NM <= 4 ? 4 : (NM <= 8 ? 8 : 16);

// Whether the ray hits child `c` of the node.
template <int NM, int FMT>
BVHGPU_DEV bool team_child_hit(const uint8_t* rec, const PoolRay& r, int c) {
  using F = PackFmt<NM, FMT>;
  if (c >= NM) return false;
  const bool exact = (r.bits >> 3) & 1u;
  float lo[3], hi[3];
  if (FMT == kFmtFP32) {
    const float* b = reinterpret_cast<const float*>(rec) + c;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      lo[a] = __ldg(b + a * NM);
      hi[a] = __ldg(b + (3 + a) * NM);
    }
    if (exact && c >= (int)(ldgu(rec + F::COUNT) & 0xFFu)) return false;
  } else {
    const uint4 h = ldgu4(rec);
    if (c >= (int)(h.w >> 24)) return false;
    const uint32_t org[3] = {h.x, h.y, h.z};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const float o = __uint_as_float(org[a]), st = exp2i((int)(int8_t)(h.w >> (8 * a)));
      lo[a] = __fadd_rd(o, (float)__ldg(rec + F::BOX + a * NM + c) * st);
      hi[a] = __fadd_ru(o, (float)__ldg(rec + F::BOX + (3 + a) * NM + c) * st);
    }
  }
  if (exact) return slab_exact(lo[0], lo[1], lo[2], hi[0], hi[1], hi[2], r);
  float n[3], f[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float x = (lo[a] - r.o[a]) * r.inv[a], y = (hi[a] - r.o[a]) * r.inv[a];
    n[a] = r.inv[a] >= 0.0f ? x : y;
    f[a] = r.inv[a] >= 0.0f ? y : x;
  }
  return fmaxf(max3f(n[0], n[1], n[2]), 0.0f) <= fminf(min3f(f[0], f[1], f[2]), r.tmax);
}

// One leaf visit of a team, as pool_leaf. c: the lane in its team; mask: the
// team's lanes; base: its first lane.
template <int T, int PROFILE, int KIND>
BVHGPU_DEV bool team_leaf(const PackView& v, uint32_t e, const PoolRay pr, const float4& k, int c,
                          unsigned mask, int base, float& tmax) {
  const int cnt = (int)((e >> kLeafCountShift) & 15u) + 1;
  const uint32_t slot = __float_as_uint(k.w);
  const bool exact = (pr.bits >> 3) & 1u;
  Ray r;
#pragma unroll
  for (int a = 0; a < 3; ++a) { r.o[a] = pr.o[a]; r.inv[a] = pr.inv[a]; }
  r.code = (int)(pr.bits & 3u);
  r.kx = r.code == 2 ? 0 : r.code + 1;
  r.ky = r.code == 0 ? 2 : r.code - 1;
  if (PROFILE == BVHGPU_PROFILE_INSTRUMENTED) {
    r.sx = k.x; r.sy = k.y; r.sz = k.z;
  } else {
    r.d[0] = k.x; r.d[1] = k.y; r.d[2] = k.z;
  }
  bool any = false;
  // Fast profile: the leaf's first minimum per gang lane (visit_leaf_points).
  float best = 1000000.0f, wu = 0.f, wv = 0.f, wprim = 0.f;
  int winner = -1;
  uint32_t lanes_at_best = 0;
  for (int g = 0; g < cnt; g += T) {
    const int i = g + c;
    const bool mine = i < cnt;
    const float4* b = v.blocks + ((size_t)(e & kLeafIndexMask) + ((mine ? i : g) >> 2)) * kBlockWords;
    const float4* tri = b + kBlockTris + 3 * (i & 3);
    const float4 t0 = __ldg(tri), t1 = __ldg(tri + 1), t2 = __ldg(tri + 2);
    float t = 0.f, b1 = 0.f, b2 = 0.f;
    bool h = mine;
    if (PROFILE == BVHGPU_PROFILE_INSTRUMENTED) {
      // The triangle's part in the leaf's pre-test (with the tMax the leaf was
      // entered with), and its tMax condition, repeated below.
      float tmin = 0.0f;
      if (!exact) {
        const float* bf = reinterpret_cast<const float*>(b) + (i & 3);
        float n[3], f[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          const float x = (__ldg(bf + 4 * a) - r.o[a]) * r.inv[a];
          const float y = (__ldg(bf + 4 * (3 + a)) - r.o[a]) * r.inv[a];
          n[a] = r.inv[a] >= 0.0f ? x : y;
          f[a] = r.inv[a] >= 0.0f ? y : x;
        }
        tmin = max3f(n[0], n[1], n[2]);
        h = h && fmaxf(tmin, 0.0f) <= fminf(min3f(f[0], f[1], f[2]), pr.tmax);
      }
      // The triangles one after the other, each with the tMax that the
      // accepted ones before it left: the first hit is accepted, and those
      // behind it are tested again if they passed, or all of them if its t is
      // not below the old tMax (it may round up, or be no number).
      bool todo = h;
      while (true) {
        h = todo && (exact || !(tmax < tmin)) &&
            (exact ? pool_watertight<false>(t0, t1, t2, r, tmax, t, b1, b2)
                   : pool_watertight<true>(t0, t1, t2, r, tmax, t, b1, b2));
        const unsigned hits = __ballot_sync(mask, h) & mask;
        if (hits == 0) break;
        any = true;
        if (KIND == BVHGPU_ANY) return true;
        const int first = __ffs(hits) - 1;
        const float ti = __shfl_sync(mask, t, first);
        const bool fell = ti < tmax;
        tmax = ti;
        if (base + c == first) static_cast<float4*>(v.out)[slot] = make_float4(t2.y, t, b1, b2);
        __syncwarp(mask);
        todo = todo && base + c > first && (h || !fell);
        if ((__ballot_sync(mask, todo) & mask) == 0) break;
      }
      continue;
    }
    const float q[3][3] = {{t0.x, t0.y, t0.z}, {t0.w, t1.x, t1.y}, {t1.z, t1.w, t2.x}};
    h = h && moller_trumbore(q, r, tmax, t, b1, b2);
    unsigned hits = __ballot_sync(mask, h) & mask;
    any = any || hits != 0;
    if (KIND == BVHGPU_ANY) {
      if (any) return true;
      continue;
    }
    while (hits) {
      const int from = __ffs(hits) - 1;
      hits &= hits - 1u;
      const float ti = __shfl_sync(mask, t, from);
      const int id = g + from - base;
      const uint32_t lane_bit = 1u << (id % v.gang);
      if (ti < best || (winner >= 0 && ti == best && !(lanes_at_best & lane_bit))) {
        lanes_at_best = ti < best ? lane_bit : lanes_at_best | lane_bit;
        best = ti < best ? ti : best;
        winner = id;
        wu = __shfl_sync(mask, b1, from);
        wv = __shfl_sync(mask, b2, from);
        wprim = __shfl_sync(mask, t2.y, from);
      }
    }
  }
  if (PROFILE == BVHGPU_PROFILE_FAST && KIND == BVHGPU_CLOSEST && winner >= 0) {
    tmax = best;
    if (c == 0) static_cast<float4*>(v.out)[slot] = make_float4(wprim, best, wu, wv);
  }
  return any;
}

template <int NM, int PROFILE, int KIND, int FMT, bool ORDERED, typename SRC>
__global__ void __launch_bounds__(128) trace_team_kernel(const __grid_constant__ SRC p) {
  using F = PackFmt<NM, FMT>;
  using W = PoolWord<NM>;
  constexpr int T = kTeam<NM>;
  extern __shared__ __align__(16) uint8_t pool_smem[];
  typename W::T* stack = reinterpret_cast<typename W::T*>(pool_smem) + threadIdx.x;
  const int stride = (int)blockDim.x;
  // p.slots teams of each warp have a ray.
  const int lane = (int)(threadIdx.x & 31u), c = lane & (T - 1), base = lane & ~(T - 1);
  const unsigned mask = ((1u << T) - 1u) << base;
  const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint64_t i = warp * (uint32_t)p.slots + (uint32_t)(lane / T);
  if (lane / T >= p.slots || i >= p.n) return;
  uint32_t slot, job;
  const bvhgpu_ray_t in = p.ray(i, slot, job);
  const PackView v = p.view(job);
  if (KIND == BVHGPU_CLOSEST && c == 0)
    static_cast<float4*>(v.out)[slot] = make_float4(__int_as_float(-1), in.tmax, 0.f, 0.f);
  __syncwarp(mask);
  bool hit = false;
  if (!isnan(in.ox)) {
    float4 k;
    PoolRay r = pool_ray<PROFILE>(in, slot, k);
    uint32_t e = v.root, sp = 0;
    while (true) {
      const uint32_t node = e;
      uint32_t left = 0;
      bool fresh = false;
      if (!(e & kLeafBit)) {
        const uint8_t* rec = v.nodes + (size_t)node * F::REC;
        const bool h = team_child_hit<NM, FMT>(rec, r, c);
        left = (__ballot_sync(mask, h) & mask) >> base;
        fresh = left != 0;
        if (ORDERED && fresh) left = pool_positions<NM>(pool_sequence<NM, FMT>(rec, r.bits & 3u), left);
      } else if (team_leaf<T, PROFILE, KIND>(v, e, r, k, c, mask, base, r.tmax)) {
        hit = true;
        if (KIND == BVHGPU_ANY) break;
      }
      if (!pool_take<NM, FMT, ORDERED, false>(v, stack, stride, r, node, left, fresh, sp, e)) break;
    }
  }
  if (KIND == BVHGPU_ANY && c == 0) static_cast<uint8_t*>(v.out)[slot] = hit ? 1 : 0;
}

}  // namespace dev
}  // namespace bvhgpu
