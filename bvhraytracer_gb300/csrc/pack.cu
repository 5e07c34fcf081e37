// Packs a scene for the ray-pool kernel (see pack.cuh).
#include "pack.cuh"

namespace bvhgpu {
namespace dev {

namespace {

// One thread per node. Runs once per scene.
template <int N, int FMT>
__global__ void __launch_bounds__(128) pack_nodes_kernel(SceneDev sc, uint32_t n,
                                                         const uint32_t* leaf_block, uint8_t* out) {
  using S = NodeFmt<N, FMT>;
  using D = PackFmt<N, FMT>;
  const uint32_t g = blockIdx.x * 128u + threadIdx.x;
  if (g >= n) return;
  const uint8_t* rec = sc.nodes + (size_t)g * S::REC;
  uint8_t* dst = out + (size_t)g * D::REC;
  const uint32_t* meta = reinterpret_cast<const uint32_t*>(rec + S::META);
  const int count = (int)((meta[2] >> 16) & 0xFFu);
  if (FMT == kFmtFP32) {
    const float* box = reinterpret_cast<const float*>(rec);
    float* b = reinterpret_cast<float*>(dst);
    const float inf = __int_as_float(0x7F800000);
    for (int a = 0; a < 6; ++a)
      for (int c = 0; c < N; ++c)
        b[a * N + c] = c < count ? box[a * N + c] : (a < 3 ? inf : -inf);
  } else {
    const uint32_t* head = reinterpret_cast<const uint32_t*>(rec);
    uint32_t* h = reinterpret_cast<uint32_t*>(dst);
    h[0] = head[0];
    h[1] = head[1];
    h[2] = head[2];
    h[3] = (head[3] & 0xFFFFFFu) | ((uint32_t)count << 24);
    for (int i = 0; i < 6 * N; ++i) dst[D::BOX + i] = rec[S::QBOX + i];
  }
  const uint32_t* ent = sc.child_entry + (size_t)g * N;
  uint32_t* entry = reinterpret_cast<uint32_t*>(dst + D::ENTRY);
  uint32_t* sorted = reinterpret_cast<uint32_t*>(dst + D::SORTED);
  uint32_t* seq = reinterpret_cast<uint32_t*>(dst + D::SEQ);
  for (int c = 0; c < N; ++c) {
    const uint32_t e = c < count ? ent[c] : 0u;
    entry[c] = (e & kLeafBit) ? (e & ~kLeafIndexMask) | leaf_block[e & kLeafIndexMask] : e;
  }
  const uint8_t* perm = FMT == kFmtFP32 ? rec + S::PERM : sc.q8_perm + (size_t)g * S::PSB;
  for (int a = 0; a < 3; ++a) {
    uint64_t fwd = 0, inv = 0;
    const uint8_t* w = perm + a * 2 * S::PW;
    for (int k = 0; k < S::PW; ++k) {
      fwd |= (uint64_t)w[k] << (8 * k);
      inv |= (uint64_t)w[S::PW + k] << (8 * k);
    }
    for (int k = 0; k < N; ++k)
      sorted[a * N + k] = k < count ? entry[(fwd >> (4 * k)) & 15u] : 0u;
    if (N <= 8) {
      // Positions past the count select the bytes of the empty slots, whose
      // hit bits are never set.
      uint32_t s = 0;
      for (int k = 0; k < N; ++k)
        s |= (uint32_t)(k < count ? (fwd >> (4 * k)) & 15u : (uint64_t)k) << (4 * k);
      seq[a] = s;
    } else {
      seq[2 * a] = (uint32_t)fwd;
      seq[2 * a + 1] = (uint32_t)(fwd >> 32);
      seq[6 + 2 * a] = (uint32_t)inv;
      seq[6 + 2 * a + 1] = (uint32_t)(inv >> 32);
    }
  }
  *reinterpret_cast<uint32_t*>(dst + D::COUNT) = (uint32_t)count | (meta[2] >> 24) << 8;
}

struct LeafSource {
  const float* blk;
  int cnt, stride;
};
__device__ __forceinline__ LeafSource leaf_source(const SceneDev& sc, uint32_t leaf,
                                                  const uint8_t* leaf_count) {
  LeafSource l;
  l.blk = sc.leaves + (size_t)leaf * 9 * sc.leaf_memory;
  l.cnt = (int)leaf_count[leaf];
  l.stride = ((l.cnt - 1) / sc.gang + 1) * sc.gang;
  return l;
}

// One thread per leaf and group of four triangle slots: its block if the leaf
// has one for the group, and its part of the general kernels' bounds.
__global__ void __launch_bounds__(128) pack_leaves_kernel(SceneDev sc, uint32_t n,
                                                          const uint32_t* leaf_block,
                                                          const uint8_t* leaf_count,
                                                          float4* blocks, float* bounds) {
  const uint64_t id = (uint64_t)blockIdx.x * 128u + threadIdx.x;
  const int L = sc.leaf_memory;
  const uint32_t groups = (uint32_t)L / 4u;
  const uint32_t leaf = (uint32_t)(id / groups);
  const int first = (int)(id % groups) * 4;
  if (leaf >= n) return;
  const LeafSource l = leaf_source(sc, leaf, leaf_count);
  float* b = bounds + (size_t)leaf * leaf_bounds_floats(L);
  float4* out = blocks != nullptr && first < l.cnt
                    ? blocks + (size_t)(leaf_block[leaf] + first / 4) * kBlockWords
                    : nullptr;
  for (int k = 0; k < 4; ++k) {
    const int i = first + k;
    float v[9];
    for (int q = 0; q < 9; ++q) v[q] = i < l.cnt ? l.blk[q * l.stride + i] : 0.0f;
    for (int a = 0; a < 3; ++a) {
      const float lo = fminf(fminf(v[a], v[3 + a]), v[6 + a]);
      const float hi = fmaxf(fmaxf(v[a], v[3 + a]), v[6 + a]);
      b[a * L + i] = lo;
      b[(3 + a) * L + i] = hi;
      if (out) {
        reinterpret_cast<float*>(out + a)[k] = lo;
        reinterpret_cast<float*>(out + 3 + a)[k] = hi;
      }
    }
    if (!out) continue;
    const uint32_t prim = i < l.cnt ? sc.leaf_prim[(size_t)leaf * L + i] : 0xFFFFFFFFu;
    float4* t = out + kBlockTris + 3 * k;
    t[0] = make_float4(v[0], v[1], v[2], v[3]);
    t[1] = make_float4(v[4], v[5], v[6], v[7]);
    t[2] = make_float4(v[8], __uint_as_float(prim), 0.0f, 0.0f);
  }
  for (int k = 0; k < 4 && first == 0; ++k) b[6 * L + k] = 0.0f;
  if (out)
    out[kBlockWords - 1] = make_float4(
        __uint_as_float(first == 0 ? (uint32_t)sc.leaf_depth[leaf] : 0u), 0.f, 0.f, 0.f);
}

template <int N, int FMT>
cudaError_t nodes_for(const SceneDev& sc, uint32_t n, const uint32_t* leaf_block, uint8_t* out,
                      cudaStream_t s) {
  pack_nodes_kernel<N, FMT><<<(n + 127) / 128, 128, 0, s>>>(sc, n, leaf_block, out);
  return cudaGetLastError();
}

template <int N>
cudaError_t nodes_for_width(const SceneDev& sc, int fmt, uint32_t n, const uint32_t* leaf_block,
                            uint8_t* out, cudaStream_t s) {
  return fmt == kFmtFP32 ? nodes_for<N, kFmtFP32>(sc, n, leaf_block, out, s)
                         : nodes_for<N, kFmtQ8>(sc, n, leaf_block, out, s);
}

template <int N>
int bytes_for_width(int fmt) {
  return fmt == kFmtFP32 ? PackFmt<N, kFmtFP32>::REC : PackFmt<N, kFmtQ8>::REC;
}

}  // namespace

int pack_node_bytes(int nm, int fmt) {
  switch (nm) {
    case 4: return bytes_for_width<4>(fmt);
    case 8: return bytes_for_width<8>(fmt);
    case 12: return bytes_for_width<12>(fmt);
    default: return bytes_for_width<16>(fmt);
  }
}

cudaError_t pack_nodes(const SceneDev& sc, int nm, int fmt, uint32_t n_inner,
                       const uint32_t* leaf_block, uint8_t* out, cudaStream_t s) {
  if (n_inner == 0) return cudaSuccess;
  switch (nm) {
    case 4: return nodes_for_width<4>(sc, fmt, n_inner, leaf_block, out, s);
    case 8: return nodes_for_width<8>(sc, fmt, n_inner, leaf_block, out, s);
    case 12: return nodes_for_width<12>(sc, fmt, n_inner, leaf_block, out, s);
    case 16: return nodes_for_width<16>(sc, fmt, n_inner, leaf_block, out, s);
  }
  return cudaErrorInvalidValue;
}

cudaError_t pack_leaves(const SceneDev& sc, uint32_t n_leaves, const uint32_t* leaf_block,
                        const uint8_t* leaf_count, float4* blocks, float* bounds,
                        cudaStream_t s) {
  if (n_leaves == 0) return cudaSuccess;
  const uint64_t groups = (uint64_t)n_leaves * (uint32_t)(sc.leaf_memory / 4);
  pack_leaves_kernel<<<(unsigned)((groups + 127) / 128), 128, 0, s>>>(sc, n_leaves, leaf_block,
                                                                      leaf_count, blocks, bounds);
  return cudaGetLastError();
}

}  // namespace dev
}  // namespace bvhgpu
