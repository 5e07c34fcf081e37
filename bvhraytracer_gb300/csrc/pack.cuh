// Packed scene of the ray-pool kernel (pool.cuh), made on the device from the
// scene's node records, stack entries and leaf blocks.
//
// A gather of 16 bytes per lane runs at the L1's full rate (8 cycles per warp
// load) only when the records' stride is an odd multiple of 16 bytes: at 240
// bytes a load takes 10.9 cycles, at 192 bytes 20, at 128 or 256 bytes 31
// (every lane then reads the same four banks). So every record here has an
// odd number of 16-byte words.
#pragma once
#include <cuda_runtime.h>

#include "traverse.cuh"

namespace bvhgpu {
namespace dev {

// Node record of N child slots (N rounded up to 4):
//   FP32: float box[6][N]; empty slots have lo = +inf, hi = -inf (no ray
//         without NaN hits them)
//   Q8:   float origin[3], int8 exp[3], uint8 count | uint8 q[6][N]
//   uint32 entry[N]       stack entry of each child
//   uint32 sorted[3][N]   the entries in the push sequence of each axis
//   uint32 (N > 8: uint64) seq[3]   the child at each position (nibbles)
//   N > 8: uint64 inv[3]            the position of each child (nibbles)
//   uint32 count         child count | depth << 8
template <int N, int FMT>
struct PackFmt {
  static constexpr int BOX = FMT == kFmtFP32 ? 0 : 16;
  static constexpr int ENTRY = FMT == kFmtFP32 ? 24 * N : (16 + 6 * N + 15) / 16 * 16;
  static constexpr int SORTED = ENTRY + 4 * N;
  static constexpr int SEQ = SORTED + 12 * N;
  static constexpr int INV = SEQ + 24;  // N > 8
  static constexpr int COUNT = SEQ + (N <= 8 ? 12 : 48);
  static constexpr int WORDS = (COUNT + 4 + 15) / 16;
  static constexpr int REC = (WORDS | 1) * 16;
};

// Leaf block: four triangles of a leaf, 19 words of 16 bytes. A leaf is
// consecutive blocks, and the stack entries of the packed records hold the
// leaf's first block instead of its index, so a leaf visit loads nothing
// before the bounds and the triangles themselves.
//   words 0-5    bounds of the four triangles: lo.x lo.y lo.z hi.x hi.y hi.z
//   words 6-17   triangle i at 6 + 3 i: 9 floats (p0 p1 p2), input id, 0, 0
//   word 18      first block: the leaf's depth (uint32), 0, 0, 0
constexpr int kBlockWords = 19;
constexpr int kBlockTris = 6;  // first triangle word
constexpr uint32_t kMaxBlocks = 1u << kLeafCountShift;

// Bounds of the general kernels' leaf pre-test (SceneDev::leaf_bounds): float
// lo[3][L], hi[3][L] and 4 floats of padding per leaf (24 L + 16 bytes, an odd
// number of 16-byte words for every L).
__host__ __device__ inline int leaf_bounds_floats(int leaf_memory) { return 6 * leaf_memory + 4; }

// Bytes of a packed node record.
int pack_node_bytes(int nm, int fmt);

// Fills the packed node records from the scene's records and stack entries.
// leaf_block: first block of each leaf.
cudaError_t pack_nodes(const SceneDev& sc, int nm, int fmt, uint32_t n_inner,
                       const uint32_t* leaf_block, uint8_t* out, cudaStream_t s);
// Fills the leaf blocks (null: none) and the general kernels' bounds from the leaves.
// leaf_count: triangles of each leaf.
cudaError_t pack_leaves(const SceneDev& sc, uint32_t n_leaves, const uint32_t* leaf_block,
                        const uint8_t* leaf_count, float4* blocks, float* bounds,
                        cudaStream_t s);

}  // namespace dev
}  // namespace bvhgpu
