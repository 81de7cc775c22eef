// Merkle trees (src/core/merkle/merkle.zig) built on the device.
#pragma once
#include <vector>

#include "common.cuh"

namespace zs {

// All levels of a tree over 2^log_n leaves in one buffer: level k (2^(log_n-k)
// digests) starts at digest 2N - (2N >> k), so the leaves come first and the root
// is the last digest. Digests are 8 little-endian u32 words (the Blake3 bytes).
struct DeviceTree {
  unsigned log_n = 0;
  uint32_t* words = nullptr;  // (2N - 1) * 8 words
  // Finished subtrees of a launch in which the last one's CTA goes on to the top
  // (k_tree): one word, zero before the tree's first launch and again after each.
  uint32_t* done = nullptr;
  uint32_t* root_out = nullptr;  // where else the root goes when the tree is finished (8 words)
  static size_t words_for(unsigned log_n) { return (((size_t)2 << log_n) - 1) * 8; }
  size_t level_offset(unsigned k) const {
    const size_t N2 = (size_t)2 << log_n;
    return N2 - (N2 >> k);
  }
  const uint32_t* level(unsigned k) const { return words + 8 * level_offset(k); }
  uint32_t* level(unsigned k) { return words + 8 * level_offset(k); }
  const uint32_t* root() const { return level(log_n); }
};

// A fold as the source of a layer's values (fri.cuh): out[j], j < half, from `in` (2 half
// values of layer `layer`), the challenge read from device memory.
struct FoldSource {
  const qm31* in;
  qm31* out;
  const qm31* alpha;
  const qm31* tables;  // FoldTables::tables
  qm31 off_inv;        // FoldTables::offset_inv(layer)
  uint32_t half;
  unsigned layer;
};
// A transcript step after a root: absorb it, sample a folding challenge.
struct Channel;
struct TranscriptStep {
  Channel* ch;  // the transcript, in device memory
  qm31* alpha;  // the challenge
};

// Leaves hashQM31(values[i]) for 2^log_n QM31 values plus the whole tree.
void build_qm31_tree(const qm31* d_values, DeviceTree& tree, cudaStream_t st, const TranscriptStep* tx = nullptr);
// The same over the outputs of a fold, which are stored as well.
void build_fold_tree(const FoldSource& f, DeviceTree& tree, cudaStream_t st, const TranscriptStep* tx = nullptr);

// Most trees that one launch builds (blockIdx.y picks the tree).
constexpr uint32_t kTreeBatch = 64;
// build_qm31_tree for `count` trees of one size: tree k over the values at
// d_values + k * v_stride.
void build_qm31_trees(const qm31* d_values, size_t v_stride, DeviceTree* const* trees, uint32_t count,
                      cudaStream_t st);
// Trees of several sizes up to 2^kSmallTreeLog, each over its own values: small trees are
// chains of levels, so one launch takes the time of its largest; but it waits for the last
// layer's fold, and trees of more leaves take their levels faster in launches of their own.
// From 2^13 down: a commit of 8 x 2^18 520 us against 511, of 37 x 2^15 247 against 243; from
// 2^15 down: 499 and 246, but 16 x 2^13 115 against 105 (8 x 2^10: equal).
constexpr unsigned kSmallTreeLog = 14;
void build_small_trees(const qm31* const* d_values, DeviceTree* const* trees, uint32_t count, cudaStream_t st);
// Completes the levels above `from_level` (levels <= from_level must be written).
void tree_finish(DeviceTree& tree, unsigned from_level, cudaStream_t st);
// Number of launches that a tree from its leaves' digests or values takes.
uint32_t tree_launches(unsigned log_n);

// Row leaves of C columns x 2^log_n M31 values (column c at d_cols + c * col_stride):
// leaf r = hashM31s(col_0[r], ..., col_{C-1}[r]) (src/m31/hash.zig:15-25), C <= 256.
// Also writes g[r] = sum_c gammas[c] * col_c[r] when `d_gammas` is not null. The leaf level
// only; finish with tree_finish.
void build_row_leaves(const uint32_t* d_cols, size_t col_stride, uint32_t C, DeviceTree& tree, const qm31* d_gammas,
                      qm31* g_out, cudaStream_t st);

}  // namespace zs
