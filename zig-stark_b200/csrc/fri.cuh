// FRI folding over QM31 on the device (src/m31/fri.zig).
#pragma once
#include "merkle.cuh"

namespace zs {

// Inverse domain points of the FRI layers of a size-2^dlog domain
// (D_i[j] = FRI_OFFSET^(2^i) * w_{dlog-i}^j, fri.zig:96-117): w_0^-k is the
// product of three 2^11-entry tables, so any k < 2^33 costs two QM31 products.
struct FoldTables {
  unsigned dlog = 0;
  qm31* tables = nullptr;  // 3 * 2048 entries
  cudaStream_t st = nullptr;  // freed in stream order
  explicit FoldTables(unsigned dlog, cudaStream_t st);
  ~FoldTables();
  FoldTables(const FoldTables&) = delete;
  FoldTables& operator=(const FoldTables&) = delete;
  // (FRI_OFFSET^(2^layer))^-1, host-side.
  qm31 offset_inv(unsigned layer) const;
};

// One fold (fri.zig:209-219): out[j] = (y0 + y1)/2 + alpha * (y0 - y1) / (2 D_layer[j]),
// y0 = in[j], y1 = in[j + half], for j < half, with the challenge given or (`d_alpha`) read
// from device memory.
void fri_fold(const qm31* d_in, qm31* d_out, uint32_t half, const qm31& alpha, const qm31* d_alpha, unsigned layer,
              const FoldTables& tabs, cudaStream_t st);

// A chain of folds with given challenges, from a layer of at most 2^kChainLog values down,
// in one CTA: each fold of so few values is a launch's latency otherwise (about 2 us, as much
// as the CTA takes for 2^12 values: a 16 x 2^13 commit takes 105 us with it, 103 us from 2^11
// down, 112 us from 2^13 down; the other commits are equal).
constexpr unsigned kChainLog = 12;
struct FoldChain {
  unsigned first, count;  // folds of layers first .. first + count - 1
  unsigned log_size;      // log2 of layer `first`'s length
  const qm31* tables;
  qm31 c[kChainLog];                // alpha_i * offset_inv(i)
  qm31* layer[kChainLog + 1];       // layer[0] is only read
};
void fri_fold_chain(const FoldChain& chain, cudaStream_t st);

// The small layers of the commit phase in one CTA (fri.zig:195-227): for layers
// first .. first + count - 1 (the first holding at most kTailMax values): fold the layer
// before into it, commit it (hashQM31 leaves and the whole tree), absorb its root into the
// device transcript `ch` and sample the folding challenge; at the end the fold into the
// layer after the last. Every step is a barrier apart, so the chain of small dependent
// steps costs no launches. Above 2^9 values a layer's widest levels fill more than one SM:
// SeededFib 2^12 634-638 us with it, 650 us from 2^8 down, 638 us from 2^10 down.
constexpr unsigned kTailLog = 9;
constexpr uint32_t kTailMax = 1u << kTailLog;
constexpr uint32_t kTailLayers = kTailLog + 1;
struct FriTail {
  uint32_t first, count;  // absolute index of the first layer, layers handled
  unsigned log_size;      // log2 of the first layer's length
  const qm31* tables;     // FoldTables::tables
  qm31 off_inv[kTailLayers + 1];  // of layer first - 1 + c
  // layer[c] is layer first - 1 + c; layer[0] may be null (first = 0); layer[count + 1],
  // 2^(log_size - count) values, is only written
  qm31* layer[kTailLayers + 2];
  uint32_t* tree[kTailLayers];  // DeviceTree words of layer first + c
  uint32_t* roots;              // 8 words per handled layer
  qm31* alphas;                 // one per handled layer; alphas[-1] is layer first - 1's
};
struct Channel;
// `ft` and `ch` are in device memory.
void fri_tail(const FriTail* ft, Channel* ch, cudaStream_t st);

}  // namespace zs
