// Merkle trees on the device (src/core/merkle/merkle.zig:17-68).
//
// A leaf is one Blake3 compression (hashQM31) or a few (hashM31s of a row: 4 for 64
// values), a node two (hash2 = Blake3("zig-stark:pair" || L || R), 78 bytes), each in one
// thread's registers. Every node is written, because openings need all levels.
//   k_row_leaves: one thread per row;
//   k_tree: subtrees in CTAs, level by level, up to the root.
#include <algorithm>

#include "blake3.cuh"
#include "merkle.cuh"
#include "transcript.cuh"
#include "tree.cuh"

namespace zs {

namespace {
constexpr unsigned kThreads = 256;

}  // namespace

// Row leaves hashM31s(col_0[r], ..., col_{C-1}[r]) (src/m31/hash.zig:15-25), and
// optionally g[r] = sum_c gammas[c] * col_c[r]. The four
// coordinates of g accumulate unreduced 62-bit products in 64 bits (one wide
// multiply-add each). p 2^32 is a multiple of p, so where the high word has reached p it can
// be taken off there: one ALU operation (a minimum) after every second product, where a
// Mersenne fold of 64 bits takes five after every fourth. After it the high word is at most
// p + 1, and two products of words below p keep the sum below 2^64.
__device__ __forceinline__ uint64_t fold64(uint64_t x) { return (x & P) + (x >> 31); }
__device__ __forceinline__ uint64_t fold_high(uint64_t x) {
  const uint32_t hi = (uint32_t)(x >> 32);
  return (uint64_t)umin32(hi, hi - P) << 32 | (uint32_t)x;
}
__device__ __forceinline__ uint32_t canon64(uint64_t x) {
  x = fold64(fold64(x));  // < 2^31 + 8
  const uint32_t s = (uint32_t)x;
  return umin32(s, s - P);
}

__global__ void __launch_bounds__(kThreads) k_row_leaves(const uint32_t* __restrict__ cols, size_t col_stride,
                                                         uint32_t C, uint32_t* tree_words, uint64_t n,
                                                         const qm31* __restrict__ gammas, qm31* g_out) {
  __shared__ uint4 sg[256];
  const bool comb = gammas != nullptr;
  if (comb)
    for (uint32_t c = threadIdx.x; c < C; c += blockDim.x) sg[c] = reinterpret_cast<const uint4*>(gammas)[c];
  __syncthreads();
  const uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  const uint32_t row_bytes = (uint32_t)r * 4;  // fits: a plan has at most 2^28 rows
  uint64_t acc0 = 0, acc1 = 0, acc2 = 0, acc3 = 0;
  uint32_t cv[8];
  b3::iv(cv);
  const uint32_t nblocks = C * 4 <= 64 ? 1 : (C * 4 + 63) / 64;
  // The next block's 16 column loads are issued before the current block is
  // compressed, so their latency hides behind ~700 integer instructions. Only a row's last
  // block can be a part of one: the others take their loads and products without a
  // comparison of the column, from column addresses that are the same in every thread.
  // Bound by the ALU pipe and the issue slots at once: 64 columns x 2^22 rows 761 -> 644 us,
  // 4950 -> 4230 instructions a row, 2460 -> 2150 of them on the ALU (1792 in the four
  // compressions). With one copy of the product code for whole and partial blocks (a test
  // every four columns) 663-687 us.
  uint32_t nxt[16];
  auto load_block = [&](uint32_t blk) {
    const char* col = reinterpret_cast<const char*>(cols) + (size_t)blk * 64 * col_stride;
    const uint32_t left = C - blk * 16;
    if (left >= 16) {
#pragma unroll
      for (int k = 0; k < 16; ++k)
        nxt[k] = __ldg(reinterpret_cast<const uint32_t*>(col + (size_t)k * 4 * col_stride + row_bytes));
    } else {
#pragma unroll
      for (int k = 0; k < 16; ++k)
        nxt[k] = (uint32_t)k < left
                     ? __ldg(reinterpret_cast<const uint32_t*>(col + (size_t)k * 4 * col_stride + row_bytes))
                     : 0u;
    }
  };
  auto add_product = [&](uint32_t w, uint32_t v) {
    const uint4 g = sg[w];
    acc0 += (uint64_t)g.x * v;
    acc1 += (uint64_t)g.y * v;
    acc2 += (uint64_t)g.z * v;
    acc3 += (uint64_t)g.w * v;
  };
  auto fold_sums = [&] {
    acc0 = fold_high(acc0);
    acc1 = fold_high(acc1);
    acc2 = fold_high(acc2);
    acc3 = fold_high(acc3);
  };
  load_block(0);
  for (uint32_t blk = 0; blk < nblocks; ++blk) {
    uint32_t m[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) m[k] = nxt[k];
    if (blk + 1 < nblocks) load_block(blk + 1);
    if (comb && blk * 16 + 16 <= C) {
#pragma unroll
      for (int k = 0; k < 16; ++k) {
        add_product(blk * 16 + k, m[k]);
        if (k & 1) fold_sums();
      }
    } else if (comb) {
#pragma unroll
      for (int k = 0; k < 16; ++k) {
        if (blk * 16 + k < C) add_product(blk * 16 + k, m[k]);
        if (k & 1) fold_sums();
      }
    }
    const int rem = (int)(C * 4) - (int)(blk * 64);
    const uint32_t len = rem >= 64 ? 64u : (uint32_t)rem;
    const uint32_t flags = (blk == 0 ? b3::CHUNK_START : 0u) | (blk == nblocks - 1 ? (b3::CHUNK_END | b3::ROOT) : 0u);
    b3::compress_cv(cv, m, len, flags);
  }
  put_digest(tree_words, r, cv);
  if (!comb) return;
  const qm31 acc = qmake(canon64(acc0), canon64(acc1), canon64(acc2), canon64(acc3));
  reinterpret_cast<uint4*>(g_out)[r] = u4_of(acc);
}

// The trees of one launch: of one size, or (from their leaves, narrow) of several.
struct TreeSet {
  uint32_t* words[kTreeBatch];
  uint32_t* done[kTreeBatch];
  const qm31* vals[kTreeBatch];    // the leaves' values (kValues)
  uint32_t* root_out[kTreeBatch];  // where else the root goes (8 words), or null
  uint8_t log_n[kTreeBatch];
};

// Levels level0 + 1 .. level0 + levels over the 2^span digests of CTA b's subtree
// (cta_levels; a smaller tree takes one CTA). With `top` (levels = span) the CTA that
// finishes the tree's last subtree goes on from the subtrees' roots to the tree's root:
// each CTA counts itself in `done` after its root is visible, nobody waits. TX: the CTA
// that has the root takes the transcript's step with it.
constexpr unsigned kTreeThreads = 256;
template <int SRC, bool TX>
__global__ void __launch_bounds__(kTreeThreads, SRC == kValues ? 4 : 3)
    k_tree(const __grid_constant__ TreeSet ts, unsigned level0, unsigned span, unsigned levels, unsigned top,
           const __grid_constant__ FoldSource f, const __grid_constant__ TranscriptStep tx) {
  extern __shared__ uint4 s_dig[];
  let_next_start();
  after_previous();
  uint32_t* words = ts.words[blockIdx.y];
  const unsigned log_n = ts.log_n[blockIdx.y];
  if (level0 + span > log_n) span = levels = log_n - level0;
  size_t cta = blockIdx.x;
  if (cta >> (log_n - level0 - span)) return;  // the set has larger trees
  qm31 fold_c = qzero();
  if constexpr (SRC == kFold) fold_c = qmul(q_of(__ldcg(reinterpret_cast<const uint4*>(f.alpha))), f.off_inv);
#pragma unroll 1
  for (;;) {
    cta_levels<SRC>(words, log_n, level0, span, levels, cta, s_dig, ts.vals[blockIdx.y], f, fold_c);
    if (!top || level0 + levels == log_n) break;
    uint32_t& s_last = reinterpret_cast<uint32_t*>(s_dig)[0];  // the digests there are done with
    if (threadIdx.x == 0) {  // wrote the subtree's root
      __threadfence();
      const uint32_t n_ctas = 1u << (log_n - level0 - levels);
      const bool last = atomicAdd(ts.done[blockIdx.y], 1u) == n_ctas - 1;
      if (last) {
        *ts.done[blockIdx.y] = 0;
        __threadfence();
      }
      s_last = last;
    }
    __syncthreads();
    const bool go_on = s_last != 0;
    __syncthreads();  // read before the digests overwrite it
    if (!go_on) return;
    level0 += levels;
    span = levels = log_n - level0;
    cta = 0;
  }
  if (level0 + levels != log_n) return;
  const uint32_t* root = words + 8 * (((size_t)2 << log_n) - 2);
  uint32_t* root_out = ts.root_out[blockIdx.y];
  if (root_out && threadIdx.x < 8) root_out[threadIdx.x] = __ldcg(root + threadIdx.x);
  if constexpr (TX) {
    if (threadIdx.x >= 32) return;
    __shared__ wtx::Shared s_tx;
    wtx::load(s_tx, tx.ch);
    const qm31 alpha = wtx::step(s_tx, root);
    wtx::store(s_tx, tx.ch);
    if (threadIdx.x == 0) *reinterpret_cast<uint4*>(tx.alpha) = u4_of(alpha);
  }
}

// The launches that take trees of 2^log_n leaves from level `level0` (its digests, or with
// leaves to hash first) to their roots.
namespace {
struct TreeLaunch {
  unsigned level0, span, levels, threads;
  unsigned top_levels;  // levels that the last CTA adds
  size_t smem() const {  // two levels in turn of the wider of the subtrees and the top
    const unsigned w = levels < 2 && top_levels == 0 ? 0 : std::max(span, top_levels);
    return w < 2 ? 0 : ((size_t)3 << (w - 2)) * 32;
  }
};

// While the trees' digests fill the device a launch is bound by the ALU: it stops after
// three or four levels, before a CTA's levels become narrower than its warps, and its
// CTAs are the larger the more there are. From there on the levels are a chain of two
// compressions each (1.3 us), so one launch takes 2^8 digests per CTA, one warp per
// scheduler at its widest level, and its last CTA the levels above. Measured over spans of
// 8..11, 2..11 levels and 128 or 256 threads, with leaves: one tree of 2^22 372 us (544 us
// in narrow launches only, 562 us with three levels per thread), 2^20 116 us (126 us with
// spans of 2^11), 2^18 53 us (60 us narrow), 2^14 27 us, 2^12 24.7 us; 32 trees of 2^17
// 365 us (537 us narrow), 12 of 2^14 43 us (51 us narrow, 47 us with spans of 2^11).
TreeLaunch plan_narrow(unsigned log_n, unsigned level0) {
  const unsigned rem = log_n - level0, span = std::min(rem, 8u);
  return {level0, span, span, 128, rem - span <= 8 ? rem - span : 0};
}

std::vector<TreeLaunch> plan_tree(unsigned log_n, unsigned level0, uint32_t count) {
  std::vector<TreeLaunch> v;
  while (level0 < log_n) {
    const unsigned rem = log_n - level0;
    const uint64_t digests = (uint64_t)count << rem;
    TreeLaunch t{level0, 0, 0, 0, 0};
    if (rem >= 13 && digests >= ((uint64_t)1 << 21)) {
      t.span = 11, t.levels = 4, t.threads = 256;
    } else if (rem >= 13 && digests >= ((uint64_t)1 << 20)) {
      t.span = 10, t.levels = 4, t.threads = 256;
    } else if (rem >= 13 && digests >= ((uint64_t)1 << 17)) {
      t.span = 9, t.levels = 3, t.threads = 128;
    } else {
      t = plan_narrow(log_n, level0);
    }
    v.push_back(t);
    level0 += t.levels + t.top_levels;
  }
  return v;
}

// All launches from level0 to the roots: the first from `src`, the last with the
// transcript's step when `tx` is given.
void finish_set(const TreeSet& ts, uint32_t count, unsigned log_n, unsigned level0, TreeSource src, cudaStream_t st,
                const FoldSource& f = {}, const TranscriptStep* tx = nullptr) {
  if (log_n == 0) throw Error(ZS_EGENERIC, "a tree of one leaf");
  const std::vector<TreeLaunch> plan = plan_tree(log_n, level0, count);
  for (const TreeLaunch& t : plan) {
    const dim3 grid(1u << (log_n - t.level0 - t.span), count);
    const TreeSource from = &t == &plan.front() ? src : kDigests;
    const bool with_tx = tx && &t == &plan.back();
    auto* k = from == kFold     ? (with_tx ? k_tree<kFold, true> : k_tree<kFold, false>)
              : from == kValues ? (with_tx ? k_tree<kValues, true> : k_tree<kValues, false>)
                                : (with_tx ? k_tree<kDigests, true> : k_tree<kDigests, false>);
    if (tx) {  // a chain of launches that wait for one another
      unsigned level0 = t.level0, span = t.span, levels = t.levels, top = t.top_levels > 0;
      void* args[] = {const_cast<TreeSet*>(&ts), &level0, &span, &levels, &top, const_cast<FoldSource*>(&f),
                      const_cast<TranscriptStep*>(tx)};
      launch_overlapped((const void*)k, grid, dim3(t.threads), args, t.smem(), st);
    } else {
      k<<<grid, t.threads, t.smem(), st>>>(ts, t.level0, t.span, t.levels, t.top_levels > 0, f, {});
    }
  }
  ZS_CUDA(cudaGetLastError());
}

void add_tree(TreeSet& ts, uint32_t k, const DeviceTree& tree, const qm31* vals) {
  ts.words[k] = tree.words, ts.done[k] = tree.done, ts.vals[k] = vals;
  ts.root_out[k] = tree.root_out, ts.log_n[k] = (uint8_t)tree.log_n;
}

TreeSet single(const DeviceTree& tree, const qm31* vals = nullptr) {
  TreeSet ts{};
  add_tree(ts, 0, tree, vals);
  return ts;
}
}  // namespace

void tree_finish(DeviceTree& tree, unsigned from_level, cudaStream_t st) {
  finish_set(single(tree), 1, tree.log_n, from_level, kDigests, st);
}

uint32_t tree_launches(unsigned log_n) { return (uint32_t)plan_tree(log_n, 0, 1).size(); }

void build_qm31_tree(const qm31* d_values, DeviceTree& tree, cudaStream_t st, const TranscriptStep* tx) {
  finish_set(single(tree, d_values), 1, tree.log_n, 0, kValues, st, {}, tx);
}

void build_fold_tree(const FoldSource& f, DeviceTree& tree, cudaStream_t st, const TranscriptStep* tx) {
  if (f.half != 1u << tree.log_n) throw Error(ZS_EGENERIC, "fold and tree of different sizes");
  finish_set(single(tree), 1, tree.log_n, 0, kFold, st, f, tx);
}

void build_qm31_trees(const qm31* d_values, size_t v_stride, DeviceTree* const* trees, uint32_t count,
                      cudaStream_t st) {
  for (uint32_t t0 = 0; t0 < count; t0 += kTreeBatch) {
    const uint32_t c = std::min<uint32_t>(kTreeBatch, count - t0);
    const unsigned log_n = trees[t0]->log_n;
    TreeSet ts{};
    for (uint32_t k = 0; k < c; ++k) {
      if (trees[t0 + k]->log_n != log_n) throw Error(ZS_EGENERIC, "build_qm31_trees: trees of different sizes");
      add_tree(ts, k, *trees[t0 + k], d_values + (size_t)(t0 + k) * v_stride);
    }
    finish_set(ts, c, log_n, 0, kValues, st);
  }
}

void build_small_trees(const qm31* const* d_values, DeviceTree* const* trees, uint32_t count, cudaStream_t st) {
  for (uint32_t t0 = 0; t0 < count; t0 += kTreeBatch) {
    const uint32_t c = std::min<uint32_t>(kTreeBatch, count - t0);
    TreeSet ts{};
    unsigned log_n = 0;
    for (uint32_t k = 0; k < c; ++k) {
      if (trees[t0 + k]->log_n > kSmallTreeLog || trees[t0 + k]->log_n == 0)
        throw Error(ZS_EGENERIC, "build_small_trees: tree size");
      add_tree(ts, k, *trees[t0 + k], d_values[t0 + k]);
      log_n = std::max(log_n, trees[t0 + k]->log_n);
    }
    const TreeLaunch t = plan_narrow(log_n, 0);
    k_tree<kValues, false><<<dim3(1u << (log_n - t.span), c), t.threads, t.smem(), st>>>(ts, 0, t.span, t.levels, 1,
                                                                                       {}, {});
  }
  ZS_CUDA(cudaGetLastError());
}

void build_row_leaves(const uint32_t* d_cols, size_t col_stride, uint32_t C, DeviceTree& tree, const qm31* d_gammas,
                      qm31* g_out, cudaStream_t st) {
  if (C == 0 || C > 256) throw Error(ZS_EMALFORMED, "row leaves need 1..256 columns");
  const uint64_t n = (uint64_t)1 << tree.log_n;
  k_row_leaves<<<(unsigned)((n + kThreads - 1) / kThreads), kThreads, 0, st>>>(d_cols, col_stride, C, tree.words, n,
                                                                               d_gammas, g_out);
  ZS_CUDA(cudaGetLastError());
}

}  // namespace zs
