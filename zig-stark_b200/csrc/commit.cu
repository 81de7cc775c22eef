// The circle commit workload as one device-resident plan: circle LDE of all columns, row
// leaves with the gamma combination, then the folds on one stream and the large trees
// beside them; the small layers' folds in one launch and their trees in another.
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <memory>
#include <vector>

#include "circle.cuh"
#include "commit.cuh"
#include "fri.cuh"

namespace zs {

CommitPlan::CommitPlan(uint32_t C_, unsigned L_, unsigned B_, unsigned F_) : C(C_), L(L_), B(B_), F(F_) {
  if (C == 0 || C > 256) throw Error(ZS_EMALFORMED, "n_columns must be in [1, 256]");
  if (L < 1 || L + B > 28) throw Error(ZS_EMALFORMED, "log_rows + log_blowup must be in [1, 28]");
  if (F > L + B) throw Error(ZS_EMALFORMED, "more folds than domain bits");
  ZS_CUDA(cudaStreamCreateWithFlags(&setup, cudaStreamNonBlocking));
  ZS_CUDA(cudaStreamCreateWithFlags(&copy, cudaStreamNonBlocking));
  for (auto& s : sides) ZS_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
  // Group sizes grow by about 4/3 from 2 columns at the end, so each group's LDE is
  // done before the next group's copy (the LDE of a column takes about 0.6 of its
  // copy over PCIe) and the step waits for a small group's LDE after the last copy.
  for (uint32_t g = 2, used = 0; used < C; g = std::max(g + 1, (g * 4 + 2) / 3)) {
    upload_groups.push_back(std::min(g, C - used));
    used += upload_groups.back();
  }
  std::sort(upload_groups.begin(), upload_groups.end(), std::greater<uint32_t>());
  up_events.resize(upload_groups.size() + 1);
  for (auto& e : up_events) ZS_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  events.resize(F + 2 + kSides);
  for (auto& e : events) ZS_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  const size_t n = (size_t)1 << L, N = (size_t)1 << (L + B);
  small = std::make_unique<CircleDomain>(L, setup);
  big = std::make_unique<CircleDomain>(L + B, setup);
  tabs = std::make_unique<FoldTables>(L + B, setup);
  layers.resize(F + 1);
  layer_trees.resize(F);
  // Every buffer of the plan lies in one allocation: a stream-ordered pool that keeps no
  // memory maps each block anew, so a plan of forty small blocks took longer to make than
  // one large one.
  struct Part {
    void** p;
    size_t bytes;
  };
  std::vector<Part> parts = {{(void**)&trace, C * n * sizeof(uint32_t)},
                             {(void**)&lde, C * N * sizeof(uint32_t)},
                             {(void**)&scratch, lde_scratch_words(L, B, C) * sizeof(uint32_t)},
                             {(void**)&gammas, C * sizeof(qm31)},
                             {(void**)&row_tree.words, DeviceTree::words_for(L + B) * sizeof(uint32_t)},
                             {(void**)&done, (F + 1) * sizeof(uint32_t)}};
  for (unsigned i = 0; i < F; ++i) {
    parts.push_back({(void**)&layers[i], (N >> i) * sizeof(qm31)});
    parts.push_back({(void**)&layer_trees[i].words, DeviceTree::words_for(L + B - i) * sizeof(uint32_t)});
  }
  parts.push_back({(void**)&roots, (F + 1) * 32});  // side by side: results() takes both in one copy
  parts.push_back({(void**)&layers[F], (N >> F) * sizeof(qm31)});
  size_t total = 0;
  for (const Part& q : parts) total += (q.bytes + 255) & ~(size_t)255;
  ZS_CUDA(cudaMallocAsync((void**)&base, total, setup));
  total = 0;
  for (const Part& q : parts) *q.p = base + total, total += (q.bytes + 255) & ~(size_t)255;
  ZS_CUDA(cudaMemsetAsync(done, 0, (F + 1) * sizeof(uint32_t), setup));
  row_tree.log_n = L + B, row_tree.done = done, row_tree.root_out = roots;
  for (unsigned i = 0; i < F; ++i) {
    DeviceTree& t = layer_trees[i];
    t.log_n = L + B - i, t.done = done + 1 + i, t.root_out = roots + 8 * (1 + i);
  }
  alphas.assign(F, qzero());
  const char* env = std::getenv("ZS_NO_GRAPH");
  use_graph = !(env && env[0] == '1');
  ZS_CUDA(cudaStreamSynchronize(setup));
}

CommitPlan::~CommitPlan() {
  cudaDeviceSynchronize();
  drop_graph();
  small.reset();
  big.reset();
  tabs.reset();
  cudaFreeAsync(base, setup);
  cudaStreamSynchronize(setup);  // the pool gives back what it does not keep
  for (auto& e : events) cudaEventDestroy(e);
  for (auto& e : up_events) cudaEventDestroy(e);
  cudaStreamDestroy(copy);
  for (auto& s : sides) cudaStreamDestroy(s);
  cudaStreamDestroy(setup);
}

void CommitPlan::set_challenges(const uint32_t* h_gammas, const uint32_t* h_alphas) {
  std::vector<qm31> g(C);
  for (uint32_t c = 0; c < C; ++c) g[c] = qmake(h_gammas[4 * c], h_gammas[4 * c + 1], h_gammas[4 * c + 2], h_gammas[4 * c + 3]);
  for (unsigned i = 0; i < F; ++i)
    alphas[i] = qmake(h_alphas[4 * i], h_alphas[4 * i + 1], h_alphas[4 * i + 2], h_alphas[4 * i + 3]);
  ZS_CUDA(cudaMemcpy(gammas, g.data(), C * sizeof(qm31), cudaMemcpyHostToDevice));
  drop_graph();  // fold challenges are baked into the captured launches
}

void CommitPlan::run_phase(int phase, const uint32_t* d_trace, cudaStream_t st) {
  const size_t n = (size_t)1 << L, N = (size_t)1 << (L + B);
  if (!d_trace) d_trace = trace;
  switch (phase) {
    case PHASE_LDE:
      circle_lde(d_trace, n, lde, N, C, L, B, *small, *big, scratch, st);
      break;
    case PHASE_ROW_TREE:
      build_row_leaves(lde, N, C, row_tree, gammas, layers[0], st);
      tree_finish(row_tree, 0, st);
      if (F > 0) build_qm31_tree(layers[0], layer_trees[0], st);
      break;
    case PHASE_FOLDS:
      for (unsigned i = 0; i < big_layers(); ++i) {
        fold(i, st);
        if (i + 1 < big_layers()) build_qm31_tree(layers[i + 1], layer_trees[i + 1], st);
      }
      small_layers(1, st);
      break;
    default:
      throw Error(ZS_EMALFORMED, "unknown phase");
  }
}

// The layers of more than 2^kSmallTreeLog values: each has its own launches.
unsigned CommitPlan::big_layers() const {
  return std::min(F, L + B > kSmallTreeLog ? L + B - kSmallTreeLog : 0);
}

void CommitPlan::fold(unsigned i, cudaStream_t st) {
  fri_fold(layers[i], layers[i + 1], 1u << (L + B - i - 1), alphas[i], nullptr, i, *tabs, st);
}

// The folds from layer big_layers() on and the trees of those layers: the folds of few
// values in one CTA, the trees in one launch (their levels are chains of 1.3 us, whatever
// the number of trees), from layer `first_tree` on.
void CommitPlan::small_layers(unsigned first_tree, cudaStream_t st) {
  unsigned i = big_layers();
  std::vector<const qm31*> vals;
  std::vector<DeviceTree*> trees;
  for (unsigned k = std::max(i, first_tree); k < F; ++k) vals.push_back(layers[k]), trees.push_back(&layer_trees[k]);
  for (; i < F && L + B - i > kChainLog; ++i) fold(i, st);
  FoldChain fc{};
  fc.first = i, fc.count = F - i, fc.log_size = L + B - i, fc.tables = tabs->tables;
  for (unsigned k = 0; k < fc.count; ++k) fc.c[k] = qmul(alphas[i + k], tabs->offset_inv(i + k));
  for (unsigned k = 0; k <= fc.count && fc.count; ++k) fc.layer[k] = layers[i + k];
  fri_fold_chain(fc, st);
  if (!trees.empty()) build_small_trees(vals.data(), trees.data(), (uint32_t)trees.size(), st);
}

// The step as a DAG: the LDE, the row leaves and the fold chain run on `st`; each
// large tree (the row tree above its leaves, the large fold layers') is built on a side
// stream as soon as its values exist, so the narrow tops of the trees overlap with each
// other and with the folds.
void CommitPlan::run_direct(const uint32_t* d_trace, cudaStream_t st) {
  const size_t n = (size_t)1 << L, N = (size_t)1 << (L + B);
  if (!d_trace) d_trace = trace;
  circle_lde(d_trace, n, lde, N, C, L, B, *small, *big, scratch, st);
  after_lde(st);
}

// Column group g is copied on `copy` and its LDE waits for that copy only; the groups'
// LDEs run in order on `st` and share the scratch buffer (sized for all C columns).
void CommitPlan::run_host_direct(const uint32_t* h_trace, cudaStream_t st) {
  const size_t n = (size_t)1 << L, N = (size_t)1 << (L + B);
  const size_t G = upload_groups.size();
  ZS_CUDA(cudaEventRecord(up_events[G], st));  // the previous step is done with `trace`
  ZS_CUDA(cudaStreamWaitEvent(copy, up_events[G], 0));
  for (size_t g = 0, c0 = 0; g < G; c0 += upload_groups[g++]) {
    ZS_CUDA(cudaMemcpyAsync(trace + c0 * n, h_trace + c0 * n, (size_t)upload_groups[g] * n * sizeof(uint32_t),
                            cudaMemcpyHostToDevice, copy));
    ZS_CUDA(cudaEventRecord(up_events[g], copy));
  }
  for (size_t g = 0, c0 = 0; g < G; c0 += upload_groups[g++]) {
    ZS_CUDA(cudaStreamWaitEvent(st, up_events[g], 0));
    circle_lde(trace + c0 * n, n, lde + c0 * N, N, upload_groups[g], L, B, *small, *big, scratch, st);
  }
  after_lde(st);
}

void CommitPlan::run_host(const uint32_t* h_trace, cudaStream_t st) {
  if (!use_graph) return run_host_direct(h_trace, st);
  if (!host_exec || host_trace != h_trace) {
    if (host_exec) cudaGraphExecDestroy(host_exec);
    host_exec = nullptr;
    cudaGraph_t g = nullptr;
    ZS_CUDA(cudaStreamBeginCapture(setup, cudaStreamCaptureModeThreadLocal));
    try {
      run_host_direct(h_trace, setup);
    } catch (...) {
      cudaStreamEndCapture(setup, &g);
      if (g) cudaGraphDestroy(g);
      throw;
    }
    ZS_CUDA(cudaStreamEndCapture(setup, &g));
    const cudaError_t e = cudaGraphInstantiate(&host_exec, g, 0);
    cudaGraphDestroy(g);
    ZS_CUDA(e);
    host_trace = h_trace;
  }
  ZS_CUDA(cudaGraphLaunch(host_exec, st));
}

// The roots lie just before the final layer: one copy brings both back where the layer is
// small. A copy into pageable memory is a wait of its own (15 us for a kilobyte, 20 for 64 KB,
// 33 for 256), three through pinned memory with one wait 18; but pinning takes over a
// millisecond, so a call that pins has to keep the memory when it returns. The copy lands in a
// buffer that the thread keeps (at most 257 KB of plain memory), because into fresh pages it is
// slower: results of 64, 128 and 256 KB 35, 45 and 70 us against 39, 58 and 90.
void CommitPlan::results(cudaStream_t st, uint8_t* lde_root, uint8_t* layer_roots, uint32_t* final_layer) {
  constexpr size_t kTogether = (size_t)256 << 10;
  static thread_local std::vector<uint8_t> back;
  const size_t final_bytes = ((size_t)1 << (L + B - F)) * sizeof(qm31), roots_bytes = (F + 1) * 32;
  const size_t at = reinterpret_cast<unsigned char*>(layers[F]) - reinterpret_cast<unsigned char*>(roots);
  const bool together = final_layer && final_bytes <= kTogether;
  if (final_layer && !together)
    ZS_CUDA(cudaMemcpyAsync(final_layer, layers[F], final_bytes, cudaMemcpyDeviceToHost, st));
  if (lde_root || layer_roots || together) {
    const size_t bytes = together ? at + final_bytes : roots_bytes;
    if (back.size() < bytes) back.resize(bytes);
    ZS_CUDA(cudaMemcpyAsync(back.data(), roots, bytes, cudaMemcpyDeviceToHost, st));
    ZS_CUDA(cudaStreamSynchronize(st));
    if (lde_root) std::memcpy(lde_root, back.data(), 32);
    if (layer_roots) std::memcpy(layer_roots, back.data() + 32, roots_bytes - 32);
    if (together) std::memcpy(final_layer, back.data() + at, final_bytes);
  }
  ZS_CUDA(cudaStreamSynchronize(st));
}

// Everything after the LDE: row leaves with the gamma combination, the trees, the folds.
void CommitPlan::after_lde(cudaStream_t st) {
  const size_t N = (size_t)1 << (L + B);
  build_row_leaves(lde, N, C, row_tree, gammas, layers[0], st);
  unsigned side = 0;
  bool used[kSides] = {};
  auto branch = [&](auto&& build) {
    cudaEvent_t e = events[ev_used++];
    ZS_CUDA(cudaEventRecord(e, st));
    used[side % kSides] = true;
    cudaStream_t s = sides[side++ % kSides];
    ZS_CUDA(cudaStreamWaitEvent(s, e, 0));
    build(s);
  };
  ev_used = 0;
  branch([&](cudaStream_t s) { tree_finish(row_tree, 0, s); });
  for (unsigned i = 0; i < big_layers(); ++i) {
    branch([&](cudaStream_t s) { build_qm31_tree(layers[i], layer_trees[i], s); });
    fold(i, st);
  }
  small_layers(0, st);
  for (unsigned k = 0; k < kSides; ++k) {
    if (!used[k]) continue;  // only streams forked from `st` may join it (graph capture)
    cudaEvent_t e = events[ev_used++];
    ZS_CUDA(cudaEventRecord(e, sides[k]));
    ZS_CUDA(cudaStreamWaitEvent(st, e, 0));
  }
}

void CommitPlan::drop_graph() {
  if (graph_exec) cudaGraphExecDestroy(graph_exec);
  graph_exec = nullptr;
  graph_trace = nullptr;
  if (host_exec) cudaGraphExecDestroy(host_exec);
  host_exec = nullptr;
  host_trace = nullptr;
}

// The whole step is one CUDA graph (35 launches for 64 columns of 2^20 at blowup 4 with 16
// folds, 7 for 8 of 2^10 with 6), captured on the plan's own stream and replayed on the
// caller's; it is recaptured when the trace pointer or the challenges change.
void CommitPlan::run(const uint32_t* d_trace, cudaStream_t st) {
  if (!d_trace) d_trace = trace;
  if (!use_graph) return run_direct(d_trace, st);
  if (!graph_exec || graph_trace != d_trace) {
    drop_graph();
    cudaGraph_t g = nullptr;
    ZS_CUDA(cudaStreamBeginCapture(setup, cudaStreamCaptureModeThreadLocal));
    try {
      run_direct(d_trace, setup);
    } catch (...) {
      cudaStreamEndCapture(setup, &g);
      if (g) cudaGraphDestroy(g);
      throw;
    }
    ZS_CUDA(cudaStreamEndCapture(setup, &g));
    const cudaError_t e = cudaGraphInstantiate(&graph_exec, g, 0);
    cudaGraphDestroy(g);
    ZS_CUDA(e);
    graph_trace = d_trace;
  }
  ZS_CUDA(cudaGraphLaunch(graph_exec, st));
}

uint32_t CommitPlan::launches() const {
  // circle_lde: 3; row leaves: 1 and the row tree's; each large layer a fold and its tree's;
  // then small_layers.
  const unsigned LB = L + B;
  uint32_t k = 3 + 1 + tree_launches(LB);
  for (unsigned i = 0; i < big_layers(); ++i) k += 1 + tree_launches(LB - i);
  unsigned i = big_layers();
  if (i < F) ++k;  // the trees
  for (; i < F && LB - i > kChainLog; ++i) ++k;
  if (i < F) ++k;  // the chain
  return k;
}

}  // namespace zs
